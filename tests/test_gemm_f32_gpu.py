"""Products in true 32-bit at the edges of the two kernels' tiles, against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(M, N, K, activation):
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    want = x.double() @ w.double().T
    # K products and sums, each rounded to 2^-24 of a running sum that |x| |w| bounds
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5)
    y = ops.linear(x, w, gated=activation is not None, activation=activation or "silu")
    assert torch.equal(ops.linear(x, w, gated=activation is not None, activation=activation or "silu"), y)
    if activation is None:
        assert y.shape == (M, N) and bool(((y.double() - want).abs() <= bound).all())
        return
    gate, up = want[:, 0::2], want[:, 1::2]
    act = {"silu": lambda z: z * torch.sigmoid(z), "none": lambda z: z,
           "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh")}[activation]
    # the activations' slope is at most 1.13, they are evaluated within 2^-21 of their value, and 1 + tanh(z)
    # near zero keeps 2^-24 absolute, times |g|
    slack = 1.2 * bound[:, 0::2] * (up.abs() + bound[:, 1::2]) + gate.abs() * bound[:, 1::2] \
        + (2.0 ** -21 + 2.0 ** -22) * (gate * up).abs()
    assert y.shape == (M, N // 2) and bool(((y.double() - act(gate) * up).abs() <= slack).all())


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 15, 16])
@pytest.mark.parametrize("N, K", [(1, 4), (3, 36), (147, 1024), (149, 1028), (320, 128), (2371, 132), (4738, 2052), (2050, 8192)])
def test_a_few_rows(M, N, K):
    _check(M, N, K, None)


@pytest.mark.parametrize("M", [17, 31, 33, 64, 65, 128, 129, 500])
@pytest.mark.parametrize("N, K", [(1, 4), (63, 12), (66, 36), (129, 68), (320, 128), (3001, 516), (20000, 20)])
def test_more_rows(M, N, K):
    _check(M, N, K, None)


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh", "none"])
@pytest.mark.parametrize("M, N, K", [(1, 2, 4), (3, 302, 64), (8, 16384, 256), (16, 4742, 132), (17, 66, 36), (70, 640, 128), (300, 3002, 132)])
def test_gated(M, N, K, activation):
    _check(M, N, K, activation)
