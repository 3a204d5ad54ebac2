"""Products of 17 to 128 bfloat16 rows whose K is split over a cluster: every number of parts, slabs cut short, outputs that
leave eight rows at a time and such that cannot."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [17, 32, 33, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("N, K", [(8, 512), (136, 2048), (2048, 264), (2052, 1032), (3072, 2048), (5120, 768), (6144, 512), (9000, 1024)])
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
def test_split_products(M, N, K, out):
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).bfloat16() for n in (M, N))
    want = x.double() @ w.double().T
    y = ops.linear(x, w, out_dtype=out)
    assert torch.equal(ops.linear(x, w, out_dtype=out), y)
    # products of bfloat16 numbers are exact; sums are rounded (or cut) to 2^-23 of a running sum that |x| |w| bounds, some sqrt(K)
    # of them, and the result once to its type
    bound = 2.0 ** -23 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5) + (2.0 ** -8 if out == torch.bfloat16 else 2.0 ** -24) * want.abs()
    assert y.shape == (M, N) and bool(((y.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("act", ["silu", "relu_squared"])
def test_split_products_with_an_activation(act):
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w = (torch.randn(n, 1024, device="cuda", generator=g).mul_(0.2).bfloat16() for n in (100, 2048))
    z = x.double() @ w.double().T
    want = torch.nn.functional.silu(z) if act == "silu" else z.clamp(min=0).square()
    y = ops.linear(x, w, plain_act=act).double()
    assert bool(((y - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("M", [17, 31, 33, 64, 65, 128])
@pytest.mark.parametrize("N, K", [(6, 64), (34, 136), (1000, 512), (2050, 264)])
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
def test_gated_outputs_that_leave_one_by_one(M, N, K, out):
    """Gated products whose outputs are no whole sixteen bytes, or 32-bit."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).bfloat16() for n in (M, N))
    z = x.double() @ w.double().T
    gate, up = z[:, 0::2], z[:, 1::2]
    y = ops.linear(x, w, out_dtype=out, gated=True)
    # sums within `off` as above; silu's slope is at most 1.1, its exponential and division are good to 2^-20
    off = 2.0 ** -23 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5)
    want = torch.nn.functional.silu(gate) * up
    bound = 1.1 * off[:, 0::2] * (up.abs() + off[:, 1::2]) + gate.abs() * off[:, 1::2] + \
        (2.0 ** -20 + (2.0 ** -8 if out == torch.bfloat16 else 0.0)) * (gate * up).abs()
    assert y.shape == (M, N // 2) and bool(((y.double() - want).abs() <= bound).all())
