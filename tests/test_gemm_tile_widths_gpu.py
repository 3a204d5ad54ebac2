"""Products of more than 128 bfloat16 rows, whose tiles are as wide as shares the matrix out best: widths of 128 to 256,
the last tile whole, partly and barely filled, against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, N", [(129, 128), (300, 1000), (543, 5120), (543, 16384), (600, 3080), (543, 3072), (900, 4098),
                                  (2048, 3072), (2011, 6144), (2000, 4100), (3000, 2222), (1503, 8192), (2011, 28672), (554, 6144), (1200, 4096)])
@pytest.mark.parametrize("gated, out_dtype", [(False, torch.bfloat16), (False, torch.float32), (True, torch.bfloat16), (True, torch.float32)])
@pytest.mark.parametrize("K", [72, 640])
def test_widths(M, N, K, gated, out_dtype):
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).to(torch.bfloat16) for n in (M, N))
    y = ops.linear(x, w, out_dtype=out_dtype, gated=gated)
    want = x.double() @ w.double().T
    tol = 2.0 ** -21 * K                       # sums of K products in 32-bit, of size sqrt(K), each step rounded to 2^-24 of them
    if gated:
        # the sums' errors times the other factor (silu's slope is at most 1.1), and silu by way of ex2 and a quick
        # division: 2 + 1.2 |g| units in the last place for the exponential, a few for the rest
        gate, up = want[:, 0::2], want[:, 1::2]
        want = gate * torch.sigmoid(gate) * up
        tol = tol * (1.1 * up.abs() + gate.abs() + tol) + 2.0 ** -23 * (8 + 1.2 * gate.abs()) * want.abs()
    if out_dtype == torch.bfloat16:
        tol = tol + 2.0 ** -8 * want.abs()     # (rounded once more)
    assert y.shape == want.shape and y.dtype == out_dtype and bool(((y.double() - want).abs() <= tol).all())
    for _ in range(5):
        assert torch.equal(ops.linear(x, w, out_dtype=out_dtype, gated=gated), y)
    ops.check_status()


@pytest.mark.parametrize("M, N, K", [(4200, 8192, 2112), (2900, 4100, 2112), (1290, 8192, 4104), (385, 28672, 2112), (200, 16384, 4104), (2048, 3072, 4104),
                                     (3000, 2222, 4104), (1400, 4098, 4104), (1000, 2048, 8200), (1000, 1900, 8200)])
@pytest.mark.parametrize("gated, out_dtype", [(False, torch.bfloat16), (False, torch.float32), (True, torch.bfloat16)])
def test_pairs_of_blocks(M, N, K, gated, out_dtype):
    """Long products, whose tiles pairs of blocks share: odd numbers of row tiles, and last tiles and K blocks cut short."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).to(torch.bfloat16) for n in (M, N))
    assert ops._lib("gemm_tc").lsb_gemm_tc_pairs(M, N, K, int(gated))        # (on the 148 SMs of a B200)
    y = ops.linear(x, w, out_dtype=out_dtype, gated=gated)
    want = x.double() @ w.double().T
    tol = 2.0 ** -25 * K * K ** 0.5            # each 16 products a cut to 2^-23 of sums that stay below 4 sqrt(K)
    if gated:
        gate, up = want[:, 0::2], want[:, 1::2]
        want = gate * torch.sigmoid(gate) * up
        tol = tol * (1.1 * up.abs() + gate.abs() + tol) + 2.0 ** -23 * (8 + 1.2 * gate.abs()) * want.abs()
    if out_dtype == torch.bfloat16:
        tol = tol + 2.0 ** -8 * want.abs()
    assert y.shape == want.shape and bool(((y.double() - want).abs() <= tol).all())
    for _ in range(5):
        assert torch.equal(ops.linear(x, w, out_dtype=out_dtype, gated=gated), y)
    ops.check_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_behind_a_long_kernel(dtype):
    """A product that is launched beside a long kernel: its waits' limits do not count that kernel's time."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(3)
    # one block, some 25,000 slices one behind the other
    a, b = (torch.randn(64, 400001, device="cuda", generator=g) for _ in range(2))
    x, w = (torch.randn(n, 2112, device="cuda", generator=g).to(dtype) for n in (700, 4096))
    want = ops.linear(x, w)
    for _ in range(3):
        ops.linear(a, b)
        assert torch.equal(ops.linear(x, w), want)
    ops.check_status()
