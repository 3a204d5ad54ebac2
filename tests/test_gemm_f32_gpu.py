"""Products in true 32-bit at the edges of the three kernels' tiles, against 64-bit sums."""
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


@pytest.mark.parametrize("M, N, K", [(17, 64, 4100), (129, 66, 4096), (130, 2050, 516), (300, 3002, 540), (257, 9000, 512), (500, 2048, 2052), (1000, 130, 8192), (200, 20002, 544)])
@pytest.mark.parametrize("activation", [None, "silu", "gelu_tanh"])
def test_split_products(M, N, K, activation):
    """K from 512: whole, short and barely filled tiles, last stages cut short, odd numbers of chunks."""
    _check(M, N, K, activation)


def split_plan(M, N, K):
    """(columns, parts of K, tiles whose blocks take all of K, tiles) as the product makes them."""
    import ctypes
    from llm_singularity_b200 import kernels as ops
    plan = (ctypes.c_longlong * 4)()
    ops._lib("gemm_f32").lsb_gemm_f32_split_plan(M, N, K, plan)
    return tuple(plan)


def test_split_products_are_made_in_both_widths():
    """The shapes above take blocks of 64 columns and of 128, whole and shared out (on the 148 SMs of a B200)."""
    kinds = {(columns, parts > 1, whole > 0) for columns, parts, whole, _ in
             (split_plan(*s) for s in ((17, 64, 4100), (129, 66, 4096), (300, 3002, 540), (500, 2048, 2052), (257, 9000, 512), (200, 20002, 544)))}
    assert {(64, True, False), (64, False, True), (128, True, False), (128, True, True)} <= kinds


@pytest.mark.parametrize("N", [700, 20000])
def test_split_products_out_of_range(N):
    """Values that the parts cannot hold: infinities, NaN, rows near and below the smallest normal number, the largest numbers."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = (torch.randn(n, 520, device="cuda", generator=g) for n in (200, N))
    x[3, 5], x[10, 7], w[9, 1], w[11, 2] = float("inf"), float("nan"), -float("inf"), 0.0
    x[20] *= 1e-38
    x[21] *= 1e-42
    x[22] = 0.0
    x[40] *= 1e-30
    x[41, ::2] *= 1e-37
    w[7] *= 2.0 ** -100
    w[8] *= 1e-39
    w[12] *= 1e10                                                    # (with x's 1e-38: 24 bits of it)
    x[31], w[33] = 1e25, -1e25           # sums of one sign beyond the range (of both signs 32-bit sums make NaN, 64-bit ones don't)
    y = ops.linear(x, w)
    want = x.double() @ w.double().T
    assert torch.equal(y.isnan(), want.isnan())
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + 520 ** 0.5) + 520 * 2.0 ** -149    # (and subnormal sums' own steps)
    sure = want.abs() + bound < 3.4028234e38
    assert bool(((y.double() - want).abs() <= bound)[sure].all()) and bool(sure.float().mean() > 0.95)
    beyond = (want.abs() - bound > 3.4028236e38) & ~want.isnan()
    assert torch.equal(y[beyond].double(), want[beyond].sign() * float("inf"))


@pytest.mark.parametrize("M, N, K", [(1, 64, 64), (8, 2048, 512), (16, 300, 2048), (100, 128, 512)])
def test_weights_that_the_kernel_in_front_makes(M, N, K):
    """A product's weights may be another product's result: not read before that kernel has ended."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, a, b = (torch.randn(n, k, device="cuda", generator=g) for n, k in ((M, K), (N, 256), (K, 256)))
    w = ops.linear(a, b)
    want = x.double() @ w.double().T
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5)
    for _ in range(20):
        made = ops.linear(a, b)
        y = ops.linear(x, made)
        assert torch.equal(made, w) and bool(((y.double() - want).abs() <= bound).all())
        made.zero_()                             # (its memory goes to the next turn's weights)
        del made


@pytest.mark.parametrize("N", [300, 20000])
@pytest.mark.parametrize("K", [512, 2052])
def test_split_products_of_small_values_beside_large_ones(N, K):
    """Rows with ordinary numbers and ones whose parts bfloat16 has no numbers for, against rows that are zero at the
    ordinary ones, or so large at the small ones that they count; and products near the smallest normal number."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g) for n in (140, N))
    x[:, 9] = (1 + torch.rand(140, device="cuda", generator=g)) * 2.0 ** torch.linspace(-126, -80, 140, device="cuda").round()
    w[:, 3] = (1 + torch.rand(N, device="cuda", generator=g)) * 2.0 ** torch.linspace(-120, -60, N, device="cuda").round()
    w[5], x[7] = 0.0, 0.0
    w[5, 9], x[7, 3] = 1.0, 1.0                                      # selections
    x[11, ::2] *= 2.0 ** -110
    w[13, ::2], w[13, 1::2] = w[13, ::2] * 1e30, 0.0                 # the small ones of x's row 11 times large ones
    x[20] *= 2.0 ** -62
    w[21] *= 2.0 ** -60
    w[22] *= 2.0 ** -75
    y, want = ops.linear(x, w), x.double() @ w.double().T
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5) + K * 2.0 ** -149
    assert bool(((y.double() - want).abs() <= bound).all())
    for m, n in [(slice(None), 5), (7, slice(None))]:                # a selection is the number itself
        assert torch.equal(y[m, n], want[m, n].float())


@pytest.mark.parametrize("M, N, K", [(17, 64, 512), (130, 2050, 516), (500, 2048, 2048), (129, 66, 8192), (1000, 130, 4100)])
def test_split_products_keep_24_bits(M, N, K):
    """The error of whole results, where a part of an operand left out would show (2^-17 of it or more)."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    want = x.double() @ w.double().T
    # (multiply-adds: 1.6e-7 at K = 512, 8e-7 at 8,192)
    assert ((ops.linear(x, w).double() - want).norm() / want.norm()).item() < 4e-7


@pytest.mark.parametrize("M, N, K", [(17, 70, 512), (130, 2050, 1028), (300, 9000, 544)])
def test_every_part_of_a_split_counts(M, N, K):
    """One number a row of x, with all 24 bits in use: each result is one product."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    w = torch.randn(N, K, device="cuda", generator=g)
    x, at = torch.zeros(M, K, device="cuda"), (37 * torch.arange(M, device="cuda")) % K
    parts = 1.0 + torch.tensor([2.0 ** -9 + 2.0 ** -18 + 2.0 ** -23, -2.0 ** -9 - 2.0 ** -17 - 2.0 ** -23, 2.0 ** -10 + 2.0 ** -22, 2.0 ** -23], device="cuda")
    x[torch.arange(M), at] = parts[torch.arange(M, device="cuda") % 4] * 2.0 ** (torch.arange(M, device="cuda") % 9 - 4)
    want = x.double() @ w.double().T
    # six of the nine products of parts: what is left out is below 2^-25; the sums of the six are cut to 2^-23, twice
    assert bool(((ops.linear(x, w).double() - want).abs() <= 2.0 ** -22 * want.abs()).all())
