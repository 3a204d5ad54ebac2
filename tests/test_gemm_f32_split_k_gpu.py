"""32-bit products whose K is shared out over a cluster: two to eight parts, the last of them short, whole tiles beside such, and
numbers that only one part of K knows to be small."""
import pytest
import torch

from test_gemm_f32_gpu import _check, split_plan

pytestmark = pytest.mark.gpu


SHAPES = [(17, 64, 4100), (17, 130, 640), (40, 2048, 8192), (129, 2050, 1156), (150, 2048, 2048), (300, 3074, 2052), (500, 2048, 1540),
          (500, 9600, 1024), (640, 4098, 772), (129, 66, 4096)]


def test_the_shapes_take_what_they_are_for():
    plans = [split_plan(*s) for s in SHAPES]
    parts = {p for _, p, _, _ in plans}
    assert {2, 4, 5, 6, 7, 8} <= parts
    assert any(p > 1 and 0 < whole < tiles for _, p, whole, tiles in plans)                  # whole tiles and shared-out ones
    assert any(-(-K // 128) % p for (_, _, K), (_, p, _, _) in zip(SHAPES, plans))           # a last part that is short


@pytest.mark.parametrize("M, N, K", SHAPES)
@pytest.mark.parametrize("activation", [None, "silu"])
def test_parts_of_k(M, N, K, activation):
    _check(M, N, K, activation)


@pytest.mark.parametrize("M, N, K", [(40, 2048, 4096), (300, 3072, 2048), (500, 9600, 1024)])
@pytest.mark.parametrize("at", [0.0, 0.6, 0.99])
def test_small_numbers_in_one_part(M, N, K, at):
    """A row of x, and one of w, that are zero but for a number whose parts bfloat16 has no numbers for, against ones there."""
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    k, m, n = int(at * K), M - 3, N - 5
    x[m], w[n] = 0.0, 0.0
    x[m, k], w[n, k] = 1.2345678 * 2.0 ** -120, 1.7654321 * 2.0 ** -118
    x[m - 1], w[n - 1] = 0.0, 0.0
    x[m - 1, k], w[n - 1, k] = 1.0, 1.0
    y, want = ops.linear(x, w), x.double() @ w.double().T
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5) + K * 2.0 ** -149
    assert bool(((y.double() - want).abs() <= bound).all())
    assert torch.equal(y[m, n - 1], x[m, k]) and torch.equal(y[m - 1, n], w[n, k])          # a selection is the number itself
    x[m, k] = float("inf")
    y = ops.linear(x, w)
    assert y[m, n - 1].item() == float("inf") and bool(torch.isfinite(y[:m]).all())
