"""Products of a few rows whose groups of weight rows are short, after one whose operands were no numbers: what an earlier kernel
leaves in shared memory (in the places of rows that a group lacks) must not show."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 7, 8, 16])
@pytest.mark.parametrize("N, K", [(149, 1536), (2371, 1028), (3072, 2048)])
def test_left_over_values(M, N, K):
    from llm_singularity_b200 import kernels as ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    ops.linear(torch.full((M, 2048), float("nan"), device="cuda"), torch.full((16384, 2048), float("nan"), device="cuda"))
    y = ops.linear(x, w)
    # K products and sums, each rounded to 2^-24 of a running sum that |x| |w| bounds
    bound = 2.0 ** -24 * (x.abs().double() @ w.abs().double().T) * (2 + K ** 0.5)
    assert bool(((y.double() - x.double() @ w.double().T).abs() <= bound).all())
