"""Rows normed in groups and gated: four values a thread and turn where sizes and places allow, one otherwise, against
float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, groups", [(4, 1), (2048, 1), (2052, 1), (2048, 16), (1040, 5), (96, 24), (1536, 3), (8192, 64), (30, 5), (90, 1)])
@pytest.mark.parametrize("shared_weight", [False, True])
@pytest.mark.parametrize("gate", ["none", "aligned", "odd"])
def test_against_float64(dtype, n, groups, shared_weight, gate):
    from llm_singularity_b200 import kernels as K
    g = torch.Generator().manual_seed(n + groups)
    T, eps = 7, 3e-5
    x = 2 * torch.randn(T, n, generator=g)
    w = 1 + 0.3 * torch.randn(n // groups if shared_weight else n, generator=g)
    wide = torch.randn(T, n + 16, generator=g).to(dtype)
    z = {"none": None, "aligned": wide[:, 8:8 + n], "odd": wide[:, 3:3 + n]}[gate]
    parts = x.double().view(T, groups, -1)
    want = (parts / torch.sqrt((parts ** 2).mean(-1, keepdim=True) + eps)).view(T, n) * w.double().repeat(n // w.shape[0])
    if z is not None:
        want = want * torch.sigmoid(z.double())
    out, cuda = torch.full((T, n), float("nan"), dtype=dtype, device="cuda"), wide.cuda()
    K.rows_norm_gate(x.cuda(), w.cuda(), groups, eps, None if z is None else cuda[:, 3 if gate == "odd" else 8:][:, :n], out)
    # the sum's chain of n / (groups * 128) roundings and a dozen more of 2^-24 each; a bfloat16 result is rounded once more
    tol = (2.0 ** -24 * (12 + n / groups / 128) + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)) * want.abs() + 1e-30
    assert bool(((out.double().cpu() - want).abs() <= tol).all())
