"""The sampler's cuts where a row is split over the blocks of a cluster: slices' edges, buckets too full to
list, rows whose values are equal, masked or stretched by an outlier, and a vocabulary whose slices stay in memory."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COMBOS = [(1.0, 0, 1.0), (0.7, 5, 1.0), (1.3, 0, 0.8), (0.9, 40, 0.6), (0.8, 2000, 0.999), (2.5, 0, 0.3), (1.0, 1, 1.0),
          (1.0, 0, 0.0)]


def pick(row, t, k, p, u):
    """The token the rules name, in 64-bit: ties at the k-th value are all kept."""
    x = (row / np.float32(t)).astype(np.float64)
    kept = x >= np.sort(x)[-k] if 0 < k < len(x) else np.ones(len(x), bool)
    m = np.where(kept & (x > -np.inf), np.exp(x - x.max()), 0.0)
    if p < 1.0:
        order = np.argsort(-x, kind="stable")
        before = np.cumsum(m[order]) - m[order]
        cut = x[order][before <= p * m.sum()].min() if p > 0 else x.max()
        m = np.where(x >= cut, m, 0.0)
    c = np.cumsum(m)
    return int(min(np.searchsorted(c, u * c[-1]), np.nonzero(m)[0][-1]))


def check(rows, combos, seed=0):
    from llm_singularity_b200 import kernels as ops
    R, u = len(rows), np.random.RandomState(seed).rand(len(rows)).astype(np.float32)
    params = torch.tensor([[t, p, 1.0, float(u[r])] for r, (t, _, p) in enumerate(combos)], device="cuda")
    out = torch.full((R,), -1, dtype=torch.int32, device="cuda")
    ops.sample(torch.from_numpy(rows).cuda(), params, torch.tensor([k for _, k, _ in combos], dtype=torch.int32, device="cuda"),
               None, None, out)
    for r, got in enumerate(out.tolist()):
        t, k, p = combos[r]
        # (equal unless u falls within the rounding of exp, 2 ulp of a 32-bit sum's terms, of a boundary)
        near = {pick(rows[r], t, k, p, min(max(float(u[r]) + d, 0.0), 1.0)) for d in (0.0, -1e-6, 1e-6)}
        assert got in near, (r, combos[r], got, near)


@pytest.mark.parametrize("vocab", [1, 5, 513, 8192, 8193, 16385, 32770, 65539, 128256, 377003])
def test_cuts_at_the_edges_of_the_slices(vocab):
    rows = (np.random.RandomState(vocab).randn(len(COMBOS), vocab) * 3).astype(np.float32)
    check(rows, COMBOS)


@pytest.mark.parametrize("kind", ["equal", "two values", "masked", "outlier", "wide"])
def test_cuts_of_rows_that_the_histogram_does_not_spread(kind):
    rng = np.random.RandomState(7)
    rows = (rng.randn(len(COMBOS), 40000) * 2).astype(np.float32)
    if kind == "equal":
        rows[:] = 0.25
    elif kind == "two values":
        rows = np.where(rows > 2.0, np.float32(1.0), np.float32(-1.0))
    elif kind == "masked":
        rows[:, 300:] = -np.inf
    elif kind == "outlier":
        rows[:, 17] = -1e30
    else:
        rows[:, ::1000] = np.float32(3e38) * np.sign(rows[:, ::1000])
        rows = np.clip(rows, -3e38, 60.0)
    check(rows, COMBOS, seed=3)


@pytest.mark.parametrize("vocab", [5, 32770, 128256, 377003])
def test_rows_without_a_value_name_the_first_token(vocab):
    from llm_singularity_b200 import kernels as ops
    rows = np.full((6, vocab), -np.inf, dtype=np.float32)
    rows[1::3] = np.nan
    rows[2, ::2] = np.nan
    rows[5, vocab - 2] = -1e30                             # (one value: it is the maximum, whatever surrounds it)
    rows[5, :vocab - 2:3] = np.nan
    want = [0, 0, 0, 0, 0, vocab - 2]
    for t, k, p in [(0.0, 0, 1.0), (0.0, 3, 0.5)] + COMBOS:
        params = torch.tensor([[t, p, 1.0, 0.3]] * 6, device="cuda")
        out = torch.full((6,), -1, dtype=torch.int32, device="cuda")
        ops.sample(torch.from_numpy(rows).cuda(), params, torch.full((6,), k, dtype=torch.int32, device="cuda"), None, None, out)
        got = out.tolist()
        # (a NaN counts as the largest value of a top-k cut, which may leave nothing else: any token then)
        assert got[:5] == want[:5] and (k and t or got[5] == want[5]) and 0 <= got[5] < vocab, (t, k, p, got)
