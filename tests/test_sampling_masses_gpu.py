"""A cut by mass keeps the 24 bits of its exponentials: rows whose mass above a value is what top_p allows but for 2^-25 of it, to either
side.  The values are such that their exponentials have an exact 24-bit form (within 1/40 of its last place), an odd one where
the mass above is concerned, so that no rounding of a right one decides; places of 2^-23, or a bucket's end that is off by a 32-bit
rounding, do."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32
STEP, INV = F(10.0) / F(1023.0), F(1023.0) / F(10.0)           # of the histogram near the maximum


def _distance(at, odd, rng):
    """A distance d (float32) to the maximum near `at` whose e^-d over its bucket's upper end is 1 less an odd (even) number of 2^-24."""
    d = (F(at) + np.arange(200000, dtype=np.float64) * 2.0 ** -22).astype(F)
    d = rng.permutation(np.unique(d))
    b = np.floor(d * INV)                                      # (a bucket as 32-bit arithmetic finds it)
    lack = -np.expm1(b.astype(np.float64) * np.float64(STEP) - d.astype(np.float64)) * 2.0 ** 24
    whole = np.rint(lack)
    ok = (np.abs(lack - whole) < 0.025) & (whole % 2 == odd) & (whole > 1000) & (whole < 150000)
    return d[ok][0]


def _row(vocab, seed, side):
    rng = np.random.RandomState(seed)
    n = 900
    upper, lower = _distance(1.0 + 0.31 * seed, 1, rng), _distance(1.4 + 0.31 * seed, 0, rng)
    a, b = np.exp(-np.float64(upper)), np.exp(-np.float64(lower))
    above = 1.0 + n * a
    # above == p (above + m b + c) (1 + side 2^-25): p as a 32-bit number, c one value well below the others
    m = 850
    p = F(above / (above + m * b + 0.3 * b))
    c = above / (np.float64(p) * (1.0 + side * 2.0 ** -25)) - above - m * b
    row = np.full(vocab, -60.0, dtype=F)                       # (their mass is no place of 2^-44)
    at = np.sort(rng.choice(vocab - 1, n + m + 2, replace=False))
    row[at[0]] = 0.0
    row[at[1:1 + n]] = -upper
    row[at[1 + n:1 + n + m]] = -lower
    row[at[-1]] = np.log(c)
    got = np.exp(row[at].astype(np.float64)).sum() * np.float64(p) / above - 1.0
    assert abs(got - (-side) * 2.0 ** -25) < 2.0 ** -28        # (p of the mass, short of what lies above by the side)
    return row, p, int(at[1 + n]), int(at[1 + n + m - 1])


@pytest.mark.parametrize("rows", [24, 60])                     # (values kept on chip, or read again)
@pytest.mark.parametrize("vocab", [9000, 60000, 256000, 377003])
def test_cuts_within_a_rounding(vocab, rows):
    from llm_singularity_b200 import kernels as ops
    cases = [_row(vocab, s // 2 % 12, 1 if s % 2 else -1) for s in range(24)]
    cases = [cases[r % 24] for r in range(rows)]
    logits = torch.from_numpy(np.stack([c[0] for c in cases])).cuda()
    params = torch.tensor([[1.0, float(c[1]), 1.0, 0.999999] for c in cases], device="cuda")
    out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    ops.sample(logits, params, torch.zeros(rows, dtype=torch.int32, device="cuda"), None, None, out)
    for r, (got, (_, p, first, last)) in enumerate(zip(out.tolist(), cases)):
        kept = first <= got <= last                            # (the draw names the last value that is kept)
        assert kept == (r % 2 == 0), (r, got, first, last, float(p))


@pytest.mark.parametrize("vocab", [65536, 204000, 393216, 409600])
def test_a_slice_in_one_bucket(vocab):
    """As much as a bucket can lack, by all values of a block's slice: the sums still fit."""
    from llm_singularity_b200 import kernels as ops
    half, d = vocab // 2, F(0.00977)
    rows = np.full((2, vocab), -3.0, dtype=F)
    rows[:, :half] = -d
    rows[:, 5] = 0.0
    a, b = 1.0 + (half - 1) * np.exp(-np.float64(d)), (vocab - half) * np.exp(-3.0)
    share = a / (a + b)
    params = torch.tensor([[1.0, share * 1.001, 1.0, 0.9999], [1.0, share * 0.999, 1.0, 0.9999]], dtype=torch.float32, device="cuda")
    out = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    ops.sample(torch.from_numpy(rows).cuda(), params, torch.zeros(2, dtype=torch.int32, device="cuda"), None, None, out)
    assert out[0].item() >= half > out[1].item() >= 0
