"""A small k, whose cuts and draw are made among the values that the maxima of a row's stretches lead to: k on both sides of
what they are looked up for, ties, masked rows, and the same tokens however many rows share the device."""
import numpy as np
import pytest
import torch

from test_sampling_cuts_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 63, 64, 127, 128, 129, 300])
@pytest.mark.parametrize("vocab", [1023, 1025, 25600, 32000, 128256, 262145])
def test_small_k(vocab, k):
    rows = (np.random.RandomState(vocab + k).randn(4, vocab) * 3).astype(np.float32)
    check(rows, [(0.8, k, 1.0), (1.7, k, 0.9), (0.01, k, 0.5), (1.0, k, 0.05)], seed=k)


@pytest.mark.parametrize("kind", ["ties", "few values", "negative", "tiny", "huge", "infinite"])
def test_small_k_of_rows_out_of_the_ordinary(kind):
    rng = np.random.RandomState(11)
    rows = (rng.randn(4, 60000) * 3).astype(np.float32)
    if kind == "ties":
        rows = np.round(rows)                                  # (a thousand values and more equal the k-th)
    elif kind == "few values":
        rows[:, 30:] = -np.inf
    elif kind == "negative":
        rows -= 1000.0
    elif kind == "tiny":
        rows *= np.float32(1e-30)
    elif kind == "huge":
        rows *= np.float32(1e30)
    else:
        rows[:, 41234] = np.inf
        check_infinite(rows)
        return
    check(rows, [(0.8, 40, 1.0), (1.0, 40, 0.9), (3.0, 100, 1.0), (0.5, 1, 1.0)], seed=5)


def check_infinite(rows):
    """No value has a mass beside an infinity: the maximum is named."""
    from llm_singularity_b200 import kernels as ops
    for k in (1, 40):
        out = torch.full((4,), -1, dtype=torch.int32, device="cuda")
        ops.sample(torch.from_numpy(rows).cuda(), torch.tensor([[0.8, 0.9, 1.0, 0.3]] * 4, device="cuda"),
                   torch.full((4,), k, dtype=torch.int32, device="cuda"), None, None, out)
        assert out.tolist() == [41234] * 4


@pytest.mark.parametrize("vocab", [50257, 128256])
def test_tokens_do_not_depend_on_the_rows_beside_them(vocab):
    from llm_singularity_b200 import kernels as ops
    kinds = [(0.0, 0, 1.0), (0.8, 0, 1.0), (0.8, 50, 1.0), (1.0, 0, 0.9), (0.7, 40, 0.95), (1.5, 500, 0.95), (2.0, 0, 0.9999)]
    rng = np.random.RandomState(vocab)
    logits = torch.from_numpy((rng.randn(200, vocab) * 3).astype(np.float32)).cuda()
    kd = [kinds[r % len(kinds)] for r in range(200)]
    params = torch.tensor([[t, p, 1.0, float(u)] for (t, _, p), u in zip(kd, rng.rand(200))], device="cuda")
    top_k = torch.tensor([k for _, k, _ in kd], dtype=torch.int32, device="cuda")
    out = {}
    for n in (200, 50, 7):
        got = torch.full((200,), -1, dtype=torch.int32, device="cuda")
        for r in range(0, 200, n):
            e = min(200, r + n)
            ops.sample(logits[r:e], params[r:e], top_k[r:e], None, None, got[r:e])
        out[n] = got.tolist()
    assert out[200] == out[50] == out[7]


@pytest.mark.parametrize("rows, vocab", [(3, 32000), (30, 128256), (3, 377003)])
def test_penalties_beside_rows_without(rows, vocab):
    """Rows with tokens to penalise are what the same rows are with their logits changed beforehand."""
    from llm_singularity_b200 import kernels as ops
    rng = np.random.RandomState(rows)
    logits = torch.from_numpy((rng.randn(rows, vocab) * 3).astype(np.float32)).cuda()
    kinds = [(0.0, 0, 1.0, 1.3), (0.8, 40, 0.9, 1.3), (1.0, 0, 0.9, 0.7), (0.8, 0, 1.0, 1.0), (0.7, 400, 1.0, 1.2)]
    kd = [kinds[r % len(kinds)] for r in range(rows)]
    u = rng.rand(rows)
    top_k = torch.tensor([k for _, k, _, _ in kd], dtype=torch.int32, device="cuda")
    changed, prev, start = logits.clone(), [], [0]
    for r, (_, _, _, pen) in enumerate(kd):
        tokens = torch.topk(logits[r], 20).indices.tolist() + rng.randint(0, vocab, 30).tolist()
        prev += tokens
        start.append(len(prev))
        for t in tokens:
            x = changed[r, t]
            changed[r, t] = x / pen if x > 0 else x * pen
    got, want = (torch.full((rows,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    ops.sample(logits, torch.tensor([[t, p, pen, float(v)] for (t, _, p, pen), v in zip(kd, u)], device="cuda"), top_k,
               torch.tensor(start, dtype=torch.int32, device="cuda"), torch.tensor(prev, dtype=torch.int32, device="cuda"), got)
    ops.sample(changed, torch.tensor([[t, p, 1.0, float(v)] for (t, _, p, _), v in zip(kd, u)], device="cuda"), top_k, None, None, want)
    assert got.tolist() == want.tolist()
