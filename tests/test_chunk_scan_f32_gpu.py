"""Prompt portions of a memory with a fixed decay, in chunks in 32-bit, against the token-by-token recurrence in float64:
what 32-bit keeps, the edges of the chunks, decays of one and of zero, and values that are no numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SLOTS = (1, 3, 0)


def _step(q_lens):
    from llm_singularity_b200.engine.batch import ContextBuilder
    R = len(q_lens)
    return ContextBuilder("cuda", 4096, 8).build([[0] * n for n in q_lens], [3] * R, [SLOTS[r] for r in range(R)], [[]] * R)[0]


def _inputs(q_lens, heads, key_heads, N, V, seed):
    g = torch.Generator().manual_seed(seed)
    rows = torch.randn(sum(q_lens), 2 * key_heads * N + heads * V, generator=g).to(torch.bfloat16)
    return rows, torch.randn(4, heads, V, N, generator=g)


def _recurrence(rows, start, decay, q_lens, heads, key_heads, N, V):
    qk = key_heads * N
    q, k = (rows[:, i * qk:(i + 1) * qk].double().view(-1, key_heads, N).repeat_interleave(heads // key_heads, 1) for i in (0, 1))
    v, d = rows[:, 2 * qk:].double().view(-1, heads, V), decay.double()[:, None, None]
    want, end, t = torch.empty(rows.shape[0], heads, V, dtype=torch.float64), start.double(), 0
    for r, n in enumerate(q_lens):
        S = end[SLOTS[r]]
        for _ in range(n):
            S = d * S + v[t][:, :, None] * k[t][:, None, :]
            want[t] = torch.einsum("hvn,hn->hv", S, q[t])
            t += 1
        end[SLOTS[r]] = S
    return want.view(rows.shape[0], -1), end


def _chunks(rows, start, decay, q_lens, heads, key_heads, N, V):
    from llm_singularity_b200 import kernels as K
    state, out, qk = start.cuda(), torch.zeros(rows.shape[0], heads * V, device="cuda"), key_heads * N
    K.chunk_scan(rows.cuda(), 0, qk, 2 * qk, heads, key_heads, N, V, state, _step(q_lens), out, 0,
                 log_decay=torch.log(decay.double()).float().cuda())
    K.check_status()
    return out.double().cpu(), state.double().cpu()


def _off(y, want):
    return ((y - want).norm() / want.norm()).item()


@pytest.mark.parametrize("q_lens", [[48], [64], [65, 1, 127], [128, 3, 2], [1500]])
@pytest.mark.parametrize("heads, key_heads, N, V", [(3, 3, 128, 128), (4, 2, 64, 72), (1, 1, 8, 128), (2, 2, 104, 16)])
def test_keeps_32_bits(q_lens, heads, key_heads, N, V):
    from llm_singularity_b200 import kernels as K
    rows, start = _inputs(q_lens, heads, key_heads, N, V, N + V + sum(q_lens))
    decay = torch.tensor([1.0 - 2.0 ** -7, 0.97, 1e-3, 0.9][:heads])
    want, end = _recurrence(rows, start, decay, q_lens, heads, key_heads, N, V)
    y, state = _chunks(rows, start, decay, q_lens, heads, key_heads, N, V)
    # Sums of some hundred 32-bit terms of either sign: 2^-24 a rounding, a few of them a term.  (Operands held as two
    # bfloat16 numbers, 2^-17 each, would give some 5e-6.)
    assert _off(y, want) < 5e-7 and _off(state, end) < 5e-7
    # no further off than the walk
    walked, out, ctx = start.cuda(), torch.zeros(rows.shape[0], heads * V, device="cuda"), _step(q_lens)
    K.linear_scan(rows.cuda(), 0, key_heads * N, 2 * key_heads * N, heads, N, V, "fixed_decay", decay.cuda(), None, None,
                  "none", "none", "none", walked, ctx, out, key_heads=key_heads)
    assert _off(y, want) < 1.25 * _off(out.double().cpu(), want) and _off(state, end) < 1.25 * _off(walked.double().cpu(), end) + 1e-8


@pytest.mark.parametrize("a", [0.0, 1.0])
def test_decays_at_the_ends(a):
    q_lens, decay = [130, 5], torch.tensor([a, 0.5])
    rows, start = _inputs(q_lens, 2, 2, 64, 64, 5)
    want, end = _recurrence(rows, start, decay, q_lens, 2, 2, 64, 64)
    y, state = _chunks(rows, start, decay, q_lens, 2, 2, 64, 64)
    assert _off(y, want) < 5e-7 and _off(state, end) < 5e-7


@pytest.mark.parametrize("column", ["q", "k", "v"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_what_is_no_number_touches_no_earlier_token(column, bad):
    q_lens, decay, at = [150, 90], torch.tensor([0.9, 0.99]), 100
    rows, start = _inputs(q_lens, 2, 2, 64, 128, 6)
    rows[at, {"q": 5, "k": 128 + 5, "v": 256 + 5}[column]] = bad          # (the first head's)
    want, end = _recurrence(rows, start, decay, q_lens, 2, 2, 64, 128)
    y, state = _chunks(rows, start, decay, q_lens, 2, 2, 64, 128)
    # (an infinity and its successors may have become NaN: infinities of either sign meet)
    assert torch.equal(y.isfinite(), want.isfinite()) and torch.equal(state.isfinite(), end.isfinite())
    fine = want.isfinite()
    assert bool(fine[:at].all()) and bool(fine[150:].all()) and not bool(fine[at].all())
    assert _off(y[fine], want[fine]) < 5e-7
