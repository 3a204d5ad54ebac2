"""The chain through a portion's chunks takes 8 or 24 at a time: lengths around one and two such batches, beside a short request,
against the token-by-token recurrence in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [8 * 64, 8 * 64 + 1, 24 * 64 - 1, 24 * 64, 24 * 64 + 1, 25 * 64, 48 * 64 + 1])
def test_chunks_in_batches(tokens):
    from llm_singularity_b200 import kernels as K
    from llm_singularity_b200.engine.batch import ContextBuilder
    N, V, heads, lens, slots = 16, 24, 2, (70, tokens), (2, 0)
    g = torch.Generator().manual_seed(tokens)
    rows = torch.randn(sum(lens), heads * (2 * N + V), generator=g).to(torch.bfloat16)
    start, decay = torch.randn(3, heads, V, N, generator=g), torch.tensor([1.0 - 2.0 ** -7, 0.97])
    q, k = (rows[:, i * heads * N:(i + 1) * heads * N].double().view(-1, heads, N) for i in (0, 1))
    v, d = rows[:, 2 * heads * N:].double().view(-1, heads, V), decay.double()[:, None, None]
    want, end, t = torch.empty(len(rows), heads, V, dtype=torch.float64), start.double(), 0
    for slot, n in zip(slots, lens):
        S = end[slot]
        for _ in range(n):
            S = d * S + v[t][:, :, None] * k[t][:, None, :]
            want[t] = (S * q[t][:, None, :]).sum(-1)
            t += 1
        end[slot] = S
    ctx = ContextBuilder("cuda", 4096, 8).build([[0] * n for n in lens], [3, 3], list(slots), [[]] * 2)[0]
    state, out = start.cuda(), torch.zeros(len(rows), heads * V, device="cuda")
    K.chunk_scan(rows.cuda(), 0, heads * N, 2 * heads * N, heads, heads, N, V, state, ctx, out, 0,
                 log_decay=torch.log(decay.double()).float().cuda())
    K.check_status()
    # (the bound of the other lengths: sums of some hundred 32-bit terms of either sign, 2^-24 a rounding)
    for y, w in ((out.double().cpu().view_as(want), want), (state.double().cpu(), end)):
        assert ((y - w).norm() / w.norm()).item() < 5e-7
