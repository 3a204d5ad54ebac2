"""A memory with a fixed decay whose queries, keys and values pass silu on their way into the chunked form, against the
token-by-token recurrence in float64, beside the walk."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("acts", [("silu", "silu", "silu"), ("silu", "silu", "none"), ("none", "none", "silu"), ("none", "silu", "none")])
@pytest.mark.parametrize("q_lens", [[48], [1, 1, 129], [1, 128, 60], [300, 1, 2]])
@pytest.mark.parametrize("heads, N, V", [(3, 128, 128), (2, 64, 72), (1, 8, 128), (2, 104, 16)])
def test_against_the_recurrence(acts, q_lens, heads, N, V):
    from llm_singularity_b200 import kernels as K
    from llm_singularity_b200.engine.batch import ContextBuilder
    g = torch.Generator().manual_seed(N + V + len(q_lens))
    R, T, qk = len(q_lens), sum(q_lens), heads * N
    ctx, _ = ContextBuilder("cuda", 1024, 8).build([[0] * n for n in q_lens], [3] * R, [(1, 3, 0)[r] for r in range(R)], [[]] * R)
    rows = torch.randn(T, 2 * qk + heads * V, generator=g).to(torch.bfloat16)
    start = torch.randn(4, heads, V, N, generator=g)
    decay = torch.tensor([1.0, 0.97, 1e-3][:heads])
    q, k, v = (torch.nn.functional.silu(x) if a == "silu" else x
               for x, a in zip((rows[:, :qk].double(), rows[:, qk:2 * qk].double(), rows[:, 2 * qk:].double()), acts))
    want, end, t = torch.empty(T, heads, V, dtype=torch.float64), start.double(), 0
    for r, n in enumerate(q_lens):
        S = end[(1, 3, 0)[r]]
        for _ in range(n):
            S = decay.double()[:, None, None] * S + v[t].view(heads, V, 1) * k[t].view(heads, 1, N)
            want[t] = torch.einsum("hvn,hn->hv", S, q[t].view(heads, N))
            t += 1
        end[(1, 3, 0)[r]] = S
    log_decay = torch.log(decay.double()).float().cuda()
    # silu is good to 2^-20, up to three of them in a term, the terms' errors of either sign (what 32-bit sums keep is
    # held far closer where no silu stands in front, tests/test_chunk_scan_f32_gpu.py)
    tol = 3e-5
    for chunked in (False, True):
        state, out = start.cuda(), torch.zeros(T, heads * V, device="cuda")
        first = K.chunk_scan_first(ctx, torch.bfloat16, N, V) if chunked else None
        if first != 0:
            K.linear_scan(rows.cuda(), 0, qk, 2 * qk, heads, N, V, "fixed_decay", decay.cuda(), None, None, *acts, state, ctx, out,
                          q_scale=0.5, requests=first)
        if first is not None:
            K.chunk_scan(rows.cuda(), 0, qk, 2 * qk, heads, heads, N, V, state, ctx, out, first, log_decay=log_decay, q_scale=0.5, acts=acts)
        assert (out.double().cpu() - 0.5 * want.view(T, -1)).abs().max() < tol * want.abs().max(), chunked
        assert (state.double().cpu() - end).abs().max() < tol * end.abs().max(), chunked
    K.check_status()
