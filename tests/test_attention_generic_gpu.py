"""The attention kernels of any head size: stretches of a single token's keys that are empty, one key or ragged, portions
on the edges of a block's rows, groups that need several blocks, windows and both score modifiers, against 64-bit."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 16


def _run(dtype, nh, nkv, hd, q_lens, kv_lens, window, softcap, bias, captured):
    from llm_singularity_b200 import kernels as ops
    from llm_singularity_b200.engine.batch import ContextBuilder
    from llm_singularity_b200.parts.base import KVCacheView
    g = torch.Generator(device="cuda").manual_seed(sum(kv_lens) + hd)
    R, T = len(q_lens), sum(q_lens)
    ctx, _ = ContextBuilder("cuda", 4096, 64).build([[0] * n for n in q_lens], [k - q for k, q in zip(kv_lens, q_lens)],
                                                    list(range(R)), [[] for _ in range(R)])
    ctx.fixed_launch = captured
    per = -(-max(kv_lens) // PAGE)
    table = torch.randperm(R * per, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(R, per).cuda()
    kp, vp = (torch.randn(R * per, nkv, PAGE, hd, device="cuda", generator=g).to(dtype) for _ in range(2))
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, device="cuda", generator=g).to(dtype)
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / nh) for h in range(nh)], device="cuda") if bias else None
    out = torch.full((T, nh * hd), float("nan"), dtype=dtype, device="cuda")
    scale = 1.0 / math.sqrt(hd)
    ops.paged_attention(qkv, nh, nkv, hd, ctx, KVCacheView(kp, vp, table, PAGE, window or None, 0), scale, window, out,
                        softcap=softcap, slopes=slopes)
    ops.check_status()
    t, group = 0, nh // nkv
    for r in range(R):
        n, L = q_lens[r], kv_lens[r]
        rows = table[r, :-(-L // PAGE)].long()
        K, V = (p[rows].transpose(1, 2).reshape(-1, nkv, hd)[:L].double().repeat_interleave(group, 1) for p in (kp, vp))
        q = qkv[t:t + n, :nh * hd].double().view(n, nh, hd)
        s = torch.einsum("ihd,jhd->hij", q, K) * scale
        pos, key = torch.arange(L - n, L, device="cuda")[:, None], torch.arange(L, device="cuda")
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if bias:
            s = s - slopes.double()[:, None, None] * (pos - key)
        s = s.masked_fill((key > pos) | ((key <= pos - window) if window else False), -math.inf)
        want = torch.einsum("hij,jhd->ihd", torch.softmax(s, -1), V).reshape(n, nh * hd)
        # scores of size s are off by some 2^-22 |s| (32-bit sums of hd terms), and a result by as much of |V|;
        # a bfloat16 result is rounded once more
        size = V.abs().max().item() * (1 + s[s > -math.inf].abs().max().item())
        tol = size * 2.0 ** -20 + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0)
        assert bool(((out[t:t + n].double() - want).abs() <= tol).all()), r
        t += n


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("window, softcap, bias", [(0, 0.0, False), (40, 0.0, False), (0, 2.5, True), (7, 1.5, True)])
@pytest.mark.parametrize("dtype, nh, nkv, hd", [(torch.float32, 8, 2, 64), (torch.float32, 6, 2, 48), (torch.float32, 5, 5, 128),
                                                (torch.float32, 14, 2, 256), (torch.float32, 80, 1, 16),
                                                (torch.float32, 34, 2, 64), (torch.bfloat16, 6, 1, 80)])
def test_edges(dtype, nh, nkv, hd, window, softcap, bias, captured):
    _run(dtype, nh, nkv, hd, [1, 1, 1, 1], [1, 17, 129, 1000], window, softcap, bias, captured)
    if not captured:
        _run(dtype, nh, nkv, hd, [1, 2, 16, 17, 65, 1], [64, 2, 16, 81, 130, 65], window, softcap, bias, False)


def test_many_requests_leave_the_keys_whole():
    _run(torch.float32, 4, 4, 32, [1] * 60 + [3] * 4, [5 + 37 * i % 300 for i in range(64)], 0, 0.0, False, False)


def _poisoned(what, dtype, nh, nkv, hd, q_lens, kv_lens, window, spots):
    """Attention over a cache in which request r's key or value at each of spots[r] holds numbers that are none, and what
    64-bit sums over each row's own keys alone make of it."""
    from llm_singularity_b200 import kernels as ops
    from llm_singularity_b200.engine.batch import ContextBuilder
    from llm_singularity_b200.parts.base import KVCacheView
    g = torch.Generator(device="cuda").manual_seed(sum(kv_lens) + hd)
    R, T, group = len(q_lens), sum(q_lens), nh // nkv
    ctx, _ = ContextBuilder("cuda", 4096, 64).build([[0] * n for n in q_lens], [k - q for k, q in zip(kv_lens, q_lens)],
                                                    list(range(R)), [[] for _ in range(R)])
    per = -(-max(kv_lens) // PAGE)
    table = torch.arange(R * per, dtype=torch.int32).view(R, per).cuda()
    kp, vp = (torch.randn(R * per, nkv, PAGE, hd, device="cuda", generator=g).to(dtype) for _ in range(2))
    bad = [float("nan"), float("inf"), -float("inf")]
    for r, at in enumerate(spots):
        for i, key in enumerate(at):
            (kp if what == "keys" else vp)[r * per + key // PAGE, i % nkv, key % PAGE, (5 * i) % hd] = bad[i % 3]
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, device="cuda", generator=g).to(dtype)
    out, scale = torch.zeros(T, nh * hd, dtype=dtype, device="cuda"), 1.0 / math.sqrt(hd)
    ops.paged_attention(qkv, nh, nkv, hd, ctx, KVCacheView(kp, vp, table, PAGE, window or None, 0), scale, window, out)
    ops.check_status()
    t, same = 0, 0
    for r in range(R):
        n, L = q_lens[r], kv_lens[r]
        K, V = (p[r * per:(r + 1) * per].transpose(1, 2).reshape(-1, nkv, hd).double().repeat_interleave(group, 1) for p in (kp, vp))
        for i in range(n):
            pos = L - n + i
            seen = slice(max(0, pos - window + 1) if window else 0, pos + 1)
            s = torch.einsum("hd,jhd->hj", qkv[t + i, :nh * hd].double().view(nh, hd), K[seen]) * scale
            w = torch.softmax(s, -1)
            want = torch.einsum("hj,jhd->hd", w, V[seen]).reshape(-1)
            y = out[t + i].double()
            assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf()), (r, i)
            fine = want.isfinite()
            same += int(fine.sum())
            size = 6.0 * (1 + s[s.isfinite()].abs().max().item())
            tol = size * 2.0 ** -20 + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0)
            assert bool(((y - want).abs() <= tol)[fine].all()) and torch.equal(y[want.isinf()], want[want.isinf()]), (r, i)
        t += n
    assert same > 0 and same < out.numel()


SIZES = [(torch.float32, 8, 2, 64), (torch.float32, 4, 4, 128), (torch.float32, 6, 2, 256), (torch.bfloat16, 6, 1, 80)]


@pytest.mark.parametrize("what", ["keys", "values"])
@pytest.mark.parametrize("dtype, nh, nkv, hd", SIZES)
def test_single_tokens_that_see_no_number(what, dtype, nh, nkv, hd):
    _poisoned(what, dtype, nh, nkv, hd, [1, 1, 1, 1], [1, 40, 700, 300], 0, [[], [3], [0, 500, 699], []])
    _poisoned(what, dtype, nh, nkv, hd, [1, 1], [300, 300], 50, [[100, 249], [250]])


@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("what", ["keys", "values"])
@pytest.mark.parametrize("dtype, nh, nkv, hd", SIZES)
def test_portions_beside_what_is_no_number(what, dtype, nh, nkv, hd, window):
    """Only the rows that see such a key or value are affected: not those before it, nor those whose window has passed it."""
    _poisoned(what, dtype, nh, nkv, hd, [100, 2, 33], [100, 90, 140], window, [[50, 71, 99], [], [20, 110, 130]])
