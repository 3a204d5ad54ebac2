"""Single tokens at the batch sizes around which the decode kernel takes its deeper ring or deals requests out longest first
(whole rounds of blocks on 148 SMs), ragged and alike, with a window, beside a prompt portion, against float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 16


class _Cache:
    pass


def _setup(lens, q_lens, nkv, hd, group, seed):
    g = torch.Generator().manual_seed(seed)
    need = [-(-n // PAGE) for n in lens]
    pages, order, at = sum(need), torch.randperm(sum(need), generator=g).int(), 0
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    for r, n in enumerate(need):
        table[r, :n] = order[at:at + n]
        at += n
    cache = _Cache()
    cache.k_pages, cache.v_pages = (torch.randn(pages, nkv, PAGE, hd, generator=g).bfloat16().cuda() for _ in range(2))
    cache.block_table, cache.page_size = table.cuda(), PAGE
    qkv = torch.randn(sum(q_lens), (nkv * group + 2 * nkv) * hd, generator=g).bfloat16().cuda()
    return cache, qkv


def _oracle(cache, qkv, lens, q_lens, nkv, hd, group, window):
    out, t = torch.zeros(len(qkv), nkv * group, hd, device="cuda"), 0
    for r, (n, m) in enumerate(zip(lens, q_lens)):
        own = cache.block_table[r, :-(-n // PAGE)].long()
        k, v = (x[own].transpose(1, 2).reshape(-1, nkv, hd)[:n].float().repeat_interleave(group, 1)
                for x in (cache.k_pages, cache.v_pages))
        q = qkv[t:t + m, :nkv * group * hd].float().view(m, nkv * group, hd)
        s = torch.einsum("qhd,khd->hqk", q, k) * hd ** -0.5
        place, key = torch.arange(n - m, n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
        s = s.masked_fill((key > place) | ((key <= place - window) if window else (key < 0)), float("-inf"))
        out[t:t + m] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v)
        t += m
    return out.view(len(qkv), -1)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("requests", [37, 38, 55, 56, 74, 75, 111, 112, 128, 129])
def test_rounds_of_blocks(requests, hd, monkeypatch):
    from llm_singularity_b200 import kernels as K
    from llm_singularity_b200.engine.batch import ContextBuilder
    monkeypatch.setattr(K, "_check_cache", lambda *a: None)
    nkv, g = 8, torch.Generator().manual_seed(requests + hd)
    ragged = torch.randint(1, 400, (requests,), generator=g).tolist()
    ragged[requests // 2], ragged[-1], ragged[0] = 1300, 1, ragged[1]        # the longest in the middle, two alike
    for lens, portion, group, window in ((ragged, 1, 4, 0), (ragged, 5, 3, 70), ([129] * requests, 1, 12, 0)):
        q_lens = [1] * requests
        q_lens[3], lens = portion, [max(n, portion) if r == 3 else n for r, n in enumerate(lens)]
        cache, qkv = _setup(lens, q_lens, nkv, hd, group, requests)
        ctx = ContextBuilder("cuda", 4096, 256).build([[0] * m for m in q_lens], [n - m for n, m in zip(lens, q_lens)],
                                                      list(range(requests)), [[]] * requests)[0]
        out = torch.full((len(qkv), nkv * group * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.paged_attention(qkv, nkv * group, nkv, hd, ctx, cache, hd ** -0.5, window, out)
        K.check_status()
        want = _oracle(cache, qkv, lens, q_lens, nkv, hd, group, window)
        # weights and results are rounded to bfloat16 (2^-9 each, of values up to about 4); sums of weights keep 32 bits
        assert (out.float() - want).abs().max().item() < 4 * 2.0 ** -8 + 2.0 ** -8
        assert ((out.float() - want).norm() / want.norm()).item() < 2 * 2.0 ** -8
