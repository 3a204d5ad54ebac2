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


@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("requests", [37, 56, 64, 75, 111, 112, 128, 129])
def test_rounds_that_rotate_and_store(requests, hd, store, monkeypatch):
    """The engine's form: the kernel rotates the tokens and puts their keys and values (poisoned before) into the right pages, whatever
    order the blocks take the requests in; lengths around the ring's, and as unlike as just keeps and just changes the order."""
    from llm_singularity_b200 import kernels as K
    from llm_singularity_b200.engine.batch import ContextBuilder
    monkeypatch.setattr(K, "_check_cache", lambda *a: None)
    nkv, group, rotary, apart = 8, 4, 48, 131072 // (4 * hd)
    inv_freq = 500000.0 ** (-torch.arange(rotary // 2, device="cuda") / (rotary // 2))
    ring = [1, 2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 192, 193, 255, 256, 257]
    for lens, window in (([ring[r * 5 % 17] for r in range(requests)], 0), ([40 + (r * 7 % 5 == 2) * apart for r in range(requests)], 0),
                         ([40 + (r * 7 % 5 == 2) * (apart + 1) for r in range(requests)], 0), ([200 * (1 + r % 3) for r in range(requests)], 90)):
        outs, pages = [], []
        for fuse in (False, True):
            cache, qkv = _setup(lens, [1] * requests, nkv, hd, group, requests)
            if store:
                for r, n in enumerate(lens):
                    cache.k_pages[cache.block_table[r, (n - 1) // PAGE].long(), :, (n - 1) % PAGE] = float("nan")
                    cache.v_pages[cache.block_table[r, (n - 1) // PAGE].long(), :, (n - 1) % PAGE] = float("inf")
            ctx = ContextBuilder("cuda", 4096, 256).build([[0]] * requests, [n - 1 for n in lens], list(range(requests)), [[]] * requests)[0]
            out = torch.full((requests, nkv * group * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
            monkeypatch.setattr(K, "FUSE_DECODE_ROPE", fuse)
            K.rope_store_attention(qkv, nkv * group, nkv, hd, ctx, cache, inv_freq, rotary, store, hd ** -0.5, window, out)
            K.check_status()
            outs.append(out.float())
            pages.append((cache.k_pages, cache.v_pages))
            if not fuse:
                want = _oracle(cache, qkv, lens, [1] * requests, nkv, hd, group, window)       # (qkv and pages are rotated by now)
        (ka, va), (kb, vb) = pages
        # the same rotation in 32-bit, where a sum of two products may be rounded once or twice, before it is rounded to bfloat16
        assert torch.equal(va, vb) and bool(((ka.float() - kb.float()).abs() <= 2.0 ** -7 * ka.float().abs()).all())
        for out in outs:                                       # (bounds as above)
            assert (out - want).abs().max().item() < 4 * 2.0 ** -8 + 2.0 ** -8
            assert ((out - want).norm() / want.norm()).item() < 2 * 2.0 ** -8
