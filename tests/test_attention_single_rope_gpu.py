"""Single tokens that the generic attention kernel rotates and stores by itself, against the rotary kernel and attention one after the
other: every place of the token's key in a tile and a stretch, rotations of part of a head, tokens beside portions, caches that
another layer has written, groups of heads over several blocks."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 16


def _both(dtype, nh, nkv, hd, rotary, q_lens, kv_lens, window, store, captured):
    from llm_singularity_b200 import kernels as ops
    from llm_singularity_b200.engine.batch import ContextBuilder
    from llm_singularity_b200.parts.base import KVCacheView
    R, T, per = len(q_lens), sum(q_lens), -(-max(kv_lens) // PAGE)
    inv_freq = 500000.0 ** (-torch.arange(rotary // 2, device="cuda") / (rotary // 2))
    table = torch.randperm(R * per, generator=torch.Generator().manual_seed(2)).to(torch.int32).view(R, per).cuda()
    results = []
    for fuse in (False, True):
        g = torch.Generator(device="cuda").manual_seed(sum(kv_lens) + hd)
        kp, vp = (torch.randn(R * per, nkv, PAGE, hd, device="cuda", generator=g).to(dtype) for _ in range(2))
        if store:                                              # (what lies at the tokens' own places is not to be used)
            for r, L in enumerate(kv_lens):
                kp[table[r, (L - 1) // PAGE].long(), :, (L - 1) % PAGE] = float("nan")
                vp[table[r, (L - 1) // PAGE].long(), :, (L - 1) % PAGE] = float("inf")
        qkv = torch.randn(T, (nh + 2 * nkv) * hd, device="cuda", generator=g).to(dtype)
        ctx, _ = ContextBuilder("cuda", 4096, 64).build([[0] * n for n in q_lens], [k - q for k, q in zip(kv_lens, q_lens)],
                                                        list(range(R)), [[] for _ in range(R)])
        ctx.fixed_launch = captured
        out = torch.full((T, nh * hd), float("nan"), dtype=dtype, device="cuda")
        ops.FUSE_DECODE_ROPE = fuse
        try:
            ops.rope_store_attention(qkv, nh, nkv, hd, ctx, KVCacheView(kp, vp, table, PAGE, window or None, 0), inv_freq, rotary, store,
                                     1 / math.sqrt(hd), window, out)
        finally:
            ops.FUSE_DECODE_ROPE = True
        ops.check_status()
        results.append((out, kp, vp))
    (a, ka, va), (b, kb, vb) = results
    # the same rotation in 32-bit (a sum of two products may be rounded once or twice: 2^-24 of each), rounded to the type
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    if store:
        assert torch.equal(va, vb) and bool(((ka - kb).abs() <= 4 * eps * (1 + ka.abs())).all())
    a, b = a.double().view(T, nh, hd), b.double().view(T, nh, hd)
    if dtype == torch.bfloat16:
        # results are rounded once (2^-9 of each); a rotated element that is rounded the other way is 2^-8 of it off, which moves a
        # score of size 1 and the outputs of its head by no more than that; few are, so that all outputs together agree better still
        rms = a.square().mean(-1, keepdim=True).sqrt()
        assert bool(((a - b).abs() <= 2 * eps * (a.abs() + rms)).all()) and (a - b).norm().item() <= eps * a.norm().item()
    else:
        assert bool(((a - b).abs() <= 40 * eps * (1 + a.abs())).all())
    assert not b.isnan().any()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("dtype, nh, nkv, hd, rotary", [(torch.float32, 32, 8, 64, 64), (torch.float32, 6, 2, 48, 20), (torch.float32, 34, 2, 64, 64),
                                                        (torch.float32, 5, 5, 128, 6), (torch.bfloat16, 6, 1, 80, 80), (torch.float32, 14, 2, 256, 256)])
def test_rotation_and_store_by_the_attention_kernel(dtype, nh, nkv, hd, rotary, store, captured):
    _both(dtype, nh, nkv, hd, rotary, [1] * 6, [1, 16, 17, 64, 65, 1000], 0, store, captured)
    _both(dtype, nh, nkv, hd, rotary, [1] * 2, [300, 129], 40, store, captured)
    if not captured:
        _both(dtype, nh, nkv, hd, rotary, [1, 9, 1, 70], [33, 9, 700, 100], 0, store, captured)
