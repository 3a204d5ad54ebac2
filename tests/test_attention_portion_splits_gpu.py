"""Portions whose keys are shared out over a cluster, where it can go wrong: stretches without a key, tiles cut short, windows that leave
a block nothing, groups of heads that do not fill a block's rows, and what is no number in one stretch only."""
import pytest
import torch

from test_attention_generic_gpu import _poisoned, _run

pytestmark = pytest.mark.gpu

CASES = [([40], [340], 32, 8, 64), ([2], [1000], 4, 1, 64), ([17, 1, 65], [817, 40, 65], 8, 2, 64), ([120], [420], 6, 2, 128), ([33], [700], 6, 2, 256),
         ([240], [240], 32, 8, 64), ([500], [500], 32, 8, 64), ([3], [65], 5, 1, 16)]


@pytest.mark.parametrize("q, kv, nh, nkv, hd", CASES)
@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("captured", [False, True])
def test_portions_over_a_cluster(q, kv, nh, nkv, hd, window, captured):
    _run(torch.float32, nh, nkv, hd, q, kv, window, 0.0, False, captured)


@pytest.mark.parametrize("what", ["keys", "values"])
def test_no_number_in_one_stretch(what):
    _poisoned(what, torch.float32, 8, 2, 64, [20, 3], [420, 300], 0, [[70, 415], [299]])
    _poisoned(what, torch.bfloat16, 6, 1, 80, [20], [420], 60, [[0, 200, 395, 419]])


def _portion_beside(single_keys, tokens, keys, window):
    """The outputs of one portion beside a single token with so many keys."""
    from llm_singularity_b200 import kernels as ops
    from llm_singularity_b200.engine.batch import ContextBuilder
    from llm_singularity_b200.parts.base import KVCacheView
    g = torch.Generator(device="cuda").manual_seed(keys)
    ctx, _ = ContextBuilder("cuda", 4096, 64).build([[0] * tokens, [0]], [keys - tokens, single_keys - 1], [0, 1], [[], []])
    own, per = -(-keys // 16), -(-max(keys, single_keys) // 16)
    kp, vp = (torch.randn(own, 8, 16, 64, device="cuda", generator=g) for _ in range(2))
    qkv = torch.randn(tokens + 1, 48 * 64, device="cuda", generator=g)
    table = (torch.arange(2 * per, device="cuda", dtype=torch.int32) % own).view(2, per).contiguous()
    out = torch.empty(tokens + 1, 32 * 64, device="cuda")
    ops.paged_attention(qkv, 32, 8, 64, ctx, KVCacheView(kp, vp, table, 16, window or None, 0), 0.125, window, out)
    ops.check_status()
    return out[:tokens]


@pytest.mark.parametrize("tokens, keys, window", [(300, 300, 0), (40, 340, 0), (40, 40, 0), (300, 900, 100)])
def test_a_long_single_token_leaves_a_portion_alone(tokens, keys, window):
    """How a portion's keys are shared out follows the portions' contexts: the same bits beside 40 keys and beside 4,000."""
    assert torch.equal(_portion_beside(40, tokens, keys, window), _portion_beside(4000, tokens, keys, window))


def test_parts_follow_what_blocks_walk():
    """32 / 8 heads of 64 on 148 SMs: whole blocks where there is one tile of keys, where a window leaves a few, and where they fill the
    SMs for long; several where few blocks walk many tiles.  Contexts of 0 are not known (captured), a window still is."""
    from llm_singularity_b200 import kernels as ops
    parts = ops._lib("attention").lsb_portion_splits
    for tokens, keys, window, whole in [(40, 40, 0, True), (500, 4000, 0, True), (500, 4000, 100, True), (500, 4000, 1000, True),
                                        (2000, 2000, 256, True), (500, 0, 1000, True), (2000, 0, 256, True), (40, 340, 0, False),
                                        (40, 4000, 100, False), (40, 0, 100, False), (240, 240, 0, False), (40, 4000, 0, False)]:
        assert (parts(64, 32, 8, 1, tokens, keys, window) == 1) == whole, (tokens, keys, window)
