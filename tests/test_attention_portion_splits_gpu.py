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
