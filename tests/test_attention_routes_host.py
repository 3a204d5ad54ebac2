"""Where the attention kernel of any head size rotates single tokens by itself: steps of single tokens alone whose blocks fit 148 SMs,
two each, at once."""
import types

import numpy as np
import pytest

from llm_singularity_b200 import kernels as ops


@pytest.mark.parametrize("q_lens, nh, nkv, hd, rotates", [
    ([1] * 8, 32, 8, 64, True), ([1] * 37, 32, 8, 64, True), ([1] * 38, 32, 8, 64, False),       # 8 blocks a token: 296 at most
    ([1] * 18, 128, 8, 128, True), ([1] * 19, 128, 8, 128, False),                               # two blocks a kv head, of 8 heads each
    ([1] * 74, 32, 2, 128, True), ([1] * 75, 32, 2, 128, False),
    ([1, 40], 32, 8, 64, False), ([2], 32, 8, 64, False), ([1] * 7 + [2], 4, 2, 16, False), ([1], 4, 0, 16, False)])
def test_single_tokens_rotate(q_lens, nh, nkv, hd, rotates, monkeypatch):
    monkeypatch.setattr(ops, "num_sms", lambda device: 148)
    ctx = types.SimpleNamespace(h_q_len=np.array(q_lens, dtype=np.int32), n_requests=len(q_lens))
    assert ops._single_tokens_rotate(ctx, nh, nkv, hd, None) == rotates
