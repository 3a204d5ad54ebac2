"""The rows the sampling kernel reads, packed by the host library, against the plain statement of their draws."""
import numpy as np
import pytest

from llm_singularity_b200.sampling import SamplingParams, uniform
from llm_singularity_b200.sampling.sampler import _pack


@pytest.mark.parametrize("n", [1, 2, 33])
def test_rows_are_what_the_settings_say(n):
    seeds = [0, 1, -1, 2 ** 63, 2 ** 64 - 1, 2 ** 70 + 5, -2 ** 65 + 3]
    params = [SamplingParams(temperature=0.0 if r % 3 == 0 else 0.1 + r, top_k=(0, 50, 2 ** 31 - 1)[r % 3], top_p=1.0 if r % 2 else 0.9,
                             seed=seeds[r % len(seeds)]) for r in range(n)]
    draws = [0, 7, 2 ** 40][:n] + list(range(3, n))
    host, greedy, penal = _pack(params, draws)
    rows, top_k = host[:4 * n].reshape(n, 4), host[4 * n:].view(np.int32)
    want = np.array([[p.temperature, p.top_p, 1.0, 0.5 if p.greedy else uniform(p.seed, d)] for p, d in zip(params, draws)], dtype=np.float32)
    assert np.array_equal(rows, want) and top_k.tolist() == [p.top_k for p in params]
    assert greedy == (n == 1) and not penal
    assert _pack([SamplingParams(temperature=0.0, repetition_penalty=1.1)], [0])[1:] == (True, True)


def test_what_does_not_fit_is_refused():
    with pytest.raises(OverflowError):
        _pack([SamplingParams(top_k=2 ** 31)], [0])
    with pytest.raises(ValueError):
        _pack([SamplingParams()], [])
