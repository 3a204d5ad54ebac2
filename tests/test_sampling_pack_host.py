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


def test_greedy_rows_are_not_asked_for_more_than_their_temperature():
    greedy = SamplingParams(temperature=0.0, top_k=2 ** 40)
    for draws in ([None, None], [], [2 ** 70, -1], [0.5, 1]):
        host, all_greedy, penal = _pack([greedy, greedy], draws)
        assert all_greedy and not penal and host[:8].reshape(2, 4)[:, 0].tolist() == [0.0, 0.0]
    assert _pack([greedy, SamplingParams(seed=3)], [None, 4])[0][7] == np.float32(uniform(3, 4))


@pytest.mark.parametrize("draw", [-1, 2 ** 63 - 1, 2 ** 63, 2 ** 64 + 5, 2 ** 90, np.int64(7)])
def test_any_whole_number_is_a_draw(draw):
    host, _, _ = _pack([SamplingParams(seed=11), SamplingParams(seed=12)], [draw, 1, 99])
    assert host[3] == np.float32(uniform(11, int(draw))) and host[7] == np.float32(uniform(12, 1))


def test_what_is_no_whole_number_or_too_large_is_refused():
    with pytest.raises(TypeError):
        _pack([SamplingParams()], [0.5])
    for k in (2 ** 31, 2 ** 63, 2 ** 80):
        with pytest.raises(OverflowError):
            _pack([SamplingParams(top_k=k)], [0])
