"""Sampler: one token per row of logits, on the device.

Greedy, temperature, top-k, top-p and repetition penalty in the reference's
order (core/src/sampling.cpp:11-118), done by the ``sampling`` kernel library; the
host only packs the per-row parameters and the uniform draws.  The reference
never passes previous tokens to its sampler (app/main.cpp:308-310), which leaves
its penalty without effect; here the request's generated tokens are passed.
"""
from __future__ import annotations

from array import array
from operator import index
from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from ..cache import native
from .params import SamplingParams


def _pack(params: Sequence[SamplingParams], draw_index: Sequence[int]) -> Tuple[np.ndarray, bool, bool]:
    """(float32 [5 R]: the rows of (temperature, top_p, penalty, u), then the rows' top_k as int32 bits; whether all rows
    are greedy; whether one has a repetition penalty).  ``rng.uniform`` states the draws."""
    R = len(params)
    try:
        draws = array("q", draw_index)
    except (TypeError, OverflowError):               # (a greedy row's draw is not looked at; others are whole numbers, modulo 2^64)
        draws = array("Q", [0 if p.greedy else index(n) & (1 << 64) - 1 for p, n in zip(params, draw_index)])
    if len(draws) < R:
        if not all(p.greedy for p in params[len(draws):]):
            raise ValueError("one draw index per SamplingParams")
        draws.extend([0] * (R - len(draws)))
    host = np.empty(5 * R, dtype=np.float32)
    flags = native.lib().lsbh_pack_sampling(R, b"".join([p.packed for p in params]), draws.buffer_info()[0],
                                            host.ctypes.data, host.ctypes.data + 16 * R)
    if flags < 0:
        raise OverflowError(f"top_k {params[-flags - 1].top_k} does not fit 32 bits")
    return host, not flags & 1, bool(flags & 2)


def _rows(buf: torch.Tensor, R: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """(params [R, 4], top_k [R]) in a device copy of such an array."""
    return buf[:4 * R].view(R, 4), buf[4 * R:].view(torch.int32)


class StagedSampling:
    """Per-row sampling parameters already on the device, in arrays that keep their addresses from
    step to step (one set per number of rows), and the launch that uses them.  Calling it is the
    same work every time, so a decode step captured in a CUDA graph can hold it."""

    def __init__(self, ops, buf: torch.Tensor, out: torch.Tensor):
        self.ops, self.buf, self.out = ops, buf, out
        self.params, self.top_k = _rows(buf, out.shape[0])
        self.key = ("sample", out.shape[0])

    def __call__(self, logits: torch.Tensor) -> torch.Tensor:
        self.ops.sample(logits, self.params, self.top_k, None, None, self.out)
        return self.out


class Sampler:
    def __init__(self, rt):
        self.rt = rt
        self._greedy = {}               # batch size -> device arrays for all-greedy batches
        self._staged = {}               # batch size -> StagedSampling
        prepare = getattr(rt.ops, "prepare", None)
        if prepare is not None:
            prepare(["sampling"])

    def stage(self, params: Sequence[SamplingParams], draw_index: Sequence[int]) -> Optional[StagedSampling]:
        """Put this step's per-row parameters and uniform draws into the persistent device arrays
        of their batch size and return the launch that samples with them; None where a repetition
        penalty is in use (it needs the generated tokens, packed per step by :meth:`sample`)."""
        R = len(params)
        if R == 0:
            return None
        host, greedy, penal = _pack(params, draw_index)
        if penal:
            return None
        st = self._staged.get(R)
        if st is None:
            dev = self.rt.device
            st = self._staged[R] = StagedSampling(self.rt.ops, torch.from_numpy(host).to(dev),
                                                  torch.empty(R, dtype=torch.int32, device=dev))
            st.greedy = greedy
            return st
        if greedy and st.greedy:                         # nothing has changed since the last all-greedy step
            return st
        # (a pageable host array: the copy has left it when this call returns; on the device it runs in stream
        # order, after the sampling of the step before)
        st.buf.copy_(torch.from_numpy(host), non_blocking=True)
        st.greedy = greedy
        return st

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams],
               draw_index: Sequence[int],
               previous: Optional[Sequence[Sequence[int]]] = None) -> torch.Tensor:
        """``logits`` [R, V] float32 on the device; ``draw_index[r]`` is how many tokens request
        r has generated so far (selects its uniform draw); ``previous[r]`` its generated tokens
        (used only where a repetition penalty is set).  Returns int32 [R] on the device."""
        R = logits.shape[0]
        if len(params) != R or len(draw_index) != R:
            raise ValueError("one SamplingParams and one draw index per row of logits")
        dev = self.rt.device
        host, greedy, penal = _pack(params, draw_index)
        if greedy and not penal:
            # nothing varies from step to step: keep the per-row arrays on the device
            cached = self._greedy.get(R)
            if cached is None:
                cached = self._greedy[R] = _rows(torch.from_numpy(host).to(dev), R) \
                    + (torch.empty(R, dtype=torch.int32, device=dev),)
            d_fl, d_tk, out = cached
            self.rt.ops.sample(logits, d_fl, d_tk, None, None, out)
            return out
        d_fl, d_tk = _rows(torch.from_numpy(host).to(dev, non_blocking=True), R)
        d_start = d_prev = None
        if penal and previous is not None:
            start = np.zeros(R + 1, dtype=np.int32)
            flat: List[int] = []
            for r, prev in enumerate(previous):
                if params[r].repetition_penalty != 1.0:
                    flat.extend(prev)
                start[r + 1] = len(flat)
            d_start = torch.from_numpy(start).to(dev)
            d_prev = torch.from_numpy(np.asarray(flat if flat else [0], dtype=np.int32)).to(dev)
        out = torch.empty(R, dtype=torch.int32, device=dev)
        self.rt.ops.sample(logits, d_fl, d_tk, d_start, d_prev, out)
        return out
