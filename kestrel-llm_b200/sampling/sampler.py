"""Picks the next token of every request whose logits a step returned, on the device.

Greedy rows take the first maximum.  Other rows are sampled by one kernel with their own
temperature, top-k, min-p and top-p (meanings: src/core/vllm_transformer.c:357-479 of the
reference).  The uniform number of a draw is a function of (request seed, index of the token
being generated) only - the reference draws from the process-wide, never seeded ``rand()``
(vllm_transformer.c:464) - so a request's output does not depend on what it was batched with
and can be repeated.
"""
from __future__ import annotations

from array import array
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..cache.manager import host_library
from ..csrc import ops
from .params import SamplingParams

_MASK = (1 << 64) - 1


def _mix(z: int) -> int:
    z = (z + 0x9E3779B97F4A7C15) & _MASK
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _MASK
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _MASK
    return z ^ (z >> 31)


def uniform_for(seed: int, index: int) -> float:
    """Uniform number in (0, 1] for the ``index``-th generated token of a request with ``seed``
    (two rounds of the splitmix64 finaliser; 24 bits, so the value is exact in float32)."""
    z = _mix(_mix(seed & _MASK) ^ (index & _MASK))
    return ((z >> 40) + 1) / float(1 << 24)


class _Slot:
    """A pinned buffer for the options of a call's rows, and the event behind its last copy to the device."""

    __slots__ = ("floats", "ints", "pinned", "done", "pending")

    def __init__(self, cap: int):
        self.pinned = torch.empty((5 * cap,), dtype=torch.float32).pin_memory()
        self.floats = self.pinned.numpy()
        self.ints = self.floats.view(np.int32)
        self.done, self.pending = torch.cuda.Event(), False


class Sampler:
    RING = 4        # pinned buffers for the rows' options; a buffer is reused only after its copy has run

    def __init__(self, device):
        self.device = torch.device(device)
        self._ring: List[_Slot] = []
        self._turn = 0
        self._uniforms = host_library().kbatch_uniforms

    def _slot(self, rows: int) -> _Slot:
        """A buffer with room for the rows' options whose last copy to the device has completed."""
        if not self._ring or self._ring[0].floats.size < 5 * rows:
            for s in self._ring:
                if s.pending:
                    s.done.synchronize()
            self._ring = [_Slot(max(64, 1 << (rows - 1).bit_length())) for _ in range(self.RING)]
        self._turn = (self._turn + 1) % self.RING
        slot = self._ring[self._turn]
        if slot.pending:
            slot.done.synchronize()
        return slot

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               indices: Sequence[int], generated: Optional[Sequence[Sequence[int]]] = None) -> torch.Tensor:
        """logits float32 [R, V]; row r belongs to a request with ``params[r]``, ``seeds[r]``,
        generating its ``indices[r]``-th token; ``generated[r]`` are the tokens it has generated so
        far (needed by rows with a repetition penalty, which changes ``logits`` in place).
        Returns int32 [R] on the device."""
        R = logits.shape[0]
        out = torch.empty((R,), dtype=torch.int32, device=self.device)
        if any(p.penalised for p in params):
            if generated is None:
                raise ValueError("a repetition penalty needs the tokens generated so far")
            W = 64
            hist = np.full((R, W), -1, dtype=np.int32)
            counts = np.zeros((R,), dtype=np.int32)
            pen = np.ones((R,), dtype=np.float32)
            for r, (p, g) in enumerate(zip(params, generated)):
                if not p.penalised:
                    continue
                last = list(g[-p.repetition_window:])[::-1]       # most recent first, as the reference walks them
                hist[r, :len(last)] = last
                counts[r] = len(last)
                pen[r] = p.repetition_penalty
            ops.repetition_penalty(logits, torch.from_numpy(hist).to(self.device), torch.from_numpy(counts).to(self.device),
                                   torch.from_numpy(pen).to(self.device))
        if all(p.greedy for p in params):
            ops.argmax(logits, out)
            return out
        if not len(params) == len(seeds) == len(indices) == R:          # longer ones are cut; with shorter ones rows would have no options
            if min(len(params), len(seeds), len(indices)) != R:
                raise ValueError(f"sample: {R} rows of logits, {len(params)} of options, {len(seeds)} seeds, {len(indices)} indices")
            params, seeds, indices = params[:R], seeds[:R], indices[:R]
        # rows of temperature, top-p, min-p, uniform number and top-k (int32 bits), one behind the other: a copy of what is contiguous
        # goes out of the pinned buffer itself
        slot = self._slot(R)
        host = slot.floats
        host[:R] = [0.0 if p.greedy else p.temperature for p in params]
        host[R:2 * R] = [p.top_p for p in params]
        host[2 * R:3 * R] = [p.min_p for p in params]
        slot.ints[4 * R:5 * R] = np.array([p.top_k for p in params], dtype=np.int32)
        s, i = array("Q", [x & _MASK for x in seeds]), array("Q", [x & _MASK for x in indices])
        self._uniforms(R, s.buffer_info()[0], i.buffer_info()[0], slot.pinned.data_ptr() + 12 * R)
        dev = torch.empty((5, R), dtype=torch.float32, device=self.device)
        dev.copy_(slot.pinned[:5 * R].view(5, R), non_blocking=True)
        slot.done.record()
        slot.pending = True
        ops.sample_options(logits, dev, out)
        return out
