"""Chooses the next token of every sampled row on the device.

Greedy rows take the arg-max (the smaller id wins a tie, crates/kernels/src/ops.cu:152-162).
Other rows are drawn from the reference's support (temperature, then top_k, then top_p;
crates/engine/src/lib.rs:207-244) with a counter-based generator: the n-th token of a
request is drawn with u(seed, n), whatever else is in the batch.  Where the reference keeps
a ChaCha8 stream per request, the per-request state here is the draw count alone."""
from __future__ import annotations

import struct
from functools import lru_cache
from typing import Sequence

import numpy as np
import torch

from .. import kernels
from ..errors import BackendError
from .params import SamplingParams

_MASK64 = (1 << 64) - 1


def uniform_from_counter(seed: int, index: int) -> float:
    """The kernel's u in [0, 1) for (seed, draw index), bit for bit (splitmix64 finaliser)."""
    z = (seed + 0x9E3779B97F4A7C15 * (index + 1)) & _MASK64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _MASK64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _MASK64
    z ^= z >> 31
    return (z >> 40) / 16777216.0


@lru_cache(maxsize=256)
def _words(rows: int) -> struct.Struct:
    """The words of `packed_parameters`."""
    return struct.Struct(f"={rows}Q{rows}f{rows}i{rows}f{rows}i")


def packed_bytes(params: Sequence[SamplingParams], draw_index: Sequence[int]) -> bytes:
    """The bytes of `packed_parameters` (in a third of the time that numpy's arrays take for some ten rows)."""
    temperatures = [0.0 if p.is_greedy() else p.temperature for p in params]
    try:
        return _words(len(params)).pack(*[int(p.seed) & _MASK64 for p in params], *temperatures, *[p.top_k or 0 for p in params],
                                        *[p.top_p for p in params], *draw_index)
    except (struct.error, OverflowError):
        # what a word of this kind does not hold: a float beyond float32 is infinite, an integer beyond 32 bits is refused
        rows = len(params)
        packed = np.empty(6 * rows, dtype=np.int32)
        packed[:2 * rows].view(np.uint64)[:] = np.array([int(p.seed) & _MASK64 for p in params], dtype=np.uint64)
        packed[2 * rows:3 * rows].view(np.float32)[:] = temperatures
        packed[3 * rows:4 * rows] = [p.top_k or 0 for p in params]
        packed[4 * rows:5 * rows].view(np.float32)[:] = [p.top_p for p in params]
        packed[5 * rows:] = draw_index
        return packed.tobytes()


def packed_parameters(params: Sequence[SamplingParams], draw_index: Sequence[int]) -> np.ndarray:
    """The rows' parameters as the words that the kernel reads: all seeds (the 64-bit patterns of their values, negative ones too),
    then all temperatures, top_k, top_p and draw indices, 32 bits each."""
    return np.frombuffer(packed_bytes(params, draw_index), dtype=np.int32)


class Chosen:
    """Tokens that `Sampler.launch` chose: on the device (`tokens`, for a step that goes on before the host has
    seen them) and in pinned host memory (`host`, complete when `arrived` has happened)."""

    def __init__(self, tokens: torch.Tensor, host: torch.Tensor, arrived: torch.cuda.Event):
        self.tokens, self.host, self.arrived = tokens, host, arrived


class _Turn:
    """Pinned host memory that one launch's kernel writes its tokens to.  It is used again, or given back, only behind `last`: the
    allocator of pinned memory does not know of a kernel's accesses."""

    def __init__(self, rows: int):
        self.tokens = torch.empty(rows, dtype=torch.int32, pin_memory=True)
        self.last: torch.cuda.Event | None = None

    def wait(self) -> None:
        if self.last is not None:
            self.last.synchronize()


class Sampler:
    def __init__(self, device: torch.device):
        self.device = device
        self._turns: list[_Turn | None] = [None] * 3         # two results may be outstanding
        self._at = 0
        self._recorded: list[_Turn] = []                     # of launches in graphs, which write again at every replay

    def __del__(self):
        for turn in getattr(self, "_turns", ()):
            if turn is not None:
                try:
                    turn.wait()
                except RuntimeError:         # the device is in no state to write any more
                    pass

    def _turn(self, rows: int) -> _Turn:
        """Pinned memory for `rows` rows that no launch uses any more."""
        if torch.cuda.is_current_stream_capturing():         # an event of a graph cannot be waited for
            self._recorded.append(_Turn(rows))
            return self._recorded[-1]
        self._at = (self._at + 1) % 3
        turn = self._turns[self._at]
        if turn is not None:
            turn.wait()
        if turn is None or turn.tokens.numel() < rows:
            turn = self._turns[self._at] = _Turn(max(256, 2 * rows))
        return turn

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], draw_index: Sequence[int]) -> list[int]:
        """One token per row of `logits` [rows, vocab] (float32, on the device)."""
        return self.read(self.launch(logits, params, draw_index))

    def read(self, chosen: Chosen) -> list[int]:
        """Waits for tokens that `launch` chose and returns them."""
        chosen.arrived.synchronize()
        tokens = chosen.host.tolist()
        if any(t < 0 for t in tokens):
            raise BackendError("empty/nonfinite logits")
        return tokens

    def launch(self, logits: torch.Tensor, params: Sequence[SamplingParams], draw_index: Sequence[int]) -> Chosen:
        """Queues the choice of one token per row of `logits` (int32; a row without finite logits gives -1) and
        their copy to the host, right behind it in the stream, so that work queued later does not hold the copy
        up.  Nothing is waited for."""
        rows = logits.shape[0]
        assert rows == len(params) == len(draw_index)
        out = torch.empty(rows, dtype=torch.int32, device=self.device)
        turn = self._turn(rows)
        host = turn.tokens[:rows]
        arrived = torch.cuda.Event()
        try:
            if all(p.is_greedy() for p in params):
                kernels.argmax(logits, out)
                host.copy_(out, non_blocking=True)
            else:
                # The parameters travel with the launch and the kernel writes the tokens to pinned memory: a copy each way is a launch on the
                # host and a wait on the device (with numpy's arrays and copies a launch took the host 75 us for 24 rows, the kernel 68).
                kernels.sample_words(logits, packed_bytes(params, draw_index), out, host.data_ptr())
        finally:                                             # many rows are several launches: one may fail behind others
            arrived.record()
            if turn in self._turns:
                turn.last = arrived
        return Chosen(out, host, arrived)
