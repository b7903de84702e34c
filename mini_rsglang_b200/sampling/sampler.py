"""Chooses the next token of every sampled row on the device.

Greedy rows take the arg-max (the smaller id wins a tie, crates/kernels/src/ops.cu:152-162).
Other rows are drawn from the reference's support (temperature, then top_k, then top_p;
crates/engine/src/lib.rs:207-244) with a counter-based generator: the n-th token of a
request is drawn with u(seed, n), whatever else is in the batch.  Where the reference keeps
a ChaCha8 stream per request, the per-request state here is the draw count alone."""
from __future__ import annotations

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


def packed_parameters(params: Sequence[SamplingParams], draw_index: Sequence[int]) -> np.ndarray:
    """The rows' parameters as the words of one copy: all seeds (the 64-bit patterns of their values, negative ones too), then all
    temperatures, top_k, top_p and draw indices, 32 bits each."""
    rows = len(params)
    packed = np.empty(6 * rows, dtype=np.int32)
    packed[:2 * rows].view(np.uint64)[:] = np.array([int(p.seed) & _MASK64 for p in params], dtype=np.uint64)
    packed[2 * rows:3 * rows].view(np.float32)[:] = [0.0 if p.is_greedy() else p.temperature for p in params]
    packed[3 * rows:4 * rows] = [p.top_k or 0 for p in params]
    packed[4 * rows:5 * rows].view(np.float32)[:] = [p.top_p for p in params]
    packed[5 * rows:] = draw_index
    return packed


class Chosen:
    """Tokens that `Sampler.launch` chose: on the device (`tokens`, for a step that goes on before the host has
    seen them) and on their way to pinned host memory (`host`, complete when `arrived` has happened)."""

    def __init__(self, tokens: torch.Tensor, host: torch.Tensor, arrived: torch.cuda.Event):
        self.tokens, self.host, self.arrived = tokens, host, arrived


class Sampler:
    def __init__(self, device: torch.device):
        self.device = device
        self._pinned: list[torch.Tensor] = []       # host buffers that take turns: two results may be outstanding
        self._turn = 0
        self._staging: list = []                    # (pinned host buffer, event of its last copy out), taken in turn
        self._staged = 0

    def _stage(self, rows: int):
        """A pinned host buffer for the parameters of `rows` rows whose last copy to the device has finished."""
        self._staged = (self._staged + 1) % 3
        while len(self._staging) < 3:
            self._staging.append(None)
        held = self._staging[self._staged]
        if held is None or held[0].numel() < 24 * rows:
            held = (torch.empty(24 * max(64, 2 * rows), dtype=torch.uint8, pin_memory=True), torch.cuda.Event())
            self._staging[self._staged] = held
        else:
            held[1].synchronize()
        return held

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
        if all(p.is_greedy() for p in params):
            kernels.argmax(logits, out)
        else:
            # One copy from pinned memory carries every row's parameters: five pageable ones waited for the stream each.
            packed = packed_parameters(params, draw_index)
            host, copied = self._stage(rows)
            host.numpy()[:24 * rows] = packed.view(np.uint8)
            words = torch.empty(6 * rows, dtype=torch.int32, device=self.device)
            words.view(torch.uint8).copy_(host[:24 * rows], non_blocking=True)
            copied.record()
            temperature, top_k, top_p, draws = (words[k * rows:(k + 1) * rows] for k in range(2, 6))
            kernels.sample(logits, temperature.view(torch.float32), top_k, top_p.view(torch.float32), words[:2 * rows].view(torch.int64), draws, out)
        while len(self._pinned) < 3:
            self._pinned.append(torch.empty(max(256, rows), dtype=torch.int32, pin_memory=True))
        self._turn = (self._turn + 1) % 3
        if self._pinned[self._turn].numel() < rows:
            self._pinned[self._turn] = torch.empty(2 * rows, dtype=torch.int32, pin_memory=True)
        host = self._pinned[self._turn][:rows]
        host.copy_(out, non_blocking=True)
        arrived = torch.cuda.Event()
        arrived.record()
        return Chosen(out, host, arrived)
