"""Choosing the next token: greedy, temperature, top-k, top-p.

Which tokens stay candidates follows LitInfer's sampler
(src/llaisys/models/qwen2.cpp:890-920): logits / temperature; the ``top_k``
largest if 0 < k < vocab; softmax over those; the shortest prefix (in
descending order) whose cumulative probability reaches ``top_p`` if
0 < p < 1; softmax again over what is left; draw.  Greedy when ``top_k == 1``
(the default of ``generate``, python/llaisys/models/qwen2.py:305-311) or when
``temperature <= 0`` (qwen2.cpp:893-895): the first maximum wins
(src/ops/argmax/op.cpp:28-33).

The draw differs from LitInfer's on purpose.  LitInfer consumes one shared
``mt19937`` in batch order, so a request's tokens depend on what else is
running.  Here the draw is Gumbel-max, ``argmax_i(z_i + g_i)`` over the
candidates with ``g_i = -log(-log(u_i))``, which samples exactly from their
softmax, and ``u_i`` comes from a counter-based generator keyed on (the
request's seed, the index of the output token, the token id i): the result
depends on nothing but the request itself.
"""

from __future__ import annotations

import struct
from dataclasses import dataclass
from functools import cached_property
from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from .. import kernels as K


# a row's parameters as the kernel reads them, but for the output index: temperature, top_k, top_p, seed low, seed high
_ROW = struct.Struct("=fifII")
_DRAWS, _SMALL_TOP_K, _ALONE = 1, 2, 4


def _pack(p) -> Tuple[Optional[bytes], int]:
    """A request's row of parameters, and what a row of it needs of the kernels: _DRAWS where it is not greedy,
    _SMALL_TOP_K with a top_k of 2 to 256, _ALONE where temperature may be its only option (for some vocabulary)."""
    # rows that are greedy get temperature 0, which the kernel reads as argmax
    temperature = p.temperature
    greedy = p.top_k == 1 or temperature <= 0.0
    try:
        temperature = 0.0 if greedy else float(temperature)
        top_k, top_p, seed = min(max(int(p.top_k), -1), 0x7FFF_FFFF), float(p.top_p), int(p.seed)
        try:
            row = _ROW.pack(temperature, top_k, top_p, seed & 0xFFFF_FFFF, seed >> 32 & 0xFFFF_FFFF)
        except OverflowError:                             # beyond float32: infinity
            row = _ROW.pack(np.float32(temperature), top_k, np.float32(top_p), seed & 0xFFFF_FFFF, seed >> 32 & 0xFFFF_FFFF)
    except (TypeError, ValueError):
        if greedy:                                        # a step of greedy rows alone reads nothing else of them
            return None, 0
        raise
    if greedy:
        return row, _SMALL_TOP_K if 1 < top_k <= 256 else 0
    if 1 < top_k <= 256:
        return row, _DRAWS | _SMALL_TOP_K
    # (a top_p next to 0 or 1 may be rounded to it)
    return row, _DRAWS if 1e-30 < top_p < 0.999999 else _DRAWS | _ALONE


@dataclass(frozen=True)
class SamplingParams:
    temperature: float = 1.0
    top_k: int = 1
    top_p: float = 1.0
    seed: int = 0

    @property
    def greedy(self) -> bool:
        return self.top_k == 1 or self.temperature <= 0.0

    @cached_property
    def packed(self) -> Tuple[Optional[bytes], int]:
        """:func:`_pack` of these parameters, made once for all of a request's tokens (64 rows: 45 us a step on the host
        when every step packed them anew)."""
        return _pack(self)


class Sampler:
    """Device-side sampling of one token per logits row."""

    def __init__(self, device) -> None:
        self.device = torch.device(device)
        # the rows' parameters go to the device through pinned memory, without blocking the host (two buffers in turn:
        # a step may be launched before the one before it has been read)
        self._pinned: List[torch.Tensor] = []
        self._rows: List[np.ndarray] = []                 # the same memory
        self._on_device: List[torch.Tensor] = []
        self._copied: List = []
        self._turn = 0

    def _upload(self, rows: bytes, output_index: Sequence[int]) -> torch.Tensor:
        R = len(output_index)
        packed = np.frombuffer(rows, dtype=np.int32).reshape(R, 5)
        if self.device.type != "cuda":
            return torch.from_numpy(np.column_stack([packed, np.asarray(output_index, dtype=np.int32)]))
        stream = torch.cuda.current_stream(self.device)
        if not self._pinned or self._pinned[0].shape[0] < R:
            for ev in self._copied:
                ev.synchronize()
            cap = max(64, 2 * R)
            self._pinned = [torch.empty((cap, 6), dtype=torch.int32).pin_memory() for _ in range(2)]
            self._rows = [t.numpy() for t in self._pinned]
            self._on_device = [torch.empty((cap, 6), dtype=torch.int32, device=self.device) for _ in range(2)]
            self._copied = [torch.cuda.Event() for _ in range(2)]
            for ev in self._copied:
                ev.record(stream)
        t = self._turn
        self._turn ^= 1
        self._copied[t].synchronize()                     # the copy that last used this pinned buffer has finished
        self._rows[t][:R, :5] = packed
        self._rows[t][:R, 5] = output_index
        dst = self._on_device[t][:R]
        dst.copy_(self._pinned[t][:R], non_blocking=True)
        self._copied[t].record(stream)
        return dst

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], output_index: Sequence[int]) -> torch.Tensor:
        """``logits`` float32 [R, V]; returns int32 [R] on the device."""
        R = logits.shape[0]
        if len(params) != R or len(output_index) != R:
            raise ValueError("one SamplingParams and one output index per logits row")
        out = torch.empty(R, dtype=torch.int32, device=logits.device)
        if R == 0:
            return out
        needs, rows = 0, []
        for p in params:
            row, n = p.packed if isinstance(p, SamplingParams) else _pack(p)
            rows.append(row)
            needs |= n
        if not needs & _DRAWS:
            K.argmax(logits, out)
            return out
        packed = self._upload(b"".join(rows), output_index)
        packed.small_top_k = bool(needs & _SMALL_TOP_K)
        packed.draws_alone = bool(needs & _ALONE)
        K.sample(logits, packed, out)
        return out


def _as_i32(u: int) -> int:
    return u - (1 << 32) if u >= (1 << 31) else u
