"""Runs the sampling kernel over the logits rows of a step: per-row temperature, top-k,
top-p, seed and the index of the output token travel in one pinned buffer; token ids come
back in one device-to-host copy."""
from __future__ import annotations

from typing import Sequence, Tuple

import numpy as np
import torch

from ..csrc import ops
from .params import SamplingParams


class Sampler:
    def __init__(self, device, max_rows: int):
        self.device = torch.device(device)
        self.max_rows = max_rows
        # per row: temperature f32, top_p f32, top_k i32, pad, seed i64, counter i64 -> 8 int32 words
        # (four pinned copies in turn: with a step in flight the host already writes the next one's)
        self._hosts = [torch.empty(max_rows * 8, dtype=torch.int32, pin_memory=True) for _ in range(4)]
        self._arrays = [h.numpy() for h in self._hosts]
        self._host_events = [None] * 4     # one a copy, recorded anew every time
        self._device_views = {}            # per number of rows: what the kernel is given of the device copy
        self._host_turn = 0
        self._dev = torch.empty(max_rows * 8, dtype=torch.int32, device=self.device)
        self._out = torch.empty(max_rows, dtype=torch.int32, device=self.device)
        # results: two pinned buffers (ids, then the status word), so that one step's ids can be read while
        # the next step's copy is already queued
        self._out_hosts = [torch.zeros(max_rows + 1, dtype=torch.int32, pin_memory=True) for _ in range(2)]
        self._out_turn = 0
        self._argmax_scratch = torch.zeros(ops.argmax_scratch_words(max_rows), dtype=torch.int32, device=self.device)

    def sample(self, logits: torch.Tensor, rows: Sequence[Tuple[SamplingParams, int, int]]) -> torch.Tensor:
        """``rows[r] = (params, seed, index of the output token)``; returns int32 [R] on the device."""
        R = logits.shape[0]
        if R != len(rows) or R > self.max_rows:
            raise ValueError(f"sampler got {R} logits rows for {len(rows)} requests (limit {self.max_rows})")
        out = self._out[:R]
        params = [r[0] for r in rows]
        temperature = [p.temperature for p in params]
        if not any(t > 0 for t in temperature):
            ops.argmax(logits, out, self._argmax_scratch)
            return out
        turn = self._host_turn = (self._host_turn + 1) % 4
        if self._host_events[turn] is not None:
            self._host_events[turn].synchronize()
        h = self._arrays[turn]
        n = self.max_rows
        h[0:R].view(np.float32)[:] = temperature
        h[n:n + R].view(np.float32)[:] = [p.top_p for p in params]
        h[2 * n:2 * n + R] = [p.top_k for p in params]
        h[4 * n:4 * n + 2 * R].view(np.uint64)[:] = [r[1] & 0xFFFFFFFFFFFFFFFF for r in rows]
        h[6 * n:6 * n + 2 * R].view(np.int64)[:] = [r[2] for r in rows]
        d = self._dev
        d.copy_(self._hosts[turn], non_blocking=True)
        if self._host_events[turn] is None:
            self._host_events[turn] = torch.cuda.Event()
        self._host_events[turn].record(torch.cuda.current_stream(d.device))      # where the copy is, whatever device the calling thread is at
        v = self._device_views.get(R)
        if v is None:
            v = self._device_views[R] = (d[0:R].view(torch.float32), d[n:n + R].view(torch.float32), d[2 * n:2 * n + R],
                                         d[4 * n:4 * n + 2 * R].view(torch.int64), d[6 * n:6 * n + 2 * R].view(torch.int64))
        ops.sample(logits, out, temperature=v[0], top_p=v[1], top_k=v[2], seed=v[3], counter=v[4])
        return out

    def last_ids(self) -> torch.Tensor:
        """The device buffer that ``sample`` writes its ids into (valid until the next ``sample``)."""
        return self._out

    def fetch(self, tokens: torch.Tensor, status: torch.Tensor = None):
        """Queue the device-to-host copy of the sampled ids (and of the engine's int32 status word) and
        return a handle for ``wait``; the stream is not synchronised."""
        R = tokens.numel()
        self._out_turn ^= 1
        host = self._out_hosts[self._out_turn]
        host[:R].copy_(tokens, non_blocking=True)
        if status is not None:
            host[self.max_rows:self.max_rows + 1].copy_(status, non_blocking=True)
        ev = torch.cuda.Event()
        ev.record()
        return (host, R, status is not None, ev)

    def wait(self, handle):
        """The ids of a ``fetch`` (and the status code when one was asked for), once its copy has arrived."""
        host, R, with_status, ev = handle
        ev.synchronize()
        ids = host[:R].tolist()
        return (ids, int(host[self.max_rows])) if with_status else ids

    def to_host(self, tokens: torch.Tensor, status: torch.Tensor = None):
        """Device-to-host read of the sampled ids. With ``status`` (the engine's int32 status word) both
        travel before the one wait and ``(ids, status code)`` is returned."""
        return self.wait(self.fetch(tokens, status))
