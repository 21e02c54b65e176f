"""Memory that a launch fills for the one behind it (partial results of KV splits)."""
from __future__ import annotations

import torch


class Scratch:
    """One tensor per device that calls share, grown by those that need more, until a CUDA graph holds its address.

    A captured graph writes to that address in every replay, whoever owns the memory by then, so from the first capture on the tensor is
    neither replaced nor given back.  A call that needs more takes memory of its own from the allocator: under capture that is the
    graph's pool, which lives as long as the graph."""

    def __init__(self, dtype: torch.dtype):
        self._dtype = dtype
        self._shared: dict[tuple, torch.Tensor] = {}
        self._captured: set[tuple] = set()

    def get(self, device: torch.device, numel: int) -> torch.Tensor:
        """At least ``numel`` elements; the caller holds the tensor until its launches are under way."""
        index = torch.cuda.current_device() if device.type == "cuda" and device.index is None else device.index
        key, capturing = (device.type, index), torch.cuda.is_initialized() and torch.cuda.is_current_stream_capturing()
        buf = self._shared.get(key)
        if buf is None or buf.numel() < numel:
            with torch.inference_mode(False):      # calls inside and outside of that mode share it
                own = torch.empty(max(numel, 1 << 20), dtype=self._dtype, device=device)
            if capturing or key in self._captured:
                return own
            self._shared[key] = buf = own
        if capturing:
            self._captured.add(key)
        return buf
