"""Device buffers of a step, handed out by name.

Row buffers are allocated once at their largest size. A flat buffer grows when a step asks for more
than any step before it; the smaller buffer it replaces is kept, never given back, because a
captured CUDA graph may still write to its address (and read from it in the same graph). Callers
that know their largest need say so (`capacity`), so that growth is the exception. Buffers of steps
that are never captured (`spare`) are let go when they are outgrown, and are not to be had where the
device is short of memory. Steady-state stepping allocates nothing (the reference's arena:
src/model/qwen3.cpp:109-146).
"""
from __future__ import annotations

import torch


class Workspace:
    def __init__(self, max_rows: int, device):
        self.max_rows = max_rows
        self.device = device
        self._rows: dict[tuple, torch.Tensor] = {}
        self._flat: dict[tuple, torch.Tensor] = {}
        self._retired: list[torch.Tensor] = []      # outgrown buffers: captured graphs may still use them
        self._spare_bytes = self._free_bytes() // 2 # what a spare buffer may take (asking the device costs 0.1 ms: asked once)

    def rows(self, name: str, n: int, width: int, dtype: torch.dtype) -> torch.Tensor:
        """[n, width] view of a buffer that holds max_rows rows."""
        if n > self.max_rows:
            raise ValueError(f"workspace '{name}': {n} rows asked of a workspace of {self.max_rows}")
        key = (name, width, dtype)
        buf = self._rows.get(key)
        if buf is None:
            buf = torch.empty((self.max_rows, width), dtype=dtype, device=self.device)
            self._rows[key] = buf
        return buf[:n]

    def flat(self, name: str, numel: int, dtype: torch.dtype, capacity: int = 0) -> torch.Tensor:
        """At least `numel` elements; allocated with max(numel, capacity) the first time."""
        return self._grow((name, dtype), numel, capacity, lambda n: torch.empty(n, dtype=dtype, device=self.device))

    def _grow(self, key, numel: int, capacity: int, make) -> torch.Tensor:
        buf = self._flat.get(key)
        if buf is None or buf.numel() < numel:
            if buf is not None:
                self._retired.append(buf)
            buf = make(max(numel, capacity, 2 * buf.numel() if buf is not None else 0))
            self._flat[key] = buf
        return buf

    def spare(self, name: str, numel: int, dtype: torch.dtype, capacity: int = 0) -> torch.Tensor | None:
        """At least `numel` elements for a step that is not captured and that has another way if there are none: None where the
        buffer would take more than half of what the device had left when this workspace was made (behind weights and cache; the
        buffers of other steps were still to come), or where it has no more. An outgrown buffer goes back to the allocator; the
        stream's order keeps it whole until the steps that use it are done."""
        key = (name, dtype, "spare")
        buf = self._flat.get(key)
        if buf is not None and buf.numel() >= numel:
            return buf
        size = max(numel, capacity)
        if size * dtype.itemsize > self._spare_bytes:
            return None
        self._flat.pop(key, None)
        del buf
        try:
            self._flat[key] = buf = torch.empty(size, dtype=dtype, device=self.device)
        except torch.cuda.OutOfMemoryError:
            self._spare_bytes = size * dtype.itemsize - 1
            return None
        return buf

    def _free_bytes(self) -> int:
        return torch.cuda.mem_get_info(self.device)[0] if torch.device(self.device).type == "cuda" else 1 << 62

    def zeros(self, name: str, numel: int, dtype: torch.dtype) -> torch.Tensor:
        """A buffer that is zero when first handed out (kernels that use it leave it zero)."""
        return self._grow((name, dtype, "zeros"), numel, 0, lambda n: torch.zeros(n, dtype=dtype, device=self.device))

    def bytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in list(self._rows.values()) + list(self._flat.values()) + self._retired)
