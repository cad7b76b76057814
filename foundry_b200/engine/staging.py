"""Host-to-device uploads of a step's description that may be queued ahead.

A replayed step reads its tokens, positions, lengths and page tables from
fixed device buffers that one copy from pinned memory refreshes. The copy is
asynchronous: when the host prepares steps faster than the device runs them
(device-resident decoding never waits for the device), a pinned buffer that is
rewritten for step k+1 may still be the source of step k's queued copy, and
step k would then run with step k+1's positions.

`StagingRing` therefore keeps the values in ordinary host memory (`values`)
and sends them through a ring of pinned buffers, each of which is rewritten
only after the copy that last read it has run. The host can be at most `depth`
uploads ahead of the device.
"""
from __future__ import annotations

import torch

from ..kernels import ops


class StagingRing:
    def __init__(self, count: int, dtype: torch.dtype, device: torch.device, depth: int = 4):
        self.dev = torch.zeros(count, dtype=dtype, device=device)
        self.values = torch.zeros(count, dtype=dtype).numpy()  # what the next upload sends
        self._to, self._from = self.dev.data_ptr(), self.values.ctypes.data
        self._size = count * self.values.itemsize
        self._buffers = [ops.UploadBuffer(self._size) for _ in range(depth)]
        self._next = 0

    def upload(self, start: int = 0) -> int:
        """Queue a copy of `values[start:]` to `dev[start:]` on the current
        stream; returns the bytes sent."""
        buffer = self._buffers[self._next]
        self._next = (self._next + 1) % len(self._buffers)
        skip = start * self.values.itemsize
        buffer.send(self._to + skip, self._from + skip, self._size - skip)
        return self._size - skip
