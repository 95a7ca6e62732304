"""Host arrays to the device and results back through page-locked memory.

A set of host arrays becomes one page-locked buffer (256-byte aligned
pieces) and one stream-ordered copy: a copy per array from pageable memory
makes the host wait for the device each time.  Results come back the same
way, as arrays on page-locked memory that live as long as they are used.
"""

from __future__ import annotations

import numpy as np


class Packed:
    """Host arrays packed into one page-locked buffer; immutable once built,
    so any thread may upload it on any stream."""

    def __init__(self, torch, arrays):
        arrays = [np.ascontiguousarray(a) for a in arrays]
        self.pieces, total = [], 0
        for a in arrays:
            self.pieces.append((total, a.nbytes))
            total += (a.nbytes + 255) & ~255
        self.host = torch.empty(max(total, 256), dtype=torch.uint8, pin_memory=True)
        hv = self.host.numpy()
        for a, (o, n) in zip(arrays, self.pieces):
            hv[o : o + n] = a.reshape(-1).view(np.uint8)
        self.nbytes = int(sum(n for _o, n in self.pieces))

    def upload(self, device):
        """(device buffer, address of every piece) from one copy on the
        current stream."""
        dev = self.host.to(device, non_blocking=True)
        base = dev.data_ptr()
        return dev, [base + o for o, _n in self.pieces]


def read_back(torch, stream, tensors):
    """Host copies of device tensors: page-locked, one synchronisation."""
    out = []
    for t in tensors:
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        h.copy_(t, non_blocking=True)
        out.append(h)
    stream.synchronize()
    return [h.numpy() for h in out]
