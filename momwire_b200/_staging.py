"""Host arrays to the device and results back through page-locked memory.

A set of host arrays becomes one page-locked buffer (256-byte aligned
pieces) and one stream-ordered copy: a copy per array from pageable memory
makes the host wait for the device each time.  A solver's results come back
the same way, as arrays on page-locked memory that live as long as they are
used; results that a host keeps by the thousand (``to_host``) come back as
ordinary arrays, through a page-locked buffer of fixed size.
"""

from __future__ import annotations

import threading

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


class _Bounce(threading.local):
    """Two page-locked slots and their events, per host thread and given back
    with it.  21 MB took 711 us through slots of 2 MB, 715 of 4, 599 of 8, 594
    of 16 (390 to page-locked memory): a slice costs 30 us beside its copies."""

    SLOT = 8 << 20  # bytes
    slots = events = None

    def get(self, torch):
        if self.slots is None:
            with torch.inference_mode(False):  # (a caller's mode must not stick to them)
                self.slots = [torch.empty(self.SLOT, dtype=torch.uint8, pin_memory=True) for _ in range(2)]
            self.events = {}
        return self.slots

    def event(self, torch, device, i):
        key = (device, i)
        if key not in self.events:
            self.events[key] = torch.cuda.Event()
        return self.events[key]


_bounce = _Bounce()
_SMALL = 1 << 17  # bytes: up to here one thread copies as fast as several (960 KB: 234 us a call against 176)
_NUMPY = {"torch.complex128": np.complex128, "torch.complex64": np.complex64, "torch.float64": np.float64,
          "torch.float32": np.float32, "torch.int32": np.int32}


def to_host(torch, stream, t):
    """An ordinary array with a contiguous device tensor's values: slice by
    slice through the thread's page-locked slots, one on its way from the
    device while the other is copied out (a small result, a row of a block
    say, in one piece)."""
    out = np.empty(tuple(t.shape), dtype=_NUMPY[str(t.dtype)])
    if out.size == 0:
        return out
    slots, S = _bounce.get(torch), _bounce.SLOT
    with torch.inference_mode():  # (no version counters, no autograd)
        src, n = t.view(-1).view(torch.uint8), out.nbytes
        dst = out.reshape(-1).view(np.uint8)
        if n <= _SMALL:
            slots[0][:n].copy_(src, non_blocking=True)
            stream.synchronize()
            dst[:] = slots[0].numpy()[:n]
            return out
        dst = torch.from_numpy(dst)
        cuts = [(o, min(o + S, n)) for o in range(0, n, S)]

        def fetch(i):
            a, b = cuts[i]
            slots[i % 2][: b - a].copy_(src[a:b], non_blocking=True)
            _bounce.event(torch, t.device, i % 2).record(stream)

        for i in range(min(2, len(cuts))):
            fetch(i)
        for i, (a, b) in enumerate(cuts):
            _bounce.event(torch, t.device, i % 2).synchronize()
            dst[a:b].copy_(slots[i % 2][: b - a])
            if i + 2 < len(cuts):
                fetch(i + 2)
    return out
