"""A process-wide pool of CUDA streams for the file pipelines.

torch's allocator keeps freed device memory per stream: a pipeline call that
makes a stream of its own finds none of the memory that the call before it
gave back and asks the driver for all of it again (1-20 ms for each array of
a piece).  A stream returned to the pool is handed to the next call on that
device, and its memory with it.  Thread-safe: a stream belongs to one caller
between take() and give(); at most `LIMIT` idle ones are kept per device.
"""
from __future__ import annotations

import threading

LIMIT = 4
_LOCK = threading.Lock()
_FREE: dict = {}  # device index -> idle streams


def take(device):
    """A stream of the device that no other caller of this pool holds."""
    import torch

    device = torch.device(device)
    with _LOCK:
        free = _FREE.get(device.index)
        if free:
            return free.pop()
    return torch.cuda.Stream(device=device)


def give(stream) -> None:
    """Returns a stream from take(), synchronised by its caller."""
    with _LOCK:
        free = _FREE.setdefault(stream.device.index, [])
        if len(free) < LIMIT:
            free.append(stream)
