"""Host arrays of a solve to the device.

A pageable copy goes through the driver's staging buffers on one thread, and every one of
them waits for the stream.  Here the small arrays of a solve travel packed in one
page-locked block (one copy instead of eight), and a large one in slots of a page-locked
ring that four threads fill while earlier slots are in flight.  Measured, pageable against
ring: 16 MB 1.0 against 1.2 ms, 49 MB 4.7 against 2.3 ms, 64 MB 6.1 against 2.6 ms; arrays in
between the two kinds take the pageable copy.  The threads are few and wait without
spinning: torch's own parallel copy, one thread per core, took 40 ms for 49 MB whenever
another process had a core.

The page-locked memory is at most ``SLOTS * SLOT_BYTES`` per call and belongs to torch's caching
host allocator, which does not hand a block out again before the copies that read it have
finished (on whatever stream they were enqueued); the threads belong to one pool, joined at
exit.
"""

from __future__ import annotations

import threading
from concurrent.futures import Future, ThreadPoolExecutor

import numpy as np

__all__ = ['to_device']

PACK_BYTES = 1 << 18  # arrays up to this size are packed together
RING_BYTES = 24 << 20  # arrays from this size on go through the ring
SLOT_BYTES = 2 << 20
SLOTS = 12
AHEAD = 6  # slots being filled; the copies of the others are in flight
THREADS = 4
_ALIGN = 256

_LOCK = threading.Lock()
_POOL = None


def _pool() -> ThreadPoolExecutor:
    global _POOL
    with _LOCK:
        if _POOL is None:
            _POOL = ThreadPoolExecutor(THREADS, thread_name_prefix='dqb-upload')
        return _POOL


def _submit(fn, *args) -> Future:
    """``fn(*args)`` on a thread of the pool, or here where none can be had (the interpreter is
    exiting, or the process is out of threads)."""
    try:
        return _pool().submit(fn, *args)
    except RuntimeError:
        done = Future()
        done.set_result(fn(*args))
        return done


def _host_array(x, dtype):
    """``x`` as a contiguous numpy array of the torch ``dtype``."""
    import torch

    np_dtype = {torch.complex64: np.complex64, torch.complex128: np.complex128,
                torch.float64: np.float64, torch.int32: np.int32}[dtype]
    a = np.ascontiguousarray(x)
    if a.dtype != np_dtype:
        with np.errstate(all='ignore'):
            a = a.astype(np_dtype)
    return a


def _ring_copy(dst, a) -> None:
    """The bytes of ``a`` into the device tensor ``dst``, on the current stream."""
    import torch

    src = a.reshape(-1).view(np.uint8)
    out = dst.view(-1).view(torch.uint8)
    chunks = range(0, src.size, SLOT_BYTES)
    ring = torch.empty(SLOTS * SLOT_BYTES, dtype=torch.uint8, pin_memory=True)
    host = ring.numpy()
    done = [None] * SLOTS

    def fill(i):
        o, s = chunks[i], i % SLOTS * SLOT_BYTES
        m = min(SLOT_BYTES, src.size - o)
        # This thread waits until the slot's previous contents have left: the threads of the
        # pool serve every caller, and one that waited for a busy stream would hold up uploads
        # to others.
        if done[i % SLOTS] is not None:
            done[i % SLOTS].synchronize()
        return _submit(np.copyto, host[s:s + m], src[o:o + m])

    filled = [fill(i) for i in range(min(AHEAD, len(chunks)))]
    for i, o in enumerate(chunks):
        filled[i].result()
        s, m = i % SLOTS * SLOT_BYTES, min(SLOT_BYTES, src.size - o)
        out[o:o + m].copy_(ring[s:s + m], non_blocking=True)
        done[i % SLOTS] = torch.cuda.Event()
        done[i % SLOTS].record()
        if i + AHEAD < len(chunks):
            filled.append(fill(i + AHEAD))


def to_device(items: dict, device) -> dict:
    """Device tensors of ``{name: (array, dtype)}``, copied on ``device``'s current stream (work
    on other streams must wait for it).  The arrays may be changed once this returns."""
    import torch

    out, packed, total = {}, [], 0
    with torch.cuda.device(device):
        for name, (x, dtype) in items.items():
            if isinstance(x, torch.Tensor):
                out[name] = x.to(device=device, dtype=dtype).contiguous()
                continue
            a = _host_array(x, dtype)
            if a.nbytes <= PACK_BYTES:
                packed.append((name, a, dtype, total))
                total += -(-max(a.nbytes, 1) // _ALIGN) * _ALIGN
            elif a.nbytes < RING_BYTES:
                out[name] = torch.from_numpy(a if a.flags.writeable else a.copy()).to(device)
            else:
                out[name] = torch.empty(a.shape, dtype=dtype, device=device)
                _ring_copy(out[name], a)
        if packed:
            host = torch.empty(total, dtype=torch.uint8, pin_memory=True)
            h = host.numpy()
            for _, a, _, o in packed:
                h[o:o + a.nbytes] = a.reshape(-1).view(np.uint8)
            d = host.to(device, non_blocking=True)
            for name, a, dtype, o in packed:
                out[name] = d[o:o + a.nbytes].view(dtype).view(a.shape)
    return out
