"""Host arrays of results.

Results from 256 KB on come back in page-locked memory where a bounded pool has it: 131 MB read
back in 0.7 ms (3 ms with the pages newly locked), against 16 ms through pageable memory
into a fresh numpy array (page faults); below, the pageable copy costs less than the pool's
bookkeeping.  The pool locks at most HELD_MAX bytes in all, in results that the caller still
holds and in blocks that wait for a later result, of which there are at most WAIT_MAX bytes
(release() frees them); beyond that, and where locking fails, a result is an ordinary array.
"""
import collections
import ctypes
import os
import threading

import numpy

from . import _lib

PINNED_MIN_BYTES = 256 << 10
HELD_MAX = 4 << 30
WAIT_MAX = 1 << 30

_lock = threading.Lock()
_returned = collections.deque()  # blocks given back; the collector may do so inside the pool's own code
_waiting = []                    # [(address, size)], oldest first
_held = 0                        # bytes locked


class _Block:
    """Page-locked memory of one result; back to the pool when the last array over it is gone."""

    def __init__(self, address, size, shape):
        self.address, self.size, self.pid = address, size, os.getpid()
        self.__array_interface__ = {"version": 3, "typestr": "<f8", "shape": tuple(shape), "data": (address, False)}

    def __del__(self):
        # (a forked child has the pages, but not the lock on them; at the interpreter's end the
        # pool may be gone first)
        if _returned is not None and os is not None and self.pid == os.getpid():
            _give(self.address, self.size)


def _free(size):
    """Waiting blocks freed, oldest first, at least `size` bytes if there are (with the lock)."""
    global _held
    while size > 0 and _waiting:
        address, n = _waiting.pop(0)
        _held -= n
        size -= n
        _lib.load().okg_host_free(ctypes.c_void_p(address))


def _settle():
    """Blocks given back join the waiting ones, unless the lock is taken: then its holder does it."""
    while _returned and _lock.acquire(blocking=False):
        try:
            _drain()
        finally:
            _lock.release()


def _drain():
    while _returned:
        _waiting.append(_returned.popleft())
    _free(sum(n for _, n in _waiting) - WAIT_MAX)


def _give(address, size):
    _returned.append((address, size))
    _settle()


def _locked(f):
    with _lock:
        _drain()
        out = f()
    _settle()
    return out


def _take(size):
    """(address, size) of a block of at least `size` bytes, or None."""
    def take():
        global _held
        fit = [i for i, b in enumerate(_waiting) if size <= b[1] <= 2 * size]
        if fit:
            return _waiting.pop(min(fit, key=lambda i: (_waiting[i][1], -i)))  # (the last used of the smallest)
        step = 1 << max(16, size.bit_length() - 4)  # (sizes in steps of 1/16 .. 1/8: blocks fit similar results)
        n = -(-size // step) * step
        _free(_held + n - HELD_MAX)
        if _held + n > HELD_MAX:
            return None
        p = ctypes.c_void_p()
        if _lib.load().okg_host_alloc(n, ctypes.byref(p)) != _lib.OKG_OK:
            return None
        _held += n
        return p.value, n

    return _locked(take)


def release():
    """Free the blocks that wait for a later result."""
    _locked(lambda: _free(_held))


def held():
    """Bytes of page-locked memory in results and waiting."""
    return _locked(lambda: _held)


class Result:
    """Host array of a result, filled in ranges of its last axis from device tensors."""

    def __init__(self, *shape):
        size = 8
        for v in shape:
            size *= int(v)
        block = _take(size) if size >= PINNED_MIN_BYTES else None
        self.array = numpy.asarray(_Block(*block, shape)) if block else numpy.empty(shape)
        self.address = block[0] if block else None
        self.stream = None

    def put(self, i, j, part):
        """Columns [i, j) from the contiguous device tensor `part`, on the current stream."""
        if self.address is None:
            self.array[..., i:j] = part.cpu().numpy()
            return
        import torch
        self.stream = torch.cuda.current_stream()
        n = self.array.shape[-1]
        _lib.check(_lib.load().okg_read_rows(ctypes.c_void_p(self.address + 8 * i), 8 * n, _lib.ptr(part), 8 * (j - i),
                                             self.array.size // n, _lib.stream_handle(self.stream)))

    def finish(self):
        """The array, complete."""
        if self.stream is not None:
            self.stream.synchronize()
            self.stream = None
        return self.array

    def __del__(self):
        # (an evaluation that raised: its copies end before the block has another user)
        if getattr(self, "stream", None) is not None:
            self.stream.synchronize()
