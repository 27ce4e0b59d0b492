"""Host memory of large result arrays.

From 32 MiB on the C allocator maps every array afresh.  Such an array has no
pages yet, and the download into it takes their faults one by one: 2.1 ms for a
2048² field, against 0.24 ms into memory that has its pages (300 iterations of
a 2048² FP32 film with upload and result: 22.0 -> 19.8 ms).  So the memory of
such results is mapped here and used again once its array (and every view of
it) is gone.  Smaller ones are better left to the allocator, which keeps their
memory itself (24 results of 0.1 to 2 MiB: 11.9 ms, and 12.2 from here).  New
memory of the pool comes in large pages: a first 2048² field takes 1.4 ms.
The memory stays the pool's, so ndarray.resize refuses these arrays.
"""
from __future__ import annotations

import collections
import math
import mmap
import os
import threading
import weakref

import numpy as np

MIN_BYTES = 32 << 20    # smaller arrays come from numpy's allocator
KEEP_BYTES = 256 << 20  # unused memory kept at most

_lock = threading.Lock()  # for _free and _kept; only release() waits for it
_returned: collections.deque = collections.deque()  # given back, not sorted in yet
_free: list = []  # unused mappings, oldest first
_kept = 0


def _sort_in() -> None:
    """Moves what was given back to the unused mappings, as many as are kept.

    A finalizer runs wherever the garbage collector does, also on a thread that
    holds the lock, so nothing here waits for it: whoever holds it comes back
    for what was given back meanwhile.
    """
    global _kept
    while _returned and _lock.acquire(blocking=False):
        try:
            while _returned:
                mem = _returned.popleft()
                _free.append(mem)
                _kept += len(mem)
            while _kept > KEEP_BYTES:
                _kept -= len(_free.pop(0))  # unmapped with its last reference
        finally:
            _lock.release()


def _give(mem) -> None:
    _returned.append(mem)
    _sort_in()


def _take(size: int):
    global _kept
    mem = None
    if _lock.acquire(blocking=False):  # else new memory
        try:
            for i in range(len(_free) - 1, -1, -1):
                if len(_free[i]) == size:
                    mem = _free.pop(i)
                    _kept -= size
                    break
        finally:
            _lock.release()
        _sort_in()
    if mem is not None:
        return mem
    # private, as numpy's own memory is: after a fork each process writes to its
    # own copy (and, as for numpy's, in large pages where the system has them)
    try:
        mem = mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    except OSError as e:
        raise MemoryError(f"{size} bytes for a result: {e}") from e
    try:
        mem.madvise(mmap.MADV_HUGEPAGE)
    except (AttributeError, OSError):
        pass
    return mem


def empty(shape) -> np.ndarray:
    """An uninitialised column-major Float64 array."""
    n = 8 * math.prod(shape)
    if n < MIN_BYTES:
        return np.empty(shape, dtype=np.float64, order="F")
    mem = _take(-(-n // mmap.PAGESIZE) * mmap.PAGESIZE)
    a = np.ndarray(shape, dtype=np.float64, buffer=mem, order="F")
    weakref.finalize(a, _give, mem).atexit = False
    return a


def release() -> None:
    """Gives unused memory back."""
    global _kept
    with _lock:
        _returned.clear()
        _free.clear()
        _kept = 0
    _sort_in()


def _after_fork() -> None:
    # another thread of the parent may have been inside the pool; it is not here
    global _lock, _kept
    _lock = threading.Lock()
    _returned.clear()
    _free.clear()
    _kept = 0


os.register_at_fork(after_in_child=_after_fork)
