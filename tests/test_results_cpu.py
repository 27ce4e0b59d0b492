"""Memory of large results: never shared with a live array or view, used again
after, bounded, and safe with several threads (no GPU)."""
import gc
import threading

import numpy as np

from swalbe_gb300 import _results as R


def test_reuse_only_after_every_view_is_gone():
    R.release()
    a = R.empty((8192, 600))
    assert a.flags.f_contiguous and a.flags.writeable and a.dtype == np.float64
    a[...] = 1.0
    at = a.ctypes.data
    view = a[5:7, ::2].T
    del a
    gc.collect()
    b = R.empty((8192, 600))
    assert b.ctypes.data != at
    b[...] = 2.0
    assert np.all(view == 1.0)
    del view
    gc.collect()
    c = R.empty((600, 8192))  # the same size of memory
    assert c.ctypes.data == at and np.all(b == 2.0)
    small = R.empty((3, 3))
    assert small.base is None


def test_bounded_and_released():
    R.release()
    arrays = [R.empty((4096, 1024)) for _ in range(12)]  # 32 MiB each: more than is kept
    del arrays
    gc.collect()
    assert 0 < R._kept <= R.KEEP_BYTES and R._kept == sum(len(m) for m in R._free)
    R.release()
    assert R._kept == 0 and not R._free


def test_threads_do_not_share():
    R.release()
    bad = []

    def work(k):
        for i in range(20):
            a = R.empty((2048, 2048 + (i + k) % 2))
            a[::7, ::9] = k
            if not np.all(a[::7, ::9] == k):
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
