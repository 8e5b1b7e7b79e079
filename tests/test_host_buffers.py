"""Reuse of result memory in the Python binding: a block returns only when no array refers to it, the total is
bounded, small results stay plain arrays."""
import threading

import numpy as np

from earthbyte_underworld_gb300 import uwgpu as U


def test_reuse_needs_every_view_gone():
    pool = U._HostBuffers()
    a = pool.array((1 << 18, 3), np.float64)
    assert a.shape == (1 << 18, 3) and a.flags.c_contiguous and a.flags.writeable
    a[:] = 1.0
    where, view = a.ctypes.data, a[5:, 1]
    del a
    b = pool.array((1 << 18, 3), np.float64)
    assert b.ctypes.data != where and float(view[0]) == 1.0
    del view
    c = pool.array(6 << 17, np.float64)
    assert c.ctypes.data == where
    assert pool.array(10, np.uint32).base is None


def test_bound_and_release():
    pool = U._HostBuffers()
    pool.LIMIT = 8 << 20
    arrays = [pool.array(3 << 20, np.uint8) for _ in range(6)]
    del arrays
    assert pool._held <= pool.LIMIT and sum(r.nbytes for r in pool._free) == pool._held > 0
    big = pool.array(64 << 20, np.uint8)
    del big
    assert all(r.nbytes < 64 << 20 for r in pool._free)
    pool.release()
    assert pool._held == 0 and not pool._free


def test_threads_get_distinct_memory():
    pool = U._HostBuffers()
    wrong = []

    def work(k):
        for _ in range(200):
            a = pool.array(1 << 20, np.uint8)
            a[:] = k
            if not (a == k).all():
                wrong.append(k)
            del a

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong and pool._held <= 8 << 20
