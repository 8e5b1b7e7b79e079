"""Results of the binding are ordinary arrays: they own their data, resize in place, and grow and shrink through the
pool's allocator without losing values."""
import gc
import pickle
import threading

import numpy as np

from earthbyte_underworld_gb300 import uwgpu as U


def test_results_own_their_data():
    pool = U._HostBuffers()
    for n in (10, 1 << 17, (1 << 17) + 1, 1 << 20):
        a = pool.array((n, 3), np.float64)
        assert type(a) is np.ndarray and a.base is None and a.flags.owndata and a.flags.writeable and a.flags.aligned
        a[:] = np.arange(3 * n).reshape(n, 3)
        a.resize((2 * n, 3))   # in place, zero-filled, as of any array
        assert a.flags.owndata and a[n:].sum() == 0 and np.array_equal(a[:n].reshape(-1), np.arange(3 * n))
        a.resize((5, 3))
        assert np.array_equal(a.reshape(-1), np.arange(15))
        b = pickle.loads(pickle.dumps(a))
        assert np.array_equal(a, b) and a.copy().base is None


def test_allocator_stays_with_the_results():
    """other arrays made meanwhile and afterwards come from numpy's own allocator, in every thread"""
    pool = U._HostBuffers()
    kept = pool.array(3 << 20, np.uint8)
    del kept
    assert pool._held >= 3 << 20
    before = [r.nbytes for r in pool._free]
    other = [np.empty(3 << 20, np.uint8) for _ in range(3)]
    del other
    assert [r.nbytes for r in pool._free] == before
    # a result that outlives its pool object, dropped by another thread
    a = pool.array(2 << 20, np.uint8)
    a[:] = 7
    del pool
    gc.collect()
    assert (a == 7).all()
    box = [a]
    del a
    t = threading.Thread(target=box.clear)
    t.start()
    t.join()


def test_limit_change_evicts():
    pool = U._HostBuffers()
    arrays = [pool.array(2 << 20, np.uint8) for _ in range(4)]
    del arrays
    assert len(pool._free) == 4
    pool.LIMIT = 5 << 20
    assert pool.LIMIT == 5 << 20 and len(pool._free) == 2 and pool._held <= pool.LIMIT
    pool.release()
    assert pool._held == 0
