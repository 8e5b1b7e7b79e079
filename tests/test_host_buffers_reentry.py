"""Results dropped in reference cycles while the pool of result memory is at its limit: a garbage collection that
starts inside a call of the pool finalises them, and their memory comes back in the middle of that call."""
import gc

import numpy as np

from earthbyte_underworld_gb300 import uwgpu as U


class _Cycle:
    def __init__(self, held):
        self.held, self.me = held, self


def test_collection_inside_a_call_leaves_blocks_whole():
    pool = U._HostBuffers()
    pool.LIMIT = 12 << 20
    sizes = np.array([1, 2, 3, 2, 1, 3]) << 20
    rng = np.random.default_rng(4)
    saved = gc.get_threshold()
    gc.collect()
    gc.freeze()
    gc.set_threshold(0)
    try:
        for trial in range(2000):
            # the pool at its limit, and three results that only a collection gives back
            arrays = [pool.array(int(n), np.uint8) for n in rng.permutation(sizes)]
            for n in rng.permutation(sizes)[:3]:
                _Cycle(pool.array(int(n), np.uint8))
            del arrays
            need = int(rng.choice(sizes))
            gc.set_threshold(gc.get_count()[0] + trial % 16, 1, 1)   # starts at another place of the call each time
            a = pool.array(need, np.uint8)
            gc.set_threshold(0)
            # numpy does not check the size of memory it is handed: the block has to hold the whole array
            block = getattr(a.base, "raw", None)
            assert a.nbytes == need and (block is None or block.nbytes >= need), trial
            assert sum(r.nbytes for r in pool._free) == pool._held <= pool.LIMIT, trial
            del a, block
            gc.collect()
            assert sum(r.nbytes for r in pool._free) == pool._held <= pool.LIMIT, trial
    finally:
        gc.set_threshold(*saved)
        gc.unfreeze()


def test_finaliser_that_asks_for_a_result_does_not_wait_for_itself():
    pool = U._HostBuffers()
    got = []

    class Asks(_Cycle):
        def __del__(self):
            got.append(pool.array(1 << 20, np.uint8).nbytes)
            pool.release()

    saved = gc.get_threshold()
    gc.collect()
    gc.freeze()
    gc.set_threshold(0)
    try:
        for trial in range(500):
            kept = [pool.array(1 << 20, np.uint8) for _ in range(4)]
            del kept
            Asks(None)
            gc.set_threshold(gc.get_count()[0] + trial % 16, 1, 1)
            pool.array(1 << 20, np.uint8)
            gc.set_threshold(0)
            gc.collect()
    finally:
        gc.set_threshold(*saved)
        gc.unfreeze()
    assert got == [1 << 20] * 500
