"""Page-locked output arrays of a recording (vai_b200.engine._LoanPool), on a stand-in for the two library calls."""
import ctypes
import gc
import threading

import numpy as np

from vai_b200 import engine


class FakeLib:
    def __init__(self):
        self.live = {}

    def vaicu_host_alloc_pinned(self, nbytes, out):
        buf = ctypes.create_string_buffer(nbytes)
        self.live[ctypes.addressof(buf)] = buf
        ctypes.cast(out, ctypes.POINTER(ctypes.c_void_p))[0] = ctypes.addressof(buf)
        return 0

    def vaicu_host_free_pinned(self, ptr):
        del self.live[ptr.value]
        return 0


def test_arrays_are_bounded_reused_and_freed():
    lib = FakeLib()
    pool = engine._LoanPool(lib, 64, np.float32, (4, 4))
    assert len(lib.live) == pool.FIRST
    held = [pool.array(pool.take()) for _ in range(pool.LIMIT)]
    assert pool.take() is None and len(lib.live) == pool.LIMIT
    view = held[0][1:]
    view[:] = 3.0
    del held[0]
    gc.collect()
    assert pool.take() is None            # a view keeps the memory out
    del view
    gc.collect()
    again = pool.array(pool.take())
    assert again.shape == (4, 4) and again.dtype == np.float32
    pool.close()
    assert len(lib.live) == pool.LIMIT    # all are out
    t = threading.Thread(target=held.clear)
    t.start()
    t.join()
    del again
    gc.collect()
    assert not lib.live
