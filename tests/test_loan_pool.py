"""Page-locked output arrays of a recording (vai_b200.engine._LoanPool): on a stand-in for the library, and through a net."""
import ctypes
import gc
import threading

import numpy as np
import pytest

import vai_b200
from vai_b200 import Tensor, engine, nodes


class FakeLib:
    def __init__(self):
        self.live, self.calls, self.copies_that_work = {}, [], 99

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


class FakeDevice:
    def __init__(self, lib):
        self.lib = lib

    def create_stream(self):
        return None


def _fake_net(monkeypatch):
    lib = FakeLib()

    def copy(dst, src, nbytes, stream):
        lib.calls.append("copy")
        lib.copies_that_work -= 1
        return 0 if lib.copies_that_work >= 0 else 3

    lib.vaicu_memcpy_d2h = copy
    lib.vaicu_stream_sync = lambda stream: lib.calls.append("sync") or 0
    monkeypatch.setattr(engine._lib, "_lib", None)            # the error text of a failed call needs no library
    return engine.NeuralNet(device=FakeDevice(lib)), lib


def test_a_failed_recording_gives_its_memory_back(monkeypatch):
    net, lib = _fake_net(monkeypatch)

    def fails(rec, fed):
        rec.loans["y"] = engine._LoanPool(lib, 64, np.float32, (4, 4))
        net._pinned(64, np.float32, (4, 4))
        assert len(lib.live) == 3
        raise RuntimeError("half way")

    monkeypatch.setattr(net, "_record_into", fails)
    with pytest.raises(RuntimeError, match="half way"):
        net._record({})
    assert not lib.live


def test_arrays_of_a_failed_call_go_back_after_the_stream(monkeypatch):
    net, lib = _fake_net(monkeypatch)
    rec = engine._Recording()

    class Pool(engine._LoanPool):
        def give_back(self, ptr):
            lib.calls.append("back")
            super().give_back(ptr)

    class Out:
        ptr = 0

    rec.loans = {"a": Pool(lib, 64, np.float32, (4, 4)), "b": Pool(lib, 64, np.float32, (4, 4))}
    rec.outputs = {"a": Out, "b": Out}
    lib.copies_that_work = 1
    try:
        net._finish(rec)
    except engine._lib.VaicuError:
        pass
    else:
        raise AssertionError("the failed copy was not reported")
    gc.collect()
    assert lib.calls == ["copy", "copy", "sync", "back", "back"]
    lib.copies_that_work, lib.calls = 99, []
    assert set(net._finish(rec)) == {"a", "b"} and lib.calls[:3] == ["copy", "copy", "sync"]


@pytest.mark.gpu
def test_results_of_a_net_stay_as_they_were(device):
    """Results of 64 KB and more, all held: the first four in page-locked arrays, the others in copies, each with its own values,
    also through views, after further calls and after the net is gone."""
    M, K = 256, 128
    net = vai_b200.NeuralNet()
    lin = nodes.LinearNode(in_dim=K, out_dim=K)
    lin["weight"] = Tensor.from_numpy(np.eye(K, dtype=np.float32))
    net.input("x") - lin - net.output("y")
    rng = np.random.default_rng(0)
    held = []
    for i in range(8):
        x = rng.standard_normal((M, K)).astype(np.float32)
        y = net(Tensor.from_numpy(x)).host
        held.append((x, y if i % 2 else y[1:]))
        if i == 5:
            del held[0]                     # its array is handed out again
    pool = next(iter(net._recordings.values())).loans["y"]
    assert pool.made == pool.LIMIT
    for x, y in held:
        np.testing.assert_array_equal(y, x[-len(y):])
    del net, lin, pool
    gc.collect()
    for x, y in held:
        np.testing.assert_array_equal(y, x[-len(y):])
