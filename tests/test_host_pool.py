"""CPU tests of the pool behind the host calls' output arrays, with a fake allocator."""
import ctypes as C
import gc

import numpy as np

from tritium_b200.backend import _HostPool


class FakeLib:
    def __init__(self):
        self.live = {}

    def tb_host_alloc(self, _backend, size, out):
        buf = (C.c_uint8 * size.value)()
        self.live[C.addressof(buf)] = buf
        out._obj.value = C.addressof(buf)
        return 0

    def tb_host_free(self, ptr):
        del self.live[ptr.value]


def test_buffers_are_reused_bounded_and_freed():
    lib = FakeLib()
    pool = _HostPool(lib, None)
    small = pool.array((100,), np.float32)
    assert small.base is None and not lib.live          # below the smallest size: ordinary memory
    a = pool.array((5000,), np.float32)
    a[:] = 1
    b = pool.array((2, 5000), np.float32)
    b[:] = 2
    assert len(lib.live) == 2 and (a == 1).all()
    view = a[10:]
    del a
    gc.collect()
    c = pool.array((5000,), np.float32)                 # the view still holds the first buffer
    c[:] = 3
    assert (view == 1).all() and len(lib.live) == 3
    del view
    gc.collect()
    d = pool.array((4900,), np.float32)                 # the same size class: used again
    assert len(lib.live) == 3
    pool.LIMIT = pool._pinned
    e = pool.array((1 << 20,), np.float32)              # over the limit: ordinary memory
    assert e.base is None and len(lib.live) == 3
    del b, e
    gc.collect()
    pool.LIMIT = pool._pinned - 65536 + (1 << 17)       # room for a new one only once the idle one is freed
    f = pool.array((30000,), np.float32)
    assert f.base is not None and len(lib.live) == 3
    pool.close()
    d[:] = 4
    assert len(lib.live) == 3 and (d == 4).all()
    del c, d, f
    gc.collect()
    assert not lib.live and pool._pinned == 0
