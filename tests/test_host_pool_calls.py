"""CPU tests of when the host calls' output arrays are pinned, with a fake allocator that counts."""
import gc

import numpy as np
import pytest

from test_host_pool import FakeLib
from tritium_b200.backend import _HostPool


class CountingLib(FakeLib):
    def __init__(self):
        super().__init__()
        self.pinned = 0   # allocations so far

    def tb_host_alloc(self, backend, size, out):
        self.pinned += 1
        return super().tb_host_alloc(backend, size, out)


@pytest.mark.parametrize("keeps,pinned", [("nothing", 1), ("the last", 2), ("all", 0), ("a view of each", 0)])
def test_calls_pin_memory_only_for_callers_that_drop_their_results(keeps, pinned):
    """Pinning happens inside a call, so a caller that keeps every output must not meet it, and one that
    drops them only in its first few calls."""
    lib = CountingLib()
    pool = _HostPool(lib, None)
    kept, after_four = [], None
    for i in range(20):
        out = pool.output((5000,), np.float32)
        out[:] = i
        if keeps == "all":
            kept.append(out)
        elif keeps == "a view of each":
            kept.append(out[5:10])
        elif keeps == "the last":
            kept = [out]
        del out
        gc.collect()
        if i == 3:
            after_four = lib.pinned
    assert lib.pinned == after_four == pinned
    if len(kept) == 20:
        assert all((a == i).all() for i, a in enumerate(kept))
    assert pool.output((100,), np.float32).base is None


def test_sizes_that_do_not_all_fit_are_not_pinned_in_turn():
    lib = CountingLib()
    pool = _HostPool(lib, None)
    pool.LIMIT = 1 << 18
    for _ in range(50):
        for size in (1 << 16, 1 << 18):   # bytes: the second one fills the limit alone
            pool.output((size // 4,), np.float32)
            gc.collect()
    assert lib.pinned <= 2 + 100 // pool.EVICT_EVERY
    pool.close()
    assert not lib.live and pool._pinned == 0
