"""Page-locked memory behind read-backs, with the allocator faked on the host: how much of it there is at a time, how long
a block lives, and returns from a finaliser that runs inside the pool's own code."""
import ctypes as C
import gc

import numpy as np
import pytest

from neuralrs_b200 import cuda

KB = 1024


class FakeLib:
    def __init__(self, room=1 << 40):
        self.live, self.most, self.room = {}, 0, room

    def nrs_host_alloc(self, size, out):
        if self.total() + size > self.room:
            return 3
        buf = (C.c_char * size)()
        out._obj.value = C.addressof(buf)
        self.live[C.addressof(buf)] = buf
        self.most = max(self.most, self.total())
        return 0

    def nrs_host_free(self, ptr):
        del self.live[ptr.value]
        return 0

    def total(self):
        return sum(map(len, self.live.values()))


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(cuda._lib, "lib", lambda: lib)
    monkeypatch.setattr(cuda, "_pinned", cuda._PinnedPool(limit=1024 * KB, most=4096 * KB))
    yield lib


def test_kept_results_stop_pinning_at_the_bound(fake):
    kept = [cuda._result(128 * KB) for _ in range(12)]   # 512 KB each, 6 MB in all
    for i, a in enumerate(kept):
        a[:] = i
    assert fake.total() == 4096 * KB == fake.most
    assert all((a == i).all() for i, a in enumerate(kept))
    del a
    kept.clear()
    assert fake.total() == 1024 * KB                     # idle blocks
    other = [cuda._result(256 * KB) for _ in range(4)]   # of another size: the idle ones make room
    assert fake.total() == 4096 * KB == fake.most and len(other) == 4


def test_block_lives_as_long_as_any_view_of_it(fake):
    a = cuda._result(100000)
    view = a[10:].reshape(-1, 2)
    view[:] = 7
    at = a.ctypes.data
    del a
    gc.collect()
    assert at in fake.live and (view == 7).all()
    other = cuda._result(100000)
    assert other.ctypes.data != at
    del view
    assert cuda._result(100000).ctypes.data == at        # back in the pool, handed out again


def test_return_while_the_pool_is_busy(fake):
    a = cuda._result(100000)
    at = a.ctypes.data
    with cuda._pinned.lock:                              # as when a collection runs inside take()
        del a
        gc.collect()
    assert cuda._result(100000).ctypes.data == at


def test_small_results_and_refusals_are_ordinary_memory(fake):
    assert isinstance(cuda._result(1000), np.ndarray) and fake.total() == 0
    fake.room = 0
    assert cuda._result(100000).size == 100000 and fake.total() == 0
    fake.room = 1 << 40
    assert cuda._result(100000).ctypes.data in fake.live
    assert cuda._pinned.locked == fake.total()
