"""The pool of page-locked output arrays, on a stand-in for the allocator (no device)."""
import ctypes
import gc
import threading

import numpy as np

from flarellm_b200 import LockedPool


class Memory:
    def __init__(self):
        self.live, self.calls = {}, 0

    def alloc(self, n):
        buf = ctypes.create_string_buffer(n)
        self.live[ctypes.addressof(buf)] = buf
        self.calls += 1
        return ctypes.addressof(buf)

    def free(self, p):
        del self.live[p]


def test_blocks_are_reused_bounded_and_given_back():
    m = Memory()
    pool = LockedPool(m.free, limit=3 << 20)
    pool.add_user(); pool.add_user()
    small = pool.empty(m.alloc, (8, 64), np.float32)
    assert small.shape == (8, 64) and m.calls == 0                   # the library takes care of those
    pool.empty(m.alloc, (3, 100000), np.float32)
    assert m.calls == 0                                              # a size asked for once: an ordinary array
    a = pool.empty(m.alloc, (3, 100000), np.float32)
    assert a.shape == (3, 100000) and a.dtype == np.float32 and a.flags.writeable and m.calls == 1
    held = pool.held
    assert 1200000 <= held <= 1200000 * 9 // 8
    a[:] = 7.0
    view = a.reshape(-1)[5:]
    where = a.ctypes.data
    del a; gc.collect()
    assert view[0] == 7.0 and pool.held == held                      # a view keeps the block
    b = pool.empty(m.alloc, (300000,), np.float32)
    assert b.ctypes.data != where and m.calls == 2
    c = pool.empty(m.alloc, (300000,), np.float32)                   # the limit is reached: an ordinary array
    assert m.calls == 2 and c.shape == (300000,)
    del view; gc.collect()
    d = pool.empty(m.alloc, (350000,), np.uint16)                    # another size, for the first time: the free block will do
    assert d.ctypes.data == where and d.dtype == np.uint16 and d.shape == (350000,) and m.calls == 2
    e = pool.empty(m.alloc, (100, 1000), np.float32)
    assert m.calls == 2 and e.shape == (100, 1000)                   # nothing free
    del b; gc.collect()
    pool.empty(m.alloc, (100, 1000), np.float32)                     # a block three times too large stays free
    assert m.calls == 3 and len(m.live) == 3 and pool.held <= 3 << 20
    gc.collect()
    pool.drop_user()
    assert len(m.live) == 3
    pool.drop_user()                                                 # the last user: free blocks go, held ones when dropped
    assert len(m.live) == 1 and pool.held == held
    del d; gc.collect()
    assert not m.live and pool.held == 0


def test_an_allocator_that_fails_gives_ordinary_arrays():
    pool = LockedPool(lambda p: None)
    pool.add_user()
    pool.empty(lambda n: None, (1 << 20,), np.float32)
    a = pool.empty(lambda n: None, (1 << 20,), np.float32)
    assert a.shape == (1 << 20,) and pool.held == 0


def test_several_threads():
    m = Memory()
    pool = LockedPool(m.free, limit=16 << 20)
    pool.add_user()
    bad = []

    def work(tag):
        for i in range(200):
            a = pool.empty(m.alloc, (60000 + 10000 * (i % 3),), np.float32)
            a[:] = tag
            if not (a == tag).all():
                bad.append(tag)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    gc.collect()
    assert not bad and pool.held <= 16 << 20
    pool.drop_user()
    assert not m.live and pool.held == 0
