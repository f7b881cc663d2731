"""The pool of page-locked result buffers (stratiflow_b200._ResultBuffers), on
the CPU with a fake allocator: a buffer is not handed out while a view of its
array lives, comes back when the last one is gone, the bytes held never pass
the limit, and ordinary memory serves what does not fit."""
import ctypes as C
import threading

import numpy as np
import pytest

import stratiflow_b200 as sf


class FakeLib:
    def __init__(self):
        self.live, self.allocs = {}, 0

    def sf_host_alloc(self, n, out):
        b = (C.c_char * n)()
        self.live[C.addressof(b)] = b
        out._obj.value = C.addressof(b)
        self.allocs += 1
        return 0

    def sf_host_free(self, p):
        del self.live[p.value]
        return 0


@pytest.fixture
def pool(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(sf, "load_library", lambda path=None: lib)
    p = sf._ResultBuffers()
    p.lib = lib
    return p


N = sf._ResultBuffers.SMALL // 4


def test_a_buffer_is_reused_only_after_its_last_view(pool):
    a = pool.empty((N,))
    a[:] = 1
    v = a[10:20]
    del a
    b = pool.empty((N,))
    b[:] = 2
    assert pool.lib.allocs == 2 and np.all(v == 1)
    del v
    c = pool.empty((2, N // 2))
    assert pool.lib.allocs == 2 and c.shape == (2, N // 2) and c.flags.writeable and np.all(b == 2)


def test_small_and_excess_results_are_ordinary_memory(pool):
    assert pool.empty((8,)).flags.owndata and pool.lib.allocs == 0
    big = pool.LIMIT // 4
    keep = [pool.empty((big // 4,)) for _ in range(6)]
    assert pool.lib.allocs == 4 and pool.held == pool.LIMIT
    assert all(k.flags.owndata for k in keep[4:])
    del keep
    x = pool.empty((big // 2,))   # another size: the waiting buffers make room
    assert pool.held <= pool.LIMIT and len(pool.lib.live) * 1 >= 1 and not x.flags.owndata


def test_threads_get_buffers_of_their_own(pool):
    bad = []

    def work(k):
        for i in range(200):
            a = pool.empty((N,))
            a[:] = k
            if not np.all(a == k):
                bad.append(k)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad and pool.held <= pool.LIMIT
