"""CPU tests of the host memory for results (sf_host_alloc): a forked child has a
copy of its own as of the fork, whatever parent and child write afterwards, and
the calls refuse what is not theirs."""
import ctypes as C
import os

import numpy as np

import stratiflow_b200 as sf

N = 3 << 20


def _alloc(n=N):
    L, p = sf.load_library(), C.c_void_p()
    assert L.sf_host_alloc(n, C.byref(p)) == 0
    return L, p, np.frombuffer((C.c_ubyte * n).from_address(p.value), dtype=np.uint8)


def test_a_forked_child_has_a_copy_of_its_own():
    L, p, a = _alloc()
    rng = np.random.default_rng(1)
    want = rng.integers(0, 256, N, dtype=np.uint8)
    a[:] = want
    go_r, go_w = os.pipe()
    child = os.fork()
    if child == 0:   # no assertion and no return: the test process must not run twice
        code = 1
        try:
            os.read(go_r, 1)          # the parent has written its array
            code = 0 if np.array_equal(a, want) else 2
            a[:] = 1
        finally:
            os._exit(code)
    a[:] = 0
    os.write(go_w, b"x")
    _, status = os.waitpid(child, 0)
    os.close(go_r)
    os.close(go_w)
    assert os.waitstatus_to_exitcode(status) == 0
    assert not a.any()                # the child's writes stayed with it
    del a
    assert L.sf_host_free(p) == 0


def test_blocks_are_freed_once_and_only_if_they_are_blocks():
    L, p, a = _alloc(1)
    a[0] = 7
    inside = C.c_void_p(p.value + 1)
    del a
    assert L.sf_host_free(inside) != 0
    assert L.sf_host_free(p) == 0
    assert L.sf_host_free(p) != 0
    assert L.sf_host_free(None) == 0
    assert L.sf_host_alloc(0, C.byref(p)) != 0
