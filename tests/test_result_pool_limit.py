"""CPU test of the result pool (stratiflow_b200._ResultBuffers): a result that
cannot be held, because it is larger than the limit or because too much is in
use, leaves the waiting buffers where they are."""
import numpy as np
import pytest

import stratiflow_b200 as sf
from tests.test_result_buffers import FakeLib


@pytest.fixture
def pool(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(sf, "load_library", lambda path=None: lib)
    p = sf._ResultBuffers()
    p.lib = lib
    return p


def test_a_result_that_does_not_fit_evicts_nothing(pool):
    q = pool.LIMIT // 16           # floats of a quarter of the limit
    a, b = pool.empty((q,)), pool.empty((q,))
    del a
    big = pool.empty((pool.LIMIT // 4 + 1,))          # over the limit by itself
    assert big.flags.owndata and len(pool.lib.live) == 2
    big = pool.empty((3 * q + q // 2,))               # over it beside what is in use
    assert big.flags.owndata and len(pool.lib.live) == 2
    fits = pool.empty((3 * q,))                       # fits once the waiting one is gone
    assert not fits.flags.owndata and pool.held == pool.LIMIT and len(pool.lib.live) == 2
    assert np.all(b.shape == (q,))
