"""The predictor's GEMM tiles at their edges against the CPU restatement
oracle/net_ref.py (bounds as tests/test_net_gpu.py states them): channel counts
below, at and past a tile of 128 rows and a K slice of 64, and counts that are
not multiples of 16; one level, and levels below, at and past a tile of 64."""
import numpy as np
import pytest

from oracle import net_ref as R
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ch,Z,B", [
    ([8, 24, 16], 1, 2), ([8, 8, 8], 5, 1), ([64, 128, 64], 64, 2), ([72, 136, 56], 63, 3), ([136, 264, 72], 65, 2),
    ([128, 64, 128], 130, 2),
])
def test_forward_and_gradient_at_tile_edges(ch, Z, B):
    import stratiflow_b200 as sf
    n = sf.Net(ch, Z, B, seed=5)
    p = R.init_params(ch, 5)
    n.set_params(p)
    rng = np.random.default_rng(8)
    x = rng.normal(0, 1, (B, Z, ch[0])).astype(np.float32)
    t = rng.normal(0, 1, (B, Z, ch[-1])).astype(np.float32)
    y, _ = R.forward(p, ch, x)
    assert rel_l2(n.forward(x), y) < 2e-3
    n.set_data(x, t)
    g, loss = n.gradient()
    gr, lr = R.gradient(p, ch, x, t)
    assert abs(loss - lr) <= 1e-4 * lr
    off = 0
    for l, (ci, co) in enumerate(zip(ch[:-1], ch[1:])):
        nw = co * 5 * ci
        tol = 1e-4 if l == len(ch) - 2 else 1e-2
        assert rel_l2(g[off:off + nw], gr[off:off + nw]) < tol, l
        assert rel_l2(g[off + nw:off + nw + co], gr[off + nw:off + nw + co]) < tol, l
        off += nw + co
