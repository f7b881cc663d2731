"""The live-base march (tangent-linear batches) against the slab kernels at the
row widths of four lanes, whose warps hold eight segments, some of them idle,
and with several bases, tangent r about base (r - nbase) % nbase. The bound is
that of tests/test_xmarch_modes_gpu.py: 1e-5 relative L2 per field, 5e-4 for p,
after 3 steps."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic, rel_l2
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,nrun,nbase", [
    (16, 1, 260, 33, 1), (16, 1, 388, 24, 2), (32, 1, 132, 33, 1), (32, 1, 260, 18, 2),
    (128, 1, 68, 9, 3), (256, 1, 260, 6, 2), (64, 16, 36, 6, 2),
])
def test_live_base_march_agrees_with_the_slabs(n1, n2, n3, nrun, nbase):
    cfg = dict(CONFIGS["kh2d" if n2 == 1 else "shear3d_small"], N1=n1, N2=n2, N3=n3)
    assert n2 > 1 or n1 * n3 * (nrun - nbase) >= (1 << 13 if n1 == 128 else 1 << 17)   # both kernels can run
    ics = [make_ic(cfg, seed=160 + r, amp=5e-2) for r in range(5)]

    def run(kind):
        s = gpu_solver(cfg, nrun=nrun)
        s.set_xpass_kernel(kind)
        for r in range(nrun):
            s.set_state(r, ics[r % len(ics)])
        s.set_tangent(nbase)
        s.Prepare()
        s.TimeStep(3)
        s.synchronize()
        out = s.get_state_kept()
        s.close()
        return out
    a, b = run(0), run(1)
    assert np.isfinite(a).all() and not np.array_equal(a, b)
    for r in range(nrun):
        for f in range(5):
            err = rel_l2(b[r, f], a[r, f])
            assert err <= (5e-4 if f == 4 else 1e-5), (r, f, err)
