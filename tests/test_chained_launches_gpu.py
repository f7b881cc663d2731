"""A stage's kernels launched while the one before runs out against the same
kernels launched one by one (timed steps have an event between any two): the
same kernels on the same inputs, so after many steps back to back every bit of
the state agrees. Grids whose kernels end in a partial wave, fit a few SMs, fill
tables before they wait, and a tangent batch's two x passes."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,nrun,tangent", [
    (64, 1, 64, 1, False), (256, 1, 260, 5, False), (128, 1, 132, 17, True), (64, 16, 36, 1, False),
    (64, 32, 180, 2, False), (256, 16, 132, 1, False), (64, 16, 36, 3, True),
])
def test_same_bits_as_one_by_one(n1, n2, n3, nrun, tangent):
    cfg = dict(CONFIGS["kh2d" if n2 == 1 else "shear3d_small"], N1=n1, N2=n2, N3=n3)
    out = []
    for timed in (False, True):
        s = gpu_solver(cfg, nrun=nrun)
        for r in range(nrun):
            s.set_state(r, make_ic(cfg, seed=60 + r % 3, amp=5e-2))
        if tangent:
            s.set_tangent(1)
        s.Prepare()
        if timed:
            s.profile_step(20)
        else:
            for _ in range(20):
                s.TimeStep()
        s.synchronize()
        out.append(np.asarray(s.get_state_kept()).copy())
    assert np.isfinite(out[0].view(np.float32)).all()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
