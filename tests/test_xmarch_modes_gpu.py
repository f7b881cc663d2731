"""The level-marching x passes (sf_set_xpass_kernel 1) against the slab kernels
(0) in every mode: nonlinear, frozen base, live base (tangent-linear batch) and
adjoint, 2D and 3D, every row width they take, heights that leave segments
short or lane groups idle, several runs. Both form the same products; the
transforms and the z stencils round in another order, so the states agree to
the parity tests' bound against the FP64 oracle (1e-5 relative L2 per field,
5e-4 for p) after 3 steps."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic, rel_l2
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu

# mode, N1, N2, N3, runs
CASES = [
    ("nonlinear", 16, 1, 260, 64), ("linear", 16, 1, 36, 2),
    ("nonlinear", 32, 1, 256, 33), ("nonlinear", 64, 1, 100, 41), ("nonlinear", 128, 1, 132, 16),
    ("nonlinear", 256, 1, 260, 4), ("nonlinear", 512, 1, 132, 4), ("nonlinear", 64, 16, 36, 2),
    ("linear", 32, 1, 36, 1), ("linear", 64, 1, 44, 3), ("linear", 128, 1, 68, 1), ("linear", 256, 1, 36, 2),
    ("linear", 512, 1, 68, 1), ("linear", 64, 16, 36, 2), ("linear", 128, 16, 36, 1), ("linear", 256, 16, 36, 1),
    ("tangent", 64, 1, 100, 42), ("tangent", 128, 1, 132, 17), ("tangent", 256, 1, 260, 5), ("tangent", 512, 1, 132, 5),
    ("tangent", 64, 16, 36, 3), ("tangent", 128, 16, 36, 2), ("tangent", 256, 16, 36, 2),
    ("adjoint", 32, 1, 36, 2), ("adjoint", 64, 1, 44, 1), ("adjoint", 128, 1, 68, 3), ("adjoint", 256, 1, 36, 1),
    ("adjoint", 64, 16, 36, 2), ("adjoint", 128, 16, 36, 1), ("adjoint", 256, 16, 36, 1),
]


@pytest.mark.parametrize("mode,n1,n2,n3,nrun", CASES)
def test_march_agrees_with_the_slabs(mode, n1, n2, n3, nrun):
    cfg = dict(CONFIGS["kh2d" if n2 == 1 else "shear3d_small"], N1=n1, N2=n2, N3=n3)
    ics = [make_ic(cfg, seed=60 + r, amp=5e-2) for r in range(min(nrun, 3))]

    def run(kind):
        s = gpu_solver(cfg, nrun=nrun)
        s.set_xpass_kernel(kind)
        if mode == "adjoint":
            for r in range(nrun):
                s.set_state(r, ics[(r + 1) % len(ics)])
            below = s.get_state_kept()
            for r in range(nrun):
                s.set_state(r, ics[(r + 2) % len(ics)])
            above = s.get_state_kept()
        for r in range(nrun):
            s.set_state(r, ics[r % len(ics)])
            if mode == "linear":
                b = ics[(r + 1) % len(ics)]
                s.SetBase(r, b["u1"], b["u2"], b["u3"], b["b"])
        if mode == "tangent":
            s.set_tangent(1)
        s.Prepare()
        for _ in range(3):
            if mode == "adjoint":
                s.TimeStepAdjoint(below, above)
            elif mode == "linear":
                s.TimeStepLinear()
            else:
                s.TimeStep()
        s.synchronize()
        out = s.get_state_kept()
        s.close()
        return out
    a, b = run(0), run(1)
    assert np.isfinite(a).all()
    for f in range(5):
        err = rel_l2(b[:, f], a[:, f])
        assert err <= (5e-4 if f == 4 else 1e-5), (f, err)
