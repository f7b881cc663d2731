"""A stage whose z pass is not k_z_step_f launches its x pass in the ordinary
way in 2D and chained in 3D: columns too short (k_z_step) and too tall
(k_z_step_c) for it, and the z kernels by choice. After many steps every bit
equals that of the same kernels launched one by one, as in
tests/test_chained_launches_gpu.py."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,nrun,zkernel,tangent", [
    (64, 1, 20, 1, 2, False), (256, 1, 28, 5, 2, True), (64, 1, 900, 1, 2, False), (128, 1, 68, 2, 0, False),
    (64, 16, 20, 1, 2, False), (64, 16, 700, 1, 2, False), (64, 16, 36, 3, 0, True),
])
def test_same_bits_as_one_by_one(n1, n2, n3, nrun, zkernel, tangent):
    cfg = dict(CONFIGS["kh2d" if n2 == 1 else "shear3d_small"], N1=n1, N2=n2, N3=n3)
    out = []
    for timed in (False, True):
        s = gpu_solver(cfg, nrun=nrun)
        s.set_z_kernel(zkernel)
        for r in range(nrun):
            s.set_state(r, make_ic(cfg, seed=60 + r % 3, amp=5e-2))
        if tangent:
            s.set_tangent(1)
        s.Prepare()
        if timed:
            s.profile_step(10)
        else:
            for _ in range(10):
                s.TimeStep()
        s.synchronize()
        out.append(np.asarray(s.get_state_kept()).copy())
        s.close()
    assert np.isfinite(out[0].view(np.float32)).all()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
