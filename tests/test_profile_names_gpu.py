"""GPU test: sf_profile_names names the x-pass kernel that the profiled step
launched. Small 2D grids march the linear step's rows and take the slab kernel
for the nonlinear step's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N1,N2,runs,linear,march", [
    (64, 1, 1, True, True), (64, 1, 1, False, False), (128, 1, 1, False, True), (64, 16, 1, True, True),
    (32, 16, 1, True, False),
])
def test_names_follow_the_profiled_step(N1, N2, runs, linear, march):
    import stratiflow_b200 as sf
    s = sf.IMEXRK(N1, N2, 64, 14.0, 7.0, 10.0, 1000.0, 1.0, 0.01, nrun=runs)
    if linear:
        st = s.get_state(0)
        s.SetBase(0, st["u1"], st["u2"], st["u3"], st["b"])
    names = [n.split(":")[1] for n, _ in s.profile_step(1, linear=linear)]
    assert ("k_xmarch" in names) == march and ("k_xpass" in names) == (not march)
    if linear:   # the last step profiled counts
        names = [n.split(":")[1] for n, _ in s.profile_step(1)]
        assert ("k_xmarch" in names) == (march and N2 > 1)
    s.close()
