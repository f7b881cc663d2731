"""A member's z kernel (IMEXRK.set_z_kernel) holds in its ensemble: members with
kernel 0 or 1 solve one field after the other, with chunks of their own, and so
differ in rounding from the same members left at the default, on heights where
the stage kernel's items are 8 modes and where they are 16. Both agree with the
run on its own solver within the parity tests' bounds (1e-5 relative L2 per
field, 5e-4 for p, 4 steps), and the setting may change between two calls."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic, rel_l2
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu

GRIDS = [(64, 16), (64, 36), (128, 128), (256, 484), (32, 488), (64, 1024)]


def _run(ics, first, then):
    """Two steps with z kernels `first`, two with `then`; the kept states."""
    import stratiflow_b200 as sf
    from stratiflow_b200.grid import background_profile
    c = CONFIGS["kh2d"]
    e = sf.Ensemble(GRIDS, (c["L1"], c["L3"], c["Re"], c["Pr"]), c["dt"])
    for m, (n1, n3), ic in zip(e.members, GRIDS, ics):
        U, dB = background_profile(c["bg"], c["L3"], n3)
        m.set_ri(0, c["Ri"])
        m.SetBackground(0, U, dB)
        m.set_state(0, ic)
        m.Prepare()
    for kinds in (first, then):
        for m, k in zip(e.members, kinds):
            m.set_z_kernel(k)
        e.step(2)
        e.synchronize()
    out = [m.get_state_kept()[0] for m in e.members]
    e.close()
    return out


def test_a_members_z_kernel_holds_in_the_ensemble():
    base = CONFIGS["kh2d"]
    cfgs = [dict(base, N1=n1, N3=n3) for n1, n3 in GRIDS]
    ics = [make_ic(c, seed=60, amp=5e-2) for c in cfgs]
    n = len(GRIDS)
    default = _run(ics, [2] * n, [2] * n)
    again = _run(ics, [2] * n, [2] * n)
    zero = _run(ics, [0] * n, [0] * n)
    changed = _run(ics, [2] * n, [0] * n)
    mixed = _run(ics, [0, 2, 1, 2, 0, 2], [0, 2, 1, 2, 0, 2])
    for r, c in enumerate(cfgs):
        assert np.array_equal(default[r], again[r])
        assert not np.array_equal(default[r], zero[r]), GRIDS[r]
        assert not np.array_equal(changed[r], zero[r]) and not np.array_equal(changed[r], default[r]), GRIDS[r]
        assert np.array_equal(mixed[r], default[r] if r in (1, 3, 5) else zero[r]), GRIDS[r]
        s = gpu_solver(c)
        s.set_state(0, ics[r])
        s.Prepare()
        s.set_z_kernel(0)
        s.TimeStep(4)
        s.synchronize()
        a = s.get_state_kept()[0]
        s.close()
        for b in (default[r], zero[r], changed[r]):
            for f in (0, 2, 3, 4):
                err = rel_l2(b[f], a[f])
                assert err <= (5e-4 if f == 4 else 1e-5), (GRIDS[r], f, err)
