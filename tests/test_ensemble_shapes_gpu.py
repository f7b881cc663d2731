"""The ensemble's stage kernel on every grid width and on the heights where its
z items change shape (chunks in registers up to 64 levels, fused columns up to
484, taller ones by the one-field-after-the-other body), members mixed, against
each run on its own solver: the same scheme with other segments and chunks, so
the parity tests' bound against the FP64 oracle holds between them (1e-5
relative L2 per field, 5e-4 for p), 5 steps. A member's dt changed between two
calls takes effect."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic, rel_l2
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu

MIXES = [
    [(16, 36), (32, 64), (64, 68), (128, 100), (256, 128), (512, 132)],
    [(64, 484), (64, 488), (128, 32), (32, 1024), (16, 16)],
    [(512, 36)],
    [(64, 128)] * 40,
]


@pytest.mark.parametrize("grids", MIXES, ids=["widths", "heights", "one", "many"])
def test_ensemble_matches_its_members_alone(grids):
    import stratiflow_b200 as sf
    from stratiflow_b200.grid import background_profile
    base = CONFIGS["kh2d"]
    cfgs = [dict(base, N1=n1, N3=n3, Ri=0.05 + 0.01 * r) for r, (n1, n3) in enumerate(grids)]
    e = sf.Ensemble(grids, (base["L1"], base["L3"], base["Re"], base["Pr"]), base["dt"])
    ics, made = [], {}
    for r, (c, m) in enumerate(zip(cfgs, e.members)):
        U, dB = background_profile(c["bg"], c["L3"], c["N3"])
        m.set_ri(0, c["Ri"])
        m.SetBackground(0, U, dB)
        key = (c["N1"], c["N3"])
        ics.append(made.setdefault(key, make_ic(c, seed=90, amp=5e-2)))
        m.set_state(0, ics[r])
        m.Prepare()
    e.step(3)
    e.synchronize()
    for m in e.members:
        m.UpdateForTimestep(0.5 * base["dt"])
    e.step(2)
    e.synchronize()
    for r, c in enumerate(cfgs):
        s = gpu_solver(c)
        s.set_state(0, ics[r])
        s.Prepare()
        s.TimeStep(3)
        s.UpdateForTimestep(0.5 * base["dt"])
        s.TimeStep(2)
        s.synchronize()
        a, b = s.get_state_kept()[0], e.members[r].get_state_kept()[0]
        s.close()
        assert np.isfinite(b).all()
        for f in (0, 2, 3, 4):
            err = rel_l2(b[f], a[f])
            assert err <= (5e-4 if f == 4 else 1e-5), (grids[r], f, err)
    e.close()
