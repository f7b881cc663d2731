"""The 3D adjoint x pass in slabs of levels (k_xpass_adj3), the kernel of the
row widths that do not march, against the FP64 oracle: two steps, several runs,
heights that leave the last slab short. Bounds as tests/test_adjoint_gpu.py:
1e-5 relative L2 for u1, u2, u3, b, 5e-4 for p."""
import pytest

from tests.helpers import CONFIGS, make_ic, make_oracle, rel_l2
from tests.test_adjoint_gpu import _kept
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,nrun", [(16, 16, 36, 2), (32, 32, 44, 1), (32, 16, 68, 2)])
def test_adjoint_slabs_match_oracle(n1, n2, n3, nrun):
    cfg = dict(CONFIGS["shear3d_small"], N1=n1, N2=n2, N3=n3)
    below, above, adj = ([make_ic(cfg, seed=600 + 10 * k + r, amp=1e-3 if k == 2 else 5e-2) for r in range(nrun)]
                         for k in range(3))
    s = gpu_solver(cfg, nrun=nrun)
    for r in range(nrun):
        s.set_state(r, adj[r])
    s.Prepare()
    kb, ka = _kept(cfg, below), _kept(cfg, above)
    for _ in range(2):
        s.TimeStepAdjoint(kb, ka)
    for r in range(nrun):
        o = make_oracle(cfg, 64)
        o.set_state(adj[r])
        o.prepare()
        for _ in range(2):
            o.step_adjoint(below[r], above[r])
        for k in ("u1", "u2", "u3", "b"):
            assert rel_l2(s.get_field(r, k), o.get_field(k)) < 1e-5, (r, k)
        assert rel_l2(s.get_field(r, "p"), o.get_field("p")) < 5e-4, r
