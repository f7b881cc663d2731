"""Every shape of the default z pass (k_z_step_f: 2D and 3D; short chunks in
registers, one or two blocks per SM, tall columns) against k_z_step
(sf_set_z_kernel 0) at the edges of its range: the smallest and the tallest
grid that takes it, the first one past it, chunks with a remainder, empty
chunks, and the block counts on either side of the choice between one and two
blocks per SM. Both solve the same systems with the same terms; the chunks
reassociate the recurrences, so they agree to the parity tests' bound against
the FP64 oracle (1e-5 relative L2 per field, 5e-4 for p), 4 steps."""
import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic, rel_l2
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu

# N1, N2, N3, runs
GRIDS = [
    (64, 1, 32, 1), (64, 1, 64, 2), (64, 1, 68, 1), (64, 1, 128, 3),          # 2D in registers
    (64, 1, 132, 1), (32, 1, 244, 2), (64, 1, 488, 1),                        # 2D, one block per SM
    (64, 1, 132, 50), (64, 1, 268, 50), (64, 1, 272, 50),                     # 2D, blocks for two per SM, and past it
    (64, 1, 492, 1), (32, 1, 824, 1), (32, 1, 828, 1),                        # 2D, tall, and past every shape
    (16, 16, 32, 1), (16, 16, 64, 2),                                         # 3D in registers
    (16, 16, 96, 1), (16, 16, 100, 2), (16, 16, 128, 1), (16, 16, 100, 99),   # 3D, the longer register chunks, and past the block rule
    (16, 16, 68, 1), (16, 16, 132, 1), (16, 16, 332, 1), (16, 16, 672, 1), (16, 16, 676, 1),    # 3D, one block per SM, and past it
    (16, 16, 132, 26), (32, 16, 332, 15), (32, 16, 336, 15),                   # 3D, blocks for two per SM, and past it
]


@pytest.mark.parametrize("n1,n2,n3,nrun", GRIDS)
def test_z_pass_shapes_agree_with_the_z_step(n1, n2, n3, nrun):
    cfg = dict(CONFIGS["kh2d" if n2 == 1 else "shear3d_small"], N1=n1, N2=n2, N3=n3)
    ic = make_ic(cfg, seed=77, amp=5e-2)

    def run(kind):
        s = gpu_solver(cfg, nrun=nrun)
        s.set_z_kernel(kind)
        for r in range(nrun):
            s.set_state(r, ic)
            s.set_ri(r, 0.05 + 0.01 * r)
        s.Prepare()
        s.TimeStep(4)
        s.synchronize()
        out = s.get_state_kept()
        s.close()
        return out
    a, b = run(0), run(2)
    assert np.isfinite(a).all()
    for f in range(5):
        err = rel_l2(b[:, f], a[:, f])
        assert err <= (5e-4 if f == 4 else 1e-5), (f, err)
