"""CPU test of bench.py's byte model of the z pass: k_z_step_f's mean over the
three stages, counted stage by stage."""
import types

import pytest

import bench


@pytest.mark.parametrize("N2,fields,stages", [(128, 4, (18, 22, 20)), (1, 3, (15, 18, 16))])
def test_z_step_f_bytes_are_the_mean_of_its_stages(N2, fields, stages):
    s = types.SimpleNamespace(N1=256, N2=N2, N3=384, nrun=2, K1=85, K2=2 * (N2 // 3) - 1 if N2 > 1 else 1, dim3=N2 > 1)
    S = s.N3 * s.K1 * s.K2 * 8 * s.nrun
    pivots = 2                                     # four float fields
    for k, want in enumerate(stages):
        read = fields + 1 + fields + (fields if k else 0) + pivots
        written = fields + 1 + (2 if k < 2 else 0)
        assert read + written == want
    assert bench.kernel_bytes(s, "k_z_step_f") == pytest.approx(sum(stages) / 3 * S, rel=1e-12)
    assert bench.kernel_bytes(s, "k_z_step_c") == (3 * fields + 3 + 2 * fields + 1) * S
