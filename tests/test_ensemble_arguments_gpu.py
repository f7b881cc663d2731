"""GPU test: an ensemble's stage arguments reach the device although the call
that first saw them changed was only recorded (its stream was being captured
into a graph that never runs). Bit for bit against the same calls without the
recorded one."""
import ctypes
import os

import numpy as np
import pytest

from tests.helpers import CONFIGS, make_ic

pytestmark = pytest.mark.gpu


def _recorded(stream, call):
    import nvidia.cuda_runtime
    rt = ctypes.CDLL(os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib", "libcudart.so.12"))
    graph = ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(ctypes.c_void_p(stream), 2) == 0   # relaxed
    try:
        call()
    finally:
        assert rt.cudaStreamEndCapture(ctypes.c_void_p(stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphDestroy(graph) == 0


@pytest.mark.parametrize("record", [False, True])
def test_arguments_changed_under_a_capture_still_arrive(record):
    import stratiflow_b200 as sf
    from stratiflow_b200.grid import background_profile
    c = CONFIGS["kh2d"]
    grids = [(64, 64), (128, 100)]
    out = []
    for rec in (False, record):
        e = sf.Ensemble(grids, (c["L1"], c["L3"], c["Re"], c["Pr"]), c["dt"])
        for m, (n1, n3) in zip(e.members, grids):
            U, dB = background_profile(c["bg"], c["L3"], n3)
            m.set_ri(0, c["Ri"])
            m.SetBackground(0, U, dB)
            m.set_state(0, make_ic(dict(c, N1=n1, N3=n3), seed=70, amp=5e-2))
            m.Prepare()
        e.step(1)
        e.synchronize()
        for m in e.members:
            m.UpdateForTimestep(0.5 * c["dt"])
        if rec:
            _recorded(e.stream(), lambda: e.step(0))
        e.step(2)
        e.synchronize()
        out.append([m.get_state_kept() for m in e.members])
        e.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
