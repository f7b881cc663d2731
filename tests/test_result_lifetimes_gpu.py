"""GPU tests of who owns host memory after a call of the predictor returns: a
caller may change or drop the arrays it passed in or was given, whatever is
still queued on the GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CH, Z, B = [64, 256, 512], 64, 4   # forward results of 512 KB, gradients of 2.9 MB: buffers of the pool


def _net(stream=None):
    import stratiflow_b200 as sf
    n = sf.Net(CH, Z, B, seed=3, stream=stream)
    rng = np.random.default_rng(4)
    n.set_params(rng.normal(0, 0.05, n.num_params).astype(np.float32))
    return n, rng.normal(0, 1, (B, Z, CH[0])).astype(np.float32)


def _delay():
    import torch
    torch.cuda._sleep(100_000_000)   # tens of milliseconds on the current stream


def test_set_data_has_read_its_arrays_when_it_returns():
    import torch
    st = torch.cuda.Stream()
    n, x = _net(st.cuda_stream)
    y = n.forward(x)
    y += 1.0                       # loss 1 against these targets
    with torch.cuda.stream(st):
        _delay()                   # whatever set_data queues runs after this
    n.set_data(x, y)
    y -= 1.0
    _, loss = n.gradient()
    assert abs(loss - 1.0) < 1e-4


def test_a_result_can_be_changed_or_dropped_under_a_queued_copy():
    import torch
    n, x = _net()
    y = n.forward(x)
    want = y.copy()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _delay()
        d = torch.from_numpy(y).to("cuda", non_blocking=True)
    y[:] = 0.0
    side.synchronize()
    assert torch.equal(d.cpu(), torch.from_numpy(want))
    y = n.forward(x)
    with torch.cuda.stream(side):
        _delay()
        d = torch.from_numpy(y).to("cuda", non_blocking=True)
    del y
    n.forward(-x)                  # takes the buffer that came back
    side.synchronize()
    assert torch.equal(d.cpu(), torch.from_numpy(want))


RESET = """
import ctypes, os
import numpy as np
import stratiflow_b200 as sf
import nvidia.cuda_runtime
rng = np.random.default_rng(4)

def gradient():
    n = sf.Net([64, 256, 512], 64, 4, seed=3)
    n.set_params(w)
    n.set_data(x, t)
    return n.gradient()[0]

w = rng.normal(0, 0.05, 64 * 5 * 256 + 256 + 256 * 5 * 512 + 512).astype(np.float32)
x, t = (rng.normal(0, 1, (4, 64, c)).astype(np.float32) for c in (64, 512))
a, b = gradient(), gradient()
want = a.copy()
del b                              # its buffer waits in the pool
rt = ctypes.CDLL(os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib", "libcudart.so.12"))
assert rt.cudaDeviceReset() == 0
assert np.array_equal(a, want)
assert np.array_equal(gradient(), want)
print("same")
"""


def test_results_outlive_a_reset_of_the_device():
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr


def test_states_stream_through_blocks():
    """sf_step_host_async in and out of two states inside blocks of
    sf_host_alloc, against the same states in arrays."""
    import ctypes as C
    import stratiflow_b200 as sf
    from tests.helpers import CONFIGS, make_ic
    from tests.test_gpu_parity import gpu_solver
    s = gpu_solver(CONFIGS["kh2d"])
    want, ins = [], []
    for k in range(2):
        s.set_state(0, make_ic(CONFIGS["kh2d"], seed=80 + k, amp=5e-2))
        s.Prepare()
        ins.append(s.get_state_kept())
        s.TimeStep(2)
        s.synchronize()
        want.append(s.get_state_kept())
    L, n, ptrs, bufs = sf.load_library(), ins[0].nbytes, [], []
    for _ in range(2):
        p = C.c_void_p()
        assert L.sf_host_alloc(2 * n, C.byref(p)) == 0
        ptrs.append(p)
        bufs.append(np.frombuffer((C.c_char * (2 * n)).from_address(p.value), dtype=np.complex64)
                    .reshape((2,) + s.kept_shape))
    bufs[0][0], bufs[0][1] = ins
    for k in range(2):
        s.step_host_async(bufs[0][k], bufs[1][k], 2)
    s.synchronize()
    assert np.array_equal(bufs[1][0], want[0]) and np.array_equal(bufs[1][1], want[1])
    del bufs
    for p in ptrs:
        assert L.sf_host_free(p) == 0
