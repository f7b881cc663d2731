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
