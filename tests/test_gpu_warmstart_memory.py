"""Where the rows of gb_ws_forward and gb_ws_forward_backward may lie: pageable memory, device memory, and
outputs inside the rows. A row's output does
not depend on where it was read from, so all of them give the bits of the plain call."""
import ctypes

import numpy as np
import pytest

import mlp_oracle as mo
from test_gpu_warmstart import _params

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROWS = [1, 640, 32768, 70001]


def _ptr(address):
    return ctypes.cast(ctypes.c_void_p(address), ctypes.POINTER(ctypes.c_float))


@pytest.fixture
def network(gpu_lib):
    with gpu_lib.WarmStart(seed=5) as w:
        w.set_params(_params(3))
        yield w


def _rows(n):
    return np.random.default_rng(n).uniform(-1.0, 1.0, size=(n, mo.N_IN)).astype(np.float32)


@pytest.mark.parametrize("rows", ROWS)
def test_rows_in_device_memory(network, rows):
    x = _rows(rows)
    want = network.forward(x)
    d = torch.from_numpy(x).cuda()
    y = np.empty((rows, mo.N_OUT), dtype=np.float32)
    torch.cuda.synchronize()
    network._check(network._L.gb_ws_forward(network.h, _ptr(d.data_ptr()), rows, _ptr(y.ctypes.data)))
    assert np.array_equal(y, want)


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("at", [0.0, 0.4, 0.75])
def test_outputs_inside_the_rows(network, rows, at):
    x = _rows(rows)
    want = network.forward(x)
    buf = x.copy()
    first = int(at * buf.size)                           # (the outputs are a quarter of the rows' size)
    network._check(network._L.gb_ws_forward(network.h, _ptr(buf.ctypes.data), rows, _ptr(buf.ctypes.data + 4 * first)))
    flat, n = buf.reshape(-1), rows * mo.N_OUT
    assert np.array_equal(flat[first:first + n].reshape(want.shape), want)
    assert np.array_equal(flat[:first], x.reshape(-1)[:first]) and np.array_equal(flat[first + n:], x.reshape(-1)[first + n:])
