"""Where the rows of gb_ws_forward and gb_ws_forward_backward may lie: pageable memory, pinned memory that a copy on the
default stream still fills, device memory that it still fills, and outputs inside the rows. A row's output does
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
@pytest.mark.parametrize("where", ["device", "pinned"])
def test_rows_still_being_written(network, rows, where):
    x = _rows(rows)
    want = network.forward(x)
    new = torch.from_numpy(x).cuda()
    old = torch.zeros((rows, mo.N_IN), device="cuda") if where == "device" else torch.zeros((rows, mo.N_IN), pin_memory=True)
    y = np.empty((rows, mo.N_OUT), dtype=np.float32)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)                       # some 50 ms on the default stream, then the rows
    old.copy_(new, non_blocking=True)
    network._check(network._L.gb_ws_forward(network.h, _ptr(old.data_ptr()), rows, _ptr(y.ctypes.data)))
    assert np.array_equal(y, want)


@pytest.mark.parametrize("rows", ROWS)
def test_rows_in_device_memory(network, rows):
    x = _rows(rows)
    want = network.forward(x)
    d = torch.from_numpy(x).cuda()
    y = np.empty((rows, mo.N_OUT), dtype=np.float32)
    torch.cuda.synchronize()
    network._check(network._L.gb_ws_forward(network.h, _ptr(d.data_ptr()), rows, _ptr(y.ctypes.data)))
    assert np.array_equal(y, want)


@pytest.mark.parametrize("rows", [640, 40000])
def test_gradients_of_rows_and_targets_still_being_written(network, rows):
    x, t = _rows(rows), np.random.default_rng(rows + 1).normal(size=(rows, mo.N_USED)).astype(np.float32)
    loss, grad = network.forward_backward(x, t)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    xs, ts = torch.zeros_like(xd), torch.zeros(t.shape, pin_memory=True)
    g, l = np.zeros(network.n_params, dtype=np.float32), ctypes.c_float()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    xs.copy_(xd)
    ts.copy_(td, non_blocking=True)
    network._check(network._L.gb_ws_forward_backward(network.h, _ptr(xs.data_ptr()), _ptr(ts.data_ptr()), rows, ctypes.byref(l),
                                                     _ptr(g.ctypes.data)))
    assert l.value == loss and np.array_equal(g, grad)


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
