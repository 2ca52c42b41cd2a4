"""The warm-start network on numbers of rows where the kernels' work is split: forward() runs in pieces of
32768 rows whose features the device reads from the caller's memory (16-byte loads where they are aligned), and
a block works on two tiles of 128 rows in turn, from 152 x 128 rows on. A row's output does not depend on the other
rows, so forward() on slices gives the same bits; gradients against the CPU oracle at the bound of the
gradient test (3e-2 normwise: one BF16 ulp of a stored intermediate is 4e-3)."""
import numpy as np
import pytest

import mlp_oracle as mo
from test_gpu_warmstart import _params, _rel, _split

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,shift", [(1, 0), (127, 1), (32768, 0), (32769, 0), (98304, 2), (100001, 1)])
def test_forward_in_pieces(gpu_lib, rows, shift):
    flat = np.random.default_rng(rows).uniform(-1.0, 1.0, size=rows * mo.N_IN + 4).astype(np.float32)
    base = (-flat.ctypes.data // 4) % 4                     # first 16-byte boundary
    shift = (base + shift) % 4 if shift else base
    x = flat[shift:shift + rows * mo.N_IN].reshape(rows, mo.N_IN)
    with gpu_lib.WarmStart(seed=5) as w:
        w.set_params(_params(3))
        y = w.forward(x)
        parts = [w.forward(x[a:a + 5000].copy()) for a in range(0, rows, 5000)]
    assert np.array_equal(y, np.concatenate(parts))


@pytest.mark.parametrize("rows", [129, 152 * 128 + 129])
def test_gradients_over_two_tiles(gpu_lib, rows):
    p = _params(4)
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1.0, 1.0, size=(rows, mo.N_IN)).astype(np.float32)
    t = rng.normal(size=(rows, mo.N_USED)).astype(np.float32)
    with gpu_lib.WarmStart(seed=5) as w:
        w.set_params(p)
        loss, g = w.forward_backward(x, t)
    loss_o, go = mo.loss_and_grad(p, x, t)
    assert abs(loss - loss_o) / loss_o < 1e-2
    for q, (a, b) in enumerate(zip(_split(g), _split(go))):
        if np.linalg.norm(b) == 0.0:
            assert np.all(a == 0.0), q
            continue
        assert _rel(a, b) < 3e-2, (q, _rel(a, b))
