"""Halves, quarters and the comparison with a positive bound, which the FP64 face flux forms by integer
operations, against numpy: bit for bit over all exponents, with zeros, subnormal numbers, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values():
    rng = np.random.default_rng(3)
    bits = rng.integers(0, 1 << 63, 1 << 16, dtype=np.uint64) | (rng.integers(0, 2, 1 << 16, dtype=np.uint64) << np.uint64(63))
    edge = [0.0, 5e-324, 1e-310, 2.2250738585072014e-308, 4.450147717014403e-308, 8.900295434028806e-308,
            1.7800590868057611e-307, 1e-20, np.nextafter(1e-20, 0), np.nextafter(1e-20, 1), 1.0, 1.7976931348623157e308, np.inf, np.nan]
    e = np.array(edge)
    return np.concatenate([bits.view(np.float64), e, -e])


@pytest.mark.parametrize("op,factor", [(8, 0.5), (9, 0.25)])
def test_scaled_by_powers_of_two(gpu_lib, op, factor):
    x = _values()
    with np.errstate(all="ignore"):
        want = x * factor
    assert np.array_equal(gpu_lib.fp64_arith_check(op, x), want, equal_nan=True)


@pytest.mark.parametrize("bound", [float(np.float32(1e-20)), 0.5])
def test_comparison(gpu_lib, bound):
    x = _values()
    assert np.array_equal(gpu_lib.fp64_arith_check(10, x, np.full_like(x, bound)), (x <= bound).astype(np.float64))
