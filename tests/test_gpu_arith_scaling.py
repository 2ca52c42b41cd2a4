"""Halves, quarters and comparisons, which the FP64 form takes by integer operations, and quotients from a rounded
reciprocal, against numpy: bit for bit over all exponents, with zeros, subnormal numbers, infinities and NaN."""
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


@pytest.mark.parametrize("bound", [0.0, 1e-300, 1.0, np.inf, np.nan])
def test_larger(gpu_lib, bound):
    x = _values()
    assert np.array_equal(gpu_lib.fp64_arith_check(11, x, np.full_like(x, bound)), (x > bound).astype(np.float64))


@pytest.mark.parametrize("divisor", [26.0, 0.72, 0.9, 1.0, np.nextafter(2.0, 0), 3e-7, 1e-200, 0.0, None])
def test_quotient_from_the_reciprocal(gpu_lib, divisor):
    # (the sign of a zero quotient is not kept where it is minus zero over a positive number: it equals plus zero)
    x = np.concatenate([_values(), np.random.default_rng(5).normal(size=1 << 18)])
    y = np.full_like(x, divisor) if divisor is not None else np.abs(np.random.default_rng(6).normal(size=x.size)) + 1e-3
    with np.errstate(all="ignore"):
        want = x / y
    assert np.array_equal(gpu_lib.fp64_arith_check(12, x, y), want, equal_nan=True)
