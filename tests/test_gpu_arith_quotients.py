"""Quotients from a rounded reciprocal against numpy where they, their reciprocal or the products on the way to them leave
the normal range: divisors just inside and just outside the ends of the range for which the reciprocal is kept, far
beyond them, and dividends of every exponent. Bit for bit, subnormal and infinite quotients included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENDS = [1e-60, 1e60, 1e-150, 1e150]
DIVISORS = sorted({v for e in ENDS for v in (np.nextafter(e, 0), e, np.nextafter(e, np.inf), 0.7 * e, 1.3 * e)} |
                  {2.0 ** -490, 2.0 ** 490, 3.0 * 2.0 ** -300, 1e-30, 1e30})


def _dividends():
    # two mantissas per exponent and sign, subnormal numbers included, and the edges of every exponent
    rng = np.random.default_rng(11)
    e = np.arange(0, 2047, dtype=np.uint64) << np.uint64(52)
    m = [rng.integers(0, 1 << 52, e.size, dtype=np.uint64) for _ in range(6)] + [np.zeros(e.size, np.uint64), np.full(e.size, (1 << 52) - 1, np.uint64)]
    x = np.concatenate([(e | q) for q in m]).view(np.float64)
    return np.concatenate([x, -x, [np.inf, -np.inf, np.nan]])


@pytest.mark.parametrize("divisor", DIVISORS)
def test_quotient_over_all_exponents(gpu_lib, divisor):
    x = _dividends()
    y = np.full_like(x, divisor)
    with np.errstate(all="ignore"):
        want = x / y
    assert np.array_equal(gpu_lib.fp64_arith_check(12, x, y), want, equal_nan=True)
