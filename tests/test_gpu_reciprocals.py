"""The reciprocals that multiply the pivot columns, to the bit. rustymath's `divide` multiplies by the
pivot's correctly rounded reciprocal, or divides where the pivot is subnormal. In the LU of a lower
triangular matrix whose diagonal is each column's largest item nothing is subtracted but zeros, so the
factors are that division alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pivots(n, rng, bits, low, high, tiny):
    """Random mantissas, mantissas of all ones and powers of two, of ordinary magnitude and near both
    ends of the exponent range (low .. high), and below it."""
    mantissa = 1.0 + rng.integers(0, 2 ** bits, n) * 2.0 ** -bits
    mantissa[1::5] = 2.0 - 2.0 ** -bits
    mantissa[2::7] = 1.0
    mantissa[3::11] = 2.0 - 2.0 ** (1 - bits)
    exponent = rng.integers(-3, 4, n)
    exponent[4::6] = rng.integers(high - 3, high + 1, exponent[4::6].size)
    exponent[5::6] = rng.integers(low, low + 4, exponent[5::6].size)
    d = np.ldexp(mantissa, exponent)
    d[9::13] = tiny * rng.integers(1, 1000, d[9::13].size)
    return d * rng.choice([-1.0, 1.0], n)


# one CTA a leaf (300), clusters of 4 and of 16 (700, 2500), the one-launch form (100)
@pytest.mark.parametrize("n", [100, 300, 700, 2500])
def test_float64_multipliers_are_the_division_of_the_reference(n):
    from rustymath_b200 import linalg
    rng = np.random.default_rng(n)
    d = pivots(n, rng, 52, -1022, 1023, 5e-324)
    with np.errstate(all="ignore"):
        a = np.tril(rng.uniform(-1, 1, (n, n)), -1) * d + np.diag(d)
        expect = np.where(np.abs(d) < np.finfo(np.float64).tiny, a / d, a * (1.0 / d))
    expect = np.tril(expect, -1) + np.diag(d)
    f, p = linalg.lu(a)
    assert np.array_equal(p, np.arange(n))
    np.testing.assert_array_equal(f.T, expect)
