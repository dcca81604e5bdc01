"""An infinity in the blocked float64 LU (n > 256): it stays where rustymath's substitution and products leave
it. A block row with one is substituted, as a product with an inverted diagonal block's zeros would spread it.
Pivots equal and the same items finite, infinite and NaN as the oracle's, up to the infinity's own column."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# the infinity in the first or the second block's rows, in a later block's columns or the last, short one
@pytest.mark.parametrize("n,row,col", [(300, 5, 200), (300, 100, 299), (700, 200, 640), (1100, 3, 1050)])
def test_an_infinity_stays_in_its_column(n, row, col):
    from rustymath_b200 import linalg
    rng = np.random.default_rng(n + col)
    a = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    a[row, col] = np.inf
    f, p = linalg.lu(a)
    with np.errstate(all="ignore"):
        fo, po = O.lu_factor(a)
    done = (col // 128) * 128  # columns of the blocks before the infinity's
    assert np.array_equal(p[:done], po[:done])
    f, fo = f.T, fo.T
    for got, want in ((f[:, :done], fo[:, :done]), (f[:done], fo[:done])):
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
        fine = np.isfinite(want)
        assert np.abs(got[fine] - want[fine]).max() <= 64 * n * np.finfo(np.float64).eps * np.abs(want[fine]).max()
