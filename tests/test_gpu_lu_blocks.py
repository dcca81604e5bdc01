"""The blocked float64 LU (n > 256) at the sizes where its parts change: leaves of one CTA up to 512
rows and clusters of 4, 8 and 16 beyond, the look-ahead and its persistent update from n = 1024,
leaves taller than 8192 rows, blocks and leaves that end short. Against the oracle as
test_lu_matches_oracle holds it (pivots equal; factors within 64 n eps of their scale), and the
pivot rule's special cases: equal magnitudes (the first row), a zero column (left unreduced), a
subnormal pivot (divided by, not inverted), NaN (never chosen but when nothing else is left)."""
import numpy as np
import pytest

from oracle import oracle as O
from refdata import ref_random

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def rb():
    import rustymath_b200 as rb
    return rb


@pytest.mark.parametrize("n", [257, 264, 288, 385, 511, 513, 545, 641, 1023, 1024, 1025, 1153, 1700])
def test_blocks_match_the_oracle(rb, n):
    a = ref_random(n, n, n + 1)
    f, p = rb.lu(a)
    fo, po = O.lu_factor(a)
    assert np.array_equal(p, po)
    assert np.abs(f - fo).max() <= 64 * n * EPS * max(1.0, np.abs(fo).max())


@pytest.mark.parametrize("n", [300, 700])
def test_ties_take_the_first_row(rb, n):
    """A = L U with every multiplier +-1 and integer U: each column's candidates tie with the
    diagonal, every step is exact, so the factors are L and U and no row moves."""
    rng = np.random.default_rng(n)
    lower = np.tril(rng.choice([-1.0, 1.0], (n, n)), -1) + np.eye(n)
    upper = np.triu(rng.integers(-2, 3, (n, n)).astype(float), 1) + np.diag(rng.choice([-1.0, 1.0], n))
    f, p = rb.lu(lower @ upper)
    assert np.array_equal(p, np.arange(n))
    np.testing.assert_array_equal(f.T, np.tril(lower, -1) + upper)


@pytest.mark.parametrize("n,col", [(300, 0), (300, 290), (700, 37), (1100, 130)])
def test_zero_nan_and_subnormal_columns(rb, n, col):
    a = ref_random(n, n, 3)
    zero = a.copy()
    zero[:, col] = 0.0
    nan = a.copy()
    nan[col:, col] = np.nan
    # the first pivot candidates subnormal: the reciprocal of the chosen one is not finite
    sub = a.copy()
    sub[:, 0] *= 2.0 ** -1060
    for m in (zero, nan, sub):
        f, p = rb.lu(m)
        fo, po = O.lu_factor(m)
        assert np.array_equal(p, po)
        assert np.array_equal(np.isnan(f), np.isnan(fo))
        fine = ~np.isnan(fo)
        assert np.abs(f[fine] - fo[fine]).max() <= 64 * n * EPS * max(1.0, np.abs(fo[fine]).max())


def test_leaves_taller_than_the_register_panel():
    """n = 8260: the first leaves have more than 8192 rows and take the other panel. Residual
    ||L U - P A|| (infinity norm) below 4 eps n of ||L|| ||U||, the usual backward error bound."""
    import torch

    from rustymath_b200 import linalg
    n = 8260
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    f = linalg.lu(a)
    low = torch.tril(f.factors.mT, -1)
    low.diagonal().fill_(1.0)
    up = torch.triu(f.factors.mT)
    assert torch.equal(f.p.sort().values, torch.arange(n, device="cuda"))
    assert low.abs().max().item() <= 1.0
    r = (low @ up - a[f.p]).abs().sum(1).max()
    assert (r / (low.abs().sum(1).max() * up.abs().sum(1).max())).item() < 4 * EPS * n
