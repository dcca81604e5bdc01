"""Triangular solves of many right-hand sides run as one chain per 16 columns side by side. Every
chain does what it does alone, so a wide solve equals, bit for bit, the same columns solved 16 at
a time; the widths leave remainders and exceed the CTAs that an SM array holds at once."""
import numpy as np
import pytest

from refdata import ref_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,k", [(193, 17), (257, 33), (330, 4001)])
def test_wide_solves_equal_narrow_ones(n, k, trans):
    import rustymath_b200 as rb
    from rustymath_b200.linalg import lu_solve
    f = rb.lu(ref_random(n, n, 7))
    b = np.random.default_rng(k).standard_normal((n, k))
    wide = lu_solve(f.factors, f.p, b, trans=trans)
    for c in sorted({0, 16, k // 2 // 16 * 16, (k - 1) // 16 * 16}):
        narrow = lu_solve(f.factors, f.p, np.ascontiguousarray(b[:, c:c + 16]), trans=trans)
        np.testing.assert_array_equal(wide[:, c:c + 16], narrow)
