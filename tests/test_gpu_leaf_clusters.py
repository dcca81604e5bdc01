"""The float64 LU where the device places smaller clusters than the 16 CTAs of the tallest leaves: the same
factors from clusters of 8, 4 and 2 and from single CTAs, the leaves too tall for them by the other panel.
Each item takes the same fmas in the same order either way; pivots equal, factors within 64 n eps of their
scale, as against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [513, 1100, 2100, 4200])
def test_smaller_clusters_give_the_same_factors(n, ctas):
    from rustymath_b200 import _lib, linalg
    lib = _lib.load()
    a = np.random.default_rng(n).standard_normal((n, n))
    f, p = linalg.lu(a)
    assert lib.rm_test_limit_leaf_ctas(ctas) == _lib.RM_OK
    try:
        f2, p2 = linalg.lu(a)
    finally:
        assert lib.rm_test_limit_leaf_ctas(0) == _lib.RM_OK
    assert np.array_equal(p, p2)
    assert np.abs(f - f2).max() <= 64 * n * np.finfo(np.float64).eps * max(1.0, np.abs(f).max())


def test_the_limit_is_a_power_of_two():
    from rustymath_b200 import _lib
    lib = _lib.load()
    for bad in (-1, 3, 12, 32):
        assert lib.rm_test_limit_leaf_ctas(bad) == _lib.RM_BAD_ARG
