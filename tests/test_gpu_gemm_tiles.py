"""Products at the sizes where rm_dgemm changes its tile (by the tiles per SM of a 148-SM GPU), with
remainders in every direction and each transpose: against the oracle's product bit for bit, as both
fold one fma per k in order."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(33, 31, 17), (511, 530, 33), (641, 650, 18), (700, 1100, 20), (1025, 1030, 16),
                                   (1250, 1130, 9), (1540, 1530, 40)])
def test_tiles(m, n, k, ta, tb):
    import rustymath_b200 as rb
    rng = np.random.default_rng(m + ta + 2 * tb)
    a = rng.uniform(-1, 1, (k, m) if ta else (m, k))
    b = rng.uniform(-1, 1, (n, k) if tb else (k, n))
    c = np.zeros((m, n))
    st = rb._lib.load().rm_dgemm_host(ta, tb, m, n, k, 1.0, a.ctypes.data, a.shape[1], b.ctypes.data, b.shape[1], 0.0,
                                      c.ctypes.data, n)
    assert st == rb._lib.RM_OK
    want = O.dgemm(np.ascontiguousarray(a.T) if ta else a, np.ascontiguousarray(b.T) if tb else b)
    np.testing.assert_array_equal(c, want)
