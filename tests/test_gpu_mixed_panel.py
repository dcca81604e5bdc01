"""The rank-16 updates inside the mixed solve's float32 panels keep their sums apart from C.

Row and column r of A couple to the first 16 unknowns by 1/2 and 2, so that column r's pivot becomes C - 16
by 16 products of 1, with C = 2^24 + 4: float32 numbers there lie 2 apart, so a sum that starts from C rounds
every product away (an error of 2^-20 in x_r); with four chains, one of them from C, four products are lost
(2^-22). The tolerance is 1, so that x is the float32 solve as it is. Bound: 2^-21, which leaves the solve's
own error 2^-22 (the inverse 1 / u and a product of three TF32 passes, whose factors are exact in two TF32
parts each)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the first row after a leaf, odd ones, a panel's last, and rows of a panel that is 256 rows tall
@pytest.mark.parametrize("n,r", [(32, 16), (64, 37), (100, 99), (128, 127), (300, 45), (300, 127)])
def test_the_products_do_not_all_round_at_c(n, r):
    import rustymath_b200 as rb
    from rustymath_b200 import _lib
    a = np.eye(n)
    a[r, :16] = 0.5
    a[:16, r] = 2.0
    a[r, r] = 2.0 ** 24 + 4
    b = np.zeros((n, 1))
    b[r] = 2.0 ** 24 - 12  # x_r = 1, the first 16 unknowns -2
    b[:16] = 0.0
    x = np.zeros((n, 1))
    opts = rb.linalg._options("mixed", tolerance=1.0)
    rep = _lib.SolveReport()
    st = _lib.load().rm_dsolve_host(n, a.ctypes.data, b.ctypes.data, 1, x.ctypes.data, ctypes.byref(opts),
                                    ctypes.byref(rep))
    assert st == _lib.RM_OK and rep.method_used == _lib.RM_METHOD_F32_IR and rep.iterations == 0
    assert abs(x[r, 0] - 1.0) <= 2.0 ** -21
