"""A leaf of the blocked float64 LU whose waits for the other CTAs' posts run out: the call reports a
timeout, the launches queued behind the leaf stay within the matrix, and the next calls are right.
RM_INJECT_LEAF_TIMEOUT holds back one column's posts in every CTA of a leaf, RM_INJECT_LEAF_CTA_TIMEOUT
in its last CTA only, so that the others first go on; the waits are 1 ms and nothing faults."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# n = 600: leaves of 4 CTAs, no look-ahead; 1500: 8 and look-ahead; 2500: 16 and a persistent update.
# after: the leaf that fails; 5 lies in the second block, where a first list has been used.
@pytest.mark.parametrize("kind", ["RM_INJECT_LEAF_TIMEOUT", "RM_INJECT_LEAF_CTA_TIMEOUT"])
@pytest.mark.parametrize("n,after", [(600, 0), (600, 2), (1500, 3), (1500, 5), (2500, 0), (2500, 9)])
def test_a_leaf_that_gives_up_is_reported(kind, n, after):
    import rustymath_b200 as rb
    from rustymath_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(n + after)
    a = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    b = rng.standard_normal((n, 2))
    assert lib.rm_test_inject_failure(getattr(_lib, kind), after, 1) == _lib.RM_OK
    t0 = time.perf_counter()
    try:
        with pytest.raises(_lib.RmError) as e:
            rb.solve(a, b)
        assert e.value.status == _lib.RM_TIMEOUT
        assert time.perf_counter() - t0 < 5.0
    finally:
        lib.rm_test_inject_failure(getattr(_lib, kind), 0, 0)
    x = rb.solve(a, b)
    assert np.abs(a @ x - b).max() <= 1e-10 * np.abs(b).max()
