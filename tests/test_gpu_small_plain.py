"""The two-launch plain solve (no report asked for; n <= 192, k <= 8) against the launches that a
report takes: the same bits, the same answer on irregular matrices, at the sizes where the cluster
grows (32, 64, 128 rows) and the route ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 127, 129, 191, 192, 193])
@pytest.mark.parametrize("k", [1, 3, 8, 9])
def test_same_bits_with_and_without_a_report(n, k):
    import rustymath_b200 as rb
    rng = np.random.default_rng(n * 10 + k)
    a, b = rng.standard_normal((n, n)) + 2 * np.eye(n), rng.standard_normal((n, k))
    plain = rb.solve(a, b)
    reps = []
    with_report = rb.solve(a, b, report=reps)
    assert len(reps) == 1 and reps[0].regular == 1
    np.testing.assert_array_equal(plain, with_report)


@pytest.mark.parametrize("n", [1, 5, 33, 150])
def test_irregular_matrices_are_refused(n):
    import rustymath_b200 as rb
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a[:, n // 2] = 0.0
    with pytest.raises(rb.linalg.NotRegular):
        rb.solve(a, np.ones(n))
    a = rng.standard_normal((n, n))
    a[n // 2, n // 2] = np.nan  # a NaN pivot counts as regular, as in rustymath
    assert np.isnan(rb.solve(a, np.ones(n))).any()
