"""The split-precision product's two tile shapes and its launches of two orders: 128 x 256 tiles
(products of more than one wave) against 128 x 128 tiles, which a block of their rows takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(a, b, slices):
    import torch
    import rustymath_b200 as rb
    return rb.linalg.matmul_ozaki(torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda"),
                                  slices=slices).cpu().numpy()


# n = 1400 leaves half a 256-wide tile, whose box reaches into the next plane; odd slice counts
# end with a launch of one order; k = 129 and 131 leave one and three columns of a 128 tile
@pytest.mark.parametrize("m,k,n,slices", [(1700, 200, 1400, 8), (1700, 129, 1400, 5), (1665, 128, 1537, 3),
                                          (1700, 131, 1400, 2), (1700, 64, 1400, 1)])
def test_wide_tiles_are_the_narrow_ones(m, k, n, slices):
    rng = np.random.default_rng(m + k + slices)
    a = rng.uniform(-1, 1, (m, k)) * 10.0 ** rng.uniform(-3, 3, (m, 1))
    b = rng.uniform(-1, 1, (k, n)) * 10.0 ** rng.uniform(-3, 3, (1, n))
    got = run(a, b, slices)
    # integer sums are exact and each element's float64 additions come in one order: equal bits
    assert (got[:200] == run(a[:200], b, slices)).all()
    assert (got[-130:, -300:] == run(a[-130:], b[:, -300:], slices)).all()
    bound = (3 * k * 2.0 ** (-7 * slices) * (2 * np.abs(a).max(1, keepdims=True)) * (2 * np.abs(b).max(0, keepdims=True))
             + (k + 16) * 2.0 ** -53 * (np.abs(a) @ np.abs(b)))
    assert (np.abs(got - a @ b) <= bound).all()


@pytest.mark.parametrize("m,n", [(130, 140), (1700, 1400)])
def test_scales_out_of_the_normal_range(m, n):
    rng = np.random.default_rng(m)
    k = 96
    a, b = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))
    base = run(a, b, 8)
    assert (run(a * 2.0 ** 900, b * 2.0 ** 100, 8) == base * 2.0 ** 1000).all()
    # subnormal results: each of the eight terms rounds once, the additions are exact
    low = run(a * 2.0 ** -600, b * 2.0 ** -450, 8)
    assert (np.abs(low - np.ldexp(base, -1050)) <= 8 * 2.0 ** -1074).all()
    # an infinity or a NaN stays in its row and column
    a[3, 5], b[7, 11] = np.inf, np.nan
    got = run(a, b, 8)
    keep = np.ones((m, n), bool)
    keep[3], keep[:, 11] = False, False
    assert (got[keep] == base[keep]).all()
