"""The reciprocals that multiply the pivot columns, to the bit. rustymath's `divide` multiplies by the
pivot's correctly rounded reciprocal, or divides where the pivot is subnormal. In the LU of a lower
triangular matrix whose diagonal is each column's largest item nothing is subtracted but zeros, so the
factors are that division alone. The float32 factors of the batched solver show through its solutions."""
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


def float32_solutions(a, b, adjoint=False):
    """The batched solver's float32 solutions as they are (a tolerance of 1 takes no refinement step), of
    a or (adjoint) of its transpose, with the factors of a."""
    import torch

    from rustymath_b200 import batched
    count, n = a.shape[:2]
    plan = batched.BatchPlan([n] * count, [1] * count, method="mixed", tolerance=1.0)
    ta, tb = torch.tensor(a, device="cuda").flatten(), torch.tensor(b, device="cuda").flatten()
    x = torch.empty_like(tb)
    plan.execute(ta, tb, x)
    _, iters, flags, _ = plan.results()
    assert not np.any(iters) and not np.any(flags)
    if adjoint:
        plan.adjoint(ta, x, tb, x)
    return x.cpu().numpy().reshape(count, n)


# the 64-thread build (panels of 16 columns) and the 256-thread one (16 and 32)
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("n", [5, 32, 64, 70, 200])
def test_float32_quotients_are_correctly_rounded(n, adjoint):
    """Diagonal systems: x_i = b_i / d_i, of ordinary and subnormal magnitude, and zero."""
    rng = np.random.default_rng(n)
    count = 20000 // n
    d = np.stack([pivots(n, rng, 23, -126, 127, 2.0 ** -149) for _ in range(count)])
    b = rng.uniform(1, 2, d.shape) * np.exp2(np.floor(np.log2(np.abs(d)) / 2))
    b[:, 1::4] = rng.uniform(-2, 2, b[:, 1::4].shape)
    b[: count // 2, 2::5] = 0.0
    small = rng.random(d.shape) < 0.3
    b = np.where(small, d * np.exp2(rng.uniform(-151, -124, d.shape)), b).astype(np.float32)
    with np.errstate(all="ignore"):
        b[~np.isfinite(b / d.astype(np.float32))] = 0.0  # an infinity would leave no residual to accept x by
        expect = b / d.astype(np.float32)
    x = float32_solutions(np.einsum("ci,ij->cij", d, np.eye(n)), b.astype(np.float64), adjoint)
    np.testing.assert_array_equal(x, expect.astype(np.float64))


# swap: the rows reversed, so that the route with a pivot search factors
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("n", [5, 32, 64, 70, 200])
def test_float32_multipliers_are_the_division_of_the_reference(n, swap):
    """Identities but for the first column (p, a_1, a_2, ...): with b = e_0 the unknowns after the first are
    -a_i times p's reciprocal, to the bit."""
    rng = np.random.default_rng(100 + n)
    p = pivots(400, rng, 23, -126, 127, 2.0 ** -126).astype(np.float32)
    # column diagonal dominance, for the route without a search
    col = (rng.uniform(-0.9, 0.9, (p.size, n)) / n * np.abs(p)[:, None]).astype(np.float32)
    a = np.broadcast_to(np.eye(n), (p.size, n, n)).copy()
    a[:, :, 0] = col
    a[:, 0, 0] = p
    b = np.zeros((p.size, n))
    b[:, 0] = 1.0
    reciprocal = np.float32(1) / p
    expect = -(col * reciprocal[:, None])
    expect[:, 0] = reciprocal
    if swap:
        a, b = a[:, ::-1].copy(), b[:, ::-1].copy()
    np.testing.assert_array_equal(float32_solutions(a, b), expect.astype(np.float64))
