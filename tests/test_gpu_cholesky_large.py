"""The blocked Cholesky factorization where its parts change size: the trailing update by 64 x 64 and
by 128 x 128 tiles of the lower triangle, last blocks of one, a few and all 64 columns; and a pivot
that fails in a later block. Bounds as test_gpu_cholesky.py: ||L L^T - A|| below 4 eps n of ||A||."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("n", [129, 192, 1985, 2240, 2305])
def test_blocks(n):
    import torch

    from rustymath_b200 import linalg
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    a = x @ x.T / n + torch.eye(n, device="cuda", dtype=torch.float64)
    # only the lower triangle is read
    low = linalg.cholesky(torch.tril(a) + torch.triu(torch.full_like(a, 7.0), 1))
    assert torch.equal(torch.triu(low, 1), torch.zeros_like(low))
    r = (low @ low.T - a).abs().sum(1).max() / a.abs().sum(1).max()
    assert r.item() < 4 * EPS * n


@pytest.mark.parametrize("at", [64, 79, 150, 299])
def test_a_later_pivot_fails(at):
    import torch

    from rustymath_b200 import linalg
    n = 300
    a = torch.eye(n, device="cuda", dtype=torch.float64) * 4
    a[at, 0] = 4.0  # pivot at: 4 - (4 / 2)^2 = 0, not > 0
    assert torch.isnan(linalg.cholesky(a)).all()
    a[at, 0] = 3.0
    assert torch.isfinite(linalg.cholesky(a)).all()
