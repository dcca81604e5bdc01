"""The gradient of A in the batched adjoint, -(dL/db) x^T, to the bit from the gb and x it is formed from, at
the sizes where its split over the threads changes, in plans that hold empty systems as well."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["mixed", "plain"])
def test_outer_products_of_every_width(method):
    import torch

    from rustymath_b200 import batched
    ns = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 0, 63, 64, 65, 96, 97, 128, 129, 160, 161, 224, 225, 256]
    ks = [2, 1, 8, 3, 4, 2, 1, 5, 2, 1, 0, 2, 0, 1, 2, 3, 1, 0, 2, 1, 4, 2, 1, 8, 3]
    rng = np.random.default_rng(0)
    As = [rng.standard_normal((n, n)) + n * np.eye(n) for n in ns]
    Bs = [rng.standard_normal((n, k)) for n, k in zip(ns, ks)]
    plan = batched.BatchPlan(ns, ks, method=method)
    a, b = plan.pack(As, Bs, device="cuda")
    _, g = plan.pack(As, [rng.standard_normal(m.shape) for m in Bs], device="cuda")
    x, gb, ga = torch.zeros_like(b), torch.zeros_like(b), torch.full_like(a, 7.0)
    plan.execute(a, b, x)
    plan.adjoint(a, x, g, gb, ga)
    plan.adjoint_results()
    ao = bo = 0
    ga, gb, x = ga.cpu().numpy(), gb.cpu().numpy(), x.cpu().numpy()
    for n, k in zip(ns, ks):
        u, v = gb[bo:bo + n * k].reshape(n, k), x[bo:bo + n * k].reshape(n, k)
        got = ga[ao:ao + n * n].reshape(n, n)
        if k <= 1:  # one product, rounded once
            np.testing.assert_array_equal(got, -(u @ v.T) if k else np.zeros((n, n)))
        else:  # k fused steps: k roundings of at most the sum of magnitudes
            assert np.all(np.abs(got + u @ v.T) <= 2 * k * 2.0 ** -53 * (np.abs(u) @ np.abs(v).T))
        ao, bo = ao + n * n, bo + n * k
