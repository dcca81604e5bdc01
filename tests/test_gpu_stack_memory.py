"""A stack solve's scratch: the pool keeps at most 1 GiB of it, larger stacks (2048 systems of n = 256) go in
several launches over the same scratch, with the same bits as their parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["plain", "mixed"])
def test_a_large_stack_keeps_at_most_a_gibibyte(method):
    import torch

    from rustymath_b200 import linalg
    count, n = 4600, 256  # 2.4 GB of factors
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(count, n, n, generator=g, device="cuda", dtype=torch.float64)
    a.diagonal(dim1=1, dim2=2).add_(float(n))
    b = torch.randn(count, n, 1, generator=g, device="cuda", dtype=torch.float64)
    x = torch.empty_like(b)
    for first in range(0, count, 2000):
        x[first:first + 2000] = linalg.solve(a[first:first + 2000], b[first:first + 2000], method=method)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    whole = linalg.solve(a, b, method=method)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 1 << 28  # up to 2000 systems' scratch was kept before
    assert torch.equal(whole, x)


@pytest.mark.parametrize("method", ["plain", "mixed"])
def test_uneven_systems_in_several_launches(method):
    """Systems of both kernels after a launch's end, and the report over all of them."""
    import ctypes

    import torch

    from rustymath_b200 import _lib, batched, linalg
    rng = np.random.default_rng(4)
    ns = np.concatenate([np.full(2100, 256), rng.integers(1, 70, 300), [0, 256, 64, 65]]).astype(np.int64)
    rng.shuffle(ns)
    ks = 1 + ns % 3
    plan = batched.BatchPlan(ns, ks, method=method)
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(plan.a_size, generator=g, device="cuda", dtype=torch.float64)
    b = torch.randn(plan.b_size, generator=g, device="cuda", dtype=torch.float64)
    for off, n in zip(plan.a_off, ns):
        a[off:off + n * n].view(n, n).diagonal().add_(float(n))
    expect, x = torch.zeros_like(b), torch.zeros_like(b)
    plan.execute(a, b, expect)
    _, _, _, rep = plan.results()
    opts, got = linalg._options(method), _lib.BatchReport()
    st = _lib.load().rm_dsolve_batched(len(ns), ns.ctypes.data, ks.ctypes.data, plan.a_off.ctypes.data,
                                       plan.b_off.ctypes.data, plan.b_off.ctypes.data, a.data_ptr(), b.data_ptr(),
                                       x.data_ptr(), ctypes.byref(opts), ctypes.byref(got), None)
    assert st == _lib.RM_OK
    assert torch.equal(x, expect)
    assert got.max_backward_error == rep.max_backward_error and got.max_iterations == rep.max_iterations
    assert got.fell_back == rep.fell_back and got.not_regular == rep.not_regular
