"""The calls that programs built on rustymath_b200 spend their time in, as timed cases.

Eight kinds of call, each through the public Python entry point that a program uses. The listed
cases are one or two sizes of each kind, from the smallest call to the largest system; `draw`
gives others of the same ranges, odd sizes among them.

  solve     linalg.solve of one system, by either method
  stack     linalg.solve of a stack of equal systems
  batch     BatchPlan.execute on systems of uneven size
  adjoint   autograd.solve, forward and backward
  lu        linalg.lu, then what its factors give: solutions, the inverse, the determinant
  cholesky  linalg.cholesky
  matmul    linalg.matmul
  ozaki     linalg.matmul_ozaki
"""
import math

import numpy as np
import torch

from rustymath_b200 import autograd, batched, linalg

DEVICE = "cuda"
F64 = torch.float64


def listed():
    return [
        # a control loop or a small fit: one tiny system per call, bound by the call itself
        {"name": "solve_8", "kind": "solve", "n": 8, "k": 1, "method": "plain"},
        # the size rustymath's own users solve on a CPU
        {"name": "solve_512", "kind": "solve", "n": 512, "k": 1, "method": "plain"},
        # a discretised operator of no round size with a few right-hand sides
        {"name": "solve_2047", "kind": "solve", "n": 2047, "k": 5, "method": "plain"},
        # one large dense system, by the drop-in method and by the mixed-precision one
        {"name": "solve_8192", "kind": "solve", "n": 8192, "k": 16, "method": "plain"},
        {"name": "solve_8192_mixed", "kind": "solve", "n": 8192, "k": 16, "method": "mixed"},
        # a stack of equal systems, as NumPy-style code writes it
        {"name": "stack_1000x100", "kind": "stack", "count": 1000, "n": 100, "k": 1},
        # thousands of small systems of uneven size: local fits, element matrices
        {"name": "batch_20000", "kind": "batch", "count": 20000, "n_max": 256, "k_max": 4, "method": "mixed"},
        # a differentiable solve in a training step
        {"name": "adjoint_4096x64", "kind": "adjoint", "count": 4096, "n": 64, "k": 2},
        # a factorization kept and reused
        {"name": "lu_1030", "kind": "lu", "n": 1030, "k": 3},
        # a covariance matrix factored for sampling or a likelihood
        {"name": "cholesky_2048", "kind": "cholesky", "n": 2048},
        # float64 products: a small one, and a large one by the split-precision product
        {"name": "matmul_512", "kind": "matmul", "m": 512, "k": 512, "n": 512},
        {"name": "ozaki_8192", "kind": "ozaki", "m": 8192, "k": 8192, "n": 8192},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "stack", "batch", "adjoint", "lu", "cholesky", "matmul", "ozaki"])
    if kind == "solve":
        method = rng.choice(["plain", "plain", "mixed"])
        return {"kind": kind, "n": _log_int(rng, 8 if method == "plain" else 256, 8191), "k": rng.randint(1, 16),
                "method": method}
    if kind == "stack":
        n = _log_int(rng, 8, 256)
        return {"kind": kind, "count": _log_int(rng, 16, max(32, min(4000, 40000 // n))), "n": n, "k": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 200, 20000), "n_max": _log_int(rng, 16, 256),
                "k_max": rng.randint(1, 4), "method": rng.choice(["mixed", "plain"])}
    if kind == "adjoint":
        n = _log_int(rng, 8, 128)
        return {"kind": kind, "count": _log_int(rng, 32, min(4096, 262144 // n)), "n": n, "k": rng.randint(1, 4)}
    if kind == "lu":
        return {"kind": kind, "n": _log_int(rng, 16, 3000), "k": rng.randint(1, 16)}
    if kind == "cholesky":
        return {"kind": kind, "n": _log_int(rng, 16, 5000)}
    hi = 4096 if kind == "matmul" else 8192
    lo = 64 if kind == "matmul" else 512
    return {"kind": kind, "m": _log_int(rng, lo, hi), "k": _log_int(rng, lo, hi), "n": _log_int(rng, lo, hi)}


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEVICE, dtype=F64)


def _general(g, *shape):
    """Well-conditioned general matrices: N(0,1) entries plus 2 sqrt(n) on the diagonal, the rows
    then in random order, so that pivots come from anywhere below the diagonal."""
    n = shape[-1]
    a = _randn(g, *shape)
    a.diagonal(dim1=-2, dim2=-1).add_(2.0 * math.sqrt(n))
    order = torch.randperm(n, generator=g, device=DEVICE)
    return a[..., order, :].contiguous()


def _batch_shapes(case):
    rng = np.random.default_rng(1)
    ns = rng.integers(8, case["n_max"] + 1, case["count"]).astype(np.int64)
    ks = rng.integers(1, case["k_max"] + 1, case["count"]).astype(np.int64)
    return ns, ks


def _batch_inputs(case, seed):
    """Packed diagonally dominant systems, N(0,1) + n I; their sizes belong to the case."""
    ns, ks = _batch_shapes(case)
    g = _generator(seed)
    a = _randn(g, int((ns * ns).sum()))
    b = _randn(g, int((ns * ks).sum()))
    start = np.concatenate([[0], np.cumsum(ns * ns)[:-1]])
    first = np.concatenate([[0], np.cumsum(ns)[:-1]])
    step = np.arange(int(ns.sum())) - np.repeat(first, ns)
    where = torch.as_tensor(np.repeat(start, ns) + step * np.repeat(ns + 1, ns), device=DEVICE)
    a[where] += torch.as_tensor(np.repeat(ns, ns).astype(np.float64), device=DEVICE)
    return ns, ks, a, b


def _wide_range(g, m, n, dim):
    """U(-1,1) entries, rows (dim 0) or columns (dim 1) scaled by 10^U(-3,3)."""
    x = torch.rand(m, n, generator=g, device=DEVICE, dtype=F64).mul_(2).sub_(1)
    size = (m, 1) if dim == 0 else (1, n)
    return x.mul_(10.0 ** (torch.rand(*size, generator=g, device=DEVICE, dtype=F64) * 6 - 3))


def _inputs(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("solve", "lu"):
        return _general(g, case["n"], case["n"]), _randn(g, case["n"], case["k"])
    if kind == "stack":
        shape = (case["count"], case["n"])
        return _general(g, *shape, case["n"]), _randn(g, *shape, case["k"])
    if kind == "adjoint":
        shape = (case["count"], case["n"])
        return _general(g, *shape, case["n"]), _randn(g, *shape, case["k"]), _randn(g, *shape, case["k"])
    if kind == "cholesky":
        x = _randn(g, case["n"], case["n"])
        a = (x @ x.T).div_(case["n"])
        a.diagonal().add_(1.0)
        return (a,)
    if kind == "matmul":
        a = torch.rand(case["m"], case["k"], generator=g, device=DEVICE, dtype=F64).mul_(2).sub_(1)
        b = torch.rand(case["k"], case["n"], generator=g, device=DEVICE, dtype=F64).mul_(2).sub_(1)
        return a, b
    return _wide_range(g, case["m"], case["k"], 0), _wide_range(g, case["k"], case["n"], 1)


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "batch":
        ns, ks, a, b = _batch_inputs(case, seed)
        state["plan"] = batched.BatchPlan(ns, ks, method=case["method"])
        state["args"] = (a, b, torch.empty_like(b))
    else:
        state["args"] = _inputs(case, seed)
    if case["kind"] == "adjoint":
        for t in state["args"][:2]:
            t.requires_grad_(True)
    return state


def run(state):
    case, args = state["case"], state["args"]
    kind = case["kind"]
    if kind == "solve":
        return linalg.solve(*args, method=case["method"])
    if kind == "stack":
        return linalg.solve(*args)
    if kind == "batch":
        state["plan"].execute(*args)
        return args[2]
    if kind == "adjoint":
        a, b, w = args
        x = autograd.solve(a, b)
        ga, gb = torch.autograd.grad((w * x).sum(), (a, b))
        return {"x": x.detach(), "ga": ga, "gb": gb}
    if kind == "lu":
        a, b = args
        f = linalg.lu(a)
        sign, log = f.log_determinant()
        return {"factors": f.factors, "p": f.p, "x": f.solve(b), "inverse": f.inverse(), "sign": sign, "log": log}
    if kind == "cholesky":
        return linalg.cholesky(*args)
    if kind == "matmul":
        return linalg.matmul(*args)
    return linalg.matmul_ozaki(*args)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "stack"):
        n, k, c = case["n"], case["k"], case.get("count", 1)
        return {"bytes": 8 * c * (n * n + 2 * n * k), "flops": c * (2 * n ** 3 / 3 + 2 * n * n * k)}
    if kind == "batch":
        # the mean over n ~ U{8..n_max}, k ~ U{1..k_max}
        n = np.arange(8, case["n_max"] + 1, dtype=np.float64)
        k, c = (1 + case["k_max"]) / 2, case["count"]
        return {"bytes": float(8 * c * np.mean(n * n + 2 * n * k)), "flops": float(c * np.mean(2 * n ** 3 / 3 + 2 * n * n * k))}
    if kind == "adjoint":
        # forward: a, b -> x; backward: the gradient of x -> those of a and b
        n, k, c = case["n"], case["k"], case["count"]
        return {"bytes": 8 * c * (3 * n * n + 5 * n * k), "flops": c * (2 * n ** 3 / 3 + 6 * n * n * k)}
    if kind == "lu":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * (3 * n * n + 2 * n * k + n), "flops": 2 * n ** 3 + 2 * n * n * k}
    if kind == "cholesky":
        n = case["n"]
        return {"bytes": 8 * (n * n / 2 + n * n), "flops": n ** 3 / 3}
    m, k, n = case["m"], case["k"], case["n"]
    return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * k * n}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ns, ks, a, b = _batch_inputs(case, seed)
        out = torch.empty_like(b)
        a_off = np.concatenate([[0], np.cumsum(ns * ns)[:-1]])
        b_off = np.concatenate([[0], np.cumsum(ns * ks)[:-1]])
        for n in np.unique(ns):
            for k in np.unique(ks[ns == n]):
                mine = np.flatnonzero((ns == n) & (ks == k))
                n, k = int(n), int(k)
                ia = torch.as_tensor(a_off[mine][:, None] + np.arange(n * n), device=DEVICE)
                ib = torch.as_tensor(b_off[mine][:, None] + np.arange(n * k), device=DEVICE)
                x = torch.linalg.solve(a[ia].view(-1, n, n), b[ib].view(-1, n, k))
                out[ib] = x.reshape(len(mine), n * k)
        return out
    args = _inputs(case, seed)
    if kind in ("solve", "stack"):
        return torch.linalg.solve(*args)
    if kind == "adjoint":
        a, b, w = args
        x = torch.linalg.solve(a, b)
        gb = torch.linalg.solve(a.mT, w)
        return {"x": x, "ga": -gb @ x.mT, "gb": gb}
    if kind == "lu":
        a, b = args
        f, pivots = torch.linalg.lu_factor(a)
        p = np.arange(case["n"])
        for i, j in enumerate(pivots.cpu().numpy() - 1):
            p[[i, j]] = p[[j, i]]
        sign, log = torch.linalg.slogdet(a)
        return {"factors": f.mT.contiguous(), "p": torch.as_tensor(p, device=DEVICE), "x": torch.linalg.solve(a, b),
                "inverse": torch.linalg.inv(a), "sign": sign, "log": log}
    if kind == "cholesky":
        return torch.linalg.cholesky(*args)
    return args[0] @ args[1]
