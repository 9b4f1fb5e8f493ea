"""The work that this library is timed on.

Every case is one call sequence of a user's program through the public entry
points of ``blockedbunchkaufmanldlt_b200``:

``factor_solve``  a device matrix is copied into the buffer that is factored
                  in place, factored, and solved for ``nrhs`` right-hand sides.
``factor``        the factorization alone, in the reference's summation order.
``mixed``         factor and solve with a BF16x3 trailing update and FP64 FGMRES
                  refinement against the original matrix.
``solve``         new right-hand sides against factors kept from before.
``batched``       many small KKT systems in one planned call.
``full``          the class that mirrors the reference's: host matrix in,
                  factors, pivots and the reconstructed matrix out.

Matrices: ``random`` (uniform [-1, 1] entries, N(0, 0.01) added on the
diagonal), ``kkt`` ([[H, B^T], [B, 0]], H = G G^T / h + 0.01 I with h a given
share of n), ``spectral`` (Q diag(lambda) Q^T, |lambda| log-uniform in
[1e-2, 1e2], half of them negative).
"""
import math
import random

import numpy as np
import torch

import blockedbunchkaufmanldlt_b200 as bbk

KKT_SHARE = 0.8    # order of H in a single KKT matrix, as a share of n
BATCH_SHARE = 0.75  # the same in a batch


def listed():
    return [
        # one small dense system inside a larger program: launches and latency
        {"name": "small_n320", "kind": "factor_solve", "matrix": "random", "n": 320, "block": 32, "nrhs": 1,
         "mode": "fp64"},
        # an interior-point step of odd order, a few right-hand sides
        {"name": "kkt_n1999", "kind": "factor_solve", "matrix": "kkt", "n": 1999, "block": 64, "nrhs": 3,
         "mode": "fp64"},
        # results that have to be the reference's bit for bit
        {"name": "ordered_n2000", "kind": "factor", "matrix": "random", "n": 2000, "block": 64,
         "mode": "fp64_ordered"},
        # a matrix with a wide spectrum and a block of right-hand sides
        {"name": "spectral_n4001", "kind": "factor_solve", "matrix": "spectral", "n": 4001, "block": 128, "nrhs": 16,
         "mode": "fp64"},
        # the ordinary large system: saddle point, one right-hand side
        {"name": "kkt_n10000", "kind": "factor_solve", "matrix": "kkt", "n": 10000, "block": 128, "nrhs": 1,
         "mode": "fp64"},
        # the largest dense indefinite system of the benchmark
        {"name": "random_n40000", "kind": "factor_solve", "matrix": "random", "n": 40000, "block": 256, "nrhs": 4,
         "mode": "fp64"},
        # low-precision factors refined to FP64 accuracy
        {"name": "mixed_n16000", "kind": "mixed", "matrix": "random", "n": 16000, "block": 256, "nrhs": 4,
         "mode": "bf16x3"},
        # many small KKT systems at once, the benchmark's range of orders
        {"name": "batched_4096", "kind": "batched", "count": 4096, "lo": 16, "hi": 512, "mode": "fp64"},
        # a batch of the smallest orders: under one system per multiprocessor slot
        {"name": "batched_small", "kind": "batched", "count": 300, "lo": 8, "hi": 96, "mode": "fp64"},
        # time stepping: one new right-hand side against kept factors
        {"name": "solve_n10000", "kind": "solve", "matrix": "random", "n": 10000, "block": 128, "nrhs": 1},
        # many right-hand sides against kept factors
        {"name": "solve_n5000_r64", "kind": "solve", "matrix": "random", "n": 5000, "block": 128, "nrhs": 64},
        # a program written for the reference's class, full mode
        {"name": "full_n1500", "kind": "full", "matrix": "random", "n": 1500, "block": 64, "mode": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["factor_solve", "factor_solve", "factor_solve", "mixed", "solve", "batched", "full"])
    if kind == "batched":
        lo = rng.randint(4, 64)
        return {"kind": kind, "count": _log_int(rng, 64, 4096), "lo": lo, "hi": lo + rng.randint(16, 448),
                "mode": "fp64"}
    if kind == "full":
        return {"kind": kind, "matrix": rng.choice(["random", "kkt"]), "n": _log_int(rng, 200, 2500),
                "block": rng.choice([32, 48, 64, 128]), "mode": rng.choice(["fp64", "fp64", "fp64_ordered"])}
    if kind == "solve":
        return {"kind": kind, "matrix": "random", "n": _log_int(rng, 300, 16000), "block": 128,
                "nrhs": _log_int(rng, 1, 96)}
    if kind == "mixed":
        # the BF16 updates take rows that start on 16 bytes: an even order
        return {"kind": kind, "matrix": "random", "n": 2 * _log_int(rng, 2000, 10000),
                "block": rng.choice([128, 192, 256]), "nrhs": rng.randint(1, 8), "mode": "bf16x3"}
    mode = rng.choice(["fp64", "fp64", "fp64", "fp64_ordered"])
    n = _log_int(rng, 100, 3000 if mode == "fp64_ordered" else 30000)
    matrix = rng.choice(["random", "kkt", "spectral"] if n <= 6000 else ["random", "kkt"])
    block = rng.choice([32, 48, 64] if n < 1000 else [64, 100, 128] if n < 6000 else [128, 192, 256])
    if mode == "fp64_ordered":
        return {"kind": "factor", "matrix": matrix, "n": n, "block": block, "mode": mode}
    return {"kind": kind, "matrix": matrix, "n": n, "block": block, "nrhs": _log_int(rng, 1, 16), "mode": mode}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _mirror(a):
    """The upper triangle of ``a`` copied into its lower one, in place."""
    n, step = a.shape[0], 2048
    for k in range(0, n, step):
        e = min(n, k + step)
        if e < n:
            a[e:, k:e] = a[k:e, e:].T
        d = torch.triu(a[k:e, k:e])
        a[k:e, k:e] = d + torch.triu(d, 1).T
    return a


def _matrix(case, g):
    n, dev = case["n"], "cuda"
    if case["matrix"] == "random":
        a = torch.empty(n, n, dtype=torch.float64, device=dev).uniform_(-1.0, 1.0, generator=g)
        a.diagonal().add_(torch.randn(n, generator=g, dtype=torch.float64, device=dev), alpha=0.1)
        return _mirror(a)
    if case["matrix"] == "kkt":
        h = int(round(KKT_SHARE * n))
        gm = torch.randn(h, h, generator=g, dtype=torch.float64, device=dev)
        a = torch.zeros(n, n, dtype=torch.float64, device=dev)
        a[:h, :h] = gm @ gm.T / h
        a[:h, :h].diagonal().add_(1e-2)
        a[:h, h:] = torch.randn(h, n - h, generator=g, dtype=torch.float64, device=dev)
        return _mirror(a)
    q, _ = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=torch.float64, device=dev))
    lam = torch.exp(torch.empty(n, dtype=torch.float64, device=dev).uniform_(math.log(1e-2), math.log(1e2),
                                                                             generator=g))
    lam[torch.randperm(n, generator=g, device=dev)[: n // 2]] *= -1.0
    return _mirror((q * lam) @ q.T)


def _system(case, seed):
    g = _generator(seed)
    a = _matrix(case, g)
    if case["kind"] == "factor":
        return a, None
    return a, torch.randn(case["nrhs"], case["n"], generator=g, dtype=torch.float64, device="cuda")


def _orders(case):
    """The batch's orders: a plan's, so the same whatever the data."""
    return np.random.default_rng([case["count"], case["lo"], case["hi"]]).integers(
        case["lo"], case["hi"] + 1, size=case["count"])


def _batch(case, seed):
    """Packed KKT matrices and right-hand sides.  The products G G^T of
    similar orders are formed together, padded with zeros."""
    sizes = _orders(case)
    g = _generator(seed)
    starts = np.concatenate([[0], np.cumsum(sizes.astype(np.int64) ** 2)])
    a = torch.zeros(int(starts[-1]), dtype=torch.float64, device="cuda")
    order = np.argsort(sizes, kind="stable")
    for at in range(0, len(order), 256):
        part = order[at:at + 256]
        hs = [max(1, int(round(BATCH_SHARE * sizes[k]))) for k in part]
        top = max(hs)
        gm = torch.randn(len(part), top, top, generator=g, dtype=torch.float64, device="cuda")
        bm = torch.randn(len(part), top, int(sizes[part[-1]]), generator=g, dtype=torch.float64, device="cuda")
        ht = torch.tensor(hs, device="cuda")
        keep = (torch.arange(top, device="cuda")[None, :] < ht[:, None]).to(torch.float64)
        gm *= keep[:, None, :]
        hm = torch.bmm(gm, gm.transpose(1, 2)) / ht[:, None, None]
        hm.diagonal(dim1=1, dim2=2).add_(1e-2)
        for i, k in enumerate(part):
            n, h = int(sizes[k]), hs[i]
            m = a[int(starts[k]):int(starts[k + 1])].view(n, n)
            m[:h, :h] = hm[i, :h, :h]
            m[:h, h:] = bm[i, :h, :n - h]
            m[h:, :h] = bm[i, :h, :n - h].T
    return sizes, starts, a, torch.randn(int(sizes.sum()), generator=g, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batched":
        sizes, _, a0, x0 = _batch(case, seed)
        plan = bbk.BatchedPlan(sizes)
        return {"case": case, "plan": plan, "a0": a0, "x0": x0, "a": torch.empty_like(a0), "x": torch.empty_like(x0)}
    if kind == "full":
        return {"case": case, "a": _matrix(case, _generator(seed)).cpu().numpy()}
    a0, b0 = _system(case, seed)
    state = {"case": case, "a0": a0, "b0": b0}
    if kind == "solve":
        perm, pivot_types, _ = bbk.factor_device(a0, case["block"])
        state.update(f=a0, perm=perm, pivot_types=pivot_types)
    else:
        state["f"] = torch.empty_like(a0)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batched":
        a, x = state["a"], state["x"]
        a.copy_(state["a0"])
        x.copy_(state["x0"])
        perm, pivot_types, _ = bbk.batched_factor_solve(state["plan"], a, x, mode=case["mode"])
        return {"f": a, "perm": perm, "pivot_types": pivot_types, "x": x}
    if kind == "full":
        d = bbk.BlockLdltDecomposition(state["a"], case["block"], full=True, mode=case["mode"])
        d.factorize()
        return {"f": d.compact_factors(), "perm": d.permutation(), "pivot_types": d.pivot_types(),
                "panel_end": d.panel_end(), "a": d.reconstruct_original()}
    if kind == "solve":
        return bbk.solve_device(state["f"], state["perm"], state["pivot_types"], state["b0"].clone())
    f = state["f"]
    f.copy_(state["a0"])
    perm, pivot_types, panel_end = bbk.factor_device(f, case["block"], mode=case["mode"])
    if kind == "mixed":
        # the factors only precondition: what they are good for is x
        x, _ = bbk.solve_refined_device(state["a0"], f, perm, pivot_types, state["b0"], tol=1e-12, max_iter=3,
                                        method="gmres", restart=50)
        return {"perm": perm, "pivot_types": pivot_types, "panel_end": panel_end, "x": x}
    out = {"f": f, "perm": perm, "pivot_types": pivot_types, "panel_end": panel_end}
    if kind == "factor_solve":
        out["x"] = bbk.solve_device(f, perm, pivot_types, state["b0"].clone())
    return out


def work(case):
    """FP64: the upper triangle in, the compact factors out, n^3 / 3 operations
    to factor, 2 n^2 to solve for a right-hand side, and n^3 / 3 more to
    multiply the factors out again."""
    kind = case["kind"]
    if kind == "batched":
        s = _orders(case).astype(np.float64)
        return {"bytes": float((8 * s * (s + 1) + 24 * s).sum()), "flops": float((s ** 3 / 3 + 2 * s ** 2).sum())}
    n = float(case["n"])
    tri = 4 * n * (n + 1)
    if kind == "full":
        return {"bytes": 2 * tri + 8 * n * n, "flops": 2 * n ** 3 / 3}
    r = case.get("nrhs", 0)
    if kind == "solve":
        return {"bytes": tri + 16 * n * r, "flops": 2 * n * n * r}
    return {"bytes": 2 * tri + 16 * n * r, "flops": n ** 3 / 3 + 2 * n * n * r}


def tolerance(case):
    """FP64 sums in another order, amplified by the matrix's conditioning and
    the growth of its factors.  Between the library's two FP64 orders (and
    against ``exact``) factors and solutions were seen to differ by 2e-14 at
    n = 320, 9e-13 at n = 2000, 7e-12 at n = 4001 (spectral) and 3e-10 at
    n = 40000; a random matrix's conditioning has a heavy tail, so a given
    order is allowed more than one matrix of it showed.  The largest entry
    differs by about 50 times as much.  Ordered factors are the reference's
    bit for bit."""
    if case["kind"] == "factor":
        return "exact"
    if case["kind"] == "batched":
        return {"rel": 1e-12, "max": 5e-11}
    rel = max(1e-11, 5e-14 * case["n"])
    return {"rel": rel, "max": 100 * rel}


def _solve64(a, b):
    """Rows of ``b`` solved in 64 bits, refined twice."""
    lu, piv = torch.linalg.lu_factor(a)
    x = torch.linalg.lu_solve(lu, piv, b.T)
    for _ in range(2):
        x += torch.linalg.lu_solve(lu, piv, b.T - a @ x)
    return x.T.contiguous()


def exact(case, seed):
    kind = case["kind"]
    none = {"f": None, "perm": None, "pivot_types": None}
    if kind == "batched":
        sizes, starts, a, b = _batch(case, seed)
        x = torch.empty_like(b)
        at = 0
        for k, n in enumerate(int(v) for v in sizes):
            m = a[int(starts[k]):int(starts[k + 1])].view(n, n)
            x[at:at + n] = torch.linalg.solve(m, b[at:at + n])
            at += n
        return {**none, "x": x}
    if kind == "full":
        return {**none, "panel_end": None, "a": _matrix(case, _generator(seed)).cpu().numpy()}
    if kind == "factor":
        return None
    x = _solve64(*_system(case, seed))
    if kind == "solve":
        return x
    if kind == "mixed":
        return {"perm": None, "pivot_types": None, "panel_end": None, "x": x}
    return {**none, "panel_end": None, "x": x}
