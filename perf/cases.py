"""The calls a user of this library makes, as measured cases.

Five families, each through the public entry points:

  mult    CompRowMatrix products: on host vectors (``mult``) or on device
          vectors (``mtjg_csr_mult_dev`` / ``mtjg_csr_trans_mult_dev``)
  solve   one IterativeSolver.solve on host vectors, FP64 or mixed precision
  factor  Preconditioner.setMatrix (a new matrix's ILU(0)) and one apply
  batch   a batch of independent systems, solveBatch
  serve   a backlog of requests through the solve server

Systems: 2D / 3D Poisson, 3D upwind convection-diffusion, and random graph
Laplacians (about 19 entries per row).  The right-hand side of every solve is
A x_true for a seeded x_true, so the exact answer is x_true.
"""
import ctypes
import functools
import math
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matrix-toolkits-java_gb300"))

from mtjg import serve, sparse, workloads  # noqa: E402

RTOL = 1e-10


def listed():
    return [
        # the smallest product, host vectors: the latency of one call
        {"name": "mult_small_host", "family": "mult", "system": "poisson2d", "size": 33, "device": False, "trans": False},
        # the product that bounds a large solve, on resident vectors
        {"name": "mult_poisson3d_128", "family": "mult", "system": "poisson3d", "size": 128, "device": True, "trans": False},
        # irregular rows and the transposed product (BiCG and QMR use both)
        {"name": "mult_trans_laplacian", "family": "mult", "system": "laplacian", "size": 150001, "device": True, "trans": True},
        # a small solve, as a time stepper makes thousands of: latency
        {"name": "cg_jacobi_2d_128", "family": "solve", "system": "poisson2d", "size": 128, "solver": "cg", "precond": "jacobi", "mixed": False},
        # the large memory-bound solve
        {"name": "cg_jacobi_3d_128", "family": "solve", "system": "poisson3d", "size": 128, "solver": "cg", "precond": "jacobi", "mixed": False},
        # incomplete Cholesky: few iterations, triangular sweeps; an odd grid
        {"name": "cg_icc_3d_47", "family": "solve", "system": "poisson3d", "size": 47, "solver": "cg", "precond": "icc", "mixed": False},
        # nonsymmetric solves with ILU(0), the configured size
        {"name": "bicgstab_ilu_96", "family": "solve", "system": "convdiff3d", "size": 96, "solver": "bicgstab", "precond": "ilu", "mixed": False},
        {"name": "gmres_ilu_96", "family": "solve", "system": "convdiff3d", "size": 96, "solver": "gmres", "precond": "ilu", "mixed": False},
        # FP32 inner solves inside FP64 refinement, an odd grid
        {"name": "gmres_ilu_mixed_63", "family": "solve", "system": "convdiff3d", "size": 63, "solver": "gmres", "precond": "ilu", "mixed": True},
        # a new matrix's ILU(0): what precedes the first solve on it
        {"name": "ilu_factor_apply_96", "family": "factor", "system": "convdiff3d", "size": 96},
        # a batch of uneven systems, 500 to 50000 rows each
        {"name": "batch_cg_192", "family": "batch", "count": 192, "lo": 500, "hi": 50000, "mixed": False},
        # a backlog of served requests: 2D Poisson grids and Laplacians
        {"name": "serve_backlog_48", "family": "serve", "count": 48},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mult", "mult", "cg", "cg", "icc", "krylov", "krylov", "factor", "batch", "serve"])
    if kind == "mult":
        system = rng.choice(["poisson2d", "poisson3d", "laplacian"])
        size = {"poisson2d": lambda: _log(rng, 24, 1024), "poisson3d": lambda: _log(rng, 10, 128),
                "laplacian": lambda: _log(rng, 1000, 200000)}[system]()
        return {"family": "mult", "system": system, "size": size, "device": rng.random() < 0.6, "trans": rng.random() < 0.3}
    if kind == "cg":
        system = rng.choice(["poisson2d", "poisson3d", "laplacian"])
        size = {"poisson2d": lambda: _log(rng, 24, 400), "poisson3d": lambda: _log(rng, 10, 120),
                "laplacian": lambda: _log(rng, 1000, 200000)}[system]()
        return {"family": "solve", "system": system, "size": size, "solver": "cg", "precond": "jacobi", "mixed": rng.random() < 0.3}
    if kind == "icc":
        return {"family": "solve", "system": "poisson3d", "size": _log(rng, 10, 48), "solver": "cg", "precond": "icc", "mixed": False}
    if kind == "krylov":
        return {"family": "solve", "system": "convdiff3d", "size": _log(rng, 10, 90), "solver": rng.choice(["bicgstab", "gmres"]),
                "precond": rng.choice(["ilu", "ilu", "jacobi"]), "mixed": rng.random() < 0.4}
    if kind == "factor":
        return {"family": "factor", "system": "convdiff3d", "size": _log(rng, 12, 96)}
    if kind == "batch":
        lo = _log(rng, 500, 4000)
        return {"family": "batch", "count": _log(rng, 12, 150), "lo": lo, "hi": min(50000, lo * rng.randint(3, 12)), "mixed": rng.random() < 0.4}
    return {"family": "serve", "count": _log(rng, 6, 40)}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=6)
def _stencil(system, size):
    return getattr(workloads, system)(size)


def _system(system, size, seed):
    """(n, rowptr, colind, data): a stencil depends on its size alone, a Laplacian on the seed too."""
    return workloads.laplacian(size, seed) if system == "laplacian" else _stencil(system, size)


def _factor_system(case, seed):
    """The stencil with its rows scaled by the seed: another matrix for another seed."""
    n, rp, ci, v = _system(case["system"], case["size"], seed)
    scale = np.exp(np.random.default_rng(seed).uniform(-0.05, 0.05, n))
    return n, rp, ci, v * np.repeat(scale, np.diff(rp))


def _vector(n, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, n)


def _times(sys_, x, trans=False):
    """A x (or A' x) in plain numpy; every row has its diagonal entry."""
    n, rp, ci, v = sys_
    if trans:
        rows = np.repeat(np.arange(n, dtype=np.int32), np.diff(rp))
        return np.bincount(ci, weights=v * x[rows], minlength=n)
    return np.add.reduceat(v * x[ci], rp[:-1])


def _many(make, count):
    with ThreadPoolExecutor(8) as ex:
        return list(ex.map(make, range(count)))


def _batch_systems(case, seed):
    sizes = workloads.batch_sizes(case["count"], 4, case["lo"], case["hi"])
    return _many(lambda k: workloads.laplacian(int(sizes[k]), seed * 1000 + k), case["count"])


def _served_specs(count):
    """2D Poisson grids N ~ U{64..384} and Laplacians n log-uniform in [1k, 100k], in turn."""
    r = np.random.default_rng(5)
    return [("poisson2d", int(r.integers(64, 385))) if k % 2 == 0 else
            ("laplacian", int(np.exp(r.uniform(math.log(1000.0), math.log(100000.0))))) for k in range(count)]


def _served_systems(case, seed):
    specs = _served_specs(case["count"])
    return _many(lambda k: workloads.poisson2d(specs[k][1]) if specs[k][0] == "poisson2d" else
                 workloads.laplacian(specs[k][1], seed * 1000 + k), case["count"])


def _matrix(sys_):
    n, rp, ci, v = sys_
    return sparse.CompRowMatrix(n, n, rp, ci, v)


def prepare(case, seed):
    family = case["family"]
    if family == "mult":
        sys_ = _system(case["system"], case["size"], seed)
        A, n = _matrix(sys_), sys_[0]
        x = _vector(n, seed)
        if not case["device"]:
            return {"family": family, "A": A, "x": x, "trans": case["trans"], "device": False}
        x = torch.from_numpy(x).cuda()
        y = torch.empty(n, dtype=torch.float64, device="cuda")
        z = torch.empty(n, dtype=torch.float64, device="cuda") if case["trans"] else None
        return {"family": family, "A": A, "x": x, "y": y, "z": z, "trans": case["trans"], "device": True}
    if family == "solve":
        sys_ = _system(case["system"], case["size"], seed)
        A, n = _matrix(sys_), sys_[0]
        b = _times(sys_, _vector(n, seed))
        solver = {"cg": sparse.CG, "bicgstab": sparse.BiCGstab, "gmres": sparse.GMRES}[case["solver"]](n)
        M = {"jacobi": lambda: sparse.DiagonalPreconditioner(n), "ilu": lambda: sparse.ILU(A),
             "icc": lambda: sparse.ICC(A)}[case["precond"]]()
        M.setMatrix(A)
        solver.setPreconditioner(M)
        solver.setIterationMonitor(sparse.DefaultIterationMonitor(20000, RTOL, 1e-50, 1e5))
        if case["mixed"]:
            solver.setMixedPrecision(True, 1e-6 if case["solver"] == "cg" else 1e-4, 3000)
        return {"family": family, "A": A, "M": M, "solver": solver, "b": b}
    if family == "factor":
        sys_ = _factor_system(case, seed)
        A = _matrix(sys_)
        return {"family": family, "A": A, "M": sparse.ILU(A), "b": _vector(sys_[0], seed + 1)}
    if family == "batch":
        systems = _batch_systems(case, seed)
        A = sparse.BatchCompRowMatrix(systems)
        n = A.numRows()
        solver = sparse.CG(n)
        M = sparse.DiagonalPreconditioner(n)
        M.setMatrix(A)
        solver.setPreconditioner(M)
        solver.setIterationMonitor(sparse.DefaultIterationMonitor(20000, RTOL, 1e-50, 1e5))
        if case["mixed"]:
            solver.setMixedPrecision(True, 1e-6, 2000)
        b = np.concatenate(_many(lambda k: _times(systems[k], _vector(systems[k][0], seed + k)), len(systems)))
        return {"family": family, "A": A, "M": M, "solver": solver, "b": b}
    systems = _served_systems(case, seed)
    srv = serve.Server(max_systems=256, pool_rows=1 << 23, rtol=RTOL)
    ids = [srv.addMatrix(*s) for s in systems]
    b = _many(lambda k: _times(systems[k], _vector(systems[k][0], seed + k)), len(systems))
    return {"family": family, "server": srv, "ids": ids, "b": b}


def run(state):
    family = state["family"]
    if family == "mult":
        A, x = state["A"], state["x"]
        if not state["device"]:
            return [A.mult(x), A.transMult(x)] if state["trans"] else A.mult(x)
        _dev(A, "mtjg_csr_mult_dev", x, state["y"])
        if not state["trans"]:
            return state["y"]
        _dev(A, "mtjg_csr_trans_mult_dev", x, state["z"])
        return [state["y"], state["z"]]
    if family == "factor":
        state["M"].setMatrix(state["A"])
        return state["M"].apply(state["b"])
    if family == "serve":
        srv = state["server"]
        place = {srv.submit(m, b): k for k, (m, b) in enumerate(zip(state["ids"], state["b"]))}
        srv.drain()
        done = {place[r.ticket]: r for r in srv.poll()}
        return [done[k].x for k in range(len(place))]
    x = np.zeros(len(state["b"]))
    if family == "batch":
        got = state["solver"].solveBatch(state["A"], state["b"], x)
        return {"x": x, "status": np.array([g[0] for g in got], dtype=np.int32)}
    state["solver"].solve(state["A"], state["b"], x)
    return {"x": x, "iterations": state["solver"].getIterationMonitor().iterations()}


def _dev(A, name, x, y):
    p = ctypes.POINTER(ctypes.c_double)
    code = getattr(A._lib, name)(A.h, ctypes.cast(x.data_ptr(), p), ctypes.cast(y.data_ptr(), p))
    if code:
        raise RuntimeError("%s: %d" % (name, code))


# -------------------------------------------------------------------- work
def _size(system, size):
    """Rows and entries."""
    if system == "laplacian":
        return size, 19 * size
    d = 2 if system == "poisson2d" else 3
    n = size ** d
    return n, n + 2 * d * (size - 1) * size ** (d - 1)


def _iterations(case):
    """About the iterations that these solves take (rtol 1e-10)."""
    if case["solver"] == "cg":
        if case["system"] == "laplacian":
            return 60
        return 1.05 * case["size"] if case["precond"] == "icc" else 3.2 * case["size"]
    per = {"bicgstab": 0.54, "gmres": 1.35}[case["solver"]] * case["size"]
    return per if case["precond"] == "ilu" else 3 * per


def work(case):
    family = case["family"]
    if family == "mult":
        n, nnz = _size(case["system"], case["size"])
        k = 2 if case["trans"] else 1
        return {"bytes": k * (12 * nnz + 4 * n + 16 * n), "flops": k * 2 * nnz}
    if family == "factor":  # the matrix in, the factor out and read by both sweeps
        n, nnz = _size(case["system"], case["size"])
        return {"bytes": 2 * 12 * nnz + 12 * nnz + 32 * n, "flops": 4 * nnz + 2 * nnz}
    if family == "solve":
        n, nnz = _size(case["system"], case["size"])
        its = _iterations(case)
        products = 2 if case["solver"] == "bicgstab" else 1
        sweeps = products * (12 * nnz + 16 * n) if case["precond"] in ("ilu", "icc") else 8 * n
        vectors = {"cg": 7, "bicgstab": 15, "gmres": 30}[case["solver"]] * 8 * n
        half = 0.5 if case["mixed"] else 1.0
        return {"bytes": half * its * (products * (12 * nnz + 4 * n) + sweeps + vectors),
                "flops": its * (products * 2 * nnz * (2 if case["precond"] in ("ilu", "icc") else 1) + 12 * n)}
    if family == "batch":
        n = int(workloads.batch_sizes(case["count"], 4, case["lo"], case["hi"]).sum())
        return {"bytes": (0.6 if case["mixed"] else 1.0) * 60 * (12 * 19 * n + 60 * n), "flops": 60 * (2 * 19 * n + 12 * n)}
    total = 0.0
    for system, size in _served_specs(case["count"]):
        n, nnz = _size(system, size)
        total += (60 if system == "laplacian" else 4.2 * size) * (8 * nnz + 56 * n)
    return {"bytes": total, "flops": total / 4}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    family = case["family"]
    if family == "mult":
        sys_ = _system(case["system"], case["size"], seed)
        x = _vector(sys_[0], seed)
        y = _times(sys_, x)
        return [y, _times(sys_, x, True)] if case["trans"] else y
    if family == "solve":
        n = _size(case["system"], case["size"])[0]
        return {"x": _vector(n, seed), "iterations": None}
    if family == "batch":
        sizes = workloads.batch_sizes(case["count"], 4, case["lo"], case["hi"])
        return {"x": np.concatenate([_vector(int(n), seed + k) for k, n in enumerate(sizes)]), "status": None}
    if family == "serve":
        return [_vector(_size(*s)[0], seed + k) for k, s in enumerate(_served_specs(case["count"]))]
    return _ilu_solve(_factor_system(case, seed), case["size"], _vector(case["size"] ** 3, seed + 1))


def _ilu_solve(sys_, N, b):
    """(L U) \\ b for the ILU(0) of a 7-point system on an N^3 grid, one
    wavefront x + y + z = const at a time.  No elimination step fills or
    touches an off-diagonal entry there, so only the pivots d change."""
    n, rp, ci, v = sys_
    rows = np.repeat(np.arange(n), np.diff(rp))
    steps = (1, N, N * N)
    at = {off: np.zeros(n) for s in steps for off in (s, -s)}
    at[0] = np.zeros(n)
    for off, a in at.items():
        k = ci - rows == off
        a[rows[k]] = v[k]
    g = np.arange(N)
    front = (g[:, None, None] + g[None, :, None] + g[None, None, :]).reshape(-1)
    order = np.argsort(front, kind="stable")
    fronts = np.split(order, np.cumsum(np.bincount(front))[:-1])
    d, y, x = at[0], b.copy(), np.empty(n)
    for i in fronts:
        for s in steps:
            j = np.maximum(i - s, 0)  # where there is no such neighbour the entry is 0
            w = at[-s][i] / d[j]
            d[i] -= w * at[s][j]
            y[i] -= w * y[j]
    for i in reversed(fronts):
        t = y[i]
        for s in steps:
            j = np.minimum(i + s, n - 1)
            e = at[s][i]
            t = t - np.where(e != 0, e * x[j], 0.0)
        x[i] = t / d[i]
    return x
