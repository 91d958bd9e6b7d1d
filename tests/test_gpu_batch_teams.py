"""Batched systems solved by teams of CTAs.

Systems on both sides of each team size's threshold (4096, 8192 and 16384
rows) and odd ones: the oracle's iteration count +-2 (the bar of the parity
tests), the FP64 true residual within rtol (plus 1e-13 |b| for forming it),
and the same bits alone and in a batch.
"""
import numpy as np
import pytest

import oracle as O
from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu

SIZES = [700, 4095, 4096, 8191, 8193, 16383, 16384, 20001, 33000]


def _systems():
    out = [workloads.laplacian(n, 40 + k) for k, n in enumerate(SIZES)]
    return out + [workloads.poisson2d(N) for N in (31, 64, 91, 129)]


def _solve(ctx, systems, bs, mixed):
    A = sparse.BatchCompRowMatrix(systems, ctx)
    n = A.numRows()
    solver = sparse.CG(n, ctx=ctx)
    M = sparse.DiagonalPreconditioner(n, ctx)
    M.setMatrix(A)
    solver.setPreconditioner(M)
    mon = sparse.DefaultIterationMonitor(3000 if not mixed else 60, 1e-10, 1e-50, 1e5)
    mon.setIterationReporter(sparse.IterationReporter(), history_cap=16)
    solver.setIterationMonitor(mon)
    if mixed:
        solver.setMixedPrecision(True, 1e-6, 3000)
    x = np.zeros(n)
    got = solver.solveBatch(A, np.concatenate(bs), x)
    hist = [solver.batchHistory(s)[0] for s in range(len(systems))]
    return got, [x[A.systemRows(s)[0]:A.systemRows(s)[1]] for s in range(len(systems))], hist


@pytest.mark.parametrize("strict,mixed", [(0, False), (1, False), (0, True)], ids=["fast", "strict", "mixed"])
def test_teams(ctx, strict, mixed):
    systems = _systems()
    bs = [workloads.uniform(s[0], 9 + k) for k, s in enumerate(systems)]
    ctx.setNumerics(strict)
    try:
        got, xs, hist = _solve(ctx, systems, bs, mixed)
        for k in (3, 6, 8, 12):
            g1, x1, h1 = _solve(ctx, [systems[k]], [bs[k]], mixed)
            assert g1[0] == got[k] and np.array_equal(x1[0], xs[k]) and np.array_equal(h1[0], hist[k])
    finally:
        ctx.setNumerics(0)
    for k, (n, rp, ci, v) in enumerate(systems):
        status, its, res = got[k]
        r = bs[k] - np.add.reduceat(v * xs[k][ci], rp[:-1])
        assert status == 0 and np.linalg.norm(r) <= (1e-10 + 1e-13) * np.linalg.norm(bs[k])
        if not mixed:
            pc = O.Precond(O.PC_JACOBI, n)
            A = O.Csr(n, n, rp, ci, v)
            pc.set_matrix(A)
            _, want, _, _ = O.solve(O.CG, A, bs[k], np.zeros(n), pc, max_iter=3000, rtol=1e-10)
            assert abs(its - want.iterations) <= 2
