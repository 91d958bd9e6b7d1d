"""GMRES's one-launch Gram-Schmidt gives the phases' results bit for bit.

Sizes where its split changes: one row tile, fewer tiles than SMs, the last
tile short, two tiles per sub-block (over 608 tiles of 1024 rows), tiles of
2048 rows (from 2^20 rows on), two of those per sub-block; a restart inside
the solve, convergence inside a cycle, the iteration limit, and SSOR, whose
apply starts from the vector the step leaves behind.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu


def _solve(ctx, mat, pc, graph, restart, max_iter):
    n, rp, ci, v = mat
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    M = {"identity": None, "jacobi": sparse.DiagonalPreconditioner(n, ctx), "ilu": sparse.ILU(A),
         "ssor": sparse.SSOR(A)}[pc]
    solver = sparse.GMRES(n, restart, ctx=ctx)
    solver.setGraphLaunch(graph)
    if M is not None:
        M.setMatrix(A)
        solver.setPreconditioner(M)
    mon = sparse.DefaultIterationMonitor(max_iter, 1e-10, 1e-50, 1e5)
    mon.setIterationReporter(sparse.IterationReporter(), history_cap=2 * max_iter + 64)
    solver.setIterationMonitor(mon)
    x = np.zeros(n)
    try:
        solver.solve(A, workloads.uniform(n, 3), x)
        status = "ok"
    except sparse.IterativeSolverNotConvergedException as e:
        status = e.getReason().name
    return status, x, np.array(solver.history[0]), mon.iterations()


@pytest.mark.parametrize("strict", [0, 1], ids=["fast", "strict"])
@pytest.mark.parametrize("name,size,pc,restart,max_iter", [
    ("poisson2d", 9, "identity", 5, 200), ("convdiff3d", 13, "jacobi", 30, 400), ("convdiff3d", 13, "ilu", 30, 400),
    ("convdiff3d", 13, "ssor", 7, 60), ("laplacian", 30011, "jacobi", 30, 400), ("convdiff3d", 55, "ilu", 4, 400),
    ("convdiff3d", 87, "jacobi", 5, 12), ("poisson3d", 102, "identity", 5, 12), ("poisson3d", 128, "jacobi", 4, 9)])
def test_same_bits(ctx, strict, name, size, pc, restart, max_iter):
    mat = workloads.laplacian(size, 7) if name == "laplacian" else getattr(workloads, name)(size)
    ctx.setNumerics(strict)
    try:
        got = _solve(ctx, mat, pc, False, restart, max_iter)
        want = _solve(ctx, mat, pc, True, restart, max_iter)
    finally:
        ctx.setNumerics(0)
    assert got[0] == want[0] and got[3] == want[3]
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[1], want[1])
