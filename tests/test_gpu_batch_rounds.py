"""A uniform batch that takes two CTAs per SM (csrc/batch_plan.h): each system
has the bits it has alone, the one-round and the two-round ones alike.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu


def _solve(ctx, systems, bs, mixed):
    A = sparse.BatchCompRowMatrix(systems, ctx)
    n = A.numRows()
    solver = sparse.CG(n, ctx=ctx)
    M = sparse.DiagonalPreconditioner(n, ctx)
    M.setMatrix(A)
    solver.setPreconditioner(M)
    solver.setIterationMonitor(sparse.DefaultIterationMonitor(60 if mixed else 3000, 1e-10, 1e-50, 1e5))
    if mixed:
        solver.setMixedPrecision(True, 1e-6, 3000)
    x = np.zeros(n)
    return solver.solveBatch(A, np.concatenate(bs), x), np.split(x, np.cumsum([s[0] for s in systems])[:-1])


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("size,count", [(64, 240), (91, 120)])  # teams of two and of four CTAs
def test_two_per_sm(ctx, size, count, mixed):
    mat = workloads.poisson2d(size)
    bs = [workloads.uniform(mat[0], 100 + k) for k in range(count)]
    got, xs = _solve(ctx, [mat] * count, bs, mixed)
    assert all(status == 0 for status, _, _ in got)
    for k in (0, count // 2, count - 1):
        one, x = _solve(ctx, [mat], [bs[k]], mixed)
        assert one[0] == got[k] and np.array_equal(x[0], xs[k])
