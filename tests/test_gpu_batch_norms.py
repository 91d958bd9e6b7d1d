"""Batched CG under every norm, by one CTA and by teams of two, four and eight.

The norms' sums take a shared butterfly (One, Two), the maximum and the robust
norm one of their own; the recorded residuals start at the norm of b and end
below rtol of it, and so does the true residual of x (plus 1e-12 |b| for forming
it and for the recurrence's own drift).  The first residual is compared to 1e-12: a
rounding of 1.1e-16 a level of the sums (some 30) and a square root, times 100.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu

SYSTEMS = [workloads.laplacian(n, 60 + k) for k, n in enumerate((37, 700, 5003, 9001, 17003))]
NORMS = {"One": lambda v: np.abs(v).sum(), "Two": np.linalg.norm, "TwoRobust": np.linalg.norm,
         "Infinity": lambda v: np.abs(v).max()}


# (a mixed solve's inner target is a two-norm: under One, a sum over all rows, it
# can be met before the outer test is, and the refinement then stands still)
CASES = [(name, False) for name in sorted(NORMS)] + [(name, True) for name in sorted(NORMS) if name != "One"]


@pytest.mark.parametrize("name,mixed", CASES, ids=[n + ("-mixed" if m else "") for n, m in CASES])
def test_norm(ctx, name, mixed):
    A = sparse.BatchCompRowMatrix(SYSTEMS, ctx)
    n = A.numRows()
    s = sparse.CG(n, ctx=ctx)
    M = sparse.DiagonalPreconditioner(n, ctx)
    M.setMatrix(A)
    s.setPreconditioner(M)
    mon = sparse.DefaultIterationMonitor(60 if mixed else 2000, 1e-10, 1e-50, 1e5)
    mon.setNormType(getattr(sparse.Norm, name))
    mon.setIterationReporter(sparse.IterationReporter(), history_cap=2100)
    s.setIterationMonitor(mon)
    if mixed:
        s.setMixedPrecision(True, 1e-6, 3000)
    b = workloads.uniform(n, 8)
    x = np.zeros(n)
    got = s.solveBatch(A, b, x)
    for k, (m, rp, ci, v) in enumerate(SYSTEMS):
        r0, r1 = A.systemRows(k)
        norm = NORMS[name](b[r0:r1])
        hist = s.batchHistory(k)[0]
        assert got[k][0] == 0 and hist[-1] < 1e-10 * hist[0]
        assert abs(hist[0] - norm) <= 1e-12 * norm
        r = b[r0:r1] - np.add.reduceat(v * x[r0:r1][ci], rp[:-1])
        assert NORMS[name](r) <= (1e-10 + 1e-12) * norm
