"""Which path a factor's set-up and sweeps take, and GMRES's Gram-Schmidt.

The comparisons with the oracle and with the phases hold on any path, so here
the path itself is checked by its launches.  An apply is four launches by tiles
of lines (b into plan order, two sweeps, x out of it) and three by level
schedules (one fill, two sweeps).  ILU(0) by levels launches at least once per
level of the factor; by tiles, a fixed number.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads
from test_gpu_lines import MATRICES, _matrix
from test_gpu_ticket_sweeps import apply_launches, permuted

pytestmark = pytest.mark.gpu

# rows in lines of four or more, four entries a triangle, and at most
# 2 n + 65536 places in the plan.  4 x 4 lines are mostly empty lanes: 100
# planes of them take 27,648 places, 200 of them 106,496.
REFUSED = {"thin:200", "thin:900"}
# elimination reaches off the diagonal: the factor is made by levels, of at least this many
LEVELS = {"nine:23": 3 * 22, "banded:-60,-7,-2,-1,0,1,2,7,60": 399}


@pytest.mark.parametrize("name", MATRICES)
def test_sweeps(ctx, name):
    mat = _matrix(name)
    assert apply_launches(ctx, mat, sparse.ILU)[1] == (3 if name in REFUSED else 4)


@pytest.mark.parametrize("make", [lambda: permuted(workloads.poisson3d(12), 3),
                                  lambda: permuted(workloads.poisson2d(40), 3)], ids=["3d", "2d"])
def test_permuted_grids_take_tickets(ctx, make):
    assert apply_launches(ctx, make(), sparse.ILU)[1] == 3


@pytest.mark.parametrize("name", MATRICES)
def test_factor(ctx, name):
    n, rp, ci, v = _matrix(name)
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    M = sparse.ILU(A)
    M.setMatrix(A)
    before = ctx.launchCount()
    M.setMatrix(A)
    launches = ctx.launchCount() - before
    if name in REFUSED:
        assert launches > int(name.split(":")[1])  # a level a plane, at least
    elif name in LEVELS:
        assert launches > LEVELS[name]
    else:
        assert launches <= 30


@pytest.mark.parametrize("restart", [4, 30])
def test_gram_schmidt(ctx, restart):
    """A cycle is (i + 2) phases with a finalize each and a scaling in step i, or one launch a step."""
    n, rp, ci, v = workloads.convdiff3d(13)
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    counts = {}
    for graph in (False, True):
        s = sparse.GMRES(n, restart, ctx=ctx)
        s.setGraphLaunch(graph)
        s.setIterationMonitor(sparse.DefaultIterationMonitor(2 * restart, 1e-300, 1e-300, 1e5))
        x = np.zeros(n)
        before = ctx.launchCount()
        with pytest.raises(sparse.IterativeSolverNotConvergedException):
            s.solve(A, workloads.uniform(n, 3), x)
        counts[graph] = ctx.launchCount() - before
    fewer = sum(2 * (i + 2) for i in range(restart))
    assert counts[True] - counts[False] >= fewer
