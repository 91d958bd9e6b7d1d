"""Tiles of 256 lines, and the FP32 sweeps of every tile, against other paths.

More lines than 128 for every SM (19,456) take 256 a tile.  FP64 is compared
with the oracle (STRICT bit for bit, FAST to 1e-12 of max |x|: a rounding of
1.1e-16 a level of some three hundred levels, times 30, on diagonally dominant factors).

FP32 sweeps have no entry of their own.  They are compared with the ticket
sweeps bit for bit through mixed solves of two systems: A beside a six-row
block that lets the planner accept (a line), and A beside a dense one, whose
last row has five entries below its diagonal, so that the whole factor is
refused.  b is zero on the block, so every vector is zero there, and A's rows
keep their products, tiles and sums; any differing bit of an apply would show
in the refinement's residuals and in x.
"""
import functools

import numpy as np
import pytest

import oracle as O
from mtjg import sparse, workloads
from test_gpu_lines import _matrix
from test_gpu_ticket_sweeps import apply_launches

pytestmark = pytest.mark.gpu


def lines(length, count, reads, seed=2):
    """`count` lines of `length` rows; reads(l): the earlier lines that line l reads, row by row."""
    rng = np.random.default_rng(seed)
    l, x = np.divmod(np.arange(length * count), length)
    R, C = [np.arange(length * count)], [np.arange(length * count)]
    for ok, d in [(x > 0, 1)] + [(m >= 0, (l - m) * length) for m in reads(l)]:
        i = np.arange(length * count)[ok]
        j = i - (d if np.isscalar(d) else d[ok])
        R += [i, j]
        C += [j, i]
    R, C = np.concatenate(R), np.concatenate(C)
    V = np.where(R == C, 2.0 + len(R) / (length * count), -1.0 - 0.1 * rng.random(R.size))
    o = np.lexsort((C, R))
    n = length * count
    rp = np.concatenate([[0], np.cumsum(np.bincount(R, minlength=n))]).astype(np.int32)
    return n, rp, C[o].astype(np.int32), V[o]


@functools.lru_cache(maxsize=2)
def _wide(name):
    if name == "two entries":  # planes of one line each, every line reading the one 140 before
        return lines(90, 19600, lambda l: [np.where(l >= 140, l - 140, -1)])
    # three: a 33 x 140 x 140 grid, tiles of 16 by 16 lines
    return lines(33, 19600, lambda l: [np.where(l % 140 > 0, l - 1, -1), np.where(l >= 140, l - 140, -1)])


@pytest.mark.parametrize("name", ["two entries", "three entries"])
def test_wide_tiles(ctx, name):
    mat = _wide(name)
    n, rp, ci, v = mat
    assert apply_launches(ctx, mat, sparse.ILU)[1] == 4
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    M = sparse.ILU(A)
    M.setMatrix(A)
    Mo = O.Precond(O.PC_ILU, n)
    Mo.set_matrix(O.Csr(n, n, rp, ci, v))
    assert np.array_equal(M.values(), Mo.values())
    b = workloads.uniform(n, 7)
    for trans in (False, True):
        want = Mo.trans_apply(b) if trans else Mo.apply(b)
        ctx.setNumerics(1)
        try:
            got = M.transApply(b) if trans else M.apply(b)
        finally:
            ctx.setNumerics(0)
        assert np.array_equal(got, want), trans
        fast = M.transApply(b) if trans else M.apply(b)
        assert np.max(np.abs(fast - want)) <= 1e-12 * np.max(np.abs(want)), trans


def beside(mat, dense):
    """A and a block of six rows that it is not coupled to."""
    n, rp, ci, v = mat
    D = np.full((6, 6), -0.1) if dense else -0.1 * (np.abs(np.subtract.outer(np.arange(6), np.arange(6))) == 1)
    D[np.diag_indices(6)] = 1.0
    nz = [np.nonzero(r)[0] for r in D]
    return (n + 6, np.concatenate([rp, rp[-1] + np.cumsum([c.size for c in nz])]).astype(np.int32),
            np.concatenate([ci] + [n + c for c in nz]).astype(np.int32), np.concatenate([v] + [D[i][c] for i, c in enumerate(nz)]))


def _mixed(ctx, mat, cls, b):
    n, rp, ci, v = mat
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    M = sparse.ILU(A)
    M.setMatrix(A)
    s = cls(n, ctx=ctx)
    s.setPreconditioner(M)
    s.setMixedPrecision(True, 1e-4, 12)
    mon = sparse.DefaultIterationMonitor(4, 1e-14, 1e-300, 1e5)
    mon.setIterationReporter(sparse.IterationReporter(), history_cap=16)
    s.setIterationMonitor(mon)
    x = np.zeros(n)
    try:
        s.solve(A, b, x)
    except sparse.IterativeSolverNotConvergedException:
        pass
    return x, np.array(s.history[0])


FP32 = ["poisson2d:5", "poisson2d:33", "poisson2d:130", "poisson3d:17", "convdiff3d:36", "banded:-1,0,1",
        "banded:-50,-1,0,1,50", "banded:-60,-7,-2,-1,0,1,2,7,60", "ragged:", "nine:23"]


@pytest.mark.parametrize("name", ["two entries", "three entries"])
def test_wide_fp32_sweeps(ctx, name):
    _compare_fp32(ctx, _wide(name), False, sparse.GMRES)


@pytest.mark.parametrize("solver", [sparse.GMRES, sparse.BiCGstab], ids=["gmres", "bicgstab"])
@pytest.mark.parametrize("scaled", [False, True], ids=["plain", "scaled"])
@pytest.mark.parametrize("name", FP32)
def test_fp32_sweeps(ctx, name, scaled, solver):
    _compare_fp32(ctx, _matrix(name), scaled, solver)


def _compare_fp32(ctx, mat, scaled, solver):
    n, rp, ci, v = mat
    if scaled:  # diagonals and right-hand sides beyond the short division's 2^-40 to 2^41
        e = np.random.default_rng(3).integers(-46, 47, n)
        v = np.ldexp(v, np.repeat(e, np.diff(rp)))
    b = np.concatenate([workloads.uniform(n, 11), np.zeros(6)])
    if scaled:
        b[:n] = np.ldexp(b[:n], e)
    tiles, tickets = beside((n, rp, ci, v), False), beside((n, rp, ci, v), True)
    assert apply_launches(ctx, tiles, sparse.ILU)[1] == 4
    assert apply_launches(ctx, tickets, sparse.ILU)[1] == 3
    got, want = _mixed(ctx, tiles, solver, b), _mixed(ctx, tickets, solver, b)
    assert len(got[1]) > 1
    assert np.array_equal(got[1], want[1], equal_nan=True) and np.array_equal(got[0], want[0], equal_nan=True)
