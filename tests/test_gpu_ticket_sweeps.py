"""Lookahead in the ticket sweeps, on factors that the tiles of lines refuse.

Grids in natural order form lines and take the sweeps by tiles, which know no
lookahead; a randomly permuted grid keeps the level schedules.  Its rows hold
at most four entries a triangle (2D five-point), so every pending dependency
may be computed ahead.  On (MTJG_SWEEP_LOOKAHEAD=7) and off (0) give the same
bits: FP64 ILU and ICC sweeps under both numerics, and the FP32 ILU sweeps of
the mixed solves, where lookahead is on by default.  Every test asserts that
the ticket sweeps ran: an apply is three launches by tickets, four by tiles.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads
from test_gpu_sweep_lookahead import _same, _solve, _with_lookahead

pytestmark = pytest.mark.gpu


def permuted(mat, seed, skew=0.0):
    """P A P' of a random permutation, its off-diagonals scaled by up to 1 - skew."""
    n, rp, ci, v = mat
    rng = np.random.default_rng(seed)
    q = rng.permutation(n)
    rows, cols = q[np.repeat(np.arange(n), np.diff(rp))], q[ci]
    v = np.where(rows == cols, v, v * (1.0 - skew * rng.random(v.size)))
    o = np.lexsort((cols, rows))
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return n, rp2, cols[o].astype(np.int32), v[o]


def apply_launches(ctx, mat, cls):
    n, rp, ci, v = mat
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    M = cls(A)
    M.setMatrix(A)
    b = workloads.uniform(n, 23)
    before = ctx.launchCount()
    x = M.apply(b)
    return x, ctx.launchCount() - before


SPD = permuted(workloads.poisson2d(60), 4)
SKEW = permuted(workloads.poisson2d(60), 5, skew=0.3)


@pytest.fixture(params=[0, 1], ids=["fast", "strict"])
def numerics(request, ctx):
    ctx.setNumerics(request.param)
    yield request.param
    ctx.setNumerics(0)


@pytest.mark.parametrize("mat,cls", [(SPD, sparse.ICC), (SPD, sparse.ILU), (SKEW, sparse.ILU)],
                         ids=["icc", "ilu", "ilu_skew"])
def test_applies(ctx, numerics, mat, cls):
    on, n_on = _with_lookahead(True, lambda: apply_launches(ctx, mat, cls))
    off, n_off = _with_lookahead(False, lambda: apply_launches(ctx, mat, cls))
    assert n_on == n_off == 3
    _same([on], [off])


@pytest.mark.parametrize("solver,mat,cls", [(sparse.CG, SPD, sparse.ICC), (sparse.BiCGstab, SKEW, sparse.ILU)],
                         ids=["icc_cg", "ilu_bicgstab"])
def test_solves(ctx, numerics, solver, mat, cls):
    assert apply_launches(ctx, mat, cls)[1] == 3
    on = _with_lookahead(True, lambda: _solve(ctx, mat, solver, cls))
    off = _with_lookahead(False, lambda: _solve(ctx, mat, solver, cls))
    _same(on, off)
    assert on[2] > 5


@pytest.mark.parametrize("solver", [sparse.GMRES, sparse.BiCGstab], ids=["gmres", "bicgstab"])
def test_fp32_sweeps(ctx, solver):
    assert apply_launches(ctx, SKEW, sparse.ILU)[1] == 3
    on = _with_lookahead(True, lambda: _solve(ctx, SKEW, solver, sparse.ILU, mixed=True))
    off = _with_lookahead(False, lambda: _solve(ctx, SKEW, solver, sparse.ILU, mixed=True))
    _same(on, off)
