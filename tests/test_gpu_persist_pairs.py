"""The one-launch CG with two product tiles a CTA, against the phases bit for bit.

Two CTAs of one tile fit an SM, so 305 tiles and more (of 152 SMs) take two
tiles each, up to 512.  A tridiagonal matrix has tiles of exactly 256 rows, so
its sizes lie on both sides of either limit; the rest are one-lane and four-lane
rows of uneven tiles.
"""
import numpy as np
import pytest

from mtjg import sparse, workloads
from test_gpu_persist import _same, _solve

pytestmark = pytest.mark.gpu


def tridiagonal(n):
    i = np.arange(n)
    R, C = np.concatenate([i, i[1:], i[:-1]]), np.concatenate([i, i[:-1], i[1:]])
    o = np.lexsort((C, R))
    rp = np.concatenate([[0], np.cumsum(np.bincount(R, minlength=n))]).astype(np.int32)
    return n, rp, C[o].astype(np.int32), np.where(R == C, 2.2, -1.0)[o]


@pytest.fixture(params=[0, 1], ids=["fast", "strict"])
def numerics(request, ctx):
    ctx.setNumerics(request.param)
    yield request.param
    ctx.setNumerics(0)


def _compare(ctx, mat, one_launch, **kw):
    one = _solve(ctx, mat, "jacobi", graph=False, **kw)
    many = _solve(ctx, mat, "jacobi", graph=True, **kw)
    _same(one, many)
    assert one[2] > 5
    assert (one[5] <= 5) == one_launch


@pytest.mark.parametrize("rows", [303 * 256, 304 * 256, 304 * 256 + 1, 305 * 256, 401 * 256 + 77, 512 * 256, 512 * 256 + 1])
def test_tile_counts(ctx, numerics, rows):
    _compare(ctx, tridiagonal(rows), rows <= 512 * 256)


@pytest.mark.parametrize("mat", [workloads.poisson2d(300), workloads.poisson3d(41), workloads.laplacian(25000, 3)],
                         ids=["2d", "3d", "laplacian"])
def test_uneven_tiles(ctx, numerics, mat):
    _compare(ctx, mat, True)


@pytest.mark.parametrize("norm", [sparse.Norm.One, sparse.Norm.TwoRobust, sparse.Norm.Infinity])
def test_norms(ctx, norm):
    _compare(ctx, workloads.laplacian(25000, 3), True, norm=norm)


def test_iteration_limit(ctx):
    one = _solve(ctx, workloads.poisson2d(300), "identity", graph=False, max_iter=7)
    many = _solve(ctx, workloads.poisson2d(300), "identity", graph=True, max_iter=7)
    _same(one, many)
    assert one[2] == 7 and one[5] <= 5
