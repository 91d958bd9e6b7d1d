"""A mixed solve where the FP32 records of the tiles of lines do not fit.

The FP64 tiles are made by setMatrix; their FP32 records are made by the first
mixed solve and take about 100 bytes a row, where the FP32 factor by itself
takes 28.  With room for the factor only, the solve takes the level schedules:
the same bits as by tiles (both sum a row in the same order with FMAs and round
its quotient once).
"""
import ctypes as C
import os

import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu

N = 110
MB = 1 << 20


def _cudart():
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return C.CDLL(os.path.join(home, "lib64", "libcudart.so"))


def _free(rt):
    free, total = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
    return free.value


def _fill(rt, leave):
    """Allocations that leave about `leave` bytes free."""
    held = []
    size = 1 << 36
    while size >= 4 * MB:
        p = C.c_void_p()
        if _free(rt) - leave >= size and rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
            held.append(p)
        else:
            size //= 2
    return held


def _permuted(mat, seed):
    n, rp, ci, v = mat
    q = np.random.default_rng(seed).permutation(n)
    rows, cols = q[np.repeat(np.arange(n), np.diff(rp))], q[ci]
    o = np.lexsort((cols, rows))
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return n, rp2, cols[o].astype(np.int32), v[o]


def _solver(ctx, n):
    s = sparse.GMRES(n, 10, ctx=ctx)
    mon = sparse.DefaultIterationMonitor(50, 1e-10, 1e-50, 1e5)
    mon.setIterationReporter(sparse.IterationReporter(), history_cap=64)
    s.setIterationMonitor(mon)
    s.setMixedPrecision(True, 1e-4, 200)
    return s


def _solve(ctx, s, A, M, b):
    s.setPreconditioner(M)
    x = np.zeros(b.size)
    before = ctx.launchCount()
    s.solve(A, b, x)
    return x, np.array(s.history[0]), s.innerIterations(), ctx.launchCount() - before


def test_mixed_solve_without_room_for_fp32_records(ctx):
    # every kernel of the ticket sweeps is loaded
    small = _permuted(workloads.convdiff3d(12), 1)
    As = sparse.CompRowMatrix(small[0], small[0], *small[1:], ctx)
    Ms = sparse.ILU(As)
    Ms.setMatrix(As)
    _solve(ctx, _solver(ctx, small[0]), As, Ms, workloads.uniform(small[0], 2))

    n, rp, ci, v = workloads.convdiff3d(N)
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    b = workloads.uniform(n, 3)
    M = sparse.ILU(A)
    M.setMatrix(A)
    s = _solver(ctx, n)
    J = sparse.DiagonalPreconditioner(n, ctx)
    J.setMatrix(A)
    _solve(ctx, s, A, J, b)  # the matrix's FP32 copy and the solver's own vectors are made
    tiles = _solve(ctx, s, A, M, b)
    M.setMatrix(A)  # the FP32 copies go
    rt = _cudart()
    # the FP32 factor and one vector, and half of what the records take beside them
    held = _fill(rt, 4 * (v.size + n) + 50 * n)
    try:
        tickets = _solve(ctx, s, A, M, b)
    finally:
        for p in held:
            assert rt.cudaFree(p) == 0
    assert tickets[3] < tiles[3]  # an apply: 3 launches by tickets, 4 by tiles
    assert tickets[2] == tiles[2]
    assert np.array_equal(tickets[1], tiles[1]) and np.array_equal(tickets[0], tiles[0])
    # a new matrix has room again
    M.setMatrix(A)
    again = _solve(ctx, s, A, M, b)
    assert again[3] == tiles[3] and np.array_equal(again[0], tiles[0])
