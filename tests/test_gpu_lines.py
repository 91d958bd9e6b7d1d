"""Triangular sweeps by tiles of lines against the oracle.

STRICT applies are compared bit for bit, so the tiles' edges, the ring of
recent values and the division by a prepared reciprocal must give the row by
row result; FAST applies to 1e-12 of max |x|: a unit of rounding (1.1e-16) per
level of at most a few hundred levels, on diagonally dominant factors that do
not amplify it, times 20.
"""
import numpy as np
import pytest

import oracle as O
from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu


def _banded(n, offsets, rng):
    """A diagonally dominant matrix with the given diagonals (where in range)."""
    rp, ci, v = [0], [], []
    for i in range(n):
        for o in sorted(offsets):
            if 0 <= i + o < n:
                ci.append(i + o)
                v.append(2.0 * len(offsets) if o == 0 else -1.0 - 0.5 * rng.random())
        rp.append(len(ci))
    return n, np.array(rp, dtype=np.int32), np.array(ci, dtype=np.int32), np.array(v)


def _ragged(rng):
    """Planes of different line counts, lines of different lengths: an L-shaped grid, natural order."""
    return _grid7([(x, y, z) for z in range(7) for y in range(19) for x in range(23) if not (x > 9 + z and y > 11)], rng)


def _grid7(keep, rng):
    at = {p: k for k, p in enumerate(keep)}
    rp, ci, v = [0], [], []
    for (x, y, z) in keep:
        row = [(at[q], -1.0 - 0.1 * rng.random()) for q in
               ((x, y, z - 1), (x, y - 1, z), (x - 1, y, z), (x + 1, y, z), (x, y + 1, z), (x, y, z + 1)) if q in at]
        row = sorted(row + [(at[(x, y, z)], 7.5)])
        ci += [c for c, _ in row]
        v += [w for _, w in row]
        rp.append(len(ci))
    return len(keep), np.array(rp, dtype=np.int32), np.array(ci, dtype=np.int32), np.array(v)


def _grid9(N, rng):
    rp, ci, v = [0], [], []
    for y in range(N):
        for x in range(N):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if 0 <= x + dx < N and 0 <= y + dy < N:
                        ci.append((y + dy) * N + x + dx)
                        v.append(9.0 if dx == dy == 0 else -1.0 - 0.1 * rng.random())
            rp.append(len(ci))
    return N * N, np.array(rp, dtype=np.int32), np.array(ci, dtype=np.int32), np.array(v)


def _matrix(name):
    rng = np.random.default_rng(11)
    kind, _, arg = name.partition(":")
    if kind == "banded":
        return _banded(400, [int(t) for t in arg.split(",")], rng)
    if kind == "ragged":
        return _ragged(rng)
    if kind == "nine":  # 2D nine-point: elimination reaches off the diagonal
        N = int(arg)
        return _grid9(N, rng)
    if kind == "thin":  # 4 x 4 lines: mostly empty lanes, the plan is refused (900: before its offsets are found)
        return _grid7([(x, y, z) for z in range(int(arg)) for y in range(4) for x in range(4)], rng)
    return getattr(workloads, kind)(int(arg))


MATRICES = ["poisson2d:4", "poisson2d:33", "poisson2d:130", "poisson3d:5", "poisson3d:17", "convdiff3d:9",
            "convdiff3d:36",  # tiles with empty lanes on two sides
            "banded:-1,0,1", "banded:-50,-1,0,1,50",  # one line, and a value further back than the ring
            "banded:-60,-7,-2,-1,0,1,2,7,60",  # four entries a row, two of them in the line
            "ragged:", "nine:23", "thin:100", "thin:200", "thin:900"]


def _vectors(n):
    rng = np.random.default_rng(5)
    b = rng.uniform(-1, 1, n)
    spread = b * 10.0 ** rng.integers(-300, 290, n)  # quotients beyond the short division's range
    zeros = np.where(rng.random(n) < 0.7, 0.0, b) * np.where(rng.random(n) < 0.5, 1.0, -1.0)
    return {"uniform": b, "spread": spread, "zeros": zeros}


@pytest.mark.parametrize("kind", ["ilu", "icc"])
@pytest.mark.parametrize("name", MATRICES)
def test_apply(ctx, name, kind):
    n, rp, ci, v = _matrix(name)
    if kind == "icc" and name.startswith(("banded", "ragged", "nine", "thin")):
        v = v.copy()
        rows = np.repeat(np.arange(n), np.diff(rp))
        v[ci != rows] = -1.0  # symmetric
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    Ao = O.Csr(n, n, rp, ci, v)
    M = {"ilu": sparse.ILU, "icc": sparse.ICC}[kind](A)
    Mo = O.Precond({"ilu": O.PC_ILU, "icc": O.PC_ICC}[kind], n)
    M.setMatrix(A)
    Mo.set_matrix(Ao)
    assert np.array_equal(M.values(), Mo.values())
    try:
        for label, b in _vectors(n).items():
            for trans in (False, True):
                want = Mo.trans_apply(b) if trans else Mo.apply(b)
                ctx.setNumerics(1)
                got = M.transApply(b) if trans else M.apply(b)
                assert np.array_equal(got, want, equal_nan=True), (label, trans)
                ctx.setNumerics(0)
                if label == "uniform":
                    fast = M.transApply(b) if trans else M.apply(b)
                    assert np.max(np.abs(fast - want)) <= 1e-12 * np.max(np.abs(want)), trans
    finally:
        ctx.setNumerics(0)


def test_zero_pivot(ctx):
    """A pivot that elimination makes zero: MTJ's message and row, as the oracle has them."""
    n, rp, ci, v = workloads.poisson2d(20)
    v = v.copy()
    for i in (37, 38):  # d_38 = a_38,38 - (a_38,37 / d_37) a_37,38 - ... made 0 by decoupling row 37 and 38 from above
        for k in range(rp[i], rp[i + 1]):
            v[k] = 1.0 if ci[k] in (37, 38) else 0.0
    A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
    Mo = O.Precond(O.PC_ILU, n)
    assert Mo.set_matrix(O.Csr(n, n, rp, ci, v)) != 0
    M = sparse.ILU(A)
    with pytest.raises(RuntimeError, match="Zero pivot"):
        M.setMatrix(A)
    assert M.error_row == Mo.detail
