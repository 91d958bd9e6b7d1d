"""The sweeps' quotient by a prepared reciprocal is the rounded quotient.

With y the rounded reciprocal, one residual correction of a y gives a quotient
before its last rounding that is off by at most 2^-54 d' / 2 units (d' in [1, 2)
the divisor's significand) where the exact quotient is within that of a
midpoint between two doubles; the exact quotient, by 53-bit integers, is at least
2^-53 / d' units off every midpoint.  So the closest cases are the quotients one
part in 2 d off a midpoint, here for random divisors and for the divisors
nearest to 2^53, where the two bounds meet.  A factor of diagonals alone (its
other entries are stored zeros) makes an apply one quotient a row.
"""
import random

import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu


def hard_pairs(count, seed):
    """(a, d), 53-bit integers, a 2^B = M d +- 1 or 3 with M odd: a / d beside a midpoint."""
    rng = random.Random(seed)
    out = []
    k = 0
    while len(out) < count:
        d = 2**53 - 1 - 2 * k if k < 300 else rng.randrange(2**52, 2**53) | 1
        k += 1
        for s in (1, -1, 3, -3):
            for B, top in ((54, 0), (53, 2**53)):  # quotients below and above 1
                M = (-s * pow(d, -1, 2**B)) % 2**B + top
                a, rest = divmod(M * d + s, 2**B)
                if M >= 2**53 and M % 2 and not rest and 2**52 <= a < 2**53:
                    out.append((a, d))
    return out[:count]


@pytest.mark.parametrize("numerics", [0, 1], ids=["fast", "strict"])
def test_quotients(ctx, numerics):
    n, rp, ci, _ = workloads.poisson2d(64)
    rng = np.random.default_rng(1)
    for seed in range(4):
        a, d = (np.array(t, dtype=np.float64) for t in zip(*hard_pairs(n, seed)))
        a = np.ldexp(a, rng.integers(-120, 20, n)) * rng.choice([-1.0, 1.0], n)
        d = np.ldexp(d, rng.integers(-120, 20, n)) * rng.choice([-1.0, 1.0], n)
        v = np.where(np.repeat(np.arange(n), np.diff(rp)) == ci, np.repeat(d, np.diff(rp)), 0.0)
        A = sparse.CompRowMatrix(n, n, rp, ci, v, ctx)
        M = sparse.ILU(A)
        M.setMatrix(A)
        ctx.setNumerics(numerics)
        try:
            before = ctx.launchCount()
            x = M.apply(a)
            assert ctx.launchCount() - before == 4  # by tiles of lines
        finally:
            ctx.setNumerics(0)
        assert np.array_equal(x, a / d)
