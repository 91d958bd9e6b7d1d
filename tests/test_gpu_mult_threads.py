"""Products on host vectors from several threads, one matrix each, on one context.

Every product has the bits of the same product made alone, below and above
the size of the context's pinned staging (16384 values).
"""
import threading

import numpy as np
import pytest

from mtjg import sparse, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [20, 127, 128, 129])
def test_products_from_threads(ctx, N):
    n, rp, ci, v = workloads.poisson2d(N)
    made = []
    for t in range(4):
        A = sparse.CompRowMatrix(n, n, rp, ci, v * (t + 1.0), ctx=ctx)
        x = np.random.default_rng(t).uniform(-1.0, 1.0, n)
        made.append((A, x, A.multAdd(0.5, x, A.mult(x))))
    wrong = []

    def caller(t):
        A, x, want = made[t]
        for _ in range(100):
            if not np.array_equal(A.multAdd(0.5, x, A.mult(x)), want):
                wrong.append(t)

    threads = [threading.Thread(target=caller, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
