"""Algo 5's first phase over many iterations of one launch, where every position
array is cleared and used again many times while two iterations are in work:
81 iterations in one launch against 81 launches, bit for bit (a word read
before its clear is the position of five moves before).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(1, 1), (30, 7), (500, 500), (3000, 64), (4257, 256), (12_001, 256)])
def test_one_launch_equals_many(n, batch):
    import batchlayoutcode_gb300 as B

    B.build()
    rng = np.random.default_rng(n + batch)
    u, v = np.concatenate([rng.integers(0, n, (2, n)), [np.arange(n - 1), np.arange(1, n)]], 1)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
    ci = (e % n).astype(np.int32)
    xy = rng.normal(size=(n, 2)).astype(np.float32).astype(np.float64) * 20
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        step = 1.0
        for _ in range(81):
            e1 = a.greedy_iteration(batch, step)
            step *= 0.99
        for _ in range(19):
            e1 = a.minibatch_iteration(5, batch, step)
            step *= 0.99
        x1 = a.nCoordinates
        for _ in range(3):
            a.nCoordinates = xy
            e100 = a.run_resident(5, 100, batch, 1.2, 1.0)
            assert np.array_equal(a.nCoordinates, x1) and e100 == e1
