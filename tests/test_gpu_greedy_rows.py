"""Algo 5's first phase where a vertex waits for its sources: rows of one to
several rounds of terms, rows longer than the places a lane can note, chains
through every batch, fewer vertices than warps, and several iterations in work
at once.  Forces against the oracle along the trajectory (FP32 terms: the
bound of the other algo 5 tests); a run of many iterations against the same
iterations one call each, bit for bit."""
import numpy as np
import pytest

import oracle
from test_gpu_greedy_sd import FORCE_TOL, rel_l2

pytestmark = pytest.mark.gpu


def graph(kind):
    from batchlayoutcode_gb300 import graphs as G
    if kind == "star":  # walks of 2,098 sources a leaf
        n = 2100
        u, v = np.zeros(n - 1, np.int64), np.arange(1, n)
    elif kind == "path":
        n = 300
        u, v = np.arange(n - 1), np.arange(1, n)
    elif kind == "few":
        n = 7
        u, v = np.arange(n - 1), np.arange(1, n)
    else:
        g = G.chung_lu(3001, 2.2, 10.0, seed=5)
        return g.rowptr, g.colids
    e = np.unique(np.concatenate([u * n + v, v * n + u]))
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (e % n).astype(np.int32)


@pytest.mark.parametrize("batch", [1, 7, 256])
@pytest.mark.parametrize("kind", ["star", "path", "few", "hubs"])
def test_rows(kind, batch):
    import batchlayoutcode_gb300 as B
    rp, ci = graph(kind)
    n = len(rp) - 1
    xy = np.random.default_rng(n + batch).normal(size=(n, 2)).astype(np.float32).astype(np.float64) * 20
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        e = a.greedy_iteration(batch, 1.0)
        f, x = a.prevCoordinates, a.nCoordinates
        tf, te = oracle.forces_on_trajectory(5, rp, ci, xy, x, batch)
        assert rel_l2(f, tf) <= FORCE_TOL
        assert abs(e - te) / te <= 2 * FORCE_TOL
        for total, first in ((5, 5), (16, 13)):
            a.nCoordinates = xy
            e1 = a.run_resident(5, total, batch, 1.2, 1.0)
            x1 = a.nCoordinates
            a.nCoordinates = xy
            step = 1.0
            for _ in range(first):
                e2 = a.greedy_iteration(batch, step)
                step *= 0.99
            for _ in range(total - first):
                e2 = a.minibatch_iteration(5, batch, step)
                step *= 0.99
            assert np.array_equal(x1, a.nCoordinates)
            assert e1 == e2
