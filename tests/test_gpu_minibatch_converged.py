"""The end of a converged all-pairs run (-engt): the movers learn at the end of
an iteration that no batch follows, while the sweepers and the movers' own
early teams may be at work on batches past it.  One batch (no batch before
it), two to four (every batch in the ring), odd batches, one mover, several:
the run must end with the loop count, energy, forces and positions of the same
number of single iterations, bit for bit, every time.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THRESHOLD = 0.1


@pytest.mark.parametrize("n,batch", [
    (40, 256), (200, 200), (1000, 1000), (130, 65), (193, 65), (200, 50), (257, 64), (1023, 256), (1537, 511),
    (60, 7), (300, 8), (700, 1), (3001, 256),
])
def test_converged_run_ends(n, batch):
    import batchlayoutcode_gb300 as B

    B.build()
    rng = np.random.default_rng(n + batch)
    u, v = np.concatenate([rng.integers(0, n, (2, n)), [np.arange(n - 1), np.arange(1, n)]], 1)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
    ci = (e % n).astype(np.int32)
    xy = rng.uniform(-10, 10, (n, 2)).astype(np.float32).astype(np.float64)
    with B.Algorithms(rp, ci, th=THRESHOLD) as a:
        a.nCoordinates = xy
        e0, e1, step, loops = np.finfo(np.float64).max, 0.0, 1.0, 0
        while (abs(e0 - e1) / e0 if e0 else np.inf) > THRESHOLD:
            e0, e1 = e1, a.minibatch_iteration(2, batch, step)
            step *= 0.999
            loops += 1
            assert loops < 2000
        x1, f1 = a.nCoordinates, a.prevCoordinates
        for _ in range(10):
            a.nCoordinates = xy
            energy, _ = a.cacheBlockingminiBatchForceDirectedAlgorithmConverged(0, 0, batch, 1)
            assert a.loops == loops and energy == e1
            assert np.array_equal(a.nCoordinates, x1) and np.array_equal(a.prevCoordinates, f1)
