"""The all-pairs minibatch kernel at the edges of its launch shapes.

Its blocks, lag and buffers follow from the vertex count and the batch size:
one batch (no batch before it), two to four batches (every batch in the
movers' ring, or just not), odd batches and vertex counts, shares of less
than one target and of several passes, a last batch of one vertex, rows with
more neighbours in the batch before than are staged.  Each case is one
iteration against the FP64 oracle on the device's own trajectory (forces
1e-5 relative L2, the tolerance of the other parity tests), and three
iterations in one launch against three launches, bit for bit.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5

CASES = [  # vertices, batch
    (1, 256), (2, 1), (5, 7), (9, 2), (33, 33), (65, 64), (128, 64), (131, 64), (192, 64), (193, 64), (257, 64),
    (300, 37), (511, 128), (513, 512), (1000, 1), (1025, 256), (1537, 511), (2000, 1999), (3001, 1000),
    (4100, 2048), (5000, 4096), (8200, 2048), (12289, 4096),
]


def graph(n, seed):
    """Random sparse rows plus one vertex joined to everyone (its row overflows
    the staged neighbours of the batch before, and so do its neighbours' twins)."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n, 3 * n)
    v = rng.integers(0, n, 3 * n)
    hub = n // 2
    u = np.concatenate([u, np.full(n, hub), np.arange(n - 1)])
    v = np.concatenate([v, np.arange(n), np.arange(1, n)])
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rows, cols = e // n, e % n
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), cols.astype(np.int32)


@pytest.mark.parametrize("n,batch", CASES)
def test_launch_shapes(n, batch):
    import batchlayoutcode_gb300 as B

    B.build()
    rp, ci = graph(n, n)
    xy = np.random.default_rng(n + 1).uniform(-20, 20, (n, 2)).astype(np.float32).astype(np.float64)
    model = (2, 3, 8)[n % 3]
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        e = a.minibatch_iteration(model, batch, 0.7)
        f, x1 = a.prevCoordinates, a.nCoordinates
        tf, te = oracle.forces_on_trajectory(model, rp, ci, xy, x1, batch)
        assert np.linalg.norm(f - tf) <= FORCE_TOL * max(np.linalg.norm(tf), 1e-30)
        assert abs(e - te) <= 2 * FORCE_TOL * te
        a.nCoordinates = xy
        e3 = a.run_resident(2, 3, batch, 1.2, 1.0)
        x3, f3 = a.nCoordinates, a.prevCoordinates
        a.nCoordinates = xy
        step = 1.0
        for _ in range(3):
            e1 = a.minibatch_iteration(2, batch, step)
            step *= 0.999
        assert np.array_equal(x3, a.nCoordinates) and np.array_equal(f3, a.prevCoordinates) and e3 == e1
