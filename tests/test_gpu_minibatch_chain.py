"""Long all-pairs runs in one launch, where movers run ahead of each other: a
last batch of a few vertices leaves most movers without a target, so they are
done with it while the others still store theirs, and the sweepers must not
take the batch as moved before all of them have.  Sixty iterations in one
launch against sixty launches, bit for bit: a position taken too early stays
in a sweeper's slice for an iteration and changes the forces.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [
    (1025, 512), (1281, 256), (1026, 256), (4099, 256), (7 * 200 + 1, 200), (2051, 1024), (6 * 64 + 3, 64),
    (12 * 384 + 1, 384), (20_481, 256),
])
def test_one_launch_equals_many(n, batch):
    import batchlayoutcode_gb300 as B

    B.build()
    rng = np.random.default_rng(n + batch)
    u, v = rng.integers(0, n, (2, 3 * n))
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep], np.arange(n - 1) * n + np.arange(1, n)]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
    ci = (e % n).astype(np.int32)
    xy = rng.uniform(-30, 30, (n, 2)).astype(np.float32).astype(np.float64)
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        e60 = a.run_resident(2, 60, batch, 1.2, 1.0)
        x60, f60 = a.nCoordinates, a.prevCoordinates
        a.nCoordinates = xy
        step = 1.0
        for _ in range(60):
            e1 = a.minibatch_iteration(2, batch, step)
            step *= 0.999
        assert np.array_equal(x60, a.nCoordinates)
        assert np.array_equal(f60, a.prevCoordinates) and e60 == e1
