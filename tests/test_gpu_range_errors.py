"""Layout runs that end through the device's error status: a force out of range
(two vertices 1e-15 apart, which repel with 5e14) or not a number (a coordinate
that is none).  Every wait of the kernel has to end, the call has to return the
error, no position may be moved by such a force, and the context has to give
the bits of a fresh one afterwards.  The all-pairs kernel with one batch, with
every batch in its ring, with early teams a batch ahead and not, in shares of
several passes, fixed and converged runs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BL_ERR_DEVICE_TIMEOUT = -3

CASES = [(60, 60), (130, 65), (300, 64), (1000, 7), (1025, 256), (3001, 1000), (6000, 2048)]


def layout(n):
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, (2, 2 * n))
    keep = (u != v) & ~np.isin(u, (0, n // 2)) & ~np.isin(v, (0, n // 2))  # the close pair is not joined
    u, v = np.concatenate([u[keep], [1]]), np.concatenate([v[keep], [2]])
    e = np.unique(np.concatenate([u * n + v, v * n + u]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
    xy = rng.uniform(-10, 10, (n, 2)).astype(np.float32).astype(np.float64)
    return rp, (e % n).astype(np.int32), xy


def spoiled(xy, kind):
    bad = xy.copy()
    if kind == "close":
        bad[0] = 0.0
        bad[len(xy) // 2] = 1e-15, 0.0
    else:
        bad[len(xy) // 2, 1] = np.nan
    return bad


@pytest.mark.parametrize("kind", ["close", "nan"])
@pytest.mark.parametrize("n,batch", CASES)
def test_all_pairs(n, batch, kind):
    import batchlayoutcode_gb300 as B

    B.build()
    rp, ci, xy = layout(n)
    bad = spoiled(xy, kind)
    runs = [lambda a: a.minibatch_iteration(2, batch, 1.0), lambda a: a.run_resident(2, 5, batch, 1.2, 1.0),
            lambda a: a.run_resident(7, 2, batch, 1.2, 1.0),
            lambda a: a.cacheBlockingminiBatchForceDirectedAlgorithmConverged(0, 0, batch, 1)]
    with B.Algorithms(rp, ci) as a:
        for run in runs:
            a.nCoordinates = bad
            with pytest.raises(B.BatchLayoutError) as err:
                run(a)
            assert err.value.code == BL_ERR_DEVICE_TIMEOUT
            left = a.nCoordinates
            if kind == "close":
                assert np.isfinite(left).all()
                assert np.array_equal(left[0], bad[0])
            else:  # every force of the first batch is no number: nothing in it moved
                assert np.array_equal(left[:min(batch, n)], bad[:min(batch, n)], equal_nan=True)
        a.nCoordinates = xy
        e = a.run_resident(2, 3, batch, 1.2, 1.0)
        got = a.nCoordinates
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        assert a.run_resident(2, 3, batch, 1.2, 1.0) == e
        assert np.array_equal(a.nCoordinates, got)


@pytest.mark.parametrize("kind", ["close", "nan"])
@pytest.mark.parametrize("n,batch", [(60, 60), (300, 64), (5000, 256)])
def test_greedy(n, batch, kind):
    """Algo 5's first phase: the warps wait for position words that a failed
    warp never writes.  The close pair is joined through two vertices, so that
    a walk reaches one from the other."""
    import batchlayoutcode_gb300 as B

    B.build()
    _, _, xy = layout(n)
    i, j = 0, n // 2
    u = np.concatenate([np.arange(n - 1), [i, 1, j - 1]])
    v = np.concatenate([np.arange(1, n), [1, j - 1, j]])
    keep = ~((u == i) & (v == j))
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
    ci = (e % n).astype(np.int32)
    bad = spoiled(xy, kind)
    with B.Algorithms(rp, ci) as a:
        off, src, _ = a.greedy_walks()
        assert kind == "nan" or j in src[off[i]:off[i + 1]] or i in src[off[j]:off[j + 1]]
        for run in (lambda: a.greedy_iteration(batch, 1.0), lambda: a.run_resident(5, 20, batch, 1.2, 1.0)):
            a.nCoordinates = bad
            start = a.nCoordinates
            with pytest.raises(B.BatchLayoutError) as err:
                run()
            assert err.value.code == BL_ERR_DEVICE_TIMEOUT
            assert np.array_equal(a.nCoordinates, start, equal_nan=True)
        a.nCoordinates = xy
        e1 = a.run_resident(5, 6, batch, 1.2, 1.0)
        got = a.nCoordinates
    with B.Algorithms(rp, ci) as a:
        a.nCoordinates = xy
        assert a.run_resident(5, 6, batch, 1.2, 1.0) == e1
        assert np.array_equal(a.nCoordinates, got)
