"""Rows of every length in a Barnes-Hut iteration: unmoved neighbours added by
a thread or by a warp, neighbours that moved in earlier batches taken four at
a time.  The batched layout adds both in order with one thread a vertex, so
positions are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(n, kind, rng):
    u, v = [np.arange(n - 1)], [np.arange(1, n)]
    if kind == "unmoved":  # long rows at the first ids: their neighbours come later
        rows = [(k, d) for k, d in enumerate([31, 32, 33, 34, 63, 64, 65, 96, 97, 700] * 4)]
        lo = n // 2
    elif kind == "moved":  # long rows at the last ids: their neighbours moved before
        rows = [(n - 1 - k, d) for k, d in enumerate([1, 2, 3, 4, 5, 7, 8, 9, 40, 300] * 4)]
        lo = 0
    else:  # both, anywhere
        rows = [(int(k), int(d)) for k, d in zip(rng.permutation(n)[:200], rng.integers(1, 200, 200))]
        lo = 0
    for k, d in rows:
        u.append(np.full(d, k))
        v.append(lo + rng.permutation(n // 2)[:d])
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (e % n).astype(np.int32)


@pytest.mark.parametrize("batch", [7, 256])
@pytest.mark.parametrize("n", [1500, 5003])
@pytest.mark.parametrize("kind", ["unmoved", "moved", "both"])
def test_rows(kind, n, batch):
    import batchlayoutcode_gb300 as B
    rng = np.random.default_rng(n + batch)
    g = graph(n, kind, rng)
    xy = rng.normal(size=(n, 2)).astype(np.float32).astype(np.float64) * 10
    with B.BatchedLayout([g], 4, [xy]) as bl:
        bl.run(2, batch, 1.2)
        xs, es = bl.result()
    with B.Algorithms(*g) as a:
        a.nCoordinates = xy
        a.barnes_hut_iteration(batch, 1.2, 1.0)
        e = a.barnes_hut_iteration(batch, 1.2, 0.999)
        assert np.array_equal(a.nCoordinates, xs[0])
    assert abs(e - es[0]) <= 1e-12 * e
