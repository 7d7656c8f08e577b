"""The batched layout's two block sizes: sets of graphs whose schedule takes
the larger block, and the same graphs among so many copies that it takes the
smaller one.  Positions are equal bit for bit (every sum of a vertex keeps its
order); the energies' sums over threads differ by rounding (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo,sizes,copies", [
    (2, [3, 60, 257, 400], 600),      # all pairs, smaller than a block's threads, edges of a batch
    (4, [5003, 6100, 4097], 400),     # Barnes-Hut, edges of the sort's tiles (4,096 and 8,192 keys)
    (4, [16390, 2], 400),
])
def test_block_sizes_agree(algo, sizes, copies):
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import graphs as G
    gs, xy = [], []
    for k, n in enumerate(sizes):
        u, v = np.arange(n - 1), np.arange(1, n)
        if n > 100:
            g = G.random_geometric(n, 6.0, seed=k)
            rp, ci = g.rowptr, g.colids
        else:
            e = np.unique(np.concatenate([u * n + v, v * n + u]))
            rp = np.concatenate([[0], np.cumsum(np.bincount(e // n, minlength=n))]).astype(np.int32)
            ci = (e % n).astype(np.int32)
        gs.append((rp, ci))
        xy.append(np.random.default_rng(k).normal(size=(len(rp) - 1, 2)).astype(np.float32).astype(np.float64) * 9)

    def run(m):
        with B.BatchedLayout(gs * m, algo, xy * m) as bl:
            bl.set_parts([2, 2, 2])
            bl.run(2, 256, 1.2)
            return bl.result()

    x1, e1 = run(1)
    x2, e2 = run(copies)
    for k in range(len(gs)):
        for c in (0, copies - 1):
            assert np.array_equal(x1[k], x2[c * len(gs) + k])
            assert abs(e1[k] - e2[c * len(gs) + k]) <= 1e-12 * abs(e1[k])
