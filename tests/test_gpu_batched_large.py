"""A set with an all-pairs graph so large that its shared memory leaves an SM
one block, beside Barnes-Hut graphs: the Barnes-Hut graphs' positions are those
of a set that takes two blocks an SM, bit for bit, and the large graph's are
those of the single-graph path within its FP32 sums' rounding (1e-5 of a step)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_graph_beside_small_ones():
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import graphs as G

    B.build()
    big, small = G.random_geometric(14_200, 6.0, seed=1), G.random_geometric(3000, 6.0, seed=2)
    xb = np.random.default_rng(1).uniform(-60, 60, (big.n, 2)).astype(np.float32).astype(np.float64)
    xs = np.random.default_rng(2).uniform(-25, 25, (small.n, 2)).astype(np.float32).astype(np.float64)
    gb, gs = (big.rowptr, big.colids), (small.rowptr, small.colids)

    def run(graphs, algo, xy, iterations):
        with B.BatchedLayout(graphs, algo, xy) as bl:
            bl.set_parts([2, 2, 2])
            bl.run(iterations, 256, 1.2)
            return bl.result()

    x1, _ = run([gb] + [gs] * 3, [2, 4, 4, 4], [xb] + [xs] * 3, 1)
    x2, _ = run([gs] * 700, 4, [xs] * 700, 1)
    for k in (1, 3):
        assert np.array_equal(x1[k], x2[0]) and np.array_equal(x1[k], x2[699])
    with B.Algorithms(*gb) as a:
        a.nCoordinates = xb
        a.minibatch_iteration(2, 256, 1.0)
        assert np.abs(a.nCoordinates - x1[0]).max() <= 1e-4
        assert np.linalg.norm(a.nCoordinates - x1[0]) <= 1e-5 * np.linalg.norm(x1[0] - xb)
