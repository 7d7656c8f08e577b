"""Hop distances of the learned initializer's features in every form of the
search: one block per pivot with visited bits in shared memory, the same with
a graph too large for them, the give-up when a frontier outgrows a block's
queue, the device-wide search for long rows, and a training set that mixes
the forms.  Distances are whole numbers: equal to scipy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def csr(n, u, v):
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (e % n).astype(np.int32)


def lattice(rows, cols):
    i = np.arange(rows * cols, dtype=np.int64).reshape(rows, cols)
    return (np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()]))


def make(kind):
    rng = np.random.default_rng(3)
    if kind == "line":  # one vertex a level
        n = 3000
        return csr(n, np.arange(n - 1), np.arange(1, n))
    if kind == "two-lattices":  # unreachable pivots; odd row lengths
        u, v = lattice(40, 33)
        w, x = lattice(17, 90)
        return csr(40 * 33 + 17 * 90 + 5, np.concatenate([u, w + 40 * 33]), np.concatenate([v, x + 40 * 33]))
    if kind == "rows-of-64":  # the longest row the block form takes, 17 entries at least
        n = 4000
        off = np.arange(1, 33)
        u = np.repeat(np.arange(n), 32)
        return csr(n, u, (u + np.tile(off, n)) % n)
    if kind == "rows-of-66":  # the shortest rows it does not
        n = 4000
        u = np.repeat(np.arange(n), 33)
        return csr(n, u, (u + np.tile(np.arange(1, 34), n)) % n)
    if kind == "expander":  # rows of about 6: frontiers beyond a block's queue
        n = 120_000
        return csr(n, rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n))
    u, v = lattice(1201, 1103)  # 1.32 million vertices: more than the shared visited bits
    return csr(1201 * 1103, u, v)


def distances(rp, ci, pivots):
    import scipy.sparse as sp
    from scipy.sparse.csgraph import dijkstra
    n = len(rp) - 1
    A = sp.csr_matrix((np.ones(len(ci), np.int8), ci, rp), shape=(n, n))
    d = dijkstra(A, unweighted=True, indices=pivots).T
    return np.where(np.isinf(d), 0xFFFF, np.minimum(d, 65534)).astype(np.uint16)


@pytest.mark.parametrize("kind", ["line", "two-lattices", "rows-of-64", "rows-of-66", "expander", "large"])
def test_hop_distances(kind):
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import _lib

    B.build()
    rp, ci = make(kind)
    with _lib.Mpnn() as net:
        _, d, pv = net.features(rp, ci, seed=5)
    check = range(16) if kind != "large" else (0, 7)
    assert np.array_equal(d[:, list(check)], distances(rp, ci, pv[list(check)]))


def test_training_set_of_both_forms():
    """A set with block-form and device-wide graphs trains as its graphs do
    alone in the part the distances decide: the same features give the same
    first loss as the mean over single-graph sets."""
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import _lib, learned

    B.build()
    params, _ = learned.load_model()
    sets = [make("rows-of-66"), make("line"), make("two-lattices")]
    rng = np.random.default_rng(8)
    lays = [rng.normal(size=(len(rp) - 1, 2)) for rp, _ in sets]
    first = []
    for k, (g, lay) in enumerate(zip(sets, lays)):
        with _lib.Mpnn(params) as net:
            first.append(net.train([g], [lay], 1, 1e-4, seed=1 + k)[2][0])
    with _lib.Mpnn(params) as net:
        both = net.train(sets, lays, 1, 1e-4, seed=1)[2][0]
    # FP32 sums of the same per-vertex losses (two products each way of a
    # weight 1/n against 1/(3 n)): a few units of 2^-24
    assert abs(both - np.mean(first)) <= 1e-6 * abs(both)
