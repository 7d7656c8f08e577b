"""The network's gathers at the row lengths where their form changes: empty
rows, one entry, 8 / 9 and 16 / 17 (the entries loaded at a time), 64 / 65 (the
longest row one group sums) and rows of thousands, in graphs with and without
long rows, with vertex counts that leave tiles part empty.  Against the CPU
oracle with the tolerances of the other network tests."""
import numpy as np
import pytest

from oracle import mpnn as M

pytestmark = pytest.mark.gpu


def rows_graph(n, lengths, seed):
    """Symmetric graph in which vertex k has about lengths[k % len] entries."""
    rng = np.random.default_rng(seed)
    want = np.array([lengths[k % len(lengths)] for k in range(n)])
    hubs = np.flatnonzero(want > 20)
    u, v = [], []
    for h in hubs:  # the long rows exactly, to vertices that are none
        others = np.setdiff1d(np.arange(n), hubs)
        v.append(rng.choice(others, min(want[h], len(others)), replace=False))
        u.append(np.full(len(v[-1]), h))
    small = np.flatnonzero((want > 0) & (want <= 20))
    u.append(np.repeat(small, (want[small] + 1) // 2))
    v.append(rng.choice(small, len(u[-1])))
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rp[1:])
    return rp.astype(np.int32), (e % n).astype(np.int32)


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n,lengths", [
    (1, [0]), (2, [1]), (127, [0, 1, 2]), (129, [8, 9]), (300, [16, 17, 3]), (1000, [64, 5, 5, 5, 5, 5, 0]),
    (1000, [65, 5, 5, 5, 5, 5, 0]), (4097, [3] * 1500 + [3000, 129, 64, 65, 66]),
])
def test_row_lengths(n, lengths):
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import _lib

    B.build()
    rp, ci = rows_graph(n, lengths, n)
    rng = np.random.default_rng(n + 1)
    feats = rng.normal(size=(n, M.FEATURES)).astype(np.float32)
    p = M.init_params(2)
    p[-130:] += rng.normal(0, 0.1, 130).astype(np.float32)
    target = rng.normal(size=(n, 2)).astype(np.float32)
    w = np.full(n, 1.0 / n, np.float32)
    with _lib.Mpnn(p) as net:
        out = net.run(rp, ci, feats, target=target, vweight=w, want_h=True)
    ref = M.forward(p, rp, ci, feats, mimic=True)
    h1 = (out["h"][0].astype(np.uint32) << 16).view(np.float32)
    assert np.mean(h1 == ref["h"][0].astype(np.float32)) >= 0.99
    assert rel(out["xy"], ref["xy"]) <= 1e-2
    loss, grad, _ = M.loss_and_grad(p, rp, ci, feats, target, w, mimic=True)
    assert abs(out["loss"] - loss) <= 1e-3 * loss
    o = 0
    for name, size in [("W1", 2048), ("b1", 64), ("W2", 8192), ("b2", 64), ("W3", 8192), ("b3", 64), ("Wo", 128),
                       ("bo", 2)]:
        assert rel(out["grad"][o:o + size], grad[o:o + size]) <= 2e-2, name
        o += size
