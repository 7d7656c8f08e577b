"""The training set of the learned initializer on the device: joined edges,
mean edge lengths and fitted targets, for graphs at the edges of a chunk (512
vertices) and of the MDS kernels' blocks and slices (256 vertices, 64 graphs),
rotated and mirrored targets, long and empty rows.  An untrained network's
output is zero, so its loss is the mean square of the targets, which numpy
forms in float64 (targets and weights are rounded to float32: three roundings
of 6e-8 a term, 1e-5 with the sum's); the scale model is float64 throughout
(1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(n, rng):
    u = [np.arange(n - 1)]
    v = [np.arange(1, n)]
    if n > 300:
        u += [np.zeros(200, int), rng.integers(0, n - 2, n)]
        v += [rng.integers(1, n - 2, 200), rng.integers(0, n - 2, n)]
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (e % n).astype(np.int32)


def fit(y, t):
    t = t - t.mean(0)
    u, _, vt = np.linalg.svd(t.T @ y)
    r = t @ (u @ vt)
    return r * ((r * y).sum() / (r * r).sum()) - y


@pytest.mark.parametrize("sizes", [[511, 512, 513], [255, 256, 257, 1025, 3], [5] * 65 + [700]])
def test_targets(sizes):
    from batchlayoutcode_gb300 import learned as LR
    from batchlayoutcode_gb300._lib import Mpnn
    rng = np.random.default_rng(len(sizes))
    gs = [graph(n, rng) for n in sizes]
    lays, want, rows = [], 0.0, []
    with Mpnn(LR.init_params(0)) as net:
        for g, (rp, ci) in enumerate(gs):
            n = len(rp) - 1
            y = net.features(rp, ci, seed=7 + g)[0][:, :2].astype(np.float64)
            a = rng.uniform(0, 6.28)
            rot = np.array([[np.cos(a), -np.sin(a)], [np.sin(a), np.cos(a)]]) @ np.diag([1, 1 if g % 2 else -1])
            xy = (y @ rot + 0.3 * rng.normal(size=y.shape)) * 37.0 + 1000.0
            lays.append(xy)
            want += (fit(y, xy) ** 2).sum() / n / len(gs)
            r = np.repeat(np.arange(n), np.diff(rp))
            d = xy[r] - xy[ci]
            rows.append([1.0, np.log(n), np.log(len(ci) / n), np.log(np.hypot(d[:, 0], d[:, 1]).mean())])
        _, sm, hist = net.train(gs, lays, 1, 1e-3, 7)
        assert abs(hist[0] - want) <= 1e-5 * want
        r = np.array(rows)
        A = r[:, :3].T @ r[:, :3]
        A += np.eye(3) * 1e-9 * (A[0, 0] + 1.0)
        assert np.allclose(A @ sm, r[:, :3].T @ r[:, 3], rtol=1e-9, atol=1e-9 * len(gs))


def test_colid_out_of_range_is_refused():
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import learned as LR
    rng = np.random.default_rng(1)
    gs = [graph(600, rng), graph(513, rng)]
    lays = [rng.normal(size=(len(rp) - 1, 2)) for rp, _ in gs]
    from batchlayoutcode_gb300._lib import Mpnn
    with Mpnn(LR.init_params(0)) as net:
        for bad in (-1, 513, 2147483647):
            ci = gs[1][1].copy()
            ci[-1] = bad
            with pytest.raises(B.BatchLayoutError, match="colid out of range"):
                net.train([gs[0], (gs[1][0], ci)], lays, 1, 1e-3, 7)
        net.train(gs, lays, 1, 1e-3, 7)  # the context is usable
