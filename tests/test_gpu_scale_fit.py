"""The scale of the learned start: with the positions p it leaves, the factor
that would minimise sum |k^2 A - R|^2 again (A the attraction, R the
Barnes-Hut repulsion at p) is 1.  Rows of none, a few, more than a warp's
entries at a time (192) and thousands; vertex counts at the edges of a warp's
32 rows and a block's 256.  A in float64 from the float32 positions, whose
rounding moves an edge's length by about 1e-5: bound 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(n, hubs):
    rng = np.random.default_rng(n)
    u, v = [np.arange(n - 1)], [np.arange(1, n)]
    if n > 64:
        u.append(rng.integers(0, n, 2 * n))
        v.append(rng.integers(0, n, 2 * n))
    for k, d in enumerate(hubs):
        u.append(np.full(d, 5 * k))
        v.append(rng.permutation(n)[:d])
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    e = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (e % n).astype(np.int32)


@pytest.mark.parametrize("n,hubs", [(3, []), (31, []), (256, [100]), (257, [191, 192, 193]),
                                    (5000, [3000, 385, 64])])
def test_scale_is_a_fixed_point(n, hubs):
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import learned as LR
    rp, ci = graph(n, hubs)
    _, sm = LR.load_model()
    with B.Algorithms(rp, ci, init=0) as a:
        a.learnedInit(np.zeros_like(LR.init_params(0)), sm)
        p = a.nCoordinates
        R, _ = a.bh_repulsion(1.2)
    r = np.repeat(np.arange(n), np.diff(rp))
    d = p[ci] - p[r]
    t = np.hypot(d[:, 0], d[:, 1])[:, None] * d
    A = np.stack([np.bincount(r, t[:, k], minlength=n) for k in range(2)], 1)
    k2 = (A * R).sum() / (A * A).sum()
    assert abs(k2 - 1.0) <= 1e-4
