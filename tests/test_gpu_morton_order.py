"""The sorted Morton order of the Barnes-Hut tree: keys, vertices and frame,
bit for bit, at the sizes where the tiles, the blocks and the tiles per block
change, and for every length of run of equal high halves (none, inserted by a
thread, sorted by a block in shared memory, sorted through global memory)."""
import numpy as np
import pytest

import batchlayoutcode_gb300 as B

pytestmark = pytest.mark.gpu


def spread(v):
    for s, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F),
                 (2, 0x3333333333333333), (1, 0x5555555555555555)):
        v = (v | (v << np.uint64(s))) & np.uint64(m)
    return v


def reference(xy):
    """MortonCode.h:42-97 in float64; the order is stable in the vertex."""
    lo = xy.min(0)
    mm = (xy.max(0) - lo).max()
    q = (4294967295.0 * (xy - lo) / mm).astype(np.uint64) if mm > 0 else np.zeros(xy.shape, np.uint64)
    key = (spread(q[:, 1]) << np.uint64(1)) | spread(q[:, 0])
    order = np.argsort(key, kind="stable")
    return [lo[0], lo[1], mm], key[order], order


def layout(kind, n, rng):
    if kind == "normal":
        return rng.normal(size=(n, 2)) * 1e3
    if kind == "lattice":  # coincident points: runs of every length, up to thousands
        return np.round(rng.normal(size=(n, 2)) * 8) / 8
    if kind == "cluster":  # a dense third: the runs differ in their low halves
        xy = rng.uniform(-3, 3, (n, 2))
        m = xy[n // 3:2 * n // 3].shape
        xy[n // 3:2 * n // 3] = xy[0] + rng.normal(size=m) * 1e-6
        return xy
    if kind == "line":
        x = rng.uniform(0, 1e-30, n)
        return np.stack([x, x], 1)
    return np.full((n, 2), 7.0)  # one point


# 512 keys a tile up to 304 tiles (two blocks on each of 152 SMs); 16 keys a
# thread and then two tiles a block from 2,490,369 points
@pytest.mark.parametrize("kind", ["normal", "lattice", "cluster", "line", "point"])
@pytest.mark.parametrize("n", [2, 33, 511, 512, 513, 8193, 155648, 155649])
def test_order(kind, n):
    check(kind, n)


@pytest.mark.parametrize("n", [2490368, 2490369])
def test_order_with_more_than_one_tile_a_block(n):
    check("normal", n)


def check(kind, n):
    xy = layout(kind, n, np.random.default_rng(n)).astype(np.float32).astype(np.float64)
    frame, key, order = reference(xy)
    with B.Algorithms(np.zeros(n + 1, np.int32), np.zeros(0, np.int32)) as a:
        a.nCoordinates = xy
        f, k, p = a.morton_order()
    assert list(f[:3]) == frame
    assert np.array_equal(k, key)
    assert np.array_equal(p, order)
