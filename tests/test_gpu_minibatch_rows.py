"""Row lengths of the all-pairs kernel's neighbour corrections at the edges of
their forms: rows a lane walks, rows whose entries the warps share evenly (64
at a time, several rows among them or one), enough of them for the second team
to join, empty rows among them, more neighbours in the batch before than are
staged, ids behind the end of a list; tiles of several passes; mean lengths
from which the launch shape looks at rows.  One iteration against the FP64
oracle on the device's own trajectory (forces 1e-5 relative L2, the tolerance
of the other parity tests), and three iterations in one launch against three
launches, bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5

CASES = [  # vertices, batch, row lengths in turn
    (700, 64, [3, 35, 36, 37]), (700, 64, [1, 63, 2, 64, 3, 65]), (900, 256, [127, 128, 129, 1]),
    (900, 256, [2] * 40 + [600]), (1500, 256, [2] * 31 + [449]), (1500, 256, [5] * 7 + [1000, 30]),
    (1031, 37, [4, 90, 1, 200]), (1500, 511, [1, 400]), (1200, 256, [150]), (1200, 64, [99, 101]),
    (2000, 1000, [250, 1]), (3001, 256, [2] * 255 + [3000]), (2300, 2048, [3] * 63 + [900]), (4500, 4096, [120]),
    (300, 300, [299, 20]), (520, 256, [40]),
]


def rows_graph(n, lengths, seed):
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(n):
        k = min(lengths[i % len(lengths)], n)
        # half of the long rows lie close by: many of one batch
        near = np.arange(i - k // 2, i + k - k // 2) % n
        rows.append(np.unique(near if i % 2 and k > 8 else rng.choice(n, k, replace=False)))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return rp, np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("case", range(len(CASES)))
def test_rows(case):
    import batchlayoutcode_gb300 as B

    B.build()
    n, batch, lengths = CASES[case]
    rp, ci = rows_graph(n, lengths, case)
    xy = np.random.default_rng(n + 1).uniform(-20, 20, (n, 2)).astype(np.float32).astype(np.float64)
    with B.Algorithms(rp, ci) as a:
        for model in (2, 3, 7):
            a.nCoordinates = xy
            e = a.minibatch_iteration(model, batch, 0.7)
            f, x1 = a.prevCoordinates, a.nCoordinates
            tf, te = oracle.forces_on_trajectory(model, rp, ci, xy, x1, batch)
            assert np.linalg.norm(f - tf) <= FORCE_TOL * np.linalg.norm(tf)
            assert abs(e - te) <= 2 * FORCE_TOL * te
        a.nCoordinates = xy
        e3 = a.run_resident(2, 3, batch, 1.2, 1.0)
        x3, f3 = a.nCoordinates, a.prevCoordinates
        a.nCoordinates = xy
        step = 1.0
        for _ in range(3):
            e1 = a.minibatch_iteration(2, batch, step)
            step *= 0.999
        assert np.array_equal(x3, a.nCoordinates) and np.array_equal(f3, a.prevCoordinates) and e3 == e1


@pytest.mark.parametrize("n,batch,lengths", [(600, 64, [0, 0, 70, 1, 0, 200]), (900, 256, [0, 3, 0, 36]),
                                             (500, 200, [0] * 30 + [450]), (400, 256, [130, 0])])
def test_empty_rows_and_foreign_ids(n, batch, lengths):
    """Lists handed in on the device: empty rows stay empty, ids outside the
    graph are skipped; against the sums in FP64 over the first batch, whose
    forces all use the start."""
    torch = pytest.importorskip("torch")
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import _lib

    B.build()
    L = _lib.load()
    rng = np.random.default_rng(n)
    rows = [np.unique(rng.choice(n, min(lengths[i % len(lengths)], n), replace=False)) for i in range(n)]
    lists = [np.concatenate([r, [n + i % 3, 2**30]]) if i % 4 == 0 and len(r) else r for i, r in enumerate(rows)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in lists])]).astype(np.int32)
    xy = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    dev = torch.device("cuda:0")
    d_rp, d_ci = torch.from_numpy(rp).to(dev), torch.from_numpy(np.concatenate(lists).astype(np.int32)).to(dev)
    d_xy = torch.from_numpy(xy).to(dev)
    d_f, d_e = torch.zeros((n, 2), dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    e = C.c_double()
    assert 0 == L.bl_minibatch_iteration_noalloc(n, d_rp.data_ptr(), d_ci.data_ptr(), d_xy.data_ptr(), d_f.data_ptr(),
                                                 d_e.data_ptr(), 2, batch, 1.0, 0.5, C.byref(e),
                                                 torch.cuda.current_stream().cuda_stream)
    p = xy.astype(np.float64)
    want = np.zeros((batch, 2))
    for i in range(batch):
        d = p - p[i]
        d2 = (d * d).sum(1)
        sc = np.where(d2 > 0, -1.0 / np.where(d2 > 0, d2, 1.0), 0.0)
        sc[rows[i]] = np.sqrt(d2[rows[i]])
        want[i] = (d * sc[:, None]).sum(0)
    got = d_f.cpu().numpy()[:batch]
    assert np.linalg.norm(got - want) <= FORCE_TOL * np.linalg.norm(want)
