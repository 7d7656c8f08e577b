"""Ids outside 0 .. n - 1 in the neighbour lists handed to the allocation-free
entry point: they are skipped.  The same lists without them give the same
forces but for the order of a row's float-float sum (2^-47 of the largest
term a step, far inside the 1e-6 asked for), on the forms of the kernel with
and without a batch before it.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(50, 50), (100, 7), (520, 256), (1000, 64), (3001, 200)])
def test_foreign_ids_are_skipped(n, batch):
    torch = pytest.importorskip("torch")
    import batchlayoutcode_gb300 as B
    from batchlayoutcode_gb300 import _lib

    B.build()
    L = _lib.load()
    rng = np.random.default_rng(n)
    rows = [np.unique(rng.integers(0, n, 12)) for _ in range(n)]
    foreign = np.array([-2**31, -n - 3, -1, n, n + 1, n + batch, 2**30, 2**31 - 1], np.int64)
    padded = [np.sort(np.concatenate([r, rng.choice(foreign, 1 + i % 5, replace=False)])) for i, r in enumerate(rows)]
    xy = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    dev = torch.device("cuda:0")
    out = []
    for lists in (rows, padded):
        rp = np.concatenate([[0], np.cumsum([len(r) for r in lists])]).astype(np.int32)
        d_rp = torch.from_numpy(rp).to(dev)
        d_ci = torch.from_numpy(np.concatenate(lists).astype(np.int32)).to(dev)
        d_xy = torch.from_numpy(xy).to(dev)
        d_f = torch.zeros((n, 2), dtype=torch.float64, device=dev)
        d_e = torch.zeros(n, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        e = C.c_double()
        rc = L.bl_minibatch_iteration_noalloc(n, d_rp.data_ptr(), d_ci.data_ptr(), d_xy.data_ptr(), d_f.data_ptr(),
                                              d_e.data_ptr(), 2, batch, 1.0, 0.5, C.byref(e),
                                              torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        out.append((d_f.cpu().numpy(), d_xy.cpu().numpy(), e.value))
    (f0, x0, e0), (f1, x1, e1) = out
    assert np.linalg.norm(f1 - f0) <= 1e-6 * np.linalg.norm(f0)
    assert np.abs(x1 - x0).max() <= 1e-5 and abs(e1 - e0) <= 2e-6 * e0
