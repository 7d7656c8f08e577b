"""The network's gradient where the per-block partials fill one, more than one
and all rows of the reduction (256 rows a step, 608 blocks of 128 vertices on
152 SMs), with the last tile part empty.  Against the CPU oracle with the
tolerances of the other network tests."""
import numpy as np
import pytest

from oracle import mpnn as M
from test_gpu_mpnn_rows import rel, rows_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32768, 32769, 77833])
def test_gradient(n):
    from batchlayoutcode_gb300 import _lib
    rp, ci = rows_graph(n, [3, 0, 5], n)
    rng = np.random.default_rng(n)
    feats = rng.normal(size=(n, M.FEATURES)).astype(np.float32)
    p = M.init_params(2)
    p[-130:] += rng.normal(0, 0.1, 130).astype(np.float32)
    target = rng.normal(size=(n, 2)).astype(np.float32)
    w = np.full(n, 1.0 / n, np.float32)
    with _lib.Mpnn(p) as net:
        out = net.run(rp, ci, feats, target=target, vweight=w)
    ref = M.forward(p, rp, ci, feats, mimic=True)
    assert rel(out["xy"], ref["xy"]) <= 1e-2
    loss, grad, _ = M.loss_and_grad(p, rp, ci, feats, target, w, mimic=True)
    assert abs(out["loss"] - loss) <= 1e-3 * loss
    o = 0
    for name, size in [("W1", 2048), ("b1", 64), ("W2", 8192), ("b2", 64), ("W3", 8192), ("b3", 64), ("Wo", 128),
                       ("bo", 2)]:
        assert rel(out["grad"][o:o + size], grad[o:o + size]) <= 2e-2, name
        o += size
