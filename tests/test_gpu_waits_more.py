"""The Morton sort's grid barrier and the all-pairs movers' wait for a count end
in an error code when their arrival is withheld (a block that never arrives, a
count that nothing adds to): after about their limit of 2 s of %globaltimer the
call reports BL_ERR_DEVICE_TIMEOUT and the context gives the bits of a fresh
one.  With the arrival made the same call returns at once.
"""
import time

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

BL_ERR_DEVICE_TIMEOUT = -3
LIMIT_S = 2.0


@pytest.mark.parametrize("site", [2, 3])
def test_withheld_arrival(site):
    import batchlayoutcode_gb300 as B

    B.build()
    z = load_golden("grid12")
    rp, ci, xy = z["csr_rowptr"], z["csr_colids"], z["init_xy"]

    def layout(a):
        a.nCoordinates = xy
        e = a.minibatch_iteration(2, 32, 1.0), a.barnes_hut_iteration(32, 1.2, 0.9)
        return e, a.nCoordinates

    with B.Algorithms(rp, ci) as a:
        L, ctx = a._L, a._ctx
        assert L.bl_wait_selftest(ctx, site, 1) == 0  # (loads the kernel)
        t0 = time.perf_counter()
        assert L.bl_wait_selftest(ctx, site, 1) == 0
        assert time.perf_counter() - t0 < 0.5 * LIMIT_S
        t0 = time.perf_counter()
        assert L.bl_wait_selftest(ctx, site, 0) == BL_ERR_DEVICE_TIMEOUT
        assert 0.9 * LIMIT_S <= time.perf_counter() - t0 <= LIMIT_S + 10.0
        assert "timed out" in L.bl_last_error(ctx).decode()
        assert L.bl_wait_selftest(ctx, site, 1) == 0
        e, got = layout(a)
    with B.Algorithms(rp, ci) as a:
        e1, x1 = layout(a)
        assert e == e1 and np.array_equal(got, x1)
