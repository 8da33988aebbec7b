"""A batch's heaviest-first order belongs to the step it was ranked with: another step or adaptive steps rank anew."""
import ctypes as C

import pytest

import pdds_gb300 as P
from pdds_gb300 import _capi as capi
from pdds_gb300.config import batch_instances

pytestmark = pytest.mark.gpu


def test_order_follows_the_step():
    xfer = getattr(capi.load(), "_ZN4pdds4xferEv")  # pdds::xfer(): this thread's copied bytes, to the device first
    xfer.restype, xfer.argtypes = C.POINTER(C.c_int64), []
    with P.Batch(P.BVP.HELMHOLTZ, batch_instances(3, seed=5, grid=(2, 4), nodes=(4, 9))) as b:
        def run(h, adaptive, graph=False):
            at = xfer()[0]
            b.run(256, h, seed=3, adaptive_h=adaptive, use_graph=graph)
            return xfer()[0] - at
        run(2e-3, False)
        assert run(2e-3, False) == 0
        for h, adaptive in ((1e-3, False), (1e-3, True), (2e-3, True), (2e-3, False)):
            assert run(h, adaptive) > 0
            assert run(h, adaptive) == 0
        # a captured run keeps its own order
        for _ in range(2):
            run(2e-3, False, graph=True)
            assert run(1e-3, True) > 0
            assert run(2e-3, False, graph=True) > 0
