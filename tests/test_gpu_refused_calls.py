"""A MIXED estimate that is refused leaves nothing running behind it: the layout may be replaced at once, and an earlier
estimate's results stay.  Three refusals: the knot range and histograms that no CTA size has room for (both before
anything is launched) and histograms that only the smaller CTAs have room for (after the set-up has started)."""
import ctypes as C

import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300 import _capi as capi
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu
BVP = P.BVP.poisson_sincos()
LARGE, SMALL = (8, 31), (3, 7)
N = 2000  # paths per knot: items too long for the smaller CTAs, unless asked for


def rect(nsub, nnode):
    return P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode))


def refuse(pd, **opts):
    with pytest.raises(P.PDDSError) as e:
        pd.estimate(BVP, N, 2e-3, **opts)
    assert e.value.status == capi.ERR_INVALID


def largest_bins(pd):
    """The largest bins_per_gap that 128-thread CTAs have room for: more than 256-thread ones have."""
    lo, hi = 16, 512
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            pd.estimate(BVP, 1, 2e-3, bins_per_gap=mid, cta_threads=128)
            lo = mid
        except P.PDDSError:
            hi = mid
    return lo


def rebuild(pd, nsub, nnode):
    """pd's context with another layout, as the PDDSparseGM of that layout; pd is closed."""
    other = rect(nsub, nnode)
    d = capi.LayoutDesc()
    for q in range(2):
        d.sw[q], d.ne[q] = -1.0, 1.0
    d.nsub, d.nnode = nsub, nnode
    for q, c in enumerate(fac_rule(2.0, nsub, nnode)):
        d.fac[q] = float(c)
    assert pd._lib.pdds_layout_build(pd._ctx, C.byref(d), None) == capi.OK
    other._ctx, pd._ctx = pd._ctx, other._ctx
    pd.close()
    return other


def check_same(pd, ref):
    # the factorisation in the same order on the same layout; every path's value the same
    a = pd.estimate(BVP, 64, 2e-3, mode=P.MODE_REPLAY_FP64, seed=3)
    assert np.array_equal(a.val, ref[0].val) and np.array_equal(a.B, ref[0].B)
    # FP32 sums of at most 256 deposits per bin, in any order: 256 x 2^-24 of weights of at most a few
    b = pd.estimate(BVP, 256, 2e-3, seed=3)
    np.testing.assert_allclose(b.val, ref[1].val, rtol=0, atol=1e-4)
    np.testing.assert_allclose(b.B, ref[1].B, rtol=0, atol=1e-4)


@pytest.mark.parametrize("how", ["range", "all_sizes", "one_size"])
def test_layout_replaced_after_a_refused_estimate(how):
    ref = {}
    for size in (SMALL, LARGE):
        with rect(*size) as pd:
            ref[size] = [pd.estimate(BVP, 64, 2e-3, mode=P.MODE_REPLAY_FP64, seed=3), pd.estimate(BVP, 256, 2e-3, seed=3)]
    pd = rect(*LARGE)
    opts = {"range": dict(knot_first=pd.K), "all_sizes": dict(bins_per_gap=512),
            "one_size": dict(bins_per_gap=largest_bins(pd))}[how]
    for _ in range(3):
        refuse(pd, **opts)
        check_same(pd, ref[LARGE])  # the same layout, with other bins where those were refused
        refuse(pd, **opts)
        pd = rebuild(pd, *SMALL)
        check_same(pd, ref[SMALL])
        pd = rebuild(pd, *LARGE)
    pd.close()


def test_refused_call_keeps_the_last_estimate():
    with rect(*SMALL) as pd:
        pd.estimate(BVP, 256, 2e-3, seed=3)
        u = pd.solve_interface()[0]
        refuse(pd, knot_first=pd.K)
        np.testing.assert_allclose(pd.solve_interface()[0], u, rtol=0, atol=1e-8)  # both solved to 1e-10
