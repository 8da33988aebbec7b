"""The CTA size chosen for short work items: the same paths, and the same estimate up to FP32 summation order, as with the
size forced to either; long items, Richardson pairs with wide sides and forced sizes keep theirs."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsub,nnode,npaths,opts,threads", [
    (6, 15, 5000, {}, 128), (6, 15, 5000, dict(richardson=True, dup_sum=True), 128), (4, 32, 5000, dict(want_var=True), 128),
    (4, 11, 10_000, {}, 256), (6, 15, 10_000, {}, 256), (2, 5, 300, {}, 256)])
def test_chosen_size(nsub, nnode, npaths, opts, threads):
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        bvp = P.BVP.poisson_sincos()
        a = pd.estimate(bvp, npaths, 5e-3, seed=6, **opts)
        assert a.info["cta_threads"] == threads
        for th in (128, 256):
            b = pd.estimate(bvp, npaths, 5e-3, seed=6, cta_threads=th, **opts)
            assert b.info["cta_threads"] == th
            for k in ("path_steps", "exits_global", "exits_stencil"):
                assert a.info[k] == b.info[k]
            # FP32 sums of the same terms in another order (64 products at a time)
            np.testing.assert_allclose(a.val, b.val, rtol=0, atol=64 * 2.0 ** -24)
            np.testing.assert_allclose(a.B, b.B, rtol=0, atol=1e-6 * np.max(np.abs(a.B)))


@pytest.mark.parametrize("circle", [False, True])
def test_continuation_size(circle):
    """Variance-adaptive paths: the continuation's own CTA size, the same paths."""
    opts = dict(seed=6, adaptive_n=True, npaths_max=20_000, target_stderr=4e-3, richardson=True, adaptive_h=True)
    pd = P.PDDSparseGM.circle_mesh(1.0, 3, 8, 7) if circle else \
        P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), 3, 7, fac_rule(2.0, 3, 7))
    with pd:
        bvp = P.BVP.circle_poisson() if circle else P.BVP.poisson_sincos()
        a = pd.estimate(bvp, 500, 2e-3, **opts)
        b = pd.estimate(bvp, 500, 2e-3, cta_threads=256, **opts)
        assert np.array_equal(a.npaths, b.npaths) and a.npaths.max() > 4096 + 500
        assert a.info["path_steps"] == b.info["path_steps"]
        # FP32 sums of the same terms in another order (64 products at a time)
        np.testing.assert_allclose(a.val, b.val, rtol=0, atol=64 * 2.0 ** -24)
