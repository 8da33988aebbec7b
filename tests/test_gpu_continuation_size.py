"""Variance-adaptive paths: the continuation's CTA size follows the launch's length (128 threads in long launches), and
either size runs the same paths to the same estimate, up to the order of FP32 sums."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


# 1,296 knots x 5 items: long enough for 128 threads; 16 knots: not; knots with a reflecting side take the longest items
@pytest.mark.parametrize("kind,nsub,nnode", [("poisson", 10, 9), ("poisson", 2, 5), ("robin", 4, 9), ("circle", 5, 9)])
def test_sizes_agree(kind, nsub, nnode):
    if kind == "circle":
        pd, bvp = P.PDDSparseGM.circle_mesh(1.0, nsub, 12, nnode), P.BVP.circle_poisson()
    else:
        pd = P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), nsub, nnode, fac_rule(1.0, nsub, nnode))
        bvp = P.BVP.poisson_sincos() if kind == "poisson" else P.BVP.robin_poisson("W")
    opts = dict(seed=6, adaptive_n=True, npaths_max=20_000, target_stderr=3e-4, richardson=True)
    with pd:
        a, b, c = (pd.estimate(bvp, 256, (1.0 / nsub) ** 2 * 1e-2, cta_threads=th, **opts) for th in (0, 128, 256))
        for e in (b, c):
            assert np.array_equal(a.npaths, e.npaths) and a.npaths.max() > 4096 + 256
            for k in ("path_steps", "exits_global", "exits_stencil"):
                assert a.info[k] == e.info[k]
            # FP32 sums of the same terms in another order (64 products at a time)
            np.testing.assert_allclose(a.val, e.val, rtol=0, atol=64 * 2.0 ** -24)
            np.testing.assert_allclose(a.B, e.B, rtol=0, atol=1e-6 * np.max(np.abs(a.B)))
