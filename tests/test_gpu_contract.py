"""The contraction of the exit histograms into G: side lengths around its column tiles (32 to 160 columns), knots in and
out of its 32-row tiles, one and several work items per knot, with and without variances, and split launches.

Histogram cells and product sums are FP32 sums of at most some tens of terms (error at most 64 * 2^-24 of their sum,
about one here: weights of cardinal functions times probabilities), so two runs of the same paths differ by that at
most."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu
ATOL = 64 * 2.0 ** -24


@pytest.mark.parametrize("nsub,nnode", [(2, 4), (3, 5), (3, 17), (3, 18), (2, 33), (3, 34), (3, 50), (3, 44), (3, 54)])
def test_rows_agree_over_tilings(nsub, nnode):
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        bvp = P.BVP.poisson_sincos()
        N = 1500
        a = pd.estimate(bvp, N, 2e-3, seed=7)
        v = pd.estimate(bvp, N, 2e-3, seed=7, want_var=True)  # the other tile
        np.testing.assert_allclose(v.val, a.val, rtol=0, atol=ATOL)
        first = min(3, pd.n_mc - 1)
        part = pd.estimate(bvp, N, 2e-3, seed=7, knot_first=first, knot_count=1, want_var=True)  # other items
        rows = np.flatnonzero(part.npaths)
        assert rows.size == 1
        r0, r1 = a.row_ptr[rows[0]], a.row_ptr[rows[0] + 1]
        np.testing.assert_allclose(part.val[r0:r1], a.val[r0:r1], rtol=0, atol=ATOL)
        np.testing.assert_allclose(part.var[r0:r1], v.var[r0:r1], rtol=0, atol=4 * ATOL)
        # the exits' own weights (no histogram) on the same paths, of which a few per knot exit a step apart in FP32
        f = pd.estimate(bvp, N, 2e-3, seed=7, mode=P.MODE_FP64)
        b = pd.estimate(bvp, N, 2e-3, seed=7, bins_per_gap=64)
        np.testing.assert_allclose(b.val, f.val, rtol=0, atol=4.0 / N)


def test_split_launches_match_one():
    """Histograms beyond the scratch bound: the knots in several launches."""
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), 12, 43, fac_rule(2.0, 12, 43)) as pd:
        bvp = P.BVP.poisson_sincos()
        wide = pd.estimate(bvp, 40, 2e-3, seed=7, bins_per_gap=100)
        launches = wide.info["kernel_launches"]
        k = pd.estimate(bvp, 40, 2e-3, seed=7, bins_per_gap=100, knot_first=5000, knot_count=64)
        assert launches > k.info["kernel_launches"]
        for r in np.flatnonzero(k.npaths):
            r0, r1 = k.row_ptr[r], k.row_ptr[r + 1]
            np.testing.assert_allclose(k.val[r0:r1], wide.val[r0:r1], rtol=0, atol=ATOL)
            assert abs(k.B[r] - wide.B[r]) <= 1e-6 * max(1.0, abs(wide.B[r]))
