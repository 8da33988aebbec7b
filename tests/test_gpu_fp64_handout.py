"""FP64 mode: a block's paths beyond its first 256 go to lanes by a rule that no timing enters, so G repeats to the last
bit, and does not depend on how many CTAs a block is spread over (one knot: eight; a layout of 304 knots or more: one)."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu
RECT = dict(sw=(-1.0, -1.0), ne=(1.0, 1.0), nsub=6, nnode=9)


def layout(kind):
    if kind == "circle":
        return P.PDDSparseGM.circle_mesh(1.0, 5, 12, 7), P.BVP.circle_poisson()
    pd = P.PDDSparseGM(RECT["sw"], RECT["ne"], RECT["nsub"], RECT["nnode"], fac_rule(2.0, RECT["nsub"], RECT["nnode"]))
    return pd, P.BVP.poisson_sincos() if kind == "poisson" else P.BVP.varcoef()


# at most 511 paths: one block per knot, whatever the number of knots
@pytest.mark.parametrize("npaths", [257, 264, 300, 511])
@pytest.mark.parametrize("kind,richardson", [("poisson", False), ("poisson", True), ("varcoef", False),
                                             ("circle", False)])
def test_rows_do_not_depend_on_timing(kind, richardson, npaths):
    pd, bvp = layout(kind)
    with pd:
        opts = dict(mode=P.MODE_FP64, seed=5, richardson=richardson)
        run = lambda first=0, count=0: pd.estimate(bvp, npaths, 1e-3, knot_first=first, knot_count=count, **opts)  # noqa: E731
        a, b = run(), run()
        n_mc = int(np.count_nonzero(a.npaths))
        assert n_mc >= 304
        assert np.array_equal(a.val, b.val)
        for first, count in ((0, 1), (n_mc // 2, 1), (n_mc - 60, 60), (7, 120), (40, 200)):
            c = run(first, count)
            rows = np.flatnonzero(c.npaths)
            assert len(rows) == count
            for k in rows:
                at = slice(a.row_ptr[k], a.row_ptr[k + 1])
                assert np.array_equal(a.val[at], c.val[at])


def test_single_knot_repeats():
    with P.PDDSparseGM(RECT["sw"], RECT["ne"], RECT["nsub"], RECT["nnode"], fac_rule(2.0, 6, 9)) as pd:
        sv, bvp = P.EMFKACSolver(), P.BVP.poisson_sincos()
        k = int(pd.order[5])
        st = P.Stencil.of_knot(pd, k)
        got = [sv.Solve_GPU_Analytic((pd.x[k], pd.y[k]), 5000, 1e-3, 0.0, bvp, st, seed=9, knot_id=k)[0] for _ in range(4)]
        # 19 blocks of paths, added into the row in any order: a block's sum is rounded 18 times
        for g in got[1:]:
            assert np.max(np.abs(g - got[0])) <= 19 * 2.0 ** -53 * np.max(np.abs(got[0])) * 19


def test_launches_split_where_the_sums_need_more_memory():
    # 31,597 knots, 23 KB of sums each: two launches; a quarter of the knots fits one
    nsub, nnode = 20, 43
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        run = lambda first, count: pd.estimate(P.BVP.poisson_sincos(), 300, 2e-3, mode=P.MODE_FP64, seed=5,  # noqa: E731
                                               knot_first=first, knot_count=count)
        run(0, 1)  # a context's first FP64 call also fills its tables
        a = run(0, 0)
        n_mc = int(np.count_nonzero(a.npaths))
        bounds = [n_mc * q // 4 for q in range(5)]
        parts = [run(lo, hi - lo) for lo, hi in zip(bounds, bounds[1:])]
        assert a.info["kernel_launches"] == parts[0].info["kernel_launches"] + 2
        assert np.array_equal(a.val, sum(p.val for p in parts))  # a row is zero outside its part
        interior = a.npaths > 0
        np.testing.assert_allclose(a.B[interior], sum(np.where(p.npaths > 0, p.B, 0.0) for p in parts)[interior],
                                   rtol=0, atol=1e-12)
        assert a.info["path_steps"] == sum(p.info["path_steps"] for p in parts)
