"""The interface solve that keeps its rows on chip: systems from a few rows to more than one row group per CTA, runs
of rows that share a stencil and rows that do not, against dense solves; and systems that do not fit it."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu
SQ = ((-1.0, -1.0), (1.0, 1.0))


def dense(pd, est):
    A = np.eye(pd.K)
    r, c, v = est.triplets()
    np.add.at(A, (r, c), v)
    return np.linalg.solve(A, est.B), np.linalg.norm(np.linalg.inv(A), 2)


def check(pd, est, launches=1, **kw):
    ref, inv = dense(pd, est)
    for method in (P.SOLVE_GMRES_FP32_IR, P.SOLVE_BICGSTAB_FP64):
        u, info = pd.solve_interface(method, tol=1e-11, **kw)
        assert info["rel_residual"] <= 1e-11
        assert launches is None or info["kernel_launches"] == launches
        # |u - ref| <= |A^-1| |residual|, and the dense solve's own rounding
        assert np.linalg.norm(u - ref) <= inv * (1e-11 * np.linalg.norm(est.B) + 1e-13 * np.linalg.norm(ref))


@pytest.mark.parametrize("nsub,nnode", [(2, 4), (2, 17), (3, 11), (5, 8), (6, 21), (8, 12)])
def test_layouts_against_dense(nsub, nnode):
    with P.PDDSparseGM(*SQ, nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        est = pd.estimate(P.BVP.poisson_sincos(), 600, (2.0 / nsub) ** 2 * 1e-2, seed=4, adaptive_h=True,
                          richardson=True, dup_sum=True)
        check(pd, est)
        for restart in (2, 33, 40):
            check(pd, est, restart=restart, max_refine=500)  # 30 cycles of two steps are too few for any form
        check(pd, est, launches=None, grid_ctas=3)  # rows of the larger layouts do not fit three CTAs


def test_rows_with_stencils_of_their_own():
    nsub, nnode = 3, 9
    with P.PDDSparseGM(*SQ, nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        sts = [P.Stencil.of_knot(pd, k) for k in range(pd.K)]
        with P.PDDSparseGM.from_stencils((-1.0, -1.0, 1.0, 1.0), pd.x, pd.y, sts) as q:
            check(q, q.estimate(P.BVP.poisson_sincos(), 600, 2e-3, seed=4))


def test_circle():
    with P.PDDSparseGM.circle_mesh(1.0, 3, 8, 7) as pd:
        check(pd, pd.estimate(P.BVP.circle_poisson(), 600, 5e-4, seed=4, adaptive_h=True, richardson=True))


def test_one_cta_that_cannot_hold_the_system_falls_back():
    nsub, nnode = 8, 21
    with P.PDDSparseGM(*SQ, nsub, nnode, fac_rule(2.0, nsub, nnode)) as pd:
        pd.estimate(P.BVP.poisson_sincos(), 600, 1e-3, seed=4, adaptive_h=True, richardson=True, dup_sum=True)
        a, ia = pd.solve_interface(tol=1e-12)
        b, ib = pd.solve_interface(tol=1e-12, grid_ctas=1)  # 354 k entries do not fit one CTA
        assert ia["kernel_launches"] == 1 and ib["kernel_launches"] > 1
        np.testing.assert_allclose(b, a, rtol=0, atol=1e-9)
