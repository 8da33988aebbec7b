"""Which kernel an interface solve takes, told by its number of launches, and what bounds its waits: the poll limit
counts for GMRES over the whole GPU (4,096 rows and more) only, on chip or by the grid kernel."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


def estimated(nsub, nnode, npaths=256):
    pd = P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode))
    pd.estimate(P.BVP.poisson_sincos(), npaths, 1e-3, seed=3, adaptive_h=True, richardson=True, dup_sum=True)
    return pd


def test_poll_limit_counts_for_gmres_over_the_whole_gpu_only():
    with estimated(4, 11) as small, estimated(12, 21) as large:
        assert small.K < 4096 <= large.K
        for pd, method in ((small, P.SOLVE_GMRES_FP32_IR), (small, P.SOLVE_BICGSTAB_FP64),
                           (large, P.SOLVE_BICGSTAB_FP64)):
            u, _ = pd.solve_interface(method, tol=1e-11)
            v, _ = pd.solve_interface(method, tol=1e-11, barrier_poll_limit=1)
            np.testing.assert_allclose(v, u, rtol=0, atol=1e-8)
