"""Which kernel an interface solve takes, told by its number of launches, and what bounds its waits: the poll limit
counts for GMRES over the whole GPU (4,096 rows and more) only, on chip or by the grid kernel."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300 import _capi as capi
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


# the rows on chip, and the grid kernel: the form that always takes it, and few CTAs, which cannot hold the rows
@pytest.mark.parametrize("opts,launches", [(dict(), 1), (dict(gmres_form=capi.GMRES_CLASSICAL), 3),
                                           (dict(grid_ctas=8), 3)])
def test_waits_over_the_whole_gpu_run_out(opts, launches):
    with estimated(12, 21) as pd:
        u, info = pd.solve_interface(**opts)
        assert info["kernel_launches"] == launches
        with pytest.raises(P.PDDSError) as e:
            pd.solve_interface(barrier_poll_limit=1, **opts)
        assert e.value.status == capi.ERR_TIMEOUT
        v, _ = pd.solve_interface(**opts)
        np.testing.assert_allclose(v, u, rtol=0, atol=1e-8)


def test_bicgstab_from_l2_where_the_rows_do_not_fit():
    with estimated(12, 21) as pd:
        u, a = pd.solve_interface(P.SOLVE_BICGSTAB_FP64, tol=1e-12)
        v, b = pd.solve_interface(P.SOLVE_BICGSTAB_FP64, tol=1e-12, grid_ctas=2)  # 1.0 M entries on two CTAs
        assert a["kernel_launches"] == 1 and b["kernel_launches"] > 1
        np.testing.assert_allclose(v, u, rtol=0, atol=1e-9)


def instance(nsub, nnode):
    return P.Instance((0.0, 0.0), (1.0, 1.0), nsub, nnode, fac_rule(1.0, nsub, nnode), (2.0, 1.5, -1.0))


def launches_of_last_group(b, **opts):
    """Launches beyond the cluster kernel's, which solves a group by two."""
    run = lambda form: b.run(64, 2e-3, seed=3, richardson=True, dup_sum=True, gmres_form=form, **opts)  # noqa: E731
    return run(capi.GMRES_PIPELINED)["kernel_launches"] - run(capi.GMRES_CLASSICAL)["kernel_launches"] + 2


@pytest.mark.parametrize("n,waves,expect", [(1, 1, 1), (3, 1, 3), (5, 2, 3), (4, 4, 1), (40, 1, 2)])
def test_last_group_of_a_batch_takes_the_whole_chip(n, waves, expect):
    """One launch per system of a small last group; many small systems keep the cluster kernel."""
    with P.Batch(P.BVP.HELMHOLTZ, [instance(3, 6)] * n) as b:
        assert launches_of_last_group(b, waves=waves) == expect


def test_system_of_a_batch_with_entries_beyond_the_chip():
    """The second of two systems: 19,005 rows, some of whose entries stay in L2 at their place in the batch."""
    with P.Batch(P.BVP.HELMHOLTZ, [instance(5, 12), instance(16, 41)]) as b:
        assert launches_of_last_group(b, waves=1) == 2
        b.run(64, 2e-3, seed=3, richardson=True, dup_sum=True, waves=2, gmres_form=capi.GMRES_CLASSICAL)
        ref = [b.result(i)["u"].copy() for i in range(2)]
        info = b.run(64, 2e-3, seed=3, richardson=True, dup_sum=True, waves=1)
        assert info["unconverged"] == 0
        for i in range(2):
            # both residuals are 1e-10; G and B differ in the order of FP32 sums
            assert np.max(np.abs(b.result(i)["u"] - ref[i])) <= 1e-5 * np.max(np.abs(ref[i]))
