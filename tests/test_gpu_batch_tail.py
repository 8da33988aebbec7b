"""The last group of a batch, solved on the whole chip system by system (up to three systems) or by the cluster kernel:
the same solutions whichever group an instance falls into, eager and replayed from a graph."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300 import _capi as capi
from pdds_gb300.config import batch_instances, fac_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,waves", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 2), (7, 3)])
def test_tail_solutions(n, waves):
    insts = batch_instances(n, seed=5, grid=(2, 6), nodes=(4, 15))
    opts = dict(seed=3, richardson=True, dup_sum=True)
    with P.Batch(P.BVP.HELMHOLTZ, insts) as b:
        b.run(300, 2e-3, waves=n, gmres_form=capi.GMRES_CLASSICAL, **opts)  # the cluster kernel for all
        ref = [b.result(i) for i in range(n)]
        for graph in (False, True, True):
            info = b.run(300, 2e-3, waves=waves, use_graph=graph, **opts)
            assert info["unconverged"] == 0 and info["max_rel_residual"] <= 1e-10
            for i in range(n):
                r = b.result(i)
                assert 0 < r["iterations"] and r["latency_ms"] > 0.0
                # both residuals are 1e-10; G and B differ in the order of FP32 sums
                assert np.max(np.abs(r["u"] - ref[i]["u"])) <= 1e-5 * np.max(np.abs(ref[i]["u"]))


def test_entries_beyond_the_chip():
    """A system whose entries do not all fit on chip: the rest from L2, against the FP64 method."""
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), 16, 41, fac_rule(2.0, 16, 41)) as pd:
        pd.estimate(P.BVP.poisson_sincos(), 64, 2e-3, seed=4, richardson=True, dup_sum=True)
        u, info = pd.solve_interface()
        v, _ = pd.solve_interface(P.SOLVE_BICGSTAB_FP64, tol=1e-12)
        assert info["kernel_launches"] == 1 and info["rel_residual"] <= 1e-10
        # a relative residual of 1e-10, amplified by less than the rows' count over the diagonal's dominance
        assert np.max(np.abs(u - v)) <= 1e-6 * np.max(np.abs(v))


def test_graph_replay_after_other_launch_shapes():
    """Path kernels of different CTA sizes and shared memory, launched in between, do not spoil a captured batch."""
    insts = batch_instances(2, seed=5, grid=(5, 6), nodes=(12, 15))
    opts = dict(richardson=True, dup_sum=True, use_graph=True)
    with P.Batch(P.BVP.HELMHOLTZ, insts) as b, P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), 3, 5, fac_rule(1.0, 3, 5)) as pd:
        b.run(5000, 2e-3, seed=3, **opts)
        u = b.result(1)["u"].copy()
        for th in (128, 256):
            pd.estimate(P.BVP.helmholtz(2.0, 1.0, -1.0), 300, 2e-3, cta_threads=th, richardson=True)
        info = b.run(5000, 2e-3, seed=3, **opts)
        assert info["graph_replayed"] == 1
        # the order of FP32 sums, as in the tests above
        assert np.max(np.abs(b.result(1)["u"] - u)) <= 1e-5 * np.max(np.abs(u))
