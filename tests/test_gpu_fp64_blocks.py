"""The FP64 kernel's blocks and slots: path counts around a slot's 32 and a block's 256 lanes, one knot (slots spread
over CTAs) and a layout (whole blocks per CTA), against the replay mode, which draws the same streams."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu
PROBLEMS = {"poisson": P.BVP.poisson_sincos(), "helmholtz": P.BVP.helmholtz(2.0, 1.5, -1.0), "varcoef": P.BVP.varcoef()}


@pytest.mark.parametrize("npaths", [1, 31, 33, 255, 257, 511, 513, 1000])
@pytest.mark.parametrize("kind", PROBLEMS)
def test_fp64_matches_replay(kind, npaths):
    bvp = PROBLEMS[kind]
    sw, ne, nsub, nnode = (0.0, 0.0), (1.0, 1.0), 3, 5
    with P.PDDSparseGM(sw, ne, nsub, nnode, fac_rule(1.0, nsub, nnode)) as pd, P.EMFKACSolver() as sv:
        a = pd.estimate(bvp, npaths, 2e-3, mode=P.MODE_FP64, seed=9)
        b = pd.estimate(bvp, npaths, 2e-3, mode=P.MODE_REPLAY_FP64, seed=9)
        assert a.info["path_steps"] == b.info["path_steps"]
        assert a.info["exits_global"] == b.info["exits_global"]
        # the same paths, each value rounded some 10 times per step: N(0, 1) normals, at most a few hundred steps
        tol = 1e-12
        np.testing.assert_allclose(a.B, b.B, rtol=tol, atol=tol)
        # |Psi^-1| (1e10 here at most) times the rounding of the sums
        np.testing.assert_allclose(a.val, b.val, rtol=0, atol=1e-4)
        k = int(pd.order[0])
        st = P.Stencil.of_knot(pd, k)
        G, _, gj, B, BB = sv.Solve_GPU_Analytic((pd.x[k], pd.y[k]), npaths, 2e-3, 0.0, bvp, st, seed=9, knot_id=k)
        assert abs(B - b.B[k]) <= tol * (1 + abs(b.B[k]))
        r0, r1 = b.row_ptr[k], b.row_ptr[k + 1]
        assert np.array_equal(gj, b.col[r0:r1])
        np.testing.assert_allclose(G, b.val[r0:r1], rtol=0, atol=1e-4)


@pytest.mark.parametrize("npaths", [33, 600])
def test_fp64_richardson_matches_mixed(npaths):
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), 3, 7, fac_rule(2.0, 3, 7)) as pd:
        for bvp in (P.BVP.poisson_sincos(), P.BVP.monegros(), P.BVP.robin_poisson()):
            a = pd.estimate(bvp, npaths, 2e-3, mode=P.MODE_FP64, seed=9, adaptive_h=True, richardson=True)
            b = pd.estimate(bvp, npaths, 2e-3, mode=P.MODE_MIXED, seed=9, adaptive_h=True, richardson=True)
            # FP32 paths of the same streams: a few of them leave a step earlier or later
            assert abs(a.info["path_steps"] - b.info["path_steps"]) <= 1e-3 * b.info["path_steps"]
            np.testing.assert_allclose(a.B, b.B, rtol=0, atol=5e-2)
