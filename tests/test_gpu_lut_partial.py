"""Staged table windows where some knots' windows do not fit: only with fields that are the same at every node (the outer
loops' tables) in long launches; the paths are those of nodes read through L1 (wide histograms leave no room to stage)."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule, varcoef_tables

pytestmark = pytest.mark.gpu
RICH = dict(adaptive_h=True, richardson=True, dup_sum=True)


# 2,205 knots: staged; 189 knots, 300 paths: too few items; 8,000 paths: enough
@pytest.mark.parametrize("nsub,nnode,m,npaths", [(8, 21, 32, 200), (4, 9, 32, 300), (4, 9, 32, 8000)])
def test_outer_loop_tables(nsub, nnode, m, npaths):
    with P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), nsub, nnode, fac_rule(1.0, nsub, nnode)) as pd:
        for loop in (pd.solve_semilinear, pd.solve_linear_iteration):
            a, b = (loop(1, npaths, 2e-3 / nsub, m=m, seed=3, **RICH, **o)[0]["estimate"] for o in ({}, dict(bins_per_gap=256)))
            for k in ("path_steps", "exits_global", "exits_stencil"):
                assert a.info[k] == b.info[k]
            # the same values, summed in another order
            assert np.max(np.abs(a.B - b.B)) <= 2.0 ** -20 * np.max(np.abs(b.B))


def test_varying_table_after_an_outer_loop():
    """The rule belongs to the table in use: a caller's table after the outer loop's on the same context."""
    bvp = P.BVP.lut(*varcoef_tables(257), sampler="catmull_rom")
    with P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), 8, 21, fac_rule(1.0, 8, 21)) as pd, \
            P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), 8, 21, fac_rule(1.0, 8, 21)) as fresh:
        pd.solve_semilinear(1, 64, 1e-3, m=32, seed=3, **RICH)
        a, b = (q.estimate(bvp, 200, 1e-3, seed=4, **RICH) for q in (pd, fresh))
        assert a.info["path_steps"] == b.info["path_steps"]
        assert np.max(np.abs(a.B - b.B)) <= 2.0 ** -20 * np.max(np.abs(b.B))
