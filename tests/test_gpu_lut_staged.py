"""Table nodes staged in shared memory: the paths are the same, step for step, as with nodes read through L1 (wide exit
histograms leave no room to stage), for windows at the table's edges, odd table sizes and constant diffusion fields."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule, varcoef_tables

pytestmark = pytest.mark.gpu


def tables(n, constant):
    coef, g, b = varcoef_tables(n)
    if constant:  # sigma = sqrt2 I, no drift, as the outer loops' tables
        coef = coef.copy()
        coef[..., :2] = np.float32(np.sqrt(2.0))
        coef[..., 2:4] = 0.0
    return coef, g, b


@pytest.mark.parametrize("rich", [False, True])
@pytest.mark.parametrize("constant", [False, True])
@pytest.mark.parametrize("n", [4, 5, 33, 50, 127, 400])
def test_staged_nodes_give_the_same_paths(n, constant, rich):
    opts = dict(adaptive_h=True, richardson=True, dup_sum=True) if rich else {}
    bvp = P.BVP.lut(*tables(n, constant), sampler="catmull_rom")
    with P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), 4, 9, fac_rule(1.0, 4, 9)) as pd:
        a = pd.estimate(bvp, 400, 2e-3, seed=3, **opts)
        b = pd.estimate(bvp, 400, 2e-3, seed=3, bins_per_gap=512, **opts)
    for k in ("path_steps", "exits_global", "exits_stencil"):
        assert a.info[k] == b.info[k]
    # the same values, summed in another order
    assert np.max(np.abs(a.B - b.B)) <= 2 ** -20 * np.max(np.abs(b.B))
