"""The MIXED path kernel's rounds between two looks for finished pairs: near the step limit it runs them one at a
time, and a limit that no path exceeds changes nothing."""
import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rich", [False, True])
@pytest.mark.parametrize("bvp", [P.BVP.poisson_sincos(), P.BVP.helmholtz(2.0, 1.5, -1.0)], ids=["poisson", "helmholtz"])
def test_smallest_passing_step_limit_changes_nothing(bvp, rich):
    opts = dict(adaptive_h=True, richardson=True) if rich else {}
    with P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), 2, 6, fac_rule(1.0, 2, 6)) as pd:
        ref = pd.estimate(bvp, 300, 2e-3, seed=5, **opts)

        def run(limit):
            try:
                return pd.estimate(bvp, 300, 2e-3, seed=5, max_steps=limit, **opts)
            except P.PDDSError as e:
                assert "max_steps" in str(e)
                return None
        lo, hi = 0, 1
        while run(hi) is None:
            lo, hi = hi, 2 * hi
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (lo, mid) if run(mid) is not None else (mid, hi)
        assert lo > 8  # the paths are longer than one group of rounds
        est = run(hi)
    assert est.info["path_steps"] == ref.info["path_steps"]
    # the same paths, summed in another order in FP32 per lane and bin
    assert np.max(np.abs(est.B - ref.B)) <= 2 ** -20 * np.max(np.abs(ref.B))
    assert np.max(np.abs(est.val - ref.val)) <= 2 ** -20
