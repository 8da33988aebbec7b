"""The autotuner times a whole layout's launch shapes as an estimate runs them:
with the RBF set-up beside the paths."""

import pytest

import pdds_gb300 as P


@pytest.mark.gpu
def test_whole_layout_shapes_are_timed_with_the_setup():
    bvp = P.BVP.circle_poisson()
    n, h = 256, 1e-3  # the set-up outlasts the paths
    with P.PDDSparseGM.circle_mesh(1.0, 8, 16, 11) as pd:
        pd.estimate(bvp, n, h)
        run = min(pd.estimate(bvp, n, h).info["ms_paths"] for _ in range(5))
        default_ms = pd.autotune(bvp, n, h)["default_ms"]
    # the same work; a fifth for the host's part in between
    assert default_ms > 0.8 * run
