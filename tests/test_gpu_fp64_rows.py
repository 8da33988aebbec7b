"""FP64 mode: G's rows to the last bit, against rows recorded from the kernel in its first form (one plain loop per block
of paths, the math library's functions throughout).  Psi^-1 turns a changed rounding of a position, of Y or of an RBF
value into differences of 1e-9 to 1e-5, so a faster form has to keep them.  At most 256 paths: no hand-out.

To record: python tests/test_gpu_fp64_rows.py tests/golden/fp64_rows.npz"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.environ.get("PDDS_TREE", os.path.dirname(os.path.dirname(os.path.abspath(__file__)))))
import pdds_gb300 as P  # noqa: E402
from pdds_gb300.config import fac_rule  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "fp64_rows.npz")
RICH = dict(adaptive_h=True, richardson=True, dup_sum=True)
# name -> problem, lower corner and side of the domain (None: the disk), step, options
CASES = {
    "poisson": (P.BVP.poisson_sincos, -1.0, 2.0, 4e-3, {}),
    "poisson_pairs": (P.BVP.poisson_sincos, -1.0, 2.0, 4e-3, RICH),
    "helmholtz": (lambda: P.BVP.helmholtz(2.3, 1.7, -1.5), 0.0, 1.0, 1e-3, {}),
    "helmholtz_pairs": (lambda: P.BVP.helmholtz(2.3, 1.7, -1.5), 0.0, 1.0, 1e-3, RICH),
    "varcoef": (P.BVP.varcoef, 0.0, 1.0, 1e-3, {}),
    "varcoef_pairs": (P.BVP.varcoef, 0.0, 1.0, 1e-3, RICH),
    "monegros_pairs": (P.BVP.monegros, -5.0, 10.0, 0.1, RICH),
    "robin": (lambda: P.BVP.robin_poisson("W"), 0.0, 1.0, 1e-3, {}),
    "robin_west_pairs": (lambda: P.BVP.robin_poisson("W"), 0.0, 1.0, 1e-3, RICH),
    "robin_north_pairs": (lambda: P.BVP.robin_poisson("N"), 0.0, 1.0, 1e-3, RICH),
    "table_pairs": (lambda: P.BVP.varcoef_lut(64), 0.0, 1.0, 1e-3, RICH),
    "circle": (P.BVP.circle_poisson, None, 0.0, 1e-3, {}),
    "circle_pairs": (P.BVP.circle_poisson, None, 0.0, 1e-3, RICH),
}


def rows(name, first, count):
    make, lo, side, h, opts = CASES[name]
    pd = (P.PDDSparseGM.circle_mesh(1.0, 3, 8, 7) if lo is None else
          P.PDDSparseGM((lo, lo), (lo + side, lo + side), 3, 9, fac_rule(side, 3, 9)))
    with pd:
        est = pd.estimate(make(), 200, h, mode=P.MODE_FP64, seed=77, knot_first=first, knot_count=count, **opts)
        return np.concatenate([est.val[est.row_ptr[k]:est.row_ptr[k + 1]] for k in np.flatnonzero(est.npaths)])


@pytest.mark.parametrize("name", CASES)
def test_rows_as_recorded(name):
    with np.load(GOLDEN) as z:
        want = z[name]
    assert np.array_equal(rows(name, 3, 6), want)


if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{name: rows(name, 3, 6) for name in CASES})
