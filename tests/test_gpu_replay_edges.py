"""The replay reduction at the edges of its chunks: path counts around the 256 paths that it reads and the 32 exits
that it multiplies at a time, side lengths from a few knots up, every kind, bit for bit against the CPU restatement."""
import numpy as np
import pytest

import oracle as O
import pdds_gb300 as P
from oracle import replay_ipsi
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npaths", [1, 31, 33, 255, 256, 257, 600])
@pytest.mark.parametrize("kind", ["poisson", "helmholtz", "varcoef"])
def test_replay_is_bit_exact(kind, npaths):
    sw, ne, nsub, nnode = (0.0, 0.0), (1.0, 1.0), 3, 5
    fac = fac_rule(1.0, nsub, nnode)
    bvp, prob = {"poisson": (P.BVP.poisson_sincos(), O.make_problem(O.POISSON_SINCOS)),
                 "helmholtz": (P.BVP.helmholtz(2.0, 1.5, -1.0), O.make_problem(O.HELMHOLTZ, 2.0, 1.5, -1.0)),
                 "varcoef": (P.BVP.varcoef(), O.make_problem(O.VARCOEF))}[kind]
    with P.PDDSparseGM(sw, ne, nsub, nnode, fac) as pd:
        L = O.Layout(sw, ne, nsub, nnode)
        ip, _ = replay_ipsi(L, fac)
        est = pd.estimate(bvp, npaths, 2e-3, mode=P.MODE_REPLAY_FP64, seed=9, ipsi_override=ip)
        prm = O.make_params(npaths, 2e-3, seed=9, fac=fac, portable=True, sublinear=True, threads=4)
        ref = L.run(prob, prm)
        for k, kn in enumerate(ref["knots"]):
            a, b = ref["row_ptr"][k], ref["row_ptr"][k + 1]
            r0, r1 = est.row_ptr[kn], est.row_ptr[kn + 1]
            assert est.B[kn] == ref["B"][k] and est.BB[kn] == ref["BB"][k]
            assert np.array_equal(est.val[r0:r1], ref["g"][a:b])
            assert np.array_equal(est.var[r0:r1], ref["gvar"][a:b])
        assert est.info["exits_stencil"] + est.info["exits_global"] == npaths * pd.n_mc
