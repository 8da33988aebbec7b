"""The replay reduction's terms and their ordered sums: path counts around the blocks of 512 paths that a CTA collects and
the 640 that the sums read at a time, bit for bit against the CPU restatement; and several launches of terms against one."""
import numpy as np
import pytest

import oracle as O
import pdds_gb300 as P
from oracle import replay_ipsi
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npaths", [511, 513, 640, 641, 1025, 1281])
def test_blocks_of_paths_are_bit_exact(npaths):
    sw, ne, nsub, nnode = (0.0, 0.0), (1.0, 1.0), 3, 4
    fac = fac_rule(1.0, nsub, nnode)
    with P.PDDSparseGM(sw, ne, nsub, nnode, fac) as pd:
        L = O.Layout(sw, ne, nsub, nnode)
        ip, _ = replay_ipsi(L, fac)
        est = pd.estimate(P.BVP.helmholtz(2.0, 1.5, -1.0), npaths, 2e-3, mode=P.MODE_REPLAY_FP64, seed=9,
                          ipsi_override=ip)
        prm = O.make_params(npaths, 2e-3, seed=9, fac=fac, portable=True, sublinear=True, threads=4)
        ref = L.run(O.make_problem(O.HELMHOLTZ, 2.0, 1.5, -1.0), prm)
        for k, kn in enumerate(ref["knots"]):
            a, b = ref["row_ptr"][k], ref["row_ptr"][k + 1]
            r0, r1 = est.row_ptr[kn], est.row_ptr[kn + 1]
            assert np.array_equal(est.val[r0:r1], ref["g"][a:b])
            assert np.array_equal(est.var[r0:r1], ref["gvar"][a:b])


def test_terms_in_several_launches():
    """741 knots, sides of up to 95 knots: 512 MB hold 953 paths of all knots, and all paths of one."""
    with P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), 4, 32, fac_rule(2.0, 4, 32)) as pd:
        opts = dict(mode=P.MODE_REPLAY_FP64, seed=9)
        a = pd.estimate(P.BVP.poisson_sincos(), 2500, 5e-3, **opts)
        for first in (0, 300, pd.n_mc - 1):
            b = pd.estimate(P.BVP.poisson_sincos(), 2500, 5e-3, knot_first=first, knot_count=1, **opts)
            kn = int(np.flatnonzero(b.npaths)[0])
            r = slice(a.row_ptr[kn], a.row_ptr[kn + 1])
            assert np.array_equal(a.val[r], b.val[r]) and np.array_equal(a.var[r], b.var[r])
        assert a.info["kernel_launches"] > b.info["kernel_launches"]
