"""Contexts in threads of their own at the same time: launches that ask for different amounts of shared memory (few and many
side knots, coarse and fine subdomain grids) give what each gives by itself."""
import threading

import numpy as np
import pytest

import pdds_gb300 as P
from pdds_gb300.config import fac_rule

pytestmark = pytest.mark.gpu


def in_threads(calls, repeats=30):
    """Every call in a thread of its own, again and again; the results have to stay."""
    want = [call() for call in calls]
    bad = []

    def work(i):
        try:
            for _ in range(repeats):
                if not np.array_equal(calls[i](), want[i]):
                    bad.append(i)
        except P.PDDSError as e:
            bad.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def rect(nsub, nnode):
    return P.PDDSparseGM((-1.0, -1.0), (1.0, 1.0), nsub, nnode, fac_rule(2.0, nsub, nnode))


def test_fp64_estimates():
    cases = [(2, 60, 0, 8), (6, 9, 0, 0), (3, 5, 2, 1), (8, 7, 0, 0)]
    pds = [rect(*c[:2]) for c in cases]
    in_threads([lambda pd=pd, c=c: pd.estimate(P.BVP.poisson_sincos(), 200, 2e-3, mode=P.MODE_FP64, seed=3,
                                               knot_first=c[2], knot_count=c[3]).val for pd, c in zip(pds, cases)])
    for pd in pds:
        pd.close()


def test_subdomain_solves():
    pds = [rect(3, 7) for _ in range(4)]
    for pd in pds:
        pd.estimate(P.BVP.poisson_sincos(), 200, 2e-3, seed=3)
        pd.solve_interface()
    in_threads([lambda pd=pd, m=m: pd.subdomain_solve(m)[2] for pd, m in zip(pds, (4, 64, 17, 50))], 60)
    for pd in pds:
        pd.close()
