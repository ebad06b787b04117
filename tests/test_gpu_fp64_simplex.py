"""The FP64 simplex at the edges of its row slots (32, 64, 96 and 128 rows, and
the generic loop above), with exact ties and zeros in the ratio test: every
record equal to the oracle's, bit for bit."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _tied(prob):
    """Half of the rows duplicates of the other half, and a quarter through the origin."""
    m = prob.m // 2
    prob.A[m:2 * m], prob.F[m:2 * m], prob.b[m:2 * m] = prob.A[:m], prob.F[:m], prob.b[:m]
    prob.b[:m // 2] = 0.0
    prob.b[m:m + m // 2] = 0.0
    return prob


@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("n,m,p,k", [(3, 28, 2, 2), (3, 29, 2, 2), (5, 60, 2, 2), (5, 61, 2, 2), (4, 90, 3, 2),
                                     (4, 91, 3, 2), (6, 122, 3, 1), (6, 123, 3, 1), (6, 128, 4, 1)])
def test_records_vs_oracle(n, m, p, k, tied):
    prob = P.random_mpqp(n, m, p, seed=m)
    prob = P.scale_problem(_tied(prob) if tied else prob)
    ref = O.enumerate_sets(prob, k_max=k)
    r = solver.solve([prob], precision=solver.FP64, k_max=k, record=1)
    key = lambda a: a[np.lexsort([a["mask_lo"], a["mask_hi"]])]
    got, want = key(r.rec[r.rec["level"] >= 0]), key(ref.cand)
    assert len(got) == len(want) == ref.n_cand
    for f in ("mask_lo", "mask_hi", "lp1_status", "lp1_pivots", "z", "feasible", "licq", "lp2_status", "lp2_pivots",
              "optimal", "cheb_pivots", "region"):
        assert np.array_equal(got[f], want[f]), f
    for f in ("t", "r"):
        assert np.array_equal(got[f], want[f], equal_nan=True), f
