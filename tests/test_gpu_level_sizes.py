"""Levels of every size against the oracle: a warp claims one candidate (or
parent) at a time on a small level and a longer chunk on a large one, so the
sizes run from a handful of sets to tens of thousands."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [solver.FP64, solver.MIXED])
@pytest.mark.parametrize("n,m,p,k", [(1, 1, 1, 1), (3, 5, 2, 3), (4, 33, 2, 2), (6, 64, 3, 2), (8, 65, 3, 3)])
def test_level_sizes_vs_oracle(n, m, p, k, precision):
    prob = P.scale_problem(P.random_mpqp(n, m, p, seed=1000 + m))
    ref = O.enumerate_sets(prob, k_max=k)
    r = solver.solve([prob], precision=precision, k_max=k)
    assert (r.candidates, r.total("feasible"), r.total("optimal"), r.total("regions")) == \
        (ref.n_cand, ref.n_feasible, ref.n_optimal, ref.n_region)
    want = ref.cand[ref.cand["optimal"] == 1]
    key = lambda a: a[np.lexsort([a["mask_lo"], a["mask_hi"]])]
    got, want = key(r.opt), key(want)
    assert np.array_equal(got["mask_lo"], want["mask_lo"]) and np.array_equal(got["mask_hi"], want["mask_hi"])
    assert np.array_equal(got["t"], want["t"]) and np.array_equal(got["r"], want["r"])
