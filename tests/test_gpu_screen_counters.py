"""Counters of the one-set-per-thread screen: the lanes of a warp hold sets of
several instances (a batch of one shape is not ordered by instance), and each
instance's LPs and pivots are those it has in a batch of its own."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu


# 9,880 sets at |S| = 3: beyond the levels that are evaluated in FP64 at once,
# alone as in the batch
@pytest.mark.parametrize("count", [2, 5, 24])
def test_counts_per_instance(gpu_lib, count):
    probs = [P.scale_problem(P.random_mpqp(6, 40, 3, seed=i)) for i in range(count)]
    kmax = [3] * count
    kmin = 3   # the levels below, where the batch and one instance take different routes, are not evaluated
    r = solver.solve(probs, precision=solver.MIXED, k_max=kmax, k_min=kmin)
    assert r.inst["lp2_first_stage_lps"].min() > 0
    for i, q in enumerate(probs[:6]):
        one = solver.solve([q], precision=solver.MIXED, k_max=3, k_min=kmin)
        for f in ("lp2_first_stage_lps", "lp2_first_stage_pivots", "optimal", "regions"):
            assert r.inst[f][i] == one.inst[f][0], (i, f)
