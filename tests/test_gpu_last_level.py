"""Last-level candidates settled at certified vertices of their subsets: the same
sets as the FP64 path at every depth (the last level of one run is a storing
level of the next), with more than 64 and more than 112 constraints, and where a
batch's instances end at different levels."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest", "region_digest")


def _compare(probs, kmax):
    a = solver.solve(probs, precision=solver.FP64, k_max=kmax)
    b = solver.solve(probs, precision=solver.MIXED, k_max=kmax)
    for f in FIELDS:
        assert np.array_equal(a.inst[f], b.inst[f]), f
    return b


@pytest.mark.parametrize("n,m,p,kmax", [(6, 20, 2, 1), (6, 20, 2, 2), (6, 20, 2, 3), (6, 20, 2, 6), (6, 64, 3, 3),
                                        (6, 65, 3, 3), (5, 112, 2, 3), (5, 113, 2, 3), (5, 126, 2, 2)])
def test_same_sets_as_fp64(n, m, p, kmax):
    _compare([P.scale_problem(P.random_mpqp(n, m, p, seed=m + kmax))], kmax)


def test_instances_ending_at_different_levels():
    probs = [P.scale_problem(P.random_mpqp(n, m, 3, seed=m)) for n, m in ((4, 18), (5, 24), (6, 30), (7, 16))]
    probs.append(P.scale_problem(P.mpc_mpqp(3)))
    b = _compare(probs, [4, 3, 5, 7, 2])
    assert b.total("stored") < b.total("feasible")
