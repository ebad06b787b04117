"""Last-level candidates settled from cover slots that other sets' vertices were
added to: levels large enough for that (100,000 sets and more), with singletons
as the covered sets, at both ends of the range of constraints, and in batches
whose instances end at different levels."""
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


@pytest.mark.parametrize("n,m,p,kmax", [(4, 86, 2, 3), (8, 112, 4, 3), (5, 113, 2, 3), (6, 46, 3, 4), (3, 64, 2, 4)])
def test_same_sets_as_fp64(n, m, p, kmax):
    _compare([P.scale_problem(P.random_mpqp(n, m, p, seed=m + kmax))], kmax)


@pytest.mark.parametrize("count,kmax", [(60, 2), (24, 3)])
def test_batches(count, kmax):
    probs = [P.scale_problem(P.random_mpqp(4 + i % 3, 60 + i % 7, 2, seed=i)) for i in range(count)]
    _compare(probs, kmax)
    _compare(probs, [kmax - i % 2 for i in range(count)])
