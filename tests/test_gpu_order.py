"""Levels of 40,000 candidates and more of instances of different shapes, which are
brought into the instances' order before LP1: every instance's sets and counts are
those it has alone (a batch of one is never reordered), with instances that end at
different levels, that run out of their budget in the middle of the batch, and with
more instances than one block's threads."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest",
          "region_digest", "last_level", "truncated", "stored")
PRECISIONS = [solver.FP64, solver.MIXED]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("budget", [0, 15000])
def test_mixed_shapes(precision, budget):
    probs = [P.scale_problem(P.random_mpqp(4 + i % 7, 24 + (13 * i) % 39, 2 + i % 3, seed=i)) for i in range(12)]
    kmax = [3 + i % 2 if i % 5 else 2 for i in range(12)]
    budgets = [budget if i % 3 == 1 else 1 << 22 for i in range(12)]
    r = solver.solve(probs, precision=precision, k_max=kmax, budget=budgets)
    assert budget == 0 or r.inst["truncated"].sum() > 0
    for i, q in enumerate(probs):
        one = solver.solve([q], precision=precision, k_max=[kmax[i]], budget=[budgets[i]])
        for f in FIELDS:
            assert r.inst[f][i] == one.inst[f][0], (i, f)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_many_instances(precision):
    probs = [P.scale_problem(P.random_mpqp(3 + i % 3, 11 + i % 4, 2, seed=i)) for i in range(1100)]
    r = solver.solve(probs, precision=precision, k_max=3)
    # (at most 75 x C(14, 3) = 27,300 sets a level: not reordered)
    parts = [solver.solve(probs[i:i + 75], precision=precision, k_max=3) for i in range(0, 1100, 75)]
    for f in FIELDS:
        assert np.array_equal(r.inst[f], np.concatenate([p.inst[f] for p in parts])), f
