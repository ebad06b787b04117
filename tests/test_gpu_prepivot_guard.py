"""FP64 re-solves of the mixed path do not start from a pre-pivoted root whose
pivots grew its entries (also where later pivots cancel that) or its right-hand
sides past 1e4: the rounding of such values would come near tol_feas."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest", "region_digest")


def _rescaled(seed):
    """The same problem in other units, variable by variable: entries of 2.5e4 on the way, 33 at the end."""
    prob = P.scale_problem(P.random_mpqp(10, 30, 3, seed))
    d = 10.0 ** np.random.default_rng(seed).uniform(-2, 2, prob.n)
    prob.A, prob.H, prob.c = prob.A * d, prob.H * d[:, None], prob.c * d
    prob.Q = prob.Q * np.outer(d, d)
    return prob


def _large_b():
    """Right-hand sides of 1e6, entries of single digits."""
    prob = P.scale_problem(P.random_mpqp(10, 43, 4, seed=0))
    prob.b, prob.CRb, prob.c = prob.b * 1e6, prob.CRb * 1e6, prob.c * 1e6
    return prob


def test_ordinary_problems_are_pre_pivoted(gpu_lib):
    probs = [P.scale_problem(p) for p in (P.random_n10_m43_p4(), P.mpc_mpqp(0), P.illcond_n16_m62_p8(0), P.mplp_member(0))]
    assert solver.solve(probs, precision=solver.MIXED, k_max=1).plain_roots == 0
    assert solver.solve(probs, precision=solver.FP64, k_max=1).plain_roots == 0


@pytest.mark.parametrize("make", [lambda: _rescaled(15), _large_b])
def test_grown_roots_are_refused(gpu_lib, make):
    probs = [make(), P.scale_problem(P.random_n4_m10_p2())]
    assert solver.solve(probs, precision=solver.MIXED, k_max=1).plain_roots == 1


def test_same_sets_after_cancelled_growth(gpu_lib):
    probs = [_rescaled(s) for s in (15, 1306)]
    a = solver.solve(probs, precision=solver.FP64, k_max=3)
    b = solver.solve(probs, precision=solver.MIXED, k_max=3)
    assert b.plain_roots == 2
    for f in FIELDS:
        assert np.array_equal(a.inst[f], b.inst[f]), f
