"""Instances near the limits of a block's shared memory.

The FP64 optimality kernel factors the KKT systems of four sets at a time when
its slots have room for them, and one at a time otherwise (or when the room would
leave an SM one block instead of two): problems on both sides of these limits (with |S| up to n, under a budget that ends the run at |S| =
2) and of its limit |S| = 8, in both precisions, against the oracle.

The LP1 kernel runs four warps a block with a tableau each: problems whose FP64
tableaus leave less than 4 KB of a block's shared memory.

A problem that does not fit is refused, and neither it nor a smaller one changes
what an earlier plan may launch."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("mask_lo", "mask_hi", "feasible", "licq", "optimal", "region")
FP64_FIELDS = FIELDS + ("lp1_status", "lp1_pivots", "z", "lp2_status", "lp2_pivots", "cheb_status", "cheb_pivots")


def _key(a):
    a = a[a["level"] >= 0]
    return a[np.lexsort([a["mask_lo"], a["mask_hi"]])]


def _compare(prob, ref, **kw):
    want = _key(ref.cand)
    for precision in (solver.FP64, solver.MIXED):
        r = solver.solve([prob], precision=precision, record=1, **kw)
        got = _key(r.rec)
        assert len(got) == len(want)
        for f in FP64_FIELDS if precision == solver.FP64 else ("mask_lo", "mask_hi", "feasible", "optimal", "region"):
            assert np.array_equal(got[f], want[f]), (precision, f)
        opt = want["optimal"] == 1
        for f in ("t", "r"):
            assert np.array_equal(got[f][opt], want[f][opt], equal_nan=True), (precision, f)


@pytest.mark.parametrize("make,n,m,p", [(P.random_mpqp, 16, 128, 15), (P.random_mpqp, 16, 128, 16),
                                        (P.random_mpqp, 12, 80, 21), (P.random_mpqp, 12, 80, 22),
                                        (P.random_mpqp, 16, 108, 8), (P.random_mpqp, 16, 114, 8),
                                        (P.random_mplp, 20, 128, 4), (P.random_mplp, 20, 128, 5)])
def test_both_sides_of_the_group_limit(gpu_lib, make, n, m, p):
    prob = P.scale_problem(make(n, m, p, seed=m + p))
    _compare(prob, O.enumerate_sets(prob, k_max=2, nthreads=8), k_max=n, budget=9000, opt_cap=1 << 14)


@pytest.mark.parametrize("make,n,m,p", [(P.random_mpqp, 9, 16, 5), (P.random_mplp, 9, 19, 2)])
def test_group_and_single_factors_by_level(gpu_lib, make, n, m, p):
    prob = P.scale_problem(make(n, m, p, seed=5))
    ref = O.enumerate_sets(prob, k_max=n, nthreads=8)
    assert all(((ref.cand["level"] == k) & (ref.cand["optimal"] == 1)).any() for k in (8, 9))
    _compare(prob, ref, k_max=n)


@pytest.mark.parametrize("n,m,p", [(35, 120, 13), (44, 128, 6), (59, 100, 5)])
def test_largest_lp1_tableaus(gpu_lib, n, m, p):
    prob = P.scale_problem(P.random_mpqp(n, m, p, seed=m + p))
    _compare(prob, O.enumerate_sets(prob, k_max=2, nthreads=8), k_max=2, opt_cap=1 << 14)


def test_refused_and_smaller_plans_leave_a_larger_one_alone(gpu_lib):
    large = P.scale_problem(P.random_mpqp(16, 128, 14, seed=1))      # 157 KB a block of LP1
    oversized = P.scale_problem(P.random_mpqp(16, 128, 26, seed=2))  # 250 KB
    smaller = P.scale_problem(P.random_mpqp(12, 80, 6, seed=3))      # 57 KB
    tiny = P.scale_problem(P.random_n4_m10_p2())
    want = solver.solve([tiny], precision=solver.FP64)
    plan = solver.Plan([large], precision=solver.FP64, k_max=1, use_graph=0)
    plan.run()
    first = plan.results()
    with pytest.raises(solver.MpqpError) as e:
        solver.solve([oversized], precision=solver.FP64, k_max=1)
    assert e.value.code == solver.ECUDA
    assert solver.solve([tiny], precision=solver.FP64).inst.tobytes() == want.inst.tobytes()
    solver.solve([smaller], precision=solver.FP64, k_max=1)
    plan.run()
    again = plan.results()
    plan.close()
    assert again.candidates == 129
    for f in ("feasible_digest", "optimal_digest", "region_digest"):
        assert np.array_equal(first.inst[f], again.inst[f])
