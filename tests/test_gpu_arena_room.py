"""An arena that holds the tableaus of every feasible set, but not of every
candidate, keeps them all: LP1 reserves space for candidates ahead only where it
suffices for all of them.  And where it holds a part, that part is used and the
sets are the same."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest", "region_digest")
CASES = {"mpc2-k4": (lambda: P.mpc_mpqp(2), 4), "mpc5-k4": (lambda: P.mpc_mpqp(5), 4),
         "mplp3-k5": (lambda: P.mplp_member(3), 5)}


def _tableau_bytes(prob, precision):
    nv = prob.n + prob.p
    if precision == solver.FP64:
        ld, size = (nv + 1) | 1, 8
    else:
        ld, size = (nv + 4) & ~3, 4          # 4 mod 8 floats
        ld += 0 if ld & 4 else 4
    return (((prob.m + prob.ncp + 1) * ld + 3) & ~3) * size


@pytest.mark.parametrize("precision", [solver.FP64, solver.MIXED])
@pytest.mark.parametrize("case", list(CASES))
def test_every_feasible_set_keeps_its_tableau(gpu_lib, case, precision):
    make, kmax = CASES[case]
    prob = P.scale_problem(make())
    ref = O.enumerate_sets(prob, k_max=kmax, nthreads=8).cand
    cand = np.bincount(ref["level"][ref["level"] >= 0], minlength=kmax + 1)
    feas = np.bincount(ref["level"][(ref["level"] >= 0) & (ref["feasible"] == 1)], minlength=kmax + 1)
    need = max(feas[k - 1] + feas[k] for k in range(1, kmax))        # parents and children of a storing level
    ahead = max(feas[k - 1] + cand[k] for k in range(1, kmax))
    assert need + 8 < ahead
    tab = _tableau_bytes(prob, precision)
    whole = solver.solve([prob], precision=precision, k_max=kmax)
    r = solver.solve([prob], precision=precision, k_max=kmax, arena_bytes=int(need + 4) * tab)
    assert whole.split_levels == 0 and r.split_levels == 0
    assert r.total("nodes_without_tableau") == 0 and r.total("stored") == whole.total("stored")
    # half of that: as many tableaus as the arena holds, up to one abandoned by each warp
    half = solver.solve([prob], precision=precision, k_max=kmax, arena_bytes=int(need // 2) * tab)
    assert half.split_levels > 0 and half.total("nodes_without_tableau") > 0 and half.total("lp1_cold") > 0
    for f in FIELDS:
        assert np.array_equal(whole.inst[f], r.inst[f]) and np.array_equal(whole.inst[f], half.inst[f]), f
