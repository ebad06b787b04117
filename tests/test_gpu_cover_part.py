"""Cover slots beside all, a part or none of a level's hash slots (a plan gives
them a small share of its memory): the same sets as the FP64 path, by more last-
level LPs the fewer there are."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest", "region_digest")
SLOT_PAIR, SHARE = 64, 0.05     # bytes of a slot's two sides; the share of the memory they may take


def _solve(probs, kmax, slots):
    """slots: how many the share holds (between two powers of two, as the memory in use varies)."""
    import torch
    torch.cuda.synchronize()
    solver.load().mpqp_release_cached_memory()
    free = torch.cuda.mem_get_info()[0]
    n = 1 << 19
    return solver.solve(probs, precision=solver.MIXED, k_max=kmax, cand_cap=n, node_cap=n, arena_bytes=1 << 30,
                        mem_fraction=1.4 * slots * SLOT_PAIR / SHARE / free)


@pytest.mark.parametrize("case", ["one", "batch"])
def test_part_of_the_slots(gpu_lib, case):
    if case == "one":       # 15,180 sets before the last level: 2^15 hash slots
        probs, kmax = [P.scale_problem(P.random_mpqp(6, 46, 3, seed=50))], 4
    else:                   # 20 x 780
        probs, kmax = [P.scale_problem(P.random_mpqp(4 + i % 3, 40 + i % 2, 2, seed=i)) for i in range(20)], 3
    want = solver.solve(probs, precision=solver.FP64, k_max=kmax)
    pivots = []
    for slots in (512, 1 << 12, 1 << 14, 1 << 20):      # none, an eighth, half, all
        r = _solve(probs, kmax, slots)
        for f in FIELDS:
            assert np.array_equal(want.inst[f], r.inst[f]), (slots, f)
        pivots.append(r.total("lp1_pivots"))
    assert pivots[0] > pivots[1] > pivots[2] > pivots[3], pivots
