"""The FP64 re-solves of the mixed path start from the pre-pivoted root, or from
the constraint rows where pre-pivoting grew the entries too far: the same sets
as the FP64 path either way, on near-duplicate rows (most candidates re-solved)
and with one variable rescaled so far that the pre-pivoted root is refused."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

FIELDS = ("candidates", "pruned", "feasible", "optimal", "regions", "feasible_digest", "optimal_digest", "region_digest")


def _rescaled(prob, scale):
    """The same problem in x_0' = x_0 / scale."""
    d = np.ones(prob.n)
    d[0] = scale
    prob.A, prob.H, prob.c = prob.A * d, prob.H * d[:, None], prob.c * d
    prob.Q = prob.Q * np.outer(d, d)
    return prob


@pytest.mark.parametrize("scale", [1.0, 1e-5])
@pytest.mark.parametrize("kmax", [2, 3])
def test_same_sets_as_fp64(kmax, scale):
    prob = _rescaled(P.scale_problem(P.illcond_n16_m62_p8(3)), scale)
    a = solver.solve([prob], precision=solver.FP64, k_max=kmax)
    b = solver.solve([prob], precision=solver.MIXED, k_max=kmax)
    assert b.total("fallback_lp1") > 0
    for f in FIELDS:
        assert np.array_equal(a.inst[f], b.inst[f]), f
    key = lambda x: x[np.lexsort([x["mask_lo"], x["mask_hi"]])]
    assert np.array_equal(key(a.opt)["t"], key(b.opt)["t"]) and np.array_equal(key(a.opt)["r"], key(b.opt)["r"])
