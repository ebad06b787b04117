"""d2h_bytes counts what is copied: the counters come back with the first 512
optimal sets, however many of these there are, and the others by themselves."""
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu

OPT_REC = 64     # bytes of an optimal set's record on the device


def test_bytes_copied_back(gpu_lib):
    n10, m62 = P.scale_problem(P.random_n10_m43_p4()), P.scale_problem(P.random_n12_m62_p6())
    few, more, many = (solver.solve([q], precision=solver.MIXED, k_max=k, opt_cap=1 << 16)
                       for q, k in ((n10, 1), (n10, 2), (m62, 3)))
    assert 0 < len(few.opt) < len(more.opt) <= 512 < len(many.opt)
    assert few.d2h_bytes == more.d2h_bytes > 512 * OPT_REC
    assert many.d2h_bytes == few.d2h_bytes + (len(many.opt) - 512) * OPT_REC
