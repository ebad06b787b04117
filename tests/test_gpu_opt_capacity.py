"""Calls whose sets are mostly optimal: all of them come back without a capacity
of the caller's."""
import pytest

from mpqpcudasolver_gb300 import host
from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [solver.FP64, solver.MIXED])
@pytest.mark.parametrize("n,m,p", [(16, 128, 15), (35, 120, 13)])
def test_most_sets_optimal(gpu_lib, n, m, p, precision):
    prob = P.scale_problem(P.random_mpqp(n, m, p, seed=m + p))
    ref = O.enumerate_sets(prob, k_max=2, nthreads=8, keep_records=False)
    assert ref.n_optimal > max(4096, ref.n_cand // 2)
    r = solver.solve([prob], precision=precision, k_max=2)
    assert len(r.opt) == ref.n_optimal and r.total("regions") == ref.n_region


def test_drop_in(gpu_lib):
    lib = host.load_mpqp_cuda()
    prog = host.MPQPProb.from_mpqp(P.random_mpqp(16, 128, 15, seed=143))
    prog.process_constraints(scale_method=1)
    r = host.call_mpqp(lib, host.build_lp_data(prog), k_max=2)
    ref = O.enumerate_sets(prog.to_mpqp(), k_max=2, nthreads=8, keep_records=False)
    assert r.contents.status == 0, solver.last_error()
    assert r.contents.n_final_lps == ref.n_optimal > 4096
    lib.mpqp_free(r)
