"""Device memory of single calls: the laws of many sets leave no more of it in
the plans' pool than those of a few."""
import ctypes
import itertools

import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

pytestmark = pytest.mark.gpu


def _laws(lib, prob, sets):
    ps = solver._ProblemSet([prob])
    masks = np.zeros((len(sets), 2), dtype=np.uint64)
    for i, S in enumerate(sets):
        masks[i, 0] = sum(1 << j for j in S)
    stride = lib.mpqp_region_laws_stride(ps.arr)
    laws, sizes = np.zeros((len(sets), stride)), np.zeros((len(sets), 4), dtype=np.intc)
    dp = ctypes.POINTER(ctypes.c_double)
    rc = lib.mpqp_region_laws(ps.arr, len(sets), masks.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)),
                              laws.ctypes.data_as(dp), sizes.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    assert rc == 0, solver.last_error()
    return laws, sizes


def test_large_calls_give_their_memory_back(gpu_lib):
    import torch
    prob = P.scale_problem(P.random_n12_m62_p6())
    sets = list(itertools.combinations(range(62), 3))      # 37,820: 300 MB of laws
    few = _laws(gpu_lib, prob, sets[:64])
    before = torch.cuda.mem_get_info()[0]
    many = _laws(gpu_lib, prob, sets)
    assert many[0].nbytes > 300e6
    after = torch.cuda.mem_get_info()[0]
    assert before - after < 64 << 20, (before - after) >> 20
    assert np.array_equal(many[1][:64], few[1]) and np.array_equal(many[0][:64, :20], few[0][:, :20])
    # a plan's idle memory is not given back by it
    plan = solver.Plan([prob], precision=solver.MIXED, k_max=2, arena_bytes=1 << 30)
    plan.close()
    held = torch.cuda.mem_get_info()[0]
    _laws(gpu_lib, prob, sets)
    assert torch.cuda.mem_get_info()[0] <= held + (64 << 20)
    assert gpu_lib.mpqp_release_cached_memory() == 0
    assert torch.cuda.mem_get_info()[0] > held + (512 << 20)
