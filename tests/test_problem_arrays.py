"""Problem arrays and integers as the Python front end hands them to C: whatever
converts to float64 is taken (any type, order or stride, lists), floats where the
C structure has integers are not."""
import ctypes

import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

NAMES = {"Q": "Q", "c": "c", "H": "H", "A": "A", "b": "b", "F": "F", "CRA": "At", "CRb": "bt"}


def _read(ps, i, prob):
    s = ps.arr[i]
    return {py: np.ctypeslib.as_array(ctypes.cast(getattr(s, c), ctypes.POINTER(ctypes.c_double)),
                                      shape=np.shape(getattr(prob, py))).copy() for py, c in NAMES.items()}


FORMS = {
    "integers": lambda a: np.round(a * 4).astype(np.int32),
    "float32": lambda a: a.astype(np.float32),
    "objects": lambda a: a.astype(object),
    "strings": lambda a: a.astype(str),
    "fortran": lambda a: np.asfortranarray(a),
    "strided": lambda a: np.repeat(a, 2, axis=-1)[..., ::2],
    "reversed": lambda a: a[::-1],
    "unaligned": lambda a: np.frombuffer(b"\0" + a.tobytes(), dtype=np.uint8)[1:].view(np.float64).reshape(a.shape),
}


@pytest.mark.parametrize("form", list(FORMS))
def test_arrays_arrive_as_float64(form):
    probs = [P.scale_problem(P.random_n4_m10_p2()), P.scale_problem(P.random_mpqp(3, 8, 2, seed=1))]
    for q in probs:
        for nm in NAMES:
            setattr(q, nm, FORMS[form](np.asarray(getattr(q, nm))))
    ps = solver._ProblemSet(probs)
    for i, q in enumerate(probs):
        assert (ps.arr[i].n, ps.arr[i].m, ps.arr[i].p, ps.arr[i].ncp) == (q.n, q.m, q.p, len(q.CRb))
        for nm, a in _read(ps, i, q).items():
            assert np.array_equal(a, np.ascontiguousarray(getattr(q, nm), dtype=np.float64)), nm


def test_lists_and_matrices():
    q = P.scale_problem(P.random_n4_m10_p2())
    want = q.copy()
    q.c, q.b, q.CRb = q.c.tolist(), q.b.tolist(), q.CRb.tolist()
    with pytest.warns(PendingDeprecationWarning):
        q.H = np.matrix(q.H)
    ps = solver._ProblemSet([q])
    for nm, a in _read(ps, 0, want).items():
        assert np.array_equal(a, getattr(want, nm)), nm


@pytest.mark.parametrize("kw", [dict(k_max=2.0), dict(k_max=[2.0]), dict(k_min=1.0), dict(k_max="2"), dict(k_min=None)])
def test_no_floats_for_integers(kw):
    with pytest.raises(TypeError):
        solver._ProblemSet([P.scale_problem(P.random_n4_m10_p2())], **kw)


def test_integers():
    q = P.scale_problem(P.random_n4_m10_p2())
    for k, budget in ((3, 7), (np.int64(3), np.int32(7)), (3, 7.9)):
        s = solver._ProblemSet([q], k_min=np.int16(1), k_max=k, budget=budget).arr[0]
        assert (s.k_min, s.k_max, s.budget) == (1, 3, 7)
    assert solver._ProblemSet([q], k_max=99).arr[0].k_max == q.m
