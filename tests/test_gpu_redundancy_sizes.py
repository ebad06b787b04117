"""The redundancy LPs at the sizes where their kernel changes: whole and partial
warps of rows, the largest block (128 rows, 31 columns) and the one-warp kernel
above it; every row status equal to the HiGHS restatement's."""
import numpy as np
import pytest

from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver
from oracle import preprocess as PP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,p", [(2, 5, 1), (4, 28, 2), (4, 29, 2), (6, 60, 2), (6, 92, 2), (8, 124, 2), (8, 125, 2),
                                   (28, 60, 3), (29, 60, 3)])
def test_statuses_equal_the_oracle(n, m, p):
    prob = P.random_mpqp(n, m, p, seed=m + n)
    # a third of the rows loosened until the others imply most of them
    loose = np.arange(m) % 3 == 2
    prob.b[loose] += np.random.default_rng(m).uniform(0.5, 6.0, loose.sum())
    status, _ = solver.reduce_constraints(prob)
    assert np.array_equal(status, PP.reduce_rows(prob))
    assert m < 28 or n > 8 or np.any(status[:m] == solver.ROW_REDUNDANT)
