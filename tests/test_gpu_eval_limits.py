"""Ranking criteria at the limits of the column sweep: a model whose constant is NaN (predictions of
ids outside the model are NaN) and rows of factors that fill a block's shared memory."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm

pytestmark = pytest.mark.gpu

# As the sweep gives them that searches all predictions in global memory by halves: a NaN comes last in a
# row's order and is not greater than anything.
NAN_CONSTANT = {10: 0.5242209538211974, 11: 0.5564215509463737, 12: 0.47689812132099607, 13: 0.44134506008027047}


def test_nan_constant(lib, cuda):
    rng = np.random.default_rng(7)
    m, n, k, nnz = 60, 110, 33, 900
    P, Q = ((rng.standard_normal((x, k)) * 0.4).astype(np.float32) for x in (m, n))
    u, v = rng.integers(0, m + 3, nnz), rng.integers(0, n + 4, nnz)
    prob = cm.MFProblem.from_arrays(u, v, rng.choice([-1.0, 1.0], nnz).astype(np.float32))
    model = cm.MFModel.from_arrays(P, Q, float("nan"))
    for criterion, want in NAN_CONSTANT.items():
        got = cm.evaluate(prob, model, criterion)
        assert abs(got - want) <= 1e-9, (criterion, got)


@pytest.mark.parametrize("k", [3199, 3200, 3201, 3621, 3622, 3623])
def test_long_rows_of_factors(lib, orc, cuda, k):
    """16 rows of 3,623 floats and what else a block holds are 227 KB; from 3,200 on the rows' sorted
    predictions have no room beside them."""
    rng = np.random.default_rng(k)
    m, n, nnz = 20, 11, 60
    P, Q = ((rng.standard_normal((x, k)) * 0.02).astype(np.float32) for x in (m, n))
    te = np.zeros(nnz, dtype=orc.NODE)
    te["u"], te["v"], te["r"] = rng.integers(0, m, nnz), rng.integers(0, n, nnz), rng.choice([-1, 1], nnz)
    prob = cm.MFProblem.from_arrays(te["u"], te["v"], te["r"], m=m, n=n)
    model = cm.MFModel.from_arrays(P, Q, 0.25)
    for criterion in (10, 11, 12, 13):
        assert abs(cm.evaluate(prob, model, criterion) - orc.evaluate(te, P, Q, 0.25, criterion, m, n)) <= 1e-9
