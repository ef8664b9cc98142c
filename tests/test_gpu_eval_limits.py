"""Ranking criteria at the limits of the column sweep: a model whose constant is NaN (predictions of
ids outside the model are NaN)."""
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
