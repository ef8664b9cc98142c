"""RMSE over row lengths with one, two and four ratings per turn and any length, rating counts
around the turns, and ids outside the model (predicted as b, as NaN dots are)."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [4, 32, 33, 64, 96, 128, 256])
@pytest.mark.parametrize("nnz", [1, 5, 257, 30000, 200003])
def test_dev_rmse_matches_fp64(lib, cuda, k, nnz):
    import torch
    rng = np.random.default_rng(k + nnz)
    m, n, b = 900, 300, 2.5
    rec = np.empty(nnz, dtype=cm.NODE_DTYPE)
    rec["u"], rec["v"] = rng.integers(0, m, nnz), rng.integers(0, n, nnz)
    rec["r"] = rng.integers(1, 6, nnz)
    rec["u"][::7], rec["v"][3::11] = -1, n
    P = rng.standard_normal((m, k)).astype(np.float32) / np.float32(np.sqrt(k))
    Q = rng.standard_normal((n, k)).astype(np.float32)
    Q[5, 0] = np.nan
    inside = (rec["u"] >= 0) & (rec["u"] < m) & (rec["v"] < n)
    z = np.full(nnz, b)
    dot = np.einsum("ij,ij->i", P[rec["u"][inside]].astype(np.float64), Q[rec["v"][inside]].astype(np.float64))
    z[inside] = np.where(np.isnan(dot), b, dot)
    want = np.sqrt(np.mean((rec["r"] - z) ** 2))
    dR = torch.from_numpy(rec.view(np.uint8).copy()).to(cuda)
    dP, dQ = torch.from_numpy(P).to(cuda), torch.from_numpy(Q).to(cuda)
    got = cm.dev_rmse(dR.data_ptr(), nnz, dP.data_ptr(), m, dQ.data_ptr(), n, k, b)
    # a float dot of k terms is off by at most k 2^-24 of the sum of magnitudes (about 2), the
    # square by 2^-24
    assert abs(got - want) <= (2 * k + 4) * 2.0 ** -24 * max(1.0, want)
    assert got == cm.dev_rmse(dR.data_ptr(), nnz, dP.data_ptr(), m, dQ.data_ptr(), n, k, b)
