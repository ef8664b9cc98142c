"""The user features' item rows are read by loads of 4, 2 or 1 floats, as the rows' length and
alignment allow: every width gives the same bits, and the float64 restatement's values."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 31, 32, 33, 34, 64, 66, 68, 127, 128, 130, 132, 256, 260])
def test_user_features_same_bits_for_every_load_width(lib, cuda, k):
    import torch
    rng = np.random.default_rng(k)
    n = 150
    degree = np.concatenate([np.arange(0, 70), [95, 96, 97, 128, 1000]])  # around the 32-rating fetches
    m = len(degree)
    u = rng.permutation(np.repeat(np.arange(m), degree)).astype(np.int32)
    rec = np.empty(len(u), dtype=cm.NODE_DTYPE)
    rec["u"], rec["v"] = u, rng.integers(0, n, len(u))
    rec["r"] = rng.integers(1, 6, len(u)).astype(np.float32)
    Q = (rng.standard_normal((n, k)) * 0.3).astype(np.float32)
    dR = torch.from_numpy(rec.view(np.uint8).copy()).to(cuda)
    got = []
    for shift in (0, 1, 2):  # floats that the base lies past a 16-byte boundary
        store = torch.zeros(n * k + 4, device=cuda)
        dQ = store[shift:shift + n * k]
        dQ.copy_(torch.from_numpy(Q.ravel()))
        dX = torch.full((m, k + 3), float("nan"), device=cuda)
        cm.user_features(dR.data_ptr(), len(rec), dQ.data_ptr(), n, k, m, dX.data_ptr())
        got.append(dX.cpu().numpy())
    assert (got[0] == got[1]).all() and (got[0] == got[2]).all()
    ref = mlp_oracle.user_features(rec, Q, m, k)
    assert np.abs(got[0] - ref).max() <= 1e-4 * np.abs(ref).max()
