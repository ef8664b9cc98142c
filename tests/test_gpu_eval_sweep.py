"""The column sweep of the ranking criteria at the edges of its tiles: column counts around the
thread block and the two-column step, row groups of 1, 16 and 17, rows whose positives do not
fit the shared-memory copy, factor lengths that are odd or fill shared memory, columns beyond the
model.  Against the oracle, 1e-9 (counts of exact float comparisons)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,extra,per_row", [
    (1, 255, 1, 0, 3), (16, 256, 32, 0, 5), (17, 257, 33, 0, 5), (33, 512, 64, 3, 9), (5, 513, 128, 600, 4),
    (40, 1025, 16, 0, 20), (3, 5000, 8, 0, 700), (2, 1500, 8, 10, 1100), (18, 300, 700, 0, 6), (4, 64, 3300, 0, 6),
    (20, 1, 8, 0, 1), (6, 40, 5, 0, 40),
])
def test_sweep_edges(lib, cuda, orc, m, n, k, extra, per_row):
    import cumf_sgd_gb300 as cm
    rng = np.random.default_rng(m * n + k)
    P = (rng.standard_normal((m, k)) * 0.3).astype(np.float32)
    Q = (rng.standard_normal((n, k)) * 0.3).astype(np.float32)
    if n > 3:
        Q[n // 2] = Q[n // 3]  # equal predictions
    if m > 2:
        P[1, 0] = np.nan       # predicts b
    nnz = m * per_row
    te = np.zeros(nnz, dtype=orc.NODE)
    te["u"] = np.repeat(np.arange(m), per_row)
    te["v"] = np.concatenate([rng.choice(n + extra, per_row, replace=False) if per_row <= n + extra
                              else rng.integers(0, n + extra, per_row) for _ in range(m)])
    te["r"] = rng.choice(np.array([-1, 1], dtype=np.float32), nnz, p=[0.2, 0.8])
    te = te[rng.permutation(nnz)]
    prob = cm.MFProblem.from_arrays(te["u"], te["v"], te["r"], m=m, n=n + extra)
    model = cm.MFModel.from_arrays(P, Q, 0.25)
    for c in (10, 11, 12, 13):
        ref, got = orc.evaluate(te, P, Q, 0.25, c, m, n + extra), cm.evaluate(prob, model, c)
        assert (np.isnan(ref) and np.isnan(got)) or abs(got - ref) <= 1e-9 * max(1.0, abs(ref)), (c, got, ref)
