"""The update kernel that takes two records at a time, where it can go wrong: records that share
rows with their neighbours, problems shorter than a batch (the sample wraps inside a staged
chunk), out-of-range ids beside valid ones, a last block with idle groups, and non-finite
factors under stochastic rounding.  One worker, bit-exact against the oracle."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm
from test_gpu_parity import default_lanes, dev, elem, storage_to_float

pytestmark = pytest.mark.gpu


def run(cuda, orc, rec, m, n, k, precision, workers=1, epochs=2, prefetch=-1, poison=()):
    import torch
    P = torch.empty(m * k * elem(precision), dtype=torch.uint8, device=cuda)
    Q = torch.empty(n * k * elem(precision), dtype=torch.uint8, device=cuda)
    cm.dev_init_factors(P.data_ptr(), m, k, precision, 5, 1)
    cm.dev_init_factors(Q.data_ptr(), n, k, precision, 5, 2)
    rows = P.view({"fp32": torch.float32, "fp16": torch.float16, "fp16sr": torch.float16}.get(precision, torch.bfloat16))
    for i, x in poison:
        rows[i] = x
    P0, Q0 = storage_to_float(P, precision, m, k), storage_to_float(Q, precision, n, k)
    lr = orc.lr_table(0.08, 0.3, 0.0, 8)
    d_R, d_lr, status = dev(rec, cuda), torch.from_numpy(lr).to(cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    cm.sgd_update(d_R.data_ptr(), len(rec), P.data_ptr(), m, Q.data_ptr(), n, k, precision, workers, 0, d_lr.data_ptr(),
                  0, epochs, 0.05, 0.04, 5, status.data_ptr(), prefetch=prefetch)
    torch.cuda.synchronize()
    got = storage_to_float(P, precision, m, k), storage_to_float(Q, precision, n, k)
    skipped = orc.sgd_epochs(rec, P0, Q0, precision, 1, lr, 0, epochs, 0.05, 0.04, 5, lanes=default_lanes(k, precision))
    return got, (P0, Q0), int(status.item()), skipped


def records(m, n, nnz, seed):
    rng = np.random.default_rng(seed)
    rec = np.empty(nnz, dtype=cm.NODE_DTYPE)
    rec["u"], rec["v"] = rng.integers(0, m, nnz), rng.integers(0, n, nnz)
    rec["r"] = rng.integers(1, 6, nnz).astype(np.float32) / np.float32(1.2)
    return rec


@pytest.mark.parametrize("prefetch", [0, 3])
@pytest.mark.parametrize("precision,k", [("fp16", 128), ("fp16", 32), ("fp32", 32), ("fp32", 128), ("bf16sr", 64),
                                         ("bf16", 256), ("fp16sr", 64)])
@pytest.mark.parametrize("m,n,nnz", [(1, 1, 1), (2, 1, 5), (1, 3, 127), (3, 2, 128), (2, 7, 129), (5, 4, 1000)])
def test_shared_rows_and_wraps(lib, orc, cuda, m, n, nnz, precision, k, prefetch):
    got, want, status, skipped = run(cuda, orc, records(m, n, nnz, nnz), m, n, k, precision, prefetch=prefetch)
    assert status == 0 and skipped == 0
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("precision,k", [("fp16", 128), ("fp32", 64), ("bf16sr", 32)])
@pytest.mark.parametrize("odd", [0, 1, 2])
def test_out_of_range_ids_beside_valid_ones(lib, orc, cuda, odd, precision, k):
    """First, second or both records of a pair out of range; the valid id of such a record and the
    last row (which stands in for it in flight) are in use by the neighbours."""
    m, n, nnz = 6, 5, 600
    rec = records(m, n, nnz, 7)
    bad = np.arange(nnz) % 8 == 2 + odd if odd < 2 else np.arange(nnz) % 8 // 2 == 1
    rec["u"][bad & (np.arange(nnz) % 3 == 0)] = m
    rec["u"][bad & (np.arange(nnz) % 3 == 1)] = -1
    rec["v"][bad & (np.arange(nnz) % 3 == 2)] = n + 3
    got, want, status, skipped = run(cuda, orc, rec, m, n, k, precision)
    assert skipped > 0 and status == 6  # CUMF_ERR_RANGE
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


def test_non_finite_factors_under_stochastic_rounding(lib, orc, cuda):
    m, n, k = 40, 30, 64
    rec = records(m, n, 900, 3)
    with np.errstate(all="ignore"):
        got, want, _, _ = run(cuda, orc, rec, m, n, k, "bf16sr", epochs=1,
                              poison=((5, np.inf), (3 * k + 1, -np.inf), (9 * k + 63, np.nan), (70, 3.3e38), (71, -3.3e38)))
    assert not np.isfinite(want[0]).all()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("precision,k", [("fp16", 128), ("fp32", 128), ("bf16", 32)])
def test_many_workers_touch_only_the_sampled_rows(lib, cuda, precision, k):
    """13 workers: the last block has idle groups.  Rows that no rating names stay as they were,
    the others move and stay finite."""
    import torch
    m, n, nnz = 4000, 3000, 20_000
    rec = records(m // 2, n // 2, nnz, 11)
    P = torch.empty(m * k * elem(precision), dtype=torch.uint8, device=cuda)
    Q = torch.empty(n * k * elem(precision), dtype=torch.uint8, device=cuda)
    cm.dev_init_factors(P.data_ptr(), m, k, precision, 5, 1)
    cm.dev_init_factors(Q.data_ptr(), n, k, precision, 5, 2)
    before = storage_to_float(P, precision, m, k), storage_to_float(Q, precision, n, k)
    d_R, d_lr = dev(rec, cuda), torch.from_numpy(cm.lr_schedule(0.08, 0.3, 0.0, 4)).to(cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    cm.sgd_update(d_R.data_ptr(), nnz, P.data_ptr(), m, Q.data_ptr(), n, k, precision, 13, 0, d_lr.data_ptr(), 0, 3, 0.05,
                  0.05, 5, status.data_ptr())
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for a, b, rows in ((before[0], storage_to_float(P, precision, m, k), m), (before[1], storage_to_float(Q, precision, n, k), n)):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a[rows // 2:], b[rows // 2:])
        assert (a[:rows // 2] != b[:rows // 2]).any(axis=1).mean() > 0.5
