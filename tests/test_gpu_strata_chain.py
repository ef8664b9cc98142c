"""Blocks whose ratings share rows at every distance: a row that a recent rating changed is taken
from that rating's result and stored after the last of them.  Bit for bit the serial restatement;
records outside the matrix change nothing and are reported."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm

pytestmark = pytest.mark.gpu


def epochs(torch, cuda, rec, m, n, k, precision, G, lr):
    eb = 4 if precision == "fp32" else 2
    d_R = torch.from_numpy(rec.view(np.uint8).copy()).to(cuda)
    d_S = torch.empty_like(d_R)
    d_off = torch.empty((G * G + 1) * 8, dtype=torch.uint8, device=cuda)
    cm.dev_strata_layout(d_R.data_ptr(), len(rec), G, d_S.data_ptr(), d_off.data_ptr())
    P = torch.empty(m * k * eb, dtype=torch.uint8, device=cuda)
    Q = torch.empty(n * k * eb, dtype=torch.uint8, device=cuda)
    cm.dev_init_factors(P.data_ptr(), m, k, precision, 5, 1)
    cm.dev_init_factors(Q.data_ptr(), n, k, precision, 5, 2)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    cm.dev_strata_epochs(d_S.data_ptr(), d_off.data_ptr(), G, P.data_ptr(), m, Q.data_ptr(), n, k, precision, lr,
                         0, 2, 0.05, 0.04, 5, status.data_ptr())
    torch.cuda.synchronize()
    dt = torch.float32 if precision == "fp32" else (torch.float16 if precision.startswith("fp16") else torch.bfloat16)
    return (P.view(dt).float().cpu().numpy().reshape(m, k), Q.view(dt).float().cpu().numpy().reshape(n, k),
            int(status.item()))


def ratings(rng, m, n, nnz):
    rec = np.empty(nnz, dtype=cm.NODE_DTYPE)
    rec["u"], rec["v"] = rng.integers(0, m, nnz), rng.integers(0, n, nnz)
    rec["r"] = (rng.integers(1, 6, nnz) / np.float32(1.7)).astype(np.float32)
    return rec


@pytest.mark.parametrize("k,precision", [(128, "fp16"), (128, "bf16sr"), (64, "fp16sr"), (32, "bf16"), (256, "fp16"),
                                         (128, "fp32"), (256, "fp32"), (32, "fp32")])
@pytest.mark.parametrize("m,n,nnz,G", [(1, 1, 11, 1), (9, 1, 200, 1), (3, 3, 500, 1), (40, 6, 900, 1), (12, 7, 700, 5),
                                       (64, 30, 333, 37), (5, 4, 3, 4)])
def test_strata_chains_bit_exact(lib, orc, cuda, k, precision, m, n, nnz, G):
    import torch
    rec = ratings(np.random.default_rng(k + nnz), m, n, nnz)
    lr = orc.lr_table(0.08, 0.3, 0.0, 6)
    P, Q, status = epochs(torch, cuda, rec, m, n, k, precision, G, lr)
    assert status == 0
    Po, Qo = orc.init_factors(m, k, precision, 5, 1), orc.init_factors(n, k, precision, 5, 2)
    lanes = min(32, k * (4 if precision == "fp32" else 2) // 16)
    assert orc.strata_epochs(rec, Po, Qo, precision, G, lr, 0, 2, 0.05, 0.04, 5, lanes) == 0
    np.testing.assert_array_equal(P, Po)
    np.testing.assert_array_equal(Q, Qo)


def test_strata_records_outside_the_matrix(lib, orc, cuda):
    import torch
    rng = np.random.default_rng(3)
    m, n, k, G = 12, 7, 64, 3
    rec = ratings(rng, m, n, 400)
    bad = ratings(rng, m, n, 60)
    bad["u"][::3], bad["v"][1::3], bad["u"][2::3] = m + 1, n, -2
    where = np.sort(rng.integers(0, len(rec) + 1, len(bad)))
    lr = orc.lr_table(0.08, 0.3, 0.0, 6)
    P, Q, status = epochs(torch, cuda, rec, m, n, k, "fp16", G, lr)
    Pb, Qb, status_b = epochs(torch, cuda, np.insert(rec, where, bad), m, n, k, "fp16", G, lr)
    assert status == 0 and status_b != 0
    np.testing.assert_array_equal(P, Pb)
    np.testing.assert_array_equal(Q, Qb)


@pytest.mark.parametrize("G", [700, 1200])  # fewer rows per chunk, so that all workers are resident
def test_strata_many_workers_with_long_rows(lib, orc, cuda, G):
    import torch
    rng = np.random.default_rng(G)
    m, n, k = 3 * G, 2 * G + 5, 256
    rec = ratings(rng, m, n, 3000)
    rec["u"][::4], rec["v"][::4] = G * rng.integers(0, 3, 750), G * rng.integers(0, 2, 750)  # one long block
    lr = orc.lr_table(0.08, 0.3, 0.0, 6)
    P, Q, status = epochs(torch, cuda, rec, m, n, k, "fp32", G, lr)
    assert status == 0
    Po, Qo = orc.init_factors(m, k, "fp32", 5, 1), orc.init_factors(n, k, "fp32", 5, 2)
    assert orc.strata_epochs(rec, Po, Qo, "fp32", G, lr, 0, 2, 0.05, 0.04, 5, 32) == 0
    np.testing.assert_array_equal(P, Po)
    np.testing.assert_array_equal(Q, Qo)


def test_strata_epochs_replay_from_a_graph(lib, orc, cuda):
    import torch
    m, n, k, G, precision = 40, 6, 64, 5, "fp16"
    rec = ratings(np.random.default_rng(9), m, n, 700)
    lr = orc.lr_table(0.08, 0.3, 0.0, 6)
    P, Q, _ = epochs(torch, cuda, rec, m, n, k, precision, G, lr)
    d_R = torch.from_numpy(rec.view(np.uint8).copy()).to(cuda)
    d_S, d_off = torch.empty_like(d_R), torch.empty((G * G + 1) * 8, dtype=torch.uint8, device=cuda)
    cm.dev_strata_layout(d_R.data_ptr(), len(rec), G, d_S.data_ptr(), d_off.data_ptr())
    dP = torch.empty(m * k, dtype=torch.float16, device=cuda)
    dQ = torch.empty(n * k, dtype=torch.float16, device=cuda)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cm.dev_strata_epochs(d_S.data_ptr(), d_off.data_ptr(), G, dP.data_ptr(), m, dQ.data_ptr(), n, k, precision,
                             lr, 0, 2, 0.05, 0.04, 5, 0, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        cm.dev_init_factors(dP.data_ptr(), m, k, precision, 5, 1)
        cm.dev_init_factors(dQ.data_ptr(), n, k, precision, 5, 2)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(dP.float().cpu().numpy().reshape(m, k), P)
        np.testing.assert_array_equal(dQ.float().cpu().numpy().reshape(n, k), Q)
