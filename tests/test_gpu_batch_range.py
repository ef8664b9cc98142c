"""Batched launch with ids outside the matrices: such records are skipped and the status says so,
wherever in a pair of records they are (one half of a worker's lanes each)."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm
from test_gpu_batch import as_f32, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("places", ["even", "odd", "both"])
@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_out_of_range_ids_are_reported(lib, orc, cuda, lanes, places):
    """One worker per problem, one of 100 records (a batch of 128, so a record is drawn at one place of
    its pairs or twice at places 100 apart): the oracle's bits, which skips the same records, and the
    range error from `status`."""
    import torch
    probs, host, lr, _keep = make(cuda, 3, min_k=64 if lanes == 32 else 0)
    h = host[-2]
    rec = h["rec"]
    assert len(rec) == 100
    start = orc.lib().or_batch_start(h["seed"], 0, 0, 0, len(rec))
    place = (np.arange(len(rec)) - start) % len(rec)
    bad = {"even": place % 16 == 4, "odd": place % 16 == 5, "both": place % 16 // 2 == 2}[places]
    rec["u"][bad & (place % 32 < 16)] = h["m"]
    rec["v"][bad & (place % 32 >= 16)] = -1
    h["d_R"].copy_(torch.from_numpy(rec.view(np.uint8).copy()))
    b = cm.Batch(probs)
    b.set_tuning(16, 2, 4, lanes=lanes)
    b.run(0, 1)
    torch.cuda.synchronize()
    for x in host:
        P = orc.init_factors(x["m"], x["k"], "fp16", x["seed"], 1)
        Q = orc.init_factors(x["n"], x["k"], "fp16", x["seed"], 2)
        skipped = orc.sgd_epochs(x["rec"], P, Q, "fp16", 1, lr, 0, 1, 0.05, 0.04, x["seed"], lanes=lanes)
        assert (skipped > 0) == (x is h)
        np.testing.assert_array_equal(as_f32(x["P"], x["m"], x["k"]), P)
        np.testing.assert_array_equal(as_f32(x["Q"], x["n"], x["k"]), Q)
    assert b.status() == 6  # CUMF_ERR_RANGE
