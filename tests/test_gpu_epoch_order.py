"""Several epochs in one call: every worker is resident (or the epochs are launched one by one), so
that no worker applies the first epoch's learning rate after others have run them all."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp16", "fp16sr"])
def test_last_workers_run_their_first_epoch_in_time(lib, orc, cuda, precision):
    """9,728 workers (1,024 threads on each of 152 SMs) with one batch each, every record a user and
    an item of its own, item rows and ratings zero: a draw multiplies the user's row by
    1 - lr * lambda_p, which is 0 in epoch 0 and 2^17, more than fp16 holds, in epochs 1 and 2.  A row
    drawn in epoch 0 only by workers with the last indexes, and later by others, ends at 0, or
    not finite where those workers came last.  (Workers of one wave drift, so a few may.)"""
    import torch
    workers, k, epochs = 9_728, 128, 3
    m = workers * 128
    rec = np.zeros(m, dtype=cm.NODE_DTYPE)
    rec["u"] = rec["v"] = np.arange(m)
    P, Q = torch.ones(m, k, dtype=torch.float16, device=cuda), torch.zeros(m, k, dtype=torch.float16, device=cuda)
    d_R = torch.from_numpy(rec.view(np.uint8).copy()).to(cuda)
    d_lr = torch.tensor([1.0, 1.0 - 2.0 ** 17, 1.0 - 2.0 ** 17], device=cuda)
    cm.sgd_update(d_R.data_ptr(), m, P.data_ptr(), m, Q.data_ptr(), m, k, precision, workers, 0, d_lr.data_ptr(), 0,
                  epochs, 1.0, 1.0, 3)
    torch.cuda.synchronize()
    last = workers - workers // 12
    drawn = np.zeros((2, 2, m), bool)  # [epoch 0, later][by the others, by the last]
    for e in range(epochs):
        for w in range(workers):
            a = orc.lib().or_batch_start(3, e, w, 0, m)
            d = drawn[min(e, 1), int(w >= last)]
            d[a:a + 128] = True
            d[:max(0, a + 128 - m)] = True
    rows = drawn[0, 1] & ~drawn[0, 0] & drawn[1, 0]
    assert rows.sum() > m // 100
    late = 1 - torch.isfinite(P).all(1).cpu().numpy()[rows].mean()
    print(precision, "rows", rows.sum(), "share late %.4f" % late)
    assert late < 0.5, late
