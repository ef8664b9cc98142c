"""A batch that the GPU's memory does not hold is refused, and the network goes on with smaller ones."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm

pytestmark = pytest.mark.gpu


def test_batches_after_one_that_is_too_large(lib, cuda):
    """1.5 G rows want 576 GB for the bf16 input alone, refused before anything is launched; the loss and
    the gradients of 1,000 rows are the same before and after it."""
    import torch
    d_in, d_out, rows = 131, 128, 1000
    g = torch.Generator(device=cuda)
    g.manual_seed(2)
    X, T = (torch.randn(rows, d, generator=g, device=cuda) for d in (d_in, d_out))
    mlp = cm.MLP(d_in, 512, d_out, seed=3)
    before = mlp.loss_grad(X.data_ptr(), T.data_ptr(), rows), mlp.get(1)
    with pytest.raises(cm.CumfError):
        mlp.loss_grad(X.data_ptr(), T.data_ptr(), 1_500_000_000)
    after = mlp.loss_grad(X.data_ptr(), T.data_ptr(), rows), mlp.get(1)
    assert before[0] == after[0]
    np.testing.assert_array_equal(before[1], after[1])
