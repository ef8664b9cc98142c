"""The training step's fused products against the float64 restatement at the sizes where their
tiling changes: one and several row tiles, short last tiles, one CTA per SM or two, K in one or
several parts, 64-wide layers; with unaligned targets.  A step gives the same bits every run."""
import numpy as np
import pytest

import cumf_sgd_gb300 as cm
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d_in,h,d_out", [(1, 5, 64, 64), (127, 64, 64, 64), (129, 131, 192, 64),
                                               (640, 35, 512, 128), (2500, 131, 512, 192), (5000, 67, 512, 128),
                                               (4097, 131, 128, 256), (12000, 16, 64, 64), (11000, 20, 1024, 64)])
def test_mlp_step_gradients_match_fp64(lib, cuda, rows, d_in, h, d_out):
    import torch
    rng = np.random.default_rng(rows + h)
    X = rng.standard_normal((rows, d_in)).astype(np.float32) * 0.5
    T = rng.standard_normal((rows, d_out)).astype(np.float32) * 0.2
    mlp = cm.MLP(d_in, h, d_out, seed=3)
    params = mlp.get(0)
    dX = torch.from_numpy(X).to(cuda)
    l16, g16, g64, bounds = mlp_oracle.gradient_bounds(params, X, T, d_in, h, d_out)
    got = []
    for shift in (0, 1, 0):  # floats that the targets lie past a 16-byte boundary
        store = torch.zeros(rows * d_out + 4, device=cuda)
        dT = store[shift:shift + rows * d_out]
        dT.copy_(torch.from_numpy(T.ravel()))
        loss = mlp.loss_grad(dX.data_ptr(), dT.data_ptr(), rows)
        got.append((loss, mlp.get(1)))
        assert abs(loss - l16) <= 1e-3 * l16, (loss, l16)
    for loss, grads in got[1:]:
        assert loss == got[0][0] and (grads == got[0][1]).all()
    split = [mlp_oracle.unpack(x, d_in, h, d_out) for x in (got[0][1], g16, g64)]
    for name, g, r16, r64 in zip(mlp_oracle.GRAD_NAMES, *split):
        assert mlp_oracle.rel_err(g, r16) <= 3e-3, name
        assert mlp_oracle.rel_err(g, r64) <= bounds[name], name


def test_mlp_training_gives_the_same_bits_every_run(lib, cuda):
    import torch
    rng = np.random.default_rng(8)
    rows, d_in, h, d_out = 1700, 35, 256, 64  # steps of 512 rows and a last one of 164
    dX = torch.from_numpy(rng.standard_normal((rows, d_in)).astype(np.float32)).to(cuda)
    dT = torch.from_numpy(rng.standard_normal((rows, d_out)).astype(np.float32) * 0.2).to(cuda)
    runs = []
    for _ in range(2):
        mlp = cm.MLP(d_in, h, d_out, seed=5)
        loss = mlp.train(dX.data_ptr(), dT.data_ptr(), rows, epochs=2, batch=512, lr=1e-3, seed=3)
        runs.append((loss, mlp.get(0), mlp.get(1)))
    assert runs[0][0] == runs[1][0]
    assert (runs[0][1] == runs[1][1]).all() and (runs[0][2] == runs[1][2]).all()


@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e-12, 1e20, "mixed"])
def test_mlp_loss_is_a_double_sum_at_every_magnitude(lib, cuda, scale):
    """Zero parameters: the errors are the targets.  A sum of 300 x 64 non-negative doubles is
    within 300 * 64 * 2^-53 = 2e-12 of the exact one in any order."""
    import torch
    rng = np.random.default_rng(2)
    rows, d_in, h, d_out = 300, 16, 64, 64
    factor = 10.0 ** rng.uniform(-12, 8, (rows, d_out)) if scale == "mixed" else scale
    T = (rng.standard_normal((rows, d_out)) * factor).astype(np.float32)
    mlp = cm.MLP(d_in, h, d_out, seed=1)
    mlp.set(np.zeros_like(mlp.get(0)))
    dX, dT = torch.ones(rows, d_in, device=cuda), torch.from_numpy(T).to(cuda)
    exact = float((T.astype(np.longdouble) ** 2).sum() / rows)
    assert abs(mlp.loss_grad(dX.data_ptr(), dT.data_ptr(), rows) - exact) <= 2e-12 * exact
