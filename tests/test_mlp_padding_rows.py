"""Rows that fill a batch up to a tile of the training kernels take no part in
the gradients, also where the network overflows on their zero inputs (a hidden
unit whose large bias the inputs of every row of the batch cancel)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

GRAD_RTOL = 1e-2  # the bound of the gradient test: BF16 operands, FP32 sums


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 65, 100, 127, 129, 300])
def test_gradient_where_zero_inputs_overflow(rows):
    import fvmhd3d_b200 as F
    rng = np.random.default_rng(rows)
    parts = M.unpack(M.init_params(7))
    parts[0][5] = 0.0
    parts[0][5, 0], parts[1][5] = -2.0 ** 70, 2.0 ** 70
    p = M.pack(parts).astype(np.float32)
    X = rng.normal(size=(rows, M.NIN)).astype(np.float32)
    X[:, 0] = 1.0
    T = rng.normal(size=(rows, M.NOUT)).astype(np.float32)
    s = F.System()
    s.mlp_set_weights(p)
    loss, g = s.mlp_grad(X, T)
    rloss, rg = M.loss_and_grad(p, X, T)
    assert abs(loss - rloss) <= 1e-3 * rloss
    assert np.isfinite(rg).all() and np.isfinite(g).all()
    o = 0
    for shp in M.SHAPES:
        k = int(np.prod(shp))
        assert np.linalg.norm(g[o:o + k] - rg[o:o + k]) <= GRAD_RTOL * np.linalg.norm(rg[o:o + k]), shp
        o += k
