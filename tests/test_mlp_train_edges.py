"""The fused training kernels at the edges of their 64-row chunks, 128-row
tiles and per-CTA rows, against the oracle's backward pass of the same rounded
network (the bound of the gradient test: BF16 operands, FP32 sums)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

GRAD_RTOL = 1e-2


@pytest.mark.gpu
# one tile and its remainders; rows per CTA of 128, 192 (an odd number of
# chunks) and 256 (more than 64 CTAs' worth of 128), each with a remainder
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 128, 129, 192, 257, 320, 448, 8193, 16385])
def test_gradient_at_tile_edges_vs_oracle(rows):
    import fvmhd3d_b200 as F
    rng = np.random.default_rng(rows)
    p = M.init_params(7)
    X = rng.normal(size=(rows, M.NIN)).astype(np.float32)
    T = rng.normal(size=(rows, M.NOUT)).astype(np.float32)
    wt = np.linspace(0.5, 2.0, M.NOUT)
    s = F.System()
    s.mlp_set_weights(p)
    loss, g = s.mlp_grad(X, T, wt)
    rloss, rg = M.loss_and_grad(p, X, T, wt)
    assert abs(loss - rloss) <= 1e-3 * rloss
    o = 0
    for shp in M.SHAPES:
        k = int(np.prod(shp))
        a, b = g[o:o + k], rg[o:o + k]
        assert np.linalg.norm(a - b) <= GRAD_RTOL * np.linalg.norm(b), (shp, np.linalg.norm(a - b) / np.linalg.norm(b))
        o += k


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [70, 8192])
def test_training_repeats_its_bits(batch):
    """Every sum of a training step has a fixed order: the same call gives the
    same weights and losses."""
    import fvmhd3d_b200 as F
    rng = np.random.default_rng(3)
    X = rng.normal(size=(20000, M.NIN)).astype(np.float32)
    T = np.tanh(X[:, :M.NOUT])
    got = []
    for _ in range(2):
        s = F.System()
        s.mlp_set_weights(M.init_params(5))
        loss = s.mlp_train(X, T, batch=batch, steps=8, lr=1e-3, seed=2)
        got.append((loss, s.mlp_get_weights()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
