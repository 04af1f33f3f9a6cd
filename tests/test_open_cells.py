"""The FP64 reconstruction keeps the constant n A of a cell's faces apart from
the neighbour differences; on a mesh whose cells are not closed that constant
is no round-off, and the gradient still has to be the reference's."""
import numpy as np
import pytest

from common import RTOL_FP64, setup_case
from test_gpu_parity import assert_state_close, gpu_system, oracle_system


@pytest.mark.gpu
@pytest.mark.parametrize("nside,rel", [(5, 1e-2), (8, 1e-6)])
def test_reconstruction_of_open_cells_vs_oracle(nside, rel):
    m, W = setup_case(nside, "orszag_tang", seed=nside, noise=0.05)
    rng = np.random.default_rng(nside)
    m.n = m.n * (1.0 + rel * rng.uniform(-1, 1, (m.nface, 1)))
    assert m.closure_error().max() > 0.1 * rel
    s, o = gpu_system(m, W), oracle_system(m, W)
    for _ in range(3):
        assert s.step(shared=True) == o.step(shared=True) == m.ncell
    assert_state_close(s.get_state(), o.get_state(), rtol=RTOL_FP64)
