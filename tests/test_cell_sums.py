"""FP64 global steps of large meshes sum the face contributions of every cell
in a pass of their own, in groups of 32 cells; the step has to be the oracle's
on both sides of the size where the pass takes over, with a last group that is
not full, with boundary cells, and when a context's mesh shrinks below that
size and grows again."""
import numpy as np
import pytest

from common import RTOL_FP64, setup_case
from test_gpu_parity import assert_state_close, gpu_system

CELLS = 16384  # the pass is taken from this many cells on


@pytest.mark.gpu
@pytest.mark.parametrize("nside,bounded", [(25, False), (26, False), (27, True)])
def test_steps_around_the_size_of_the_sum_pass_vs_oracle(nside, bounded):
    from oracle.pyoracle import OracleSystem
    assert (nside ** 3 >= CELLS) == (nside >= 26) and nside ** 3 % 32
    m, W = setup_case(nside, "orszag_tang", seed=nside, noise=0.05)
    bnd = np.zeros(m.ncell, np.int32)
    if bounded:
        bnd[m.pos[:, 0] < 0.1] = 1  # REFLECTING
        bnd[m.pos[:, 0] > 0.9] = 3  # DIOD
    s, o = gpu_system(m, W, bnd=bnd), OracleSystem()
    o.set_mesh(m)
    o.init_problem(W, bnd=bnd)
    for _ in range(2):
        assert s.step(shared=True) == o.step(shared=True)
    assert_state_close(s.get_state(), o.get_state(), rtol=RTOL_FP64)


@pytest.mark.gpu
def test_mesh_shrinks_and_grows_across_the_size_of_the_sum_pass():
    import fvmhd3d_b200 as F
    s = F.System()
    for nside in (10, 26, 10, 26):
        m, W = setup_case(nside, "orszag_tang", seed=nside, noise=0.05)
        s.set_mesh(m)
        s.init_problem(W)
        fresh = gpu_system(m, W)
        for _ in range(2):
            s.step(shared=True)
            fresh.step(shared=True)
        a, b = s.get_state(), fresh.get_state()
        for k in a:
            assert np.array_equal(a[k], b[k]), (nside, k)
