"""The persistent rung kernel on steps of few and of many involved cells (one
block per SM works up to 2048 of them, every block from there on): the stage
kernels' bits."""
import numpy as np
import pytest

import fvmhd3d_b200 as F


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
def test_few_and_many_involved_cells_same_bits(precision):
    m = F.build_periodic(F.jittered_lattice(22, 0.1, seed=2), 1.0)
    W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=5)
    W[m.pos[:, 0] < 0.3, 4] *= 64.0  # a third of the cells between the blast's rungs and the rest
    out, active = [], set()
    for fused in (0, m.ncell):
        s = F.System(precision=precision)
        s.set_mesh(m)
        s.init_problem(W)
        s.set_fused(fused)
        for _ in range(16):
            active.add(s.run(1, shared=False)[0])
        out.append(s.get_state())
        assert (s.fused_steps > 0) == (fused > 0)
    # an active cell has some 16 neighbours: steps on both sides of 2048
    assert min(active) * 17 < 2048 and any(2048 < a < m.ncell for a in active)
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
