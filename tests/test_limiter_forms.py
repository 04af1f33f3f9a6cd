"""Partial steps on meshes on both sides of the size from which the staged
limiter and the one over the list are launched apart (65,536 cells): the bits
of the per-thread limiter."""
import numpy as np
import pytest

import fvmhd3d_b200 as F


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
@pytest.mark.parametrize("side", [40, 41])  # 64,000 and 68,921 cells
def test_limiter_launched_together_and_apart(side, precision):
    m = F.build_periodic(F.jittered_lattice(side, 0.1, seed=1), 1.0)
    W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=5)
    W[m.pos[:, 0] < 0.3, 4] *= 64.0
    out, involved = [], set()
    for staged in (0, 1):
        s = F.System(precision=precision, static_mesh=True)
        s.set_mesh(m)
        s.init_problem(W)
        s.set_tuning(staged, 32, 32, 64)
        for _ in range(16):
            s.run(1, shared=False)
            f = s.active_faces()
            involved.add(np.unique(np.concatenate([m.s1[f], m.s2[f]])).size)
        out.append(s.get_state())
    # every cell, some, and few enough for lanes of a cell
    assert m.ncell in involved and any(4096 < k < m.ncell for k in involved) and min(involved) <= 4096
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
