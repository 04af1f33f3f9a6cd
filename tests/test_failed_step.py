"""The step after one that failed midway computes its own face flags: those
the failed partial step left are not taken for the flags of every cell."""
import numpy as np
import pytest

import fvmhd3d_b200 as F


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
def test_global_step_after_a_failed_partial_step(precision):
    m = F.build_periodic(F.jittered_lattice(8, 0.1, seed=3), 1.0)
    W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=4)
    W[m.pos[:, 0] < 0.3, 4] *= 64.0  # cells of several rungs

    def system():
        s = F.System(precision=precision)
        s.set_mesh(m)
        s.init_problem(W)
        return s

    probe = system()
    active = [probe.step(shared=False) for _ in range(40)]
    last = next(k for k in range(39) if active[k + 1] < active[k] == m.ncell)  # whole, then partial
    out = []
    for anew in (False, True):
        s = system()
        assert [s.step(shared=False) for _ in range(last + 1)] == active[:last + 1]
        s.set_reduce(lambda dt: 1 / 0)
        with pytest.raises(F.FvmError):
            s.step(shared=False)
        assert 0 < s.active_faces().size < m.nface  # the failed step was a partial one
        s.set_reduce(None)
        if anew:
            s.set_positions(m.pos)  # the same positions: the flags are computed anew
        out.append((s.step(shared=True), s.active_face_count(), s.active_faces().size, s.get_state()))
    (ca, fa, na, a), (cb, fb, nb, b) = out
    assert ca == cb and fa == fb and na == nb
    for k in a:
        assert np.array_equal(a[k], b[k]), k
