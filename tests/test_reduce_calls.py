"""A timestep reduction that makes calls of its own on the context, more than
the number after which the staging of small batches moves to pinned memory:
the step continues with the reduction's value, and nobody else's memory is
written."""
import numpy as np
import pytest

import fvmhd3d_b200 as F
from test_zz_no_alloc import face_batch


@pytest.mark.gpu
def test_reduction_that_moves_the_staging():
    m = F.build_periodic(F.jittered_lattice(5, 0.1, seed=5), 1.0)
    W = F.problems.blast(m.pos)
    args = face_batch(40, seed=6)
    held, out = [], []
    for calls in (0, 150):
        s = F.System()
        s.set_mesh(m)
        s.init_problem(W)

        def reduce(dt):
            for _ in range(calls):
                s.compute_flux(*args)
            # what the calls freed is somebody else's now
            held.extend(np.full(n, 0xa5, np.uint8) for n in (65000, 8000, 8000, 4000, 4000, 2000, 2000) * 4)
            return 0.5 * dt

        s.set_reduce(reduce)
        for _ in range(3):
            s.step(shared=True)
        s.set_reduce(None)
        out.append((s.clock(), s.get_state()))
    assert all((h == 0xa5).all() for h in held)
    assert out[0][0] == out[1][0]
    for k in out[0][1]:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
