"""First calls of a context: the kept work space is not the only block of the
device's stream-ordered pool (making and releasing that cost each context's
first call, and its destruction, 200 us), and it grows without changing results."""
import numpy as np
import pytest

import fvmhd3d_b200 as F
from fvmhd3d_b200 import learned
from test_zz_no_alloc import face_batch


def pool_peak(reset=False):
    from cuda.bindings import runtime as rt
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    if reset:
        from cuda.bindings import driver as dr
        assert rt.cudaMemPoolSetAttribute(pool, attr, dr.cuuint64_t(0))[0] == rt.cudaError_t.cudaSuccess
    err, v = rt.cudaMemPoolGetAttribute(pool, attr)
    assert err == rt.cudaError_t.cudaSuccess
    return int(v)


@pytest.mark.gpu
@pytest.mark.parametrize("faces", [1, 3000, 40000])
def test_first_calls_leave_the_pool_alone(faces):
    p = learned.init_params(2)
    X = np.random.default_rng(1).normal(size=(faces, 16)).astype(np.float32)
    want_f, want_y = None, None
    for _ in range(2):
        s = F.System()
        before = pool_peak(reset=True)
        f = s.compute_flux(*face_batch(faces, seed=3))
        s.mlp_set_weights(p)
        y = s.mlp_eval(X)
        m = F.build_periodic(F.jittered_lattice(6, 0.1, seed=3), 1.0)
        s.set_mesh(m)
        s.init_problem(F.problems.blast(m.pos))
        s.step(shared=True)
        s.close()
        assert pool_peak() <= before
        if want_f is not None:
            assert np.array_equal(y, want_y) and all(np.array_equal(a, b, equal_nan=True) for a, b in zip(f, want_f))
        want_f, want_y = f, y
