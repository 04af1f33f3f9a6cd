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


@pytest.mark.gpu
@pytest.mark.parametrize("faces,calls", [(40, 130), (400, 260)])
def test_batches_around_the_pinning_of_their_staging(faces, calls):
    """The staging of batches of up to 64 KB is pinned after 128 of them, that
    of batches of up to 1 MB after 256; the results stay the first call's."""
    s = F.System()
    args = face_batch(faces, seed=6)
    want = s.compute_flux(*args)
    for _ in range(calls):
        for a, b in zip(s.compute_flux(*args), want):
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.gpu
def test_steps_around_the_pinning_of_what_they_read():
    """What a step reads back goes to pinned memory after 128 of them."""
    m = F.build_periodic(F.jittered_lattice(4, 0.1, seed=5), 1.0)
    W = F.problems.blast(m.pos)
    s, once = F.System(), F.System()
    for x in (s, once):
        x.set_mesh(m)
        x.init_problem(W)
    for k in range(150):
        assert s.step(shared=True) == m.ncell and s.active_face_count() == m.nface
    once.run(150, shared=True)
    assert s.clock() == once.clock()
    a, b = s.get_state(), once.get_state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
