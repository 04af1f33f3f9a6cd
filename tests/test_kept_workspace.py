"""Calls on host arrays share one work space and staging of their context:
batches of changing size, over the staging's and the work space's limits, of
different entry points in turn, give what a context of their own gives; and
steps replayed after the first eager ones give the eager steps' bits."""
import numpy as np
import pytest

import fvmhd3d_b200 as F
from fvmhd3d_b200 import learned
from test_zz_no_alloc import face_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 250, 300, 3, 4800, 4900, 7), (250000, 40, 300000)])
def test_batches_of_changing_size(sizes):
    shared = F.System()
    p = learned.init_params(2)
    shared.mlp_set_weights(p)
    for rounds in range(6 if max(sizes) < 10000 else 1):  # past the calls that pin the larger staging
        for k, n in enumerate(sizes):
            own = F.System()
            args = face_batch(n, seed=10 * rounds + k)
            wij, Wi, Wj, jbnd, normal = args
            for a, b in zip(shared.compute_flux(wij, Wi, Wj, jbnd, normal), own.compute_flux(wij, Wi, Wj, jbnd, normal)):
                assert np.array_equal(a, b, equal_nan=True)
            if rounds == 0:
                own.mlp_set_weights(p)
                X = np.random.default_rng(k).normal(size=(n, 16)).astype(np.float32)
                assert np.array_equal(shared.mlp_eval(X), own.mlp_eval(X))
                T = np.tanh(X[:, :8])
                (la, ga), (lb, gb) = shared.mlp_grad(X, T), own.mlp_grad(X, T)
                assert la == lb and np.array_equal(ga, gb)


@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
def test_steps_after_the_first_eager_ones(precision):
    m = F.build_periodic(F.jittered_lattice(8, 0.1, seed=3), 1.0)
    W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=4)
    eager, later = F.System(precision=precision), F.System(precision=precision)
    for s in (eager, later):
        s.set_mesh(m)
        s.init_problem(W)
    eager.set_profiling(True)  # keeps every step eager
    for k in range(14):  # partial steps among the global ones
        assert eager.step(shared=k % 5 != 4) == later.step(shared=k % 5 != 4)
    assert later.launch_count > 0 and eager.clock() == later.clock()
    a, b = eager.get_state(), later.get_state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def test_calls_across_the_pinning_of_the_small_staging():
    """The staging of small calls becomes pinned memory after 64 of them."""
    m = F.build_periodic(F.jittered_lattice(5, 0.1, seed=5), 1.0)
    W = F.problems.blast(m.pos)
    s, plain = F.System(), F.System()
    for x in (s, plain):
        x.set_mesh(m)
        x.init_problem(W)
    args = face_batch(40, seed=6)
    want = F.System().compute_flux(*args)
    for k in range(50):
        assert s.step(shared=True) == plain.step(shared=True)
        assert s.clock() == plain.clock()
        for a, b in zip(s.compute_flux(*args), want):
            assert np.array_equal(a, b, equal_nan=True)
    a, b = s.get_state(), plain.get_state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
