"""The persistent rung kernel on steps where every block of its launch works:
such steps are run by it, and two contexts that run them at the same time do
not keep each other's blocks out (its launch is cooperative)."""
import threading

import numpy as np
import pytest

import fvmhd3d_b200 as F

pytestmark = pytest.mark.gpu
WIDE = 2048  # involved cells from which on every block works


def system(precision, fused, contrast):
    m = F.build_periodic(F.jittered_lattice(22, 0.1, seed=2), 1.0)
    W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=5)
    W[m.pos[:, 0] < 0.3, 4] *= contrast
    s = F.System(precision=precision)
    s.set_mesh(m)
    s.init_problem(W)
    s.set_fused(m.ncell if fused else 0)
    return s


@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
def test_steps_in_which_every_block_works(precision):
    s, plain = (system(precision, f, 64.0) for f in (True, False))
    wide = narrow = 0
    for _ in range(48):
        before = s.fused_steps
        assert s.run(1, shared=False) == plain.run(1, shared=False)
        f = s.active_faces()
        involved = np.unique(np.concatenate([s.mesh.s1[f], s.mesh.s2[f]])).size
        assert s.fused_steps - before == (involved < s.mesh.ncell)
        wide += WIDE <= involved < s.mesh.ncell
        narrow += involved < WIDE
    assert wide >= 3 and narrow + wide == s.fused_steps
    a, b = s.get_state(), plain.get_state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("precision", [F.FVM_PREC_FP64, F.FVM_PREC_FP32])
def test_two_contexts_at_the_same_time(precision):
    # most of its steps involve more than WIDE cells
    plain, both = system(precision, False, 1024.0), [system(precision, True, 1024.0) for _ in range(2)]
    for s in both:
        s.run(1, shared=False)  # the first call captures
    plain.run(1, shared=False)
    start, failed = threading.Barrier(2), []

    def work(s):
        try:
            start.wait()
            s.run(47, shared=False)
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in both]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    plain.run(47, shared=False)
    want = plain.get_state()
    for s in both:
        assert s.fused_steps > 10
        got = s.get_state()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
