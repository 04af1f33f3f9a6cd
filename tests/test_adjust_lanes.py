"""adjust_timesteps with several lanes per site: the rungs of strongly
jittered meshes, whose cells have from few to dozens of faces, against the
oracle's sequential sweep, exactly."""
import numpy as np
import pytest

import fvmhd3d_b200 as F


def ragged_case(nside, seed):
    rng = np.random.default_rng(seed)
    m = F.build_periodic(F.jittered_lattice(nside, 0.5, seed=seed), 1.0)
    ncell = m.ncell
    W = F.problems.perturbed(F.problems.orszag_tang(m.pos), 0.05, seed=seed)
    hot = rng.uniform(size=ncell) < 0.03  # neighbours many rungs apart
    W[hot, 4] *= 10.0 ** rng.uniform(2, 6, hot.sum())
    return m, W


@pytest.mark.gpu
@pytest.mark.parametrize("nside,fused", [(6, 0), (9, 0), (9, 700), (14, 0)])
def test_rungs_of_ragged_meshes_vs_oracle(nside, fused):
    from oracle.pyoracle import OracleSystem
    m, W = ragged_case(nside, seed=nside)
    links = np.diff(m.cell_face_off)
    assert links.min() < 10 and links.max() > 16  # from about one round of lanes to three
    s, o = F.System(), OracleSystem()
    for x in (s, o):
        x.set_mesh(m)
        x.init_problem(W)
    s.set_fused(fused)
    replays = 0
    for _ in range(12):
        assert s.step(shared=False) == o.step(shared=False)
        dirty, n, sequential = s.adjust_stats()
        replays = max(replays, n)
        a, b = s.get_state(), o.get_state()
        for k in ("rung", "tlast", "tend"):
            assert np.array_equal(a[k], b[k]), k
    assert replays >= 2
