"""The link tables built at mesh installation for cells of one to more than 64
links (one to three rounds of a warp): steps on a star of cells whose hub has
every other cell as its neighbour give the oracle's active faces and rungs,
which walk the links in both orders."""
import numpy as np
import pytest

import fvmhd3d_b200 as F


def hub_mesh(spokes):
    """A hub cell with a closed shell of `spokes` faces, one to each spoke
    cell; every spoke cell's own face closes nothing, which no table needs."""
    n = spokes + 1
    rng = np.random.default_rng(spokes)
    d = rng.normal(size=(spokes, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    order = rng.permutation(spokes) + 1  # neighbours in no order along the hub's links
    s1, s2 = np.zeros(spokes, np.int32), order.astype(np.int32)
    pos = np.full((n, 3), 0.5)
    pos[order] += 0.2 * d
    normal = 0.01 * d
    off = np.concatenate([[0, spokes], spokes + np.arange(1, spokes + 1)]).astype(np.int64)
    ids = np.concatenate([np.arange(spokes), np.argsort(order)]).astype(np.int32)
    return F.Mesh(np.ones(3), pos, s1, s2, normal, 0.5 + 0.1 * d, np.full(n, 1e-3), pos.copy(), off, ids)


@pytest.mark.gpu
@pytest.mark.parametrize("spokes", [1, 31, 32, 33, 64, 70])
def test_hub_with_many_links_vs_oracle(spokes):
    from oracle.pyoracle import OracleSystem
    m = hub_mesh(spokes)
    rng = np.random.default_rng(spokes)
    W = F.problems.perturbed(F.problems.orszag_tang(m.pos), 0.01, seed=spokes)
    W[:, 4] *= 10.0 ** rng.uniform(0, 3, m.ncell)  # neighbours some rungs apart
    s, o = F.System(static_mesh=True), OracleSystem(static_mesh=True)
    for x in (s, o):
        x.set_mesh(m)
        x.init_problem(W)
    for _ in range(4):
        assert s.step(shared=False) == o.step(shared=False)
        a, b = s.get_state(), o.get_state()
        for k in ("rung", "tlast", "tend"):
            assert np.array_equal(a[k], b[k]), k
