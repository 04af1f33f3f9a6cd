"""The diagnostics of adjust_timesteps are those of the last individual step,
also after global steps (eager, by stage calls, replayed)."""
import pytest

import fvmhd3d_b200 as F
from common import setup_case


@pytest.mark.gpu
def test_diagnostics_outlive_global_steps():
    m, W = setup_case(12, "blast", seed=9, noise=0.02)
    W = W.copy()
    W[((m.pos - 0.5) ** 2).sum(1) < 0.12 ** 2, 4] *= 1e4
    s = F.System()
    s.set_mesh(m)
    s.init_problem(W)
    for _ in range(12):
        s.step(shared=False)
        if s.adjust_stats()[0] > 0:
            break
    want = s.adjust_stats()
    assert want[0] > 0 and want[1] > 0
    s.step(shared=True)
    assert s.adjust_stats() == want
    s.begin_step()
    s.fluid_update(True, shared=True)
    s.collect_results()
    s.fluid_update(False)
    s.end_step(shared=True)
    assert s.adjust_stats() == want
    s.run(3, shared=True)
    assert s.adjust_stats() == want
