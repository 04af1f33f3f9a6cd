"""Global steps go on without a graph where none can be made: a process with a
failing fvm_graph_instantiate in place of the library's (device memory full)
steps as one whose steps are all eager, and fvm_run reports the error."""
import os
import subprocess
import sys

import pytest

from common import ROOT

FAKE = """
int calls;
int fvm_graph_instantiate(void **exec, void *graph) { (void)exec; (void)graph; calls++; return 2; }
"""

STEPS = """
import ctypes, os
import numpy as np
import fvmhd3d_b200 as F
m = F.build_periodic(F.jittered_lattice(6, 0.1, seed=3), 1.0)
W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=4)
eager, later = F.System(), F.System()
for s in (eager, later):
    s.set_mesh(m)
    s.init_problem(W)
eager.set_profiling(True)  # keeps every step eager
for _ in range(20):
    assert eager.step(shared=True) == later.step(shared=True)
calls = ctypes.c_int.in_dll(ctypes.CDLL(os.environ["LD_PRELOAD"]), "calls")
assert calls.value == 2, calls.value  # the 8th step and the 16th
try:
    later.run(1, shared=True)
    raise SystemExit("run() did not report the error")
except F.FvmError as e:
    assert "graph instantiate" in str(e), e
assert eager.step(shared=True) == later.step(shared=True)
a, b = eager.get_state(), later.get_state()
for k in a:
    assert np.array_equal(a[k], b[k]), k
"""


@pytest.mark.gpu
def test_steps_where_no_graph_can_be_made(tmp_path):
    src, so = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", STEPS], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
