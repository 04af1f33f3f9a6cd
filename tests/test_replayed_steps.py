"""Which global steps are replayed, and what the launch count says of them: a
replayed step counts the kernels of an eager one, its capture none."""
import os
import subprocess
import sys

import pytest

from common import ROOT

COUNTING = """
#define _GNU_SOURCE
#include <dlfcn.h>
int calls;
int fvm_graph_instantiate(void **exec, void *graph) {
  static void *lib;
  if (!lib) lib = dlopen(FVM_LIB, RTLD_NOW | RTLD_NOLOAD);
  calls++;
  return ((int (*)(void **, void *))dlsym(lib, "fvm_graph_instantiate"))(exec, graph);
}
"""

STEPS = """
import ctypes, os
import fvmhd3d_b200 as F
calls = ctypes.c_int.in_dll(ctypes.CDLL(os.environ["LD_PRELOAD"]), "calls")
m = F.build_periodic(F.jittered_lattice(6, 0.1, seed=3), 1.0)
W = F.problems.perturbed(F.problems.blast(m.pos), 0.02, seed=4)
s = F.System()
s.set_mesh(m)
s.init_problem(W)
made = []
for k in range(16):
    s.step(shared=True)
    if k % 3 == 2:  # a partial step in between does not count
        s.step(shared=False)
    made.append(calls.value)
    if k == 4:  # nor does a new state start the count again
        st = s.get_state()
        s.set_state(**{a: st[a] for a in ("vel", "tlast", "tend", "rung", "U", "dU", "wrec")}, tsys_ticks=s.tsys_ticks)
assert made == [0] * 7 + [1] * 9, made
n0 = s.launch_count
s.run(5, shared=True)
assert calls.value == 1
eager = F.System()
eager.set_mesh(m)
eager.init_problem(W)
eager.set_profiling(True)
n = eager.launch_count
eager.step(shared=True)
per = eager.launch_count - n
assert s.launch_count - n0 == 5 * per
total = F.System()
total.set_mesh(m)
total.init_problem(W)
n = total.launch_count
for _ in range(12):
    total.step(shared=True)
assert total.launch_count - n == 12 * per, (total.launch_count - n, per)
"""


@pytest.mark.gpu
def test_steps_replayed_and_counted(tmp_path):
    src, so = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(COUNTING)
    lib = os.path.join(ROOT, "fvmhd3d_b200", "libfvmhd3d_b200.so")
    subprocess.run(["gcc", "-shared", "-fPIC", f'-DFVM_LIB="{lib}"', "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", STEPS], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
