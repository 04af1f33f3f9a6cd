"""The persistent rung kernel's grid barrier (csrc/grid_barrier.cuh), compiled
for the host with a thread for each block: a launch whose wait gave up leaves
its error, the launches queued behind it do nothing, and once the host has
cleared the counters barriers separate the stages again."""
import os
import subprocess

from common import ROOT

HARNESS = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
struct Index { unsigned x; };
static const Index threadIdx = {0};  // one thread per block
static void __syncthreads() {}
static int __syncthreads_and(int v) { return v; }
static int __syncthreads_or(int v) { return v; }
static void __threadfence() { std::atomic_thread_fence(std::memory_order_seq_cst); }
static unsigned atomicAdd(unsigned *p, unsigned v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
static int atomicOr(int *p, int v) { return __atomic_fetch_or(p, v, __ATOMIC_SEQ_CST); }
static void __nanosleep(unsigned) { std::this_thread::sleep_for(std::chrono::microseconds(50)); }
static unsigned load_acquire(const unsigned *p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
#define FVM_BARRIER_POLLS 20000
#include "grid_barrier.cuh"

constexpr unsigned N = 4;
static unsigned bar[2];
static int err;

// A launch of N blocks of `stages` stages; block `absent` never arrives.
// Returns the blocks that ran a stage; *early: stages entered before every
// block was through the one before.
static int launch(int stages, unsigned absent, int *early) {
  std::vector<std::atomic<int>> done(stages);
  for (auto &d : done) d = 0;
  std::atomic<int> ran{0}, bad{0};
  auto block = [&](unsigned b) {
    if (grid_failed(&err)) return;
    ran++;
    unsigned passed = 0;
    for (int s = 0; s < stages; s++) {
      if (b == 0) std::this_thread::sleep_for(std::chrono::milliseconds(5));
      if (s > 0 && done[s - 1] != (int)N) bad++;
      done[s]++;
      if (!grid_barrier(bar, passed, &err, N)) return;
    }
    grid_done(bar, N);
  };
  std::vector<std::thread> t;
  for (unsigned b = 0; b < N; b++)
    if (b != absent) t.emplace_back(block, b);
  for (auto &x : t) x.join();
  *early = bad;
  return ran;
}

int main() {
  int early;
  auto check = [](bool ok, const char *what) {
    if (!ok) { std::printf("%s\n", what); std::exit(1); }
  };
  for (int k = 0; k < 2; k++) check(launch(6, N, &early) == (int)N && !early && !err, "whole launches");
  check(bar[0] == 0 && bar[1] == 0, "counters cleared by the launch");
  launch(3, N - 1, &early);
  check(err == 1 && bar[0] != 0, "a wait that gave up");
  check(launch(6, N, &early) == 0 && !early, "a launch behind the failed one");
  bar[0] = bar[1] = 0;
  err = 0;
  check(launch(6, N, &early) == (int)N && !early && !err, "after the host's clearing");
  return 0;
}
"""


def test_barriers_around_a_launch_that_gave_up(tmp_path):
    src, exe = tmp_path / "barrier.cpp", tmp_path / "barrier"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "fvmhd3d_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
