// The grid-wide barrier of the persistent rung kernel.  Included by
// fvm_fused.cu; a host test compiles it with a thread for each block.
#pragma once

// Polls of a wait before it gives up (about 100 ns each): far above the
// longest stage of a step the kernel runs (the sequential adjust_timesteps
// sweep over at most its involved cells).
#ifndef FVM_BARRIER_POLLS
#define FVM_BARRIER_POLLS (1ll << 24)
#endif

// On entry: whether a barrier of this launch or one before it gave up.  The
// counters are then not zero, and the state is that of half a step: steps
// queued behind it do nothing until the host has reported the error and
// cleared both.  Every thread of the block gets the same answer.
__device__ __forceinline__ bool grid_failed(const int *err) {
  return __syncthreads_or(*reinterpret_cast<const volatile int *>(err)) != 0;
}

// Grid-wide barrier over the nblocks working blocks of the launch (the
// first nblocks; the others have returned).  bar[0] counts arrivals, zero at
// the start of the launch: thread 0 of each block arrives after a release
// fence and waits, with bounded polls, until the count covers every block's
// passage of this barrier (`passed` of them before it).  One atomic and the
// polls are all a barrier costs; the counters are cleared at the end of the
// launch (grid_done).  Returns false on every thread of the block if the wait
// gave up (err bit 1 set).
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned &passed, int *err, unsigned nblocks) {
  __syncthreads();
  passed++;
  int ok = 1;
  if (threadIdx.x == 0) {
    const unsigned target = passed * nblocks;
    __threadfence();
    atomicAdd(&bar[0], 1u);
    long long it = 0;
    while (load_acquire(&bar[0]) < target) {
      if (++it > FVM_BARRIER_POLLS) {
        atomicOr(err, 1);
        ok = 0;
        break;
      }
      if (it > 4096) __nanosleep(64);  // short waits spin; long ones back off
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}
// After a block's last barrier: the last block of all clears the counters.
__device__ __forceinline__ void grid_done(unsigned *bar, unsigned nblocks) {
  if (threadIdx.x == 0 && atomicAdd(&bar[1], 1u) == nblocks - 1) {
    bar[0] = 0u;
    bar[1] = 0u;
  }
}
