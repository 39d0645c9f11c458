// Grid barrier of the persistent kernels, with a bounded wait.
//
// The kernels are launched cooperatively (at most the resident block count), so every block a
// barrier waits for is running.  A wait has a time budget (GRE_GRID_WAIT_MS, default 2000 ms; 0
// fails every wait at once, which the tests use; a grid of one block has nobody to wait for): one that runs out sets
// an error flag and returns false, as does every block that sees the flag, so the launch ends within about three
// budgets of the last sign of work and the context stays usable.  A warp at work that nothing splits (a row of millions of
// arcs) says so from time to time (grid_beat), and the budgets of those that wait begin again.
//
// Arrivals count up and never reset (one atomic and one polled word a barrier).  Thread 0's fences
// around the wait order the block's memory before and after it: plain loads after a barrier see
// what other blocks wrote before it (loads of such data must not go through the read-only path).
#pragma once
#include <cstdlib>

#include "gre_internal.cuh"

namespace gre {

struct GridBar {
  unsigned int arrived;  // zero at launch
  unsigned int err;
  unsigned int beat, pad;
};

// Budget of a wait in ns.
inline long long grid_wait_ns() {
  if (const char* e = getenv("GRE_GRID_WAIT_MS")) return (long long)strtoll(e, nullptr, 10) * 1000000ll;
  return 2000ll * 1000000ll;
}

#ifdef __CUDACC__
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// By one thread, within every millisecond or so of a phase that may outlast the budget.
__device__ __forceinline__ void grid_beat(GridBar* b) { atomicAdd(&b->beat, 1u); }

// `target` is thread 0's running count of arrivals (0 at the kernel's start).  `after` runs in
// thread 0 past the barrier and before the block goes on: it reads the counters that the blocks
// decide from into shared memory (read by every warp of the grid, the same few words took 7-9 us a
// barrier: one line serves a request a clock).
template <class F>
__device__ __forceinline__ bool grid_barrier(GridBar* b, unsigned int& target, long long wait_ns, F&& after) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(&b->arrived, 1u);
    int ok = 1;
    unsigned long long t0 = globaltimer_ns();
    unsigned int beat = 0;  // the last one seen when a budget ran out
    for (unsigned int spin = 0; (int)(*(volatile unsigned int*)&b->arrived - target) < 0; ++spin) {
      if (wait_ns == 0 || ((spin & 63u) == 63u && (long long)(globaltimer_ns() - t0) >= wait_ns)) {
        const unsigned int now = *(volatile unsigned int*)&b->beat;
        if (wait_ns == 0 || now == beat) atomicOr(&b->err, 1u);
        beat = now;
        t0 = globaltimer_ns();
      }
      if ((wait_ns == 0 || (spin & 63u) == 63u) && *(volatile unsigned int*)&b->err) {
        ok = 0;
        break;
      }
    }
    if (*(volatile unsigned int*)&b->err) ok = 0;
    __threadfence();
    if (ok) after();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
__device__ __forceinline__ bool grid_barrier(GridBar* b, unsigned int& target, long long wait_ns) {
  return grid_barrier(b, target, wait_ns, [] {});
}
#endif

}  // namespace gre
