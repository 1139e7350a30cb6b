// Counters that the CTAs of one cooperative launch arrive on and wait for.
//
// The launch must be cooperative (every CTA resident at once).  A counter only grows during a launch; it is
// zeroed before the launch.  Waits are bounded by the global timer (about 2 s): on a timeout the status word
// is set and the caller leaves its loop; every other CTA's own wait then runs out too.
#pragma once

#include "tcgen05.cuh"

namespace ofrr {

// all global writes of the CTA before this call are visible to a CTA that has waited for the arrival (the
// barrier orders them before thread 0's release)
__device__ __forceinline__ void grid_arrive(unsigned* ctr) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// waits until *ctr >= target; the result is the same for all threads of the CTA (s_ok: a shared word).  The
// timer, slow to read, is looked at every 64 polls only.
__device__ __forceinline__ bool grid_wait(const unsigned* ctr, unsigned target, int* s_ok, int* err, int code) {
  if (threadIdx.x == 0) {
    int ok = 1;
    uint64_t t0 = 0;
    for (unsigned polls = 1; ld_acquire(ctr) < target; ++polls) {
      if ((polls & 63u) == 0) {
        const uint64_t t = tc::globaltimer();
        if (t0 == 0) t0 = t;
        if (t - t0 > 2000000000ull) {
          atomicCAS(err, 0, code);
          ok = 0;
          break;
        }
      }
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

}  // namespace ofrr
