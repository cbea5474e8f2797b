// Grid-wide barrier for the persistent decoders (a cooperative launch: every block of
// the grid is resident).
//
// The arrival counter only grows: each barrier adds gridDim.x, and `epoch` is the
// count a block waits for.  Every wait is bounded: after limit_ns of global time, or
// as soon as another block has given up (the shared failure flag), the block records
// the failure and the barrier returns false, so that the kernel ends instead of
// waiting for a block that will never arrive.
#pragma once

#include <cuda_runtime.h>

namespace fecl {

constexpr unsigned long long kBarrierNs = 2000000000ull;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned load_acquire(const unsigned* q) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(q) : "memory");
  return v;
}

// counter and error are two words in global memory, zeroed before the launch.  `missing` more
// arrivals than there are blocks make every wait run out.
__device__ __forceinline__ bool grid_barrier(unsigned* counter, unsigned* error, unsigned& epoch,
                                             unsigned long long limit_ns = kBarrierNs, unsigned missing = 0) {
  __shared__ int ok;
  __syncthreads();
  epoch += gridDim.x + missing;
  if (threadIdx.x == 0) {
    // the block's writes, ordered before this thread by the barrier above, are released with the arrival
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    const unsigned long long t0 = global_ns();
    int good = 1;
    // the failure flag and the clock are looked at once in 64 polls: a poll costs its load alone
    for (unsigned polls = 1; load_acquire(counter) < epoch; ++polls) {
      if (polls % 64 != 0) continue;
      if (load_acquire(error) != 0u) {
        good = 0;
        break;
      }
      if (global_ns() - t0 > limit_ns) {
        atomicExch(error, 1u);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

}  // namespace fecl
