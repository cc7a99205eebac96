// Grid-wide barrier for cooperative (co-resident) launches.
#pragma once
#include <cstdint>
#include "cgc.h"

namespace cgc {

__device__ __forceinline__ uint64_t sync_globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The barrier's two words: bar[0] counts arrivals (zeroed before the launch),
// bar[1] is the launch's error word.  `target` is the arrival count that ends
// the CTA's next barrier (0 before the first one; kept per CTA, in a register).
// Waits are bounded: after `limit_ns` the waiting CTA records CGC_ERR_TIMEOUT,
// and every CTA leaves at this barrier or the next one, since a waiting CTA
// also watches the error word.  Returns false once an error was recorded.
//
// A barrier costs one release-add and the poll that sees the last one: there
// is no reset and no second round trip for a generation, and both words come
// with one 8-byte load.
__device__ __forceinline__ bool grid_barrier(uint32_t* bar, uint32_t& target, uint64_t limit_ns) {
  __shared__ int s_ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    const uint64_t t0 = sync_globaltimer_ns();
    uint32_t n, err;
    for (;;) {
      asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(n), "=r"(err) : "l"(bar) : "memory");
      if (err != 0 || (int32_t)(n - target) >= 0) break;
      if (sync_globaltimer_ns() - t0 > limit_ns) {
        atomicCAS(bar + 1, 0u, (uint32_t)CGC_ERR_TIMEOUT);
        err = CGC_ERR_TIMEOUT;
        break;
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    s_ok = err == 0;
  }
  __syncthreads();
  return s_ok != 0;
}

}  // namespace cgc
