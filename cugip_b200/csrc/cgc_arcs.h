// The arcs that one lane of a vertex walks in the generic-graph solve.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CGC_HD __host__ __device__ __forceinline__
#else
#define CGC_HD inline
#endif

namespace cgc {

// Arcs first + lane, first + lane + W, ... below end.  Unsigned, because arc
// ids go up to 2^31 - 2: as an int, the step past the last arc of such a range
// would be negative and pass for an arc below the end.
template <int W>
struct ArcWalk {
  uint32_t at = 0, end = 0;
  ArcWalk() = default;
  CGC_HD ArcWalk(int32_t first, int32_t past, int lane)
      : at((uint32_t)first + (uint32_t)lane), end((uint32_t)past) {}
  CGC_HD bool on() const { return at < end; }
  CGC_HD void step() { at += W; }
  CGC_HD void stop() { end = 0; }
};

}  // namespace cgc
