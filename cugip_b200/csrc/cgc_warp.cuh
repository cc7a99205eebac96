// Warp-per-tile seeding passes over all tiles (bfs_init_tile_w,
// reach_init_tile_w), which need no block barrier.
//
// One warp owns one 8x8x8 tile: lane l owns the 16 voxels l + 32k
// (k = 0..15), i.e. x = l&7, y = ((l>>3)&3) + 4(k&1), z = k>>1.
#pragma once
#include "cgc_kernels.cuh"

namespace cgc {

__device__ __forceinline__ int wv_index(int lane, int k) { return lane + 32 * k; }
__device__ __forceinline__ int wv_x(int lane) { return lane & 7; }
__device__ __forceinline__ int wv_y(int lane, int k) { return ((lane >> 3) & 3) | ((k & 1) << 2); }
__device__ __forceinline__ int wv_z(int k) { return k >> 1; }


// ---------------------------------------------------------------------------
// BFS seed for tile t: h = 1 where the sink residual is positive, INF
// elsewhere; the tile's seed summary (face bits, any seed, all seeds) goes to
// tflag for the second seeding step (bfs_seed_tile / bfs_queue_tile).
// A tile whose voxels were all found unable to reach the sink stays so (dead
// vertices neither receive nor send flow, and all their residual neighbours
// are dead), so it keeps INF and is never visited again.  fresh: the first
// relabel of a solve, when the heights are not set yet.  A tile whose voxels are all seeds is final
// at h = 1 and is never visited.
__device__ inline void bfs_init_tile_w(const DevPool& P, const int t, const bool fresh) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return;  // uniform over the warp
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t)t * TV;
  bool dead = !fresh, all_seed = true, any_excess = false;
  unsigned flags = 0;
  unsigned rms[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = wv_index(lane, k);
    rms[k] = __ldcg(P.rmask + base + i);
    if (!fresh) dead = dead && __ldcg(P.h + base + i) == INF;
  }
  // a tile whose voxels were all found unable to reach the sink stays so
  dead = __all_sync(FULL, dead);
  if (dead) {
    if (lane == 0) { P.tflag[t] = TF_DEAD; P.act[t] = 0; }
    return;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = wv_index(lane, k);
    const bool seed = (rms[k] & 64u) != 0;
    P.h[base + i] = seed ? 1 : INF;
    if (seed) flags |= (face_bits(wv_x(lane), wv_y(lane, k), wv_z(k)) << 1) | TF_HAS_SEED;
    all_seed = all_seed && seed;
    any_excess = any_excess || (rms[k] & 128u) != 0;
  }
  flags = __reduce_or_sync(FULL, flags);
  all_seed = __all_sync(FULL, all_seed);
  any_excess = __any_sync(FULL, any_excess);
  if (lane == 0) {
    P.tflag[t] = (uint16_t)(flags | (all_seed ? TF_ALL_SEED : 0));
    P.act[t] = (uint8_t)((all_seed && any_excess) ? 1 : 0);
  }
}

// ---------------------------------------------------------------------------
// Reachability seed for tile t: the voxels holding excess; the tile is queued
// if it has one, and so is every face neighbour next to one.
__device__ inline void reach_init_tile_w(const DevPool& P, const int t, const uint32_t id0, int32_t* list0,
                                         int32_t* cnt0) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return;  // uniform over the warp
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t)t * TV;
  // A seed only spreads along its residual edges: the tile needs a visit if
  // some seed has one inside the tile (bit 6), and the neighbour across face
  // f if a seed on that face has one through it (bit f; that neighbour's
  // visit reads the seed and the edge from its halo).  A seed without
  // residual edges -- in a maximum flow, typically an isolated excess voxel
  // whose out-edges are saturated -- is its own closure.
  unsigned flags = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = wv_index(lane, k);
    const unsigned m = __ldcg(P.rmask + base + i);
    const bool seed = (m & 128u) != 0;
    P.reach[base + i] = seed ? 1 : 0;
    if (seed) {
      const unsigned fb = (unsigned)face_bits(wv_x(lane), wv_y(lane, k), wv_z(k));
      flags |= (m & fb & 63u) | ((m & ~fb & 63u) ? 64u : 0u);
    }
  }
  flags = __reduce_or_sync(FULL, flags);
  if (lane == 0 && (flags & 64u)) queue_tile(P, P.stamp_bfs, t, id0, list0, cnt0);
  if (lane < 6 && ((flags >> lane) & 1)) {
    const int nt = __ldcg(P.nbr + lane * P.T + t);
    if (nt >= 0) queue_tile(P, P.stamp_bfs, nt, id0, list0, cnt0);
  }
}

}  // namespace cgc
