// Warp-per-tile routines, which need no block barrier: the seeding passes over
// all tiles (bfs_init_tile_w, reach_init_tile_w) and the relabel visits of
// rounds with many tiles (relabel_tile_w).
//
// In the seeding passes lane l owns the 16 voxels l + 32k
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
// Relabel visits by one warp, for rounds with more tiles than tile groups: no
// block barriers, and four times as many visits in flight, whose loads and
// queue updates are what a visit waits for.  Lane (z, j) owns the rows y = 2j,
// 2j + 1 of plane z as 16-bit heights, two to a register; the tile with its y
// and z halo rows is in the warp's 1.6 KB of shared memory and is updated in
// place, as in the group's visits (relax_row16).

constexpr int WREL_SMEM = HROWS * 8;  // 16-bit heights per warp

// The fixed point of one visit in 32-bit heights on the tile's plane in
// memory, for a tile with heights beyond 16 bits around it.  nb: in lane d the
// (checked) neighbour along d, or -1.  Returns the lane's changed faces in bits
// 0..5, bit 6: something changed.
template <bool INVAL>
__device__ __noinline__ unsigned relabel_far_w(int32_t* h, const uint8_t* rmask, int nb, int t) {
  const int lane = threadIdx.x & 31;
  volatile int32_t* const H = h;
  int nt[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) nt[d] = __shfl_sync(FULL, nb, d);
  unsigned out = 0;
  for (int it = 0; it < 1200; ++it) {
    bool ch = false;
    for (int k = 0; k < 16; ++k) {
      const int i = 16 * lane + k, x = i & 7, y = (i >> 3) & 7, z = i >> 6;
      const int64_t g = (int64_t)t * TV + i;
      const unsigned m = rmask[g];
      const int old = H[g];
      int n = INVAL ? ((m & 64u) ? 1 : INF) : old;
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if (!((m >> d) & 1u)) continue;
        int64_t u = g + loff(d);
        if (!inside(d, x, y, z)) {
          if (nt[d] < 0) continue;
          u = (int64_t)nt[d] * TV + i + xoff(d);
        }
        n = min(n, H[u] + 1);
      }
      if (INVAL && old < INF && n > old) n = INF;
      else if (INVAL) n = old;
      if (n != old) {
        H[g] = n;
        ch = true;
        out |= (unsigned)face_bits(x, y, z) | 64u;
      }
    }
    __syncwarp();
    if (!__any_sync(FULL, ch)) break;
  }
  return out;
}

// INVAL: drop unsupported voxels (inval_tile), otherwise relax (bfs_tile).
// Returns 1 for a visited tile.
template <bool INVAL>
__device__ __forceinline__ int relabel_tile_w(const DevPool& P, const int t, unsigned short* g, const uint32_t id_next,
                                              int32_t* list_next, int32_t* cnt_next, const uint32_t id_bfs,
                                              int32_t* list_bfs, int32_t* cnt_bfs) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return 0;  // uniform over the warp
  const int lane = threadIdx.x & 31, j = lane & 3, z = lane >> 2;
  const int64_t base = (int64_t)t * TV;
  const int dead = INVAL ? 0 : __ldcg(P.tflag + t) & TF_DEAD;
  int nb = lane < 6 ? __ldcg(P.nbr + lane * P.T + t) : -1;
  if (nb >= 0 && !CGC_IN_BOUNDS(P, nb, P.T)) nb = -1;
  int4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __ldcg(reinterpret_cast<const int4*>(P.h + base) + 32 * i + lane);
  const uint4 m4 = __ldcg(reinterpret_cast<const uint4*>(P.rmask + base) + lane);
  if (dead) return 0;  // uniform over the warp; nothing can change
  bool far = false;
  auto put = [&](int at, const int4& w) {  // four heights into shared memory
    const uint2 p = make_uint2(pack16(w.x, w.y), pack16(w.z, w.w));
    *reinterpret_cast<uint2*>(g + at) = p;
    far = far || far16(w.x) || far16(w.y) || far16(w.z) || far16(w.w);
    return p;
  };
  uint2 was[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = 32 * i + lane, row = k >> 1;
    was[i] = put(hrow(row & 7, row >> 3) + 4 * (k & 1), v[i]);
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {  // y, then z halo rows, half a row per lane
    const int f = PY + 2 * a + (lane >> 4), k = (lane >> 1) & 7, half = lane & 1;
    const int nt = __shfl_sync(FULL, nb, f);
    const int src = (f == PY ? 64 * k : f == MY ? 64 * k + 56 : f == PZ ? 8 * k : 8 * k + 448) + 4 * half;
    const int dst = (f == PY ? hrow(8, k) : f == MY ? hrow(-1, k) : f == PZ ? hrow(k, 8) : hrow(k, -1)) + 4 * half;
    put(dst, nt >= 0 ? __ldcg(reinterpret_cast<const int4*>(P.h + (int64_t)nt * TV + src)) : make_int4(INF, INF, INF, INF));
  }
  unsigned xl[2], xr[2];  // x halo of the lane's rows: left in the upper half, right in the lower
  {
    const int ntr = __shfl_sync(FULL, nb, PX), ntl = __shfl_sync(FULL, nb, MX);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int a = ntl >= 0 ? __ldcg(P.h + (int64_t)ntl * TV + 16 * lane + 8 * s + 7) : INF;
      const int b = ntr >= 0 ? __ldcg(P.h + (int64_t)ntr * TV + 16 * lane + 8 * s) : INF;
      xl[s] = pack16(0, a);
      xr[s] = pack16(b, 0);
      far = far || far16(a) || far16(b);
    }
  }
  unsigned faces = 0;
  bool act = false;
  if (__any_sync(FULL, far)) {
    faces = relabel_far_w<INVAL>(P.h, P.rmask, nb, t);
    if (!INVAL) {
      for (int k = 0; k < 16; ++k)
        act = act || ((P.rmask[base + 16 * lane + k] & 128u) && *(volatile int32_t*)(P.h + base + 16 * lane + k) < INF);
    }
  } else {
    __syncwarp();
    const int r0 = hrow(2 * j, z), r1 = r0 + 8;
    unsigned d[2][4], c[2][6][4], sk[2][4];
    const unsigned mw[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const uint4 w = *reinterpret_cast<const uint4*>(g + (s ? r1 : r0));
      d[s][0] = w.x; d[s][1] = w.y; d[s][2] = w.z; d[s][3] = w.w;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const unsigned b = __byte_perm(mw[2 * s + (k >> 1)], 0, (k & 1) ? 0x4342 : 0x4140);  // the two voxels' mask bytes
#pragma unroll
        for (int a = 0; a < 6; ++a)  // 1 for an open edge, CLOSED16 otherwise
          c[s][a][k] = 0x40004000u - ((b >> a) & 0x00010001u) * 0x3fffu;
        if (INVAL) sk[s][k] = 0x7fff7fffu - ((b >> 6) & 0x00010001u) * 0x7ffeu;  // the sink: 1, or nothing
        else sk[s][k] = (b >> 7) & 0x00010001u;                                  // voxels with excess
      }
    }
    const unsigned first[2] = {d[0][0], d[1][0]}, last[2] = {d[0][3], d[1][3]};
    bool moved[2] = {false, false};
    for (int it = 0; it < 1200; ++it) {  // < 512 steps
      const uint4 ym = *reinterpret_cast<const uint4*>(g + r0 - 8), yp = *reinterpret_cast<const uint4*>(g + r1 + 8);
      bool ch = false;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint4 zp4 = *reinterpret_cast<const uint4*>(g + (s ? r1 : r0) + 80);
        const uint4 zm4 = *reinterpret_cast<const uint4*>(g + (s ? r1 : r0) - 80);
        const unsigned zp[4] = {zp4.x, zp4.y, zp4.z, zp4.w}, zm[4] = {zm4.x, zm4.y, zm4.z, zm4.w};
        const unsigned yo[4] = {s ? yp.x : ym.x, s ? yp.y : ym.y, s ? yp.z : ym.z, s ? yp.w : ym.w};
        unsigned n[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          n[k] = INVAL ? sk[s][k] : d[s][k];
          n[k] = __viaddmin_s16x2(zp[k], c[s][PZ][k], n[k]);
          n[k] = __viaddmin_s16x2(zm[k], c[s][MZ][k], n[k]);
          n[k] = __viaddmin_s16x2(yo[k], c[s][s ? PY : MY][k], n[k]);
          n[k] = __viaddmin_s16x2(d[1 - s][k], c[s][s ? MY : PY][k], n[k]);
        }
        // x: the relaxation runs along the row (its own new values); the
        // invalidation compares the heights as they are
        unsigned (&q)[4] = INVAL ? d[s] : n;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          n[k] = __viaddmin_s16x2(__byte_perm(k > 0 ? q[k > 0 ? k - 1 : 0] : xl[s], q[k], 0x5432), c[s][MX][k], n[k]);
#pragma unroll
        for (int k = 3; k >= 0; --k)
          n[k] = __viaddmin_s16x2(__byte_perm(q[k], k < 3 ? q[k < 3 ? k + 1 : 3] : xr[s], 0x5432), c[s][PX][k], n[k]);
        if (INVAL) {
          // the labelling is valid, so n >= d at finite voxels, with equality
          // where supported; INF16 is all ones, and stays
#pragma unroll
          for (int k = 0; k < 4; ++k)
            n[k] = d[s][k] |
                   __viaddmin_s16x2(__viaddmax_s16x2(n[k], 0u, d[s][k]) - d[s][k], 0u, 0x00010001u) * 0x3fffu;
        }
        const bool cs = ((n[0] ^ d[s][0]) | (n[1] ^ d[s][1]) | (n[2] ^ d[s][2]) | (n[3] ^ d[s][3])) != 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) d[s][k] = n[k];
        if (cs) *reinterpret_cast<uint4*>(g + (s ? r1 : r0)) = make_uint4(n[0], n[1], n[2], n[3]);
        moved[s] = moved[s] || cs;
        ch = ch || cs;
      }
      __syncwarp();
      if (!__any_sync(FULL, ch)) break;
    }
    const bool any = moved[0] || moved[1];
    if (any) {
      faces = 64u | (((((first[0] ^ d[0][0]) | (first[1] ^ d[1][0])) & 0xffffu) != 0) ? 1u << MX : 0u) |
              (((((last[0] ^ d[0][3]) | (last[1] ^ d[1][3])) >> 16) != 0) ? 1u << PX : 0u) |
              ((j == 3 && moved[1]) ? 1u << PY : 0u) | ((j == 0 && moved[0]) ? 1u << MY : 0u) |
              (z == 7 ? 1u << PZ : 0u) | (z == 0 ? 1u << MZ : 0u);
    }
    if (!INVAL) {
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int k = 0; k < 4; ++k)  // an excess voxel with a finite height
          act = act || (__viaddmin_s16x2(d[s][k] ^ 0x3fff3fffu, 0u, 0x00010001u) & sk[s][k]) != 0;
    }
    // heights that changed, 16 bytes per lane
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 32 * i + lane, row = k >> 1;
      const uint2 p = *reinterpret_cast<const uint2*>(g + hrow(row & 7, row >> 3) + 4 * (k & 1));
      if (p.x != was[i].x || p.y != was[i].y) {
        int o[4];
        unpack16(p.x, o[0], o[1]);
        unpack16(p.y, o[2], o[3]);
        st4(P.h + base + 4 * k, o);
      }
    }
  }
  faces = __reduce_or_sync(FULL, faces);
  if (!INVAL) {
    act = __any_sync(FULL, act);
    if (lane == 0) P.act[t] = (uint8_t)(act ? 1 : 0);  // heights only drop in later visits: the last visit's value is final
  } else if (lane == 6 && (faces & 64u)) {
    queue_tile(P, P.stamp_inc, t, id_bfs, list_bfs, cnt_bfs);
  }
  if (nb >= 0 && ((faces >> lane) & 1u)) queue_tile(P, P.stamp_bfs, nb, id_next, list_next, cnt_next);
  __syncwarp();
  return 1;
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
