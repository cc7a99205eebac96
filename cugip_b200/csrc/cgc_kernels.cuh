// Tile routines and kernels of the grid push-relabel engine (sm_100a).
//
// A tile group of 128 threads owns one 8x8x8 tile at a time; thread q owns the
// four voxels 4q..4q+3 (half an x row: x = 4(q&1).., y = (q>>1)&7, z = q>>4).
// Their state (excess, height, sink residual, six out-residuals) lives in
// registers; heights of the tile plus a one-voxel halo live in shared memory
// so that neighbours can be read.  What bounds a visit is the latency of its
// steps -- a chain of shared-memory round trips and block barriers -- and, when
// many tiles are active, the instructions they issue.  Rows of four make both
// small: a y or z neighbour row is one 16-byte shared load for four voxels, the
// x neighbours are registers or one shuffle, y exchanges stay inside a warp
// (warp w owns the planes z = 2w, 2w+1), and a barrier joins 4 warps.
//
// Push sweep (replaces the per-level push of
// include/cugip/advanced_operations/detail/graph_cut_push.hpp:160-186,236-318,
// 461-482).  A visit runs up to L synchronous pulses of the Goldberg-Tarjan
// parallel push-relabel inside the tile: every active voxel (e>0, h<INF)
// pushes to the sink if h==1 and along every admissible residual edge
// (h(u)==h(v)-1), then every voxel that is still active and has no
// admissible edge relabels to 1+min over its residual neighbours.  Labels are
// fixed during a push step and relabels read the old labels, so the labelling
// stays valid.  Under the parity schedule only tiles with (tx+ty+tz) of one
// parity run at a time; face neighbours always have the other parity, so the
// halo heights are exact and the tile's pushes across a face (int32 atomics on
// the neighbour's excess, plain adds on the neighbour's reverse residual,
// which has a single writer) are ordinary valid pushes.
//
// Global relabel (replaces the level-synchronous BFS of
// detail/graph_cut_relabeling.hpp:47-112,651-751,1004-1029).  Exact BFS
// distance to the sink over reverse residual edges, computed by tile-local
// Bellman-Ford relaxation to a fixed point in shared memory; a tile whose face
// heights dropped re-queues its face neighbours.  Vertices the BFS does not
// reach keep INF, which is the gap heuristic.
//
// Exact sink flow.  Pushes to the sink are capped by the sink residual (the
// reference moves all excess of any sink-adjacent vertex,
// detail/graph_cut_push.hpp:26-41); the flow is accumulated in int64.
#pragma once
#include <cuda_runtime.h>
#include "cgc.h"
#include "cgc_device.cuh"

namespace cgc {

// offset of the neighbour along d inside a tile
__device__ __forceinline__ int loff(int d) {
  return d == PX ? 1 : d == MX ? -1 : d == PY ? 8 : d == MY ? -8 : d == PZ ? 64 : -64;
}
// local index in the neighbouring tile when stepping out of the tile along d
__device__ __forceinline__ int xoff(int d) {
  return d == PX ? -7 : d == MX ? 7 : d == PY ? -56 : d == MY ? 56 : d == PZ ? -448 : 448;
}
__device__ __forceinline__ bool inside(int d, int x, int y, int z) {
  return d == PX ? x < 7 : d == MX ? x > 0 : d == PY ? y < 7 : d == MY ? y > 0 : d == PZ ? z < 7 : z > 0;
}
// bit mask of the faces of the tile the voxel lies on
__device__ __forceinline__ int face_bits(int x, int y, int z) {
  return ((x == 7) << PX) | ((x == 0) << MX) | ((y == 7) << PY) | ((y == 0) << MY) | ((z == 7) << PZ) | ((z == 0) << MZ);
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void raise_error(const DevPool& P, int code) { atomicCAS(P.err, 0, code); }

// Bounds-checked build (-DCGC_BOUNDS_CHECK; cugip_b200/build.py --bounds-check
// builds libcgc_bounds.so): every tile, neighbour-tile and worklist index the
// tile routines compute is checked against its array.  An index out of range
// records CGC_ERR_ARG in the error word (the first one also its value in
// stats[S_BOUND_AT]) and the access is skipped; nothing traps.  The product
// build compiles the checks out.
#ifdef CGC_BOUNDS_CHECK
static __device__ __noinline__ bool bound_fail(const DevPool& P, long long i) {
  if (atomicCAS(P.err, 0, CGC_ERR_ARG) == 0) P.stats[S_BOUND_AT] = (unsigned long long)i;
  return false;
}
#define CGC_IN_BOUNDS(P, i, lim) \
  ((long long)(i) >= 0 && (long long)(i) < (long long)(lim) ? true : ::cgc::bound_fail((P), (long long)(i)))
#else
#define CGC_IN_BOUNDS(P, i, lim) true
#endif

constexpr unsigned FULL = 0xffffffffu;

// The W threads that visit a tile together, with a named barrier of their own
// (barrier 0 is __syncthreads of the whole CTA): groups of 128, numbered in the
// CTA, or the CTA's first 512 threads.
constexpr int GROUP = 128, WIDE = 512;
template <int W>
struct TileGroup {
  static constexpr int width = W;
  int q;    // thread of the group
  int bar;  // named barrier
  __device__ __forceinline__ static TileGroup of_thread() {
    if (W == WIDE) return TileGroup{(int)threadIdx.x, 15};
    return TileGroup{(int)(threadIdx.x & (W - 1)), 1 + (int)(threadIdx.x / W)};
  }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(W) : "memory"); }
  __device__ __forceinline__ bool any(bool p) const {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((int)p), "r"(bar), "n"(W)
        : "memory");
    return r != 0;
  }
};

// Heights of a tile with its y and z halo rows in shared memory: row (y, z),
// y and z in [-1, 8], is 8 ints at hrow(y, z).  The x halo is one register per
// thread (the neighbour left of x = 0 or right of x = 7).
constexpr int HROWS = 100;
__device__ __forceinline__ int hrow(int y, int z) { return ((z + 1) * 10 + (y + 1)) * 8; }

__device__ __forceinline__ int4 ld4(const int* p) { return *reinterpret_cast<const int4*>(p); }
__device__ __forceinline__ void st4(int* p, const int (&v)[4]) {
  *reinterpret_cast<int4*>(p) = make_int4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void ldcg4(const int32_t* p, int (&v)[4]) {
  const int4 a = __ldcg(reinterpret_cast<const int4*>(p));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ int at(const int4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// Heights as 16-bit numbers, two to a register, for the relaxations: a step
// then issues half the instructions (they are bound by the integer pipe).  A
// tile with a finite height above FAR16 around it uses 32-bit steps instead;
// below, no path in the tile reaches INF16.
constexpr int INF16 = 0x3fff, CLOSED16 = 0x4000, FAR16 = 15000;
__device__ __forceinline__ unsigned pack16(int lo, int hi) {
  return (unsigned)min(lo, INF16) | (unsigned)min(hi, INF16) << 16;
}
__device__ __forceinline__ void unpack16(unsigned v, int& lo, int& hi) {
  lo = (int)(v & 0xffffu);
  hi = (int)(v >> 16);
  if (lo == INF16) lo = INF;
  if (hi == INF16) hi = INF;
}
__device__ __forceinline__ bool far16(int h) { return h > FAR16 && h < INF; }

// Halo of tile t: 64 threads each load half a y or z halo row into sh0 (and
// sh1 if given) and, as 16-bit heights, into s16 (if given); every thread
// returns its x halo height (INF outside the grid).  far: set if a height the
// thread loaded does not fit 16 bits.
__device__ __forceinline__ int load_halo_heights(const DevPool& P, const int t, const int q, int* sh0, int* sh1,
                                                 unsigned short* s16, bool& far) {
  const int half = q & 1, k = (q >> 1) & 7;
  const int nx = __ldcg(P.nbr + (half ? PX : MX) * P.T + t);
  if (q < 64) {
    const int f = PY + (q >> 4);
    const int nt = __ldcg(P.nbr + f * P.T + t);
    int4 v = make_int4(INF, INF, INF, INF);
    const int src = (f == PY ? 64 * k : f == MY ? 64 * k + 56 : f == PZ ? 8 * k : 8 * k + 448) + 4 * half;
    const int dst = (f == PY ? hrow(8, k) : f == MY ? hrow(-1, k) : f == PZ ? hrow(k, 8) : hrow(k, -1)) + 4 * half;
    if (nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T)) v = __ldcg(reinterpret_cast<const int4*>(P.h + (int64_t)nt * TV + src));
    *reinterpret_cast<int4*>(sh0 + dst) = v;
    if (sh1) *reinterpret_cast<int4*>(sh1 + dst) = v;
    if (s16) *reinterpret_cast<uint2*>(s16 + dst) = make_uint2(pack16(v.x, v.y), pack16(v.z, v.w));
    far = far || far16(v.x) || far16(v.y) || far16(v.z) || far16(v.w);
  }
  const int hx = (nx >= 0 && CGC_IN_BOUNDS(P, nx, P.T)) ? __ldcg(P.h + (int64_t)nx * TV + 8 * (q >> 1) + (half ? 0 : 7)) : INF;
  far = far || far16(hx);
  return hx;
}

// Cost of a closed edge in the relaxation: INF + CLOSED does not overflow, and
// any height plus CLOSED is above INF.
constexpr int CLOSED = 0x40000000;

// One in-place Bellman-Ford step of the thread's four voxels on the heights S
// (d[] is the thread's copy of its row): d = min(d, 1 + neighbour) over the
// open edges (c[dir][k] is 1 for an open edge, CLOSED otherwise, so an edge is
// one add-min instruction and needs no predicate).  Values only drop, so
// reading a neighbour's old or new value is both correct and the fixed point
// is the same.  Returns whether d dropped (and then the row was stored).
__device__ __forceinline__ bool relax_row(int* S, const int row, const int half, const int hx, int (&d)[4],
                                          const int (&c)[6][4]) {
  const int4 yp = ld4(S + row + 8), ym = ld4(S + row - 8), zp = ld4(S + row + 80), zm = ld4(S + row - 80);
  const int xo = __shfl_xor_sync(FULL, half ? d[0] : d[3], 1);
  int n[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    n[k] = min(__viaddmin_s32(at(yp, k), c[PY][k], d[k]), __viaddmin_s32(at(ym, k), c[MY][k], at(zp, k) + c[PZ][k]));
    n[k] = __viaddmin_s32(at(zm, k), c[MZ][k], n[k]);
  }
  n[0] = __viaddmin_s32(half ? xo : hx, c[MX][0], n[0]);
  n[3] = __viaddmin_s32(half ? hx : xo, c[PX][3], n[3]);
#pragma unroll
  for (int k = 1; k < 4; ++k) n[k] = __viaddmin_s32(n[k - 1], c[MX][k], n[k]);
#pragma unroll
  for (int k = 2; k >= 0; --k) n[k] = __viaddmin_s32(n[k + 1], c[PX][k], n[k]);
  const bool ch = ((n[0] ^ d[0]) | (n[1] ^ d[1]) | (n[2] ^ d[2]) | (n[3] ^ d[3])) != 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) d[k] = n[k];
  if (ch) st4(S + row, d);
  return ch;
}

// The same step on 16-bit heights: d[0] holds the row's first two voxels, d[1]
// the others; c[dir][0..1] is 1 or CLOSED16 per half.
__device__ __forceinline__ bool relax_row16(unsigned short* S, const int row, const int half, const unsigned hx,
                                            unsigned (&d)[2], const unsigned (&c)[6][2]) {
  const uint2 yp = *reinterpret_cast<const uint2*>(S + row + 8), ym = *reinterpret_cast<const uint2*>(S + row - 8);
  const uint2 zp = *reinterpret_cast<const uint2*>(S + row + 80), zm = *reinterpret_cast<const uint2*>(S + row - 80);
  const unsigned xo = __shfl_xor_sync(FULL, half ? d[0] : d[1], 1);  // the row's other half
  const unsigned l = __byte_perm(half ? xo : hx, d[0], half ? 0x5432 : 0x5410);  // left neighbours of d[0]
  unsigned n0 = __viaddmin_s16x2(yp.x, c[PY][0], d[0]), n1 = __viaddmin_s16x2(yp.y, c[PY][1], d[1]);
  n0 = __viaddmin_s16x2(ym.x, c[MY][0], n0);
  n1 = __viaddmin_s16x2(ym.y, c[MY][1], n1);
  n0 = __viaddmin_s16x2(zp.x, c[PZ][0], n0);
  n1 = __viaddmin_s16x2(zp.y, c[PZ][1], n1);
  n0 = __viaddmin_s16x2(zm.x, c[MZ][0], n0);
  n1 = __viaddmin_s16x2(zm.y, c[MZ][1], n1);
  n0 = __viaddmin_s16x2(l, c[MX][0], n0);
  n1 = __viaddmin_s16x2(__byte_perm(n0, n1, 0x5432), c[MX][1], n1);
  n1 = __viaddmin_s16x2(__byte_perm(n1, half ? hx : xo, 0x5432), c[PX][1], n1);
  n0 = __viaddmin_s16x2(__byte_perm(n0, n1, 0x5432), c[PX][0], n0);
  const bool ch = ((n0 ^ d[0]) | (n1 ^ d[1])) != 0;
  d[0] = n0;
  d[1] = n1;
  if (ch) *reinterpret_cast<uint2*>(S + row) = make_uint2(n0, n1);
  return ch;
}

// warp-aggregated append of `pred` items to list/cnt
// (worklists hold at most T entries: stamps let a tile in once per list)
__device__ __forceinline__ void warp_append(const DevPool& P, bool pred, int32_t item, int32_t* list, int32_t* cnt) {
  const unsigned mask = __ballot_sync(0xffffffffu, pred);
  if (!mask) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(cnt, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  const int k = base + __popc(mask & ((1u << lane) - 1));
  if (pred && CGC_IN_BOUNDS(P, k, P.T)) list[k] = item;
}

__device__ __forceinline__ void queue_tile(const DevPool& P, uint32_t* stamp, int t, uint32_t id, int32_t* list,
                                           int32_t* cnt) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return;
  if (atomicExch(stamp + t, id) != id) {
    const int k = atomicAdd(cnt, 1);
    if (CGC_IN_BOUNDS(P, k, P.T)) list[k] = t;
  }
}

// Shared state of one tile group.
struct alignas(16) SweepShared {
  int h[2][HROWS * 8];  // heights, double buffered by pulse
  unsigned short g[HROWS * 8];  // 16-bit heights of the region relabel
  int out[2][TV];       // flow pushed along +z / -z in this pulse; zero between pulses
  int facc[6][64];      // flow pushed out of the tile per face entry
  unsigned char face[8];  // faces that flow left through
  int lastout;          // last pulse (1-based) that moved flow out of the tile or into the sink
};

struct alignas(16) BfsShared {
  int h[HROWS * 8];
  unsigned short g[HROWS * 8];  // 16-bit heights
  unsigned flags;  // of the visit: faces whose heights changed (bits 0..5), and bit 6 (bfs_tile, inval_tile)
};

// optional per-visit bookkeeping of the persistent schedule
struct SweepExtra {
  int32_t* sink_tiles = nullptr;  // nonzero after a sweep in which some tile delivered sink flow
  uint8_t* tr_pulses = nullptr;   // trace: pulses of the first visit in this cycle
  uint8_t* tr_sink = nullptr;     // trace: delivered sink flow in this cycle
};

// ---------------------------------------------------------------------------
// One visit of the push sweep to tile t (L pulses at most per region-relabel
// round, R rounds) by one tile group; returns the pulses it ran.
//   The tile itself (if still active) is queued for sweep id_self and the tiles
//   it pushed into for sweep id_next, with the stamps stamp_q.
//   exact: the labels are exact (no push or relabel since the last global
//   relabel), so the first region relabel would change nothing and is left out.
// The caller synchronises the group before S is used again.
//
// A pulse pushes in the order sink, +x, -x (through the thread's row, so flow
// crosses four voxels), row ends (shuffle), +-y (shuffles inside the warp), +-z
// (shared memory); flow received earlier in the pulse may be pushed on by a
// later direction, since labels do not change until the pulse's relabel.  Two
// barriers per pulse.
__device__ __forceinline__ int sweep_tile(const DevPool& P, const TileGroup<GROUP> tg, const int t, const int L, const int R,
                                          const bool exact, SweepShared& S, const uint32_t id_next, int32_t* list_next,
                                          int32_t* cnt_next, const uint32_t id_self, int32_t* list_self,
                                          int32_t* cnt_self, const SweepExtra ex, uint32_t* stamp_q) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return 0;  // uniform over the group
  const int q = tg.q, half = q & 1, y = (q >> 1) & 7, z = q >> 4;
  const int row = hrow(y, z) + 4 * half;
  const int64_t g = (int64_t)t * TV + 4 * q;
  const int64_t Np = P.Np;
  int e[4], h[4], rT[4], r[6][4];
  ldcg4(P.h + g, h);
  ldcg4(P.e + g, e);
  ldcg4(P.rT + g, rT);
#pragma unroll
  for (int d = 0; d < 6; ++d) ldcg4(P.r + d * Np + g, r[d]);
  st4(S.h[0] + row, h);
  bool far = false;
  const int hx = load_halo_heights(P, t, q, S.h[0], S.h[1], S.g, far);
  const int inst = __ldcg(P.tinst + t);
  const int hdead = P.geo[inst].hdead;
  {
    const int zero[4] = {0, 0, 0, 0};
    st4(&S.out[0][4 * q], zero);
    st4(&S.out[1][4 * q], zero);
    if (q < 96) st4(&S.facc[0][0] + 4 * q, zero);
  }
  if (q < 8) S.face[q] = 0;
  if (q == 0) S.lastout = 0;
  far = tg.any(far);

  // some voxel of the thread holds excess and may still reach the sink
  auto active = [&]() {
    return (e[0] > 0 && h[0] < INF) || (e[1] > 0 && h[1] < INF) || (e[2] > 0 && h[2] < INF) || (e[3] > 0 && h[3] < INF);
  };
  long long sink = 0;
  int pulses = 0;
  int cur = 0;
  bool dirty = false, dirty_h = false;  // the thread's excess and residuals / heights differ from memory
  bool any = true;
  for (int round = 0;; ++round) {
    if (R > 0 && !(exact && round == 0)) {
      // Region relabel: exact distance d(v) to the sink or to the (frozen)
      // halo inside the tile, then h = max(h, d).  d is a lower bound of the
      // true distance and max(h, d) keeps every residual edge valid, so this
      // is an ordinary (multi-step) relabel; d = INF means v cannot reach the
      // sink at all.
      int dd[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) dd[k] = rT[k] > 0 ? 1 : INF;
      // Bellman-Ford: < 512 steps in a tile
      if (!far) {
        unsigned d2[2] = {pack16(dd[0], dd[1]), pack16(dd[2], dd[3])}, c[6][2];
        *reinterpret_cast<uint2*>(S.g + row) = make_uint2(d2[0], d2[1]);
#pragma unroll
        for (int d = 0; d < 6; ++d)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            c[d][j] = (r[d][2 * j] > 0 ? 1u : (unsigned)CLOSED16) | (r[d][2 * j + 1] > 0 ? 1u << 16 : (unsigned)CLOSED16 << 16);
        const unsigned hx2 = pack16(hx, 0);
        tg.sync();
        for (int it = 0; it < 600; ++it) {
          const bool ch = relax_row16(S.g, row, half, hx2, d2, c);
          if (!tg.any(ch)) break;
        }
        unpack16(d2[0], dd[0], dd[1]);
        unpack16(d2[1], dd[2], dd[3]);
      } else {
        st4(S.h[cur] + row, dd);
        int c[6][4];
#pragma unroll
        for (int d = 0; d < 6; ++d)
#pragma unroll
          for (int k = 0; k < 4; ++k) c[d][k] = r[d][k] > 0 ? 1 : CLOSED;
        tg.sync();
        for (int it = 0; it < 600; ++it) {
          const bool ch = relax_row(S.h[cur], row, half, hx, dd, c);
          if (!tg.any(ch)) break;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        int hn = max(h[k], dd[k]);
        if (hn >= hdead) hn = INF;
        dirty_h = dirty_h || hn != h[k];
        h[k] = hn;
      }
      st4(S.h[cur] + row, h);
      tg.sync();
    }
    for (int p = 0; p < L; ++p) {
      // labels of the neighbours, fixed during the pulse
      const int* H = S.h[cur];
      const int4 yp = ld4(H + row + 8), ym = ld4(H + row - 8), zp = ld4(H + row + 80), zm = ld4(H + row - 80);
      const int xo = __shfl_xor_sync(FULL, half ? h[0] : h[3], 1);
      const int hl = half ? xo : hx, hr = half ? hx : xo;
      bool act = active();
      if (__any_sync(FULL, act)) {
        dirty = dirty || act;
        int out = 0;  // > 0: flow left the tile or went into the sink
        // amount voxel k pushes along d to a neighbour of height hn (a voxel
        // at INF has no neighbour at INF - 1)
        auto push = [&](int d, int k, int hn) {
          const int dl = hn + 1 == h[k] ? min(e[k], r[d][k]) : 0;
          e[k] -= dl;
          r[d][k] -= dl;
          return dl;
        };
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // a voxel with a sink residual is at height 1: the labelling is valid
          const int dl = min(e[k], rT[k]);
          e[k] -= dl;
          rT[k] -= dl;
          sink += dl;
          out |= dl;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (h[k + 1] + 1 == h[k]) {
            const int dl = min(e[k], r[PX][k]);
            e[k] -= dl;
            r[PX][k] -= dl;
            e[k + 1] += dl;
            r[MX][k + 1] += dl;
          }
#pragma unroll
        for (int k = 3; k > 0; --k)
          if (h[k - 1] + 1 == h[k]) {
            const int dl = min(e[k], r[MX][k]);
            e[k] -= dl;
            r[MX][k] -= dl;
            e[k - 1] += dl;
            r[PX][k - 1] += dl;
          }
        {  // row ends: one leaves the tile, the other goes to the row's other half
          const int ar = push(PX, 3, hr), al = push(MX, 0, hl);
          const int in = __shfl_xor_sync(FULL, half ? al : ar, 1);
          if (half) { e[0] += in; r[MX][0] += in; } else { e[3] += in; r[PX][3] += in; }
          dirty = dirty || in > 0;
          const int w = half ? ar : al;
          if (w > 0) {
            const int f = half ? PX : MX;
            S.facc[f][y + 8 * z] += w;  // this thread is the entry's only writer
            S.face[f] = 1;
            out = 1;
          }
        }
        {  // y: the warp holds all rows of its planes
          int up[4], dn[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            up[k] = push(PY, k, at(yp, k));
            dn[k] = push(MY, k, at(ym, k));
          }
          const int wu = up[0] | up[1] | up[2] | up[3], wd = dn[0] | dn[1] | dn[2] | dn[3];
          if (__any_sync(FULL, (wu | wd) > 0)) {
            const bool hi = y == 7, lo = y == 0;
            if (hi ? wu > 0 : lo && wd > 0) {
              int* fa = &S.facc[hi ? PY : MY][4 * half + 8 * z];
#pragma unroll
              for (int k = 0; k < 4; ++k) fa[k] += hi ? up[k] : dn[k];
              S.face[hi ? PY : MY] = 1;
              out = 1;
            }
            int got = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              int a = __shfl_up_sync(FULL, up[k], 2), b = __shfl_down_sync(FULL, dn[k], 2);
              a = lo ? 0 : a;
              b = hi ? 0 : b;
              e[k] += a + b;
              r[MY][k] += a;
              r[PY][k] += b;
              got |= a | b;
            }
            dirty = dirty || got > 0;
          }
        }
        {  // z: through shared memory; the receiver clears what it took
          int up[4], dn[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            up[k] = push(PZ, k, at(zp, k));
            dn[k] = push(MZ, k, at(zm, k));
          }
          if ((up[0] | up[1] | up[2] | up[3]) > 0) {
            if (z < 7) {
              st4(&S.out[0][4 * q], up);
            } else {
              int* fa = &S.facc[PZ][4 * half + 8 * y];
#pragma unroll
              for (int k = 0; k < 4; ++k) fa[k] += up[k];
              S.face[PZ] = 1;
              out = 1;
            }
          }
          if ((dn[0] | dn[1] | dn[2] | dn[3]) > 0) {
            if (z > 0) {
              st4(&S.out[1][4 * q], dn);
            } else {
              int* fa = &S.facc[MZ][4 * half + 8 * y];
#pragma unroll
              for (int k = 0; k < 4; ++k) fa[k] += dn[k];
              S.face[MZ] = 1;
              out = 1;
            }
          }
        }
        if (out > 0) {
          dirty = true;
          S.lastout = pulses + 1;  // same value from every writer of this pulse
        }
      }
      tg.sync();
      {
        const int zero[4] = {0, 0, 0, 0};
        if (z > 0) {
          int* o = &S.out[0][4 * q - 64];
          const int4 a = ld4(o);
          if (a.x | a.y | a.z | a.w) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { e[k] += at(a, k); r[MZ][k] += at(a, k); }
            st4(o, zero);
            dirty = true;
          }
        }
        if (z < 7) {
          int* o = &S.out[1][4 * q + 64];
          const int4 a = ld4(o);
          if (a.x | a.y | a.z | a.w) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { e[k] += at(a, k); r[PZ][k] += at(a, k); }
            st4(o, zero);
            dirty = true;
          }
        }
      }
      // Relabel: the labelling is valid, so the lowest residual neighbour mn is
      // at h - 1 or higher (the sink counts as height 0), and 1 + mn is h itself
      // where the voxel still has an admissible edge.
      bool still = false;
      if (__any_sync(FULL, active())) {
        int hn[4], ch = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          int mn = rT[k] > 0 ? 0 : INF;
          if (r[PX][k] > 0) mn = min(mn, k < 3 ? h[k < 3 ? k + 1 : 3] : hr);
          if (r[MX][k] > 0) mn = min(mn, k > 0 ? h[k > 0 ? k - 1 : 0] : hl);
          if (r[PY][k] > 0) mn = min(mn, at(yp, k));
          if (r[MY][k] > 0) mn = min(mn, at(ym, k));
          if (r[PZ][k] > 0) mn = min(mn, at(zp, k));
          if (r[MZ][k] > 0) mn = min(mn, at(zm, k));
          int v = mn + 1;
          if (v >= hdead) v = INF;
          hn[k] = e[k] > 0 && h[k] < INF ? v : h[k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          ch |= hn[k] ^ h[k];
          h[k] = hn[k];
        }
        dirty_h = dirty_h || ch != 0;
        still = active();
      }
      ++pulses;
      st4(S.h[cur ^ 1] + row, h);
      any = tg.any(still);
      cur ^= 1;
      if (!any) break;
    }
    if (!any || round + 1 >= max(R, 1)) break;
  }

  // The queue updates first: they are chains of two dependent atomics, and the
  // rest of the write-back runs beside them.
  if (q == 64) {
    P.act[t] = (uint8_t)(any ? 1 : 0);
    if (any) queue_tile(P, stamp_q, t, id_self, list_self, cnt_self);
    // trace label: productive pulses of the tile's first visit in the cycle
    // (255 marks a visited tile that moved nothing out)
    if (ex.tr_pulses && ex.tr_pulses[t] == 0) ex.tr_pulses[t] = (uint8_t)(S.lastout > 0 ? min(S.lastout, 254) : 255);
  }
  if (q >= 32 && q < 38 && S.face[q - 32]) {
    const int nt = __ldcg(P.nbr + (q - 32) * P.T + t);
    if (nt < 0) {
      raise_error(P, CGC_ERR_OVERFLOW);  // capacity leaving the grid
    } else if (CGC_IN_BOUNDS(P, nt, P.T)) {
      P.act[nt] = 1;
      queue_tile(P, stamp_q, nt, id_next, list_next, cnt_next);
    }
  }
  // the tile's planes, where they changed
  if (dirty_h) st4(P.h + g, h);
  if (dirty) {
    st4(P.e + g, e);
    st4(P.rT + g, rT);
    unsigned m4 = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) st4(P.r + d * Np + g, r[d]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unsigned m = (rT[k] > 0 ? 64u : 0u) | (e[k] > 0 ? 128u : 0u);
#pragma unroll
      for (int d = 0; d < 6; ++d) m |= (r[d][k] > 0 ? 1u : 0u) << d;
      m4 |= m << (8 * k);
    }
    *reinterpret_cast<unsigned*>(P.rmask + g) = m4;
  }
  // flow that left the tile: excess and reverse residual of the neighbour
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int i = q + GROUP * j, f = i >> 6, a = i & 7, b = (i >> 3) & 7;
    const int w = (&S.facc[0][0])[i];
    if (w > 0) {
      const int nt = __ldcg(P.nbr + f * P.T + t);
      if (nt < 0 || !CGC_IN_BOUNDS(P, nt, P.T)) continue;  // reported above
      const int src = f == PX ? 8 * a + 64 * b : f == MX ? 7 + 8 * a + 64 * b : f == PY ? a + 64 * b
                    : f == MY ? a + 56 + 64 * b : f == PZ ? a + 8 * b : a + 8 * b + 448;
      const int64_t ng = (int64_t)nt * TV + src;
      atomicAdd(P.e + ng, w);
      atomicAdd(P.r + (f ^ 1) * Np + ng, w);
      atomicOr((unsigned*)(P.rmask + (ng & ~(int64_t)3)), (128u | (1u << (f ^ 1))) << (8 * (int)(ng & 3)));
    }
  }
  if (__any_sync(FULL, sink > 0)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sink += __shfl_down_sync(FULL, sink, o);
    if ((q & 31) == 0) {
      atomicAdd(P.flow + inst, (unsigned long long)sink);
      if (ex.sink_tiles) atomicAdd(ex.sink_tiles, 1);
      if (ex.tr_sink) ex.tr_sink[t] = 1;
    }
  }
  return pulses;
}

// ---------------------------------------------------------------------------
// The same visit by 512 threads, one voxel each, for sweeps that leave most of
// the chip idle.  With one tile on an SM, a warp runs one instruction in about
// seven cycles (its chain of dependent instructions), so the fewest
// instructions per warp win, not the fewest in total: a relaxation step is 20
// of them instead of 60, and a warp without an active voxel skips a pulse.
//   APPEND: queue tiles as above (persistent schedule); otherwise only the
//   act[] flags are maintained (host-driven schedule).
constexpr int WH = HROWS * 8 + 128;  // a buffer of heights: the rows, then the x halo (left of x = 0, right of x = 7)
struct alignas(16) WideShared {
  int h[2][WH];      // double buffered by pulse
  int out[6][TV];    // flow pushed along d in this pulse; zero between pulses
  int facc[6][64];   // flow pushed out of the tile per face entry
  int inbox[16];     // per warp: last pulse (1-based) in which flow was pushed to its voxels
  int moved[8];      // last pulse in which flow left through face d; [6]: into the sink
  int nb[6];
};

// Predicated shared-memory updates for the six directions at once: branches
// around them cost more than the updates, and so would waiting for one
// predicate after the other.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// where v[d] > 0: *to[d] += v[d], *tell[d] = s
__device__ __forceinline__ void push_out6(const uint32_t (&to)[6], const uint32_t (&tell)[6], const int (&v)[6], int s) {
  asm volatile(
      "{\n\t.reg .pred p<6>;\n\t"
      "setp.gt.s32 p0, %12, 0;\n\tsetp.gt.s32 p1, %13, 0;\n\tsetp.gt.s32 p2, %14, 0;\n\t"
      "setp.gt.s32 p3, %15, 0;\n\tsetp.gt.s32 p4, %16, 0;\n\tsetp.gt.s32 p5, %17, 0;\n\t"
      "@p0 red.shared.add.s32 [%0], %12;\n\t@p1 red.shared.add.s32 [%1], %13;\n\t"
      "@p2 red.shared.add.s32 [%2], %14;\n\t@p3 red.shared.add.s32 [%3], %15;\n\t"
      "@p4 red.shared.add.s32 [%4], %16;\n\t@p5 red.shared.add.s32 [%5], %17;\n\t"
      "@p0 st.shared.s32 [%6], %18;\n\t@p1 st.shared.s32 [%7], %18;\n\t@p2 st.shared.s32 [%8], %18;\n\t"
      "@p3 st.shared.s32 [%9], %18;\n\t@p4 st.shared.s32 [%10], %18;\n\t@p5 st.shared.s32 [%11], %18;\n\t}" ::"r"(to[0]),
      "r"(to[1]), "r"(to[2]), "r"(to[3]), "r"(to[4]), "r"(to[5]), "r"(tell[0]), "r"(tell[1]), "r"(tell[2]), "r"(tell[3]),
      "r"(tell[4]), "r"(tell[5]), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(s)
      : "memory");
}
// v[d] = the flow pushed towards the voxel whose slot of direction 0 is at
// `from` (0 where on[d] is 0: no such neighbour in the tile)
__device__ __forceinline__ void take6(uint32_t from, const bool (&on)[6], int (&v)[6]) {
  asm volatile(
      "{\n\t.reg .pred p<6>;\n\t"
      "setp.ne.s32 p0, %7, 0;\n\tsetp.ne.s32 p1, %8, 0;\n\tsetp.ne.s32 p2, %9, 0;\n\t"
      "setp.ne.s32 p3, %10, 0;\n\tsetp.ne.s32 p4, %11, 0;\n\tsetp.ne.s32 p5, %12, 0;\n\t"
      "mov.s32 %0, 0;\n\tmov.s32 %1, 0;\n\tmov.s32 %2, 0;\n\tmov.s32 %3, 0;\n\tmov.s32 %4, 0;\n\tmov.s32 %5, 0;\n\t"
      "@p0 ld.shared.s32 %0, [%6+2052];\n\t@p1 ld.shared.s32 %1, [%6+-4];\n\t"
      "@p2 ld.shared.s32 %2, [%6+6176];\n\t@p3 ld.shared.s32 %3, [%6+4064];\n\t"
      "@p4 ld.shared.s32 %4, [%6+10496];\n\t@p5 ld.shared.s32 %5, [%6+7936];\n\t}"
      : "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]), "=&r"(v[4]), "=&r"(v[5])
      : "r"(from), "r"((int)on[0]), "r"((int)on[1]), "r"((int)on[2]), "r"((int)on[3]), "r"((int)on[4]), "r"((int)on[5])
      : "memory");
}
// clears the slots that take6 found flow in
__device__ __forceinline__ void clear6(uint32_t from, const int (&v)[6]) {
  asm volatile(
      "{\n\t.reg .pred p<6>;\n\t"
      "setp.gt.s32 p0, %1, 0;\n\tsetp.gt.s32 p1, %2, 0;\n\tsetp.gt.s32 p2, %3, 0;\n\t"
      "setp.gt.s32 p3, %4, 0;\n\tsetp.gt.s32 p4, %5, 0;\n\tsetp.gt.s32 p5, %6, 0;\n\t"
      "@p0 st.shared.s32 [%0+2052], 0;\n\t@p1 st.shared.s32 [%0+-4], 0;\n\t"
      "@p2 st.shared.s32 [%0+6176], 0;\n\t@p3 st.shared.s32 [%0+4064], 0;\n\t"
      "@p4 st.shared.s32 [%0+10496], 0;\n\t@p5 st.shared.s32 [%0+7936], 0;\n\t}" ::"r"(from),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5])
      : "memory");
}
// the offsets above: slot of direction d ^ 1 of the neighbour along d
static_assert(4 * (MX * TV + 1) == 2052 && 4 * (PX * TV - 1) == -4 && 4 * (MY * TV + 8) == 6176 &&
              4 * (PY * TV - 8) == 4064 && 4 * (MZ * TV + 64) == 10496 && 4 * (PZ * TV - 64) == 7936, "take6 / clear6");

template <bool APPEND>
__device__ __forceinline__ int sweep_tile_wide(const DevPool& P, const TileGroup<WIDE> tg, const int t, const int L,
                                               const int R, const bool exact, WideShared& S, const uint32_t id_next,
                                               int32_t* list_next, int32_t* cnt_next, const uint32_t id_self,
                                               int32_t* list_self, int32_t* cnt_self, const SweepExtra ex,
                                               uint32_t* stamp_q) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return 0;  // uniform over the group
  const int l = tg.q, lane = l & 31, wid = l >> 5;
  const int x = l & 7, y = (l >> 3) & 7, z = l >> 6;
  const int64_t g = (int64_t)t * TV + l, Np = P.Np;
  int h = __ldcg(P.h + g), e = __ldcg(P.e + g), rT = __ldcg(P.rT + g);
  int r[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) r[d] = __ldcg(P.r + d * Np + g);
  if (l >= 64 && l < 128) {  // y and z halo rows, 16 bytes per thread
    const int i = l - 64, half = i & 1, k = (i >> 1) & 7, f = PY + (i >> 4);
    const int nt = __ldcg(P.nbr + f * P.T + t);
    const int src = (f == PY ? 64 * k : f == MY ? 64 * k + 56 : f == PZ ? 8 * k : 8 * k + 448) + 4 * half;
    const int dst = (f == PY ? hrow(8, k) : f == MY ? hrow(-1, k) : f == PZ ? hrow(k, 8) : hrow(k, -1)) + 4 * half;
    int4 v = make_int4(INF, INF, INF, INF);
    if (nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T)) v = __ldcg(reinterpret_cast<const int4*>(P.h + (int64_t)nt * TV + src));
    *reinterpret_cast<int4*>(S.h[0] + dst) = v;
    *reinterpret_cast<int4*>(S.h[1] + dst) = v;
  } else if (l >= 128 && l < 256) {  // x halo
    const int i = l - 128, f = i < 64 ? MX : PX, k = i & 63;
    const int nt = __ldcg(P.nbr + f * P.T + t);
    const int v = (nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T)) ? __ldcg(P.h + (int64_t)nt * TV + 8 * k + (f == MX ? 7 : 0)) : INF;
    S.h[0][HROWS * 8 + i] = v;
    S.h[1][HROWS * 8 + i] = v;
  } else if (l >= 256 && l < 262) {
    S.nb[l - 256] = __ldcg(P.nbr + (l - 256) * P.T + t);
  }
  const int inst = __ldcg(P.tinst + t);
  const int hdead = P.geo[inst].hdead;
  const int hi = hrow(y, z) + x;
  int off[6];  // neighbours in a buffer of heights
  off[PX] = x < 7 ? hi + 1 : HROWS * 8 + 64 + (l >> 3);
  off[MX] = x > 0 ? hi - 1 : HROWS * 8 + (l >> 3);
  off[PY] = hi + 8; off[MY] = hi - 8;
  off[PZ] = hi + 80; off[MZ] = hi - 80;
  const bool in[6] = {x < 7, x > 0, y < 7, y > 0, z < 7, z > 0};
  // where a push along d goes: the voxel's slot for the neighbour (and the
  // neighbour's warp is told), or the face entry, whose only writer this is
  uint32_t to[6], tell[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    to[d] = smem_addr(in[d] ? &S.out[d][l] : &S.facc[d][d < 2 ? l >> 3 : d < 4 ? x + 8 * z : l & 63]);
    tell[d] = smem_addr(in[d] ? &S.inbox[(l + loff(d)) >> 5] : &S.moved[d]);
  }
  const uint32_t from = smem_addr(&S.out[0][l]);
  S.h[0][hi] = h;
#pragma unroll
  for (int d = 0; d < 6; ++d) S.out[d][l] = 0;
  if (l < 384) (&S.facc[0][0])[l] = 0;
  if (l < 24) S.inbox[l] = 0;  // and moved[]
  tg.sync();

  int sink = 0, pulses = 0, cur = 0;
  bool dirty = false, any = true;
  const int h0 = h;
  for (int round = 0;; ++round) {
    if (R > 0 && !(exact && round == 0)) {  // region relabel, as in sweep_tile
      int dd = rT > 0 ? 1 : INF, c[6];
      int* const H = S.h[cur];
      H[hi] = dd;
#pragma unroll
      for (int d = 0; d < 6; ++d) c[d] = r[d] > 0 ? 1 : CLOSED;
      tg.sync();
      for (int it = 0; it < 600; ++it) {  // Bellman-Ford: < 512 steps in a tile, two per barrier
        const int d0 = dd;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int a = __viaddmin_s32(H[off[0]], c[0], __viaddmin_s32(H[off[1]], c[1], dd));
          const int b = __viaddmin_s32(H[off[2]], c[2], H[off[3]] + c[3]);
          const int n = min(__viaddmin_s32(H[off[4]], c[4], a), __viaddmin_s32(H[off[5]], c[5], b));
          if (n < dd) H[hi] = n;
          dd = n;
          __syncwarp();
        }
        if (!tg.any(dd < d0)) break;
      }
      h = max(h, dd);
      if (h >= hdead) h = INF;
      H[hi] = h;
      tg.sync();
    }
    for (int p = 0; p < L; ++p) {
      const int* H = S.h[cur];
      ++pulses;
      // (a voxel at INF has no neighbour at INF - 1 and no sink residual)
      if (__any_sync(FULL, e > 0 && h < INF)) {
        int hn[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) hn[d] = H[off[d]];
        const int e0 = e;
        const int ds = min(e, rT);  // a voxel with a sink residual is at height 1: the labelling is valid
        e -= ds;
        rT -= ds;
        sink += ds;
        if (ds > 0) S.moved[6] = pulses;  // same value from every writer of this pulse
        int dl[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) dl[d] = hn[d] + 1 == h ? r[d] : 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          dl[d] = min(e, dl[d]);
          e -= dl[d];
          r[d] -= dl[d];
        }
        push_out6(to, tell, dl, pulses);
        dirty = dirty || e != e0;
      }
      tg.sync();
      if (S.inbox[wid] == pulses) {  // uniform over the warp
        int v[6], got = 0;
        take6(from, in, v);
        clear6(from, v);
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          e += v[d];
          r[d] += v[d];
          got |= v[d];
        }
        dirty = dirty || got > 0;
      }
      // Relabel, from the labels of the pulse's start: the labelling is valid,
      // so the lowest residual neighbour mn is at h - 1 or higher (the sink
      // counts as height 0), and 1 + mn is h itself where the voxel still has
      // an admissible edge.
      bool act = e > 0 && h < INF;
      if (__any_sync(FULL, act)) {
        int c[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          const int hn = H[off[d]];
          c[d] = r[d] > 0 ? hn : INF;
        }
        const int mn = min(min(min(c[0], c[1]), min(c[2], c[3])), min(c[4], c[5]));
        int v = (rT > 0 ? 0 : mn) + 1;
        if (v >= hdead) v = INF;
        if (act) h = v;
        act = act && v < INF;
      }
      S.h[cur ^ 1][hi] = h;
      any = tg.any(act);
      cur ^= 1;
      if (!any) break;
    }
    if (!any || round + 1 >= max(R, 1)) break;
  }

  // write-back, the queue updates' chains of two dependent atomics first
  if (l == 480) {
    P.act[t] = (uint8_t)(any ? 1 : 0);
    if (APPEND && any) queue_tile(P, stamp_q, t, id_self, list_self, cnt_self);
    if (ex.tr_pulses && ex.tr_pulses[t] == 0) {
      int last = 0;
      for (int d = 0; d < 7; ++d) last = max(last, S.moved[d]);
      ex.tr_pulses[t] = (uint8_t)(last > 0 ? min(last, 254) : 255);
    }
  }
  if (l >= 448 && l < 454 && S.moved[l - 448]) {
    const int nt = S.nb[l - 448];
    if (nt < 0) {
      raise_error(P, CGC_ERR_OVERFLOW);  // capacity leaving the grid
    } else if (CGC_IN_BOUNDS(P, nt, P.T)) {
      if (APPEND) queue_tile(P, stamp_q, nt, id_next, list_next, cnt_next);
      P.act[nt] = 1;
    }
  }
  if (l < 384) {  // flow that left the tile: excess and reverse residual of the neighbour
    const int w = (&S.facc[0][0])[l];
    if (w > 0) {
      const int f = l >> 6, a = l & 7, b = (l >> 3) & 7, nt = S.nb[f];
      if (nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T)) {
        const int src = f == PX ? 8 * a + 64 * b : f == MX ? 7 + 8 * a + 64 * b : f == PY ? a + 64 * b
                      : f == MY ? a + 56 + 64 * b : f == PZ ? a + 8 * b : a + 8 * b + 448;
        const int64_t ng = (int64_t)nt * TV + src;
        atomicAdd(P.e + ng, w);
        atomicAdd(P.r + (f ^ 1) * Np + ng, w);
        atomicOr((unsigned*)(P.rmask + (ng & ~(int64_t)3)), (128u | (1u << (f ^ 1))) << (8 * (int)(ng & 3)));
      }
    }
  }
  if (h != h0) P.h[g] = h;
  if (dirty) {
    P.e[g] = e;
    P.rT[g] = rT;
    unsigned m = (rT > 0 ? 64u : 0u) | (e > 0 ? 128u : 0u);
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      P.r[d * Np + g] = r[d];
      m |= (r[d] > 0 ? 1u : 0u) << d;
    }
    P.rmask[g] = (uint8_t)m;
  }
  if (__any_sync(FULL, sink > 0)) {
    long long s = sink;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
    if (lane == 0) {
      atomicAdd(P.flow + inst, (unsigned long long)s);
      if (ex.sink_tiles) atomicAdd(ex.sink_tiles, 1);
      if (ex.tr_sink) ex.tr_sink[t] = 1;
    }
  }
  return pulses;
}

// Upload of a run of up to four tiles along x of an instance, from its linear
// (x-fastest) device inputs ip[0..7] = capS, capT, fwd x/y/z, bwd x/y/z (a null
// n-link pointer is zero), fused with the preflow initialisation: the t-links
// cancel (m = min(capS, capT) goes straight to the sink, the rest of capS
// becomes excess), the residual planes and the residual bit mask are written,
// and capacities that could overflow int32 excess or residuals raise
// CGC_ERR_OVERFLOW.  Every value that needs (the capacity into the voxel from
// each neighbour: bwd[v] from +a, fwd[v - stride] from -a) is an input this
// CTA reads anyway, so the solve starts after one pass over the planes.
// Heights and reachability are not touched: the first relabel and the final
// seeding pass write them everywhere.
// Replaces initResidualsKernel and pushThroughTLinksFromSourceKernel
// (detail/graph_cut_implementation.hpp:28-40, detail/graph_cut_push.hpp:11-24).
//
// 128 threads: thread (xq, y, zh) walks four z planes, four voxels (half a
// tile row) in each.  Loads in flight bound it, so the step is kept short and
// small in registers; the run makes every access whole 128-byte lines (a warp
// reads four rows of 32 voxels and writes four rows of each of the four tiles,
// which are contiguous there); the neighbour values come from registers (z),
// the next lane (x) or the L1 (y).
//   A4: plane rows of four voxels are 16-byte aligned (aligned planes, X a
//   multiple of 4); otherwise a row is four scalars, all of a step's loads in
//   flight at once (the two aligned vectors that cover it, with a branch at the
//   plane's end, took 405x377x362 1.13 ms with both masks, scalars 0.81; without
//   the branch 0.90).  SAME: symmetric n-links, one plane per axis.
//   two_halves: the pool keeps both halves of stamp_sw.
// 512x512x128: 0.75 -> 0.29 ms, 6.3 TB/s (before: a CTA per tile, eight planes read, 64-bit
// checks per voxel); 405x377x362, whose rows are not aligned, with both masks: 2.0 -> 0.81 ms.
template <bool A4, bool SAME>
__device__ __forceinline__ void put_run_as(const DevPool& P, const int t0, const int32_t* const* ip, const InstGeo& G,
                                           const int inst, const bool two_halves) {
  __shared__ long long red[4];
  const int lt = t0 - G.tile_base;
  const int rows = lt / G.TX, tx0 = lt - rows * G.TX, tz = rows / G.TY, ty = rows - tz * G.TY;
  const int q = threadIdx.x, xq = q & 7, yl = (q >> 3) & 7, zh = q >> 6;
  const bool tile = tx0 + (xq >> 1) < G.TX;
  const int x0 = tx0 * 8 + 4 * xq, y = ty * 8 + yl;
  const int64_t N = (int64_t)G.X * G.Y * G.Z, sy = G.X, sz = (int64_t)G.X * G.Y;
  // the run lies inside the instance with a voxel to spare on every side
  const bool inner = tx0 > 0 && ty > 0 && tz > 0 && tx0 * 8 + 32 < G.X && ty * 8 + 8 < G.Y && tz * 8 + 8 < G.Z;
  // o = p[v .. v+3] (0 <= v < N; entries past the plane's end repeat one
  // inside); a null plane reads as zero
  auto row4 = [&](int (&o)[4], const int32_t* p, int64_t v) {
    if (!p) {
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = 0;
    } else if (A4) {
      const int4 w = __ldg(reinterpret_cast<const int4*>(p + v));
      o[0] = w.x; o[1] = w.y; o[2] = w.z; o[3] = w.w;
    } else {
      const int lim = (int)min((int64_t)3, N - 1 - v);
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = __ldg(p + v + min(k, lim));
    }
  };
  bool neg = false, bad = false;
  long long tot = 0;
  int fzm[4], bzm[4];  // fwd / bwd z of the plane below
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int zl = 4 * zh + i, z = tz * 8 + zl;
    const bool row = inner || (y < G.Y && z < G.Z && x0 < G.X);
    const int64_t v = row ? x0 + sy * y + sz * z : 0;
    const int64_t vy = row && y > 0 ? v - sy : v;
    const bool left = xq == 0 && row && x0 > 0;
    // r[2a]: to +a (fwd), r[2a+1]: to -a (bwd of the neighbour); bk: the
    // capacities back (symmetric n-links: the same numbers)
    int s[4], c[4], r[6][4], bk[6][4];
    row4(s, ip[0], v);
    row4(c, ip[1], v);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      row4(r[2 * a], ip[2 + a], v);
      if (!SAME) row4(bk[2 * a], ip[5 + a], v);
    }
    int fx = left && ip[2] ? __ldg(ip[2] + v - 1) : 0, bx = 0;
    row4(SAME ? r[3] : bk[3], ip[3], vy);
    if (!SAME) {
      row4(r[3], ip[6], vy);
      if (left && ip[5]) bx = __ldg(ip[5] + v - 1);
    }
    if (i == 0) {
      const int64_t vz = row && z > 0 ? v - sz : v;
      row4(fzm, ip[4], vz);
      if (!SAME) row4(bzm, ip[7], vz);
    }
    const int fl = __shfl_up_sync(FULL, r[0][3], 1);
    if (xq > 0) fx = fl;
    if (!SAME) {
      const int bl = __shfl_up_sync(FULL, bk[0][3], 1);
      if (xq > 0) bx = bl;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      (SAME ? r[1] : bk[1])[k] = k > 0 ? r[0][k > 0 ? k - 1 : 0] : fx;
      (SAME ? r[5] : bk[5])[k] = fzm[k];
      fzm[k] = r[4][k];
      if (!SAME) {
        r[1][k] = k > 0 ? bk[0][k > 0 ? k - 1 : 0] : bx;
        r[5][k] = bzm[k];
        bzm[k] = bk[4][k];
      }
    }
    if (!inner) {  // nothing outside the instance, no link across its faces
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int x = x0 + k;
        const bool ok = row && x < G.X;
        const bool has[6] = {ok && x + 1 < G.X, ok && x > 0, ok && y + 1 < G.Y, ok && y > 0, ok && z + 1 < G.Z, ok && z > 0};
        if (!ok) s[k] = c[k] = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          if (!has[d]) r[d][k] = 0;
          if (!SAME && !has[d]) bk[d][k] = 0;
        }
      }
    }
    // Checks.  Values below 2^28 are not negative and cannot overflow: a voxel
    // sums seven of them, a link two.
    unsigned any = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      any |= (unsigned)(s[k] | c[k]);
#pragma unroll
      for (int d = 0; d < 6; ++d) any |= (unsigned)(SAME ? r[d][k] : r[d][k] | bk[d][k]);
    }
    if (any >> 28) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        neg = neg || s[k] < 0 || c[k] < 0;
        long long inflow = (long long)s[k] - min(s[k], c[k]);
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          const long long back = SAME ? r[d][k] : bk[d][k];
          neg = neg || r[d][k] < 0;
          inflow += back;
          bad = bad || (long long)r[d][k] + back > 2147483647ll;
        }
        bad = bad || inflow > 2147483647ll;
      }
    }
    // t-link cancellation: min(capS, capT) flows straight through
    unsigned m4 = 0;
    int through = 0;  // below 2^30 where no value reaches 2^28
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int mcap = min(s[k], c[k]);
      s[k] -= mcap;
      c[k] -= mcap;
      if (any >> 28) tot += mcap; else through += mcap;
#pragma unroll
      for (int d = 0; d < 6; ++d) m4 |= (r[d][k] > 0 ? 1u : 0u) << (8 * k + d);
      m4 |= (c[k] > 0 ? 64u : 0u) << (8 * k) | (s[k] > 0 ? 128u : 0u) << (8 * k);
    }
    tot += through;
    if (tile) {
      const int64_t g = (int64_t)(t0 + (xq >> 1)) * TV + 64 * zl + 8 * yl + 4 * (xq & 1);
      st4(P.e + g, s);
      st4(P.rT + g, c);
#pragma unroll
      for (int d = 0; d < 6; ++d) st4(P.r + d * P.Np + g, r[d]);
      *reinterpret_cast<uint32_t*>(P.rmask + g) = m4;
    }
  }
  if (neg) raise_error(P, CGC_ERR_ARG);
  if (bad) raise_error(P, CGC_ERR_OVERFLOW);
  if (tile && (q & ~6) == 0) {  // one thread per tile
    const int t = t0 + (xq >> 1);
    P.act[t] = 0;
    P.stamp_bfs[t] = P.stamp_sw[t] = P.stamp_inc[t] = 0u;
    if (two_halves) P.stamp_sw[P.T + t] = 0u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(FULL, tot, o);
  if ((q & 31) == 0) red[q >> 5] = tot;
  __syncthreads();
  if (q == 0) {
    const long long sum = red[0] + red[1] + red[2] + red[3];
    if (sum) atomicAdd(P.flow + inst, (unsigned long long)sum);
  }
}

__device__ __forceinline__ void put_run(const DevPool& P, const int t0, const int32_t* const* ip, const bool two_halves) {
  if (!CGC_IN_BOUNDS(P, t0, P.T)) return;  // uniform over the block, as is all below
  const int inst = P.tinst[t0];
  const InstGeo G = P.geo[inst];
  uintptr_t align = 0;
  bool same = true;
#pragma unroll
  for (int a = 0; a < 8; ++a) align |= reinterpret_cast<uintptr_t>(ip[a]);
#pragma unroll
  for (int a = 0; a < 3; ++a) same = same && ip[2 + a] == ip[5 + a];
  const bool a4 = (align & 15) == 0 && (G.X & 3) == 0;
  if (a4 && same) put_run_as<true, true>(P, t0, ip, G, inst, two_halves);
  else if (a4) put_run_as<true, false>(P, t0, ip, G, inst, two_halves);
  else if (same) put_run_as<false, true>(P, t0, ip, G, inst, two_halves);
  else put_run_as<false, false>(P, t0, ip, G, inst, two_halves);
}

// ---------------------------------------------------------------------------
// Cut sets in linear voxel order, four voxels per thread: voxels v0..v0+3 of
// an instance (v0 a multiple of 4), one 32-bit store per output when the
// destination is aligned, so a warp writes whole 128-byte lines.  Where X is a
// multiple of 4 they are half a tile row, read with one 16-byte and one 4-byte
// load; else each is gathered (all loads issued at once from clamped indices).
// Bit 0 of each byte of *sink: height < INF; of *source: in the minimal
// source set.
__device__ __forceinline__ void seg_gather4(const DevPool& P, const InstGeo& G, int64_t v0, int64_t N,
                                            unsigned* sink, unsigned* source) {
  int x, y, z;
  if (N <= 0xffffffffll) {
    const unsigned v = (unsigned)v0, rest = v / (unsigned)G.X;
    x = (int)(v - rest * (unsigned)G.X);
    z = (int)(rest / (unsigned)G.Y);
    y = (int)(rest - (unsigned)z * (unsigned)G.Y);
  } else {
    const int64_t rest = v0 / G.X;
    x = (int)(v0 - rest * G.X);
    y = (int)(rest % G.Y);
    z = (int)(rest / G.Y);
  }
  if ((G.X & 3) == 0) {
    const int64_t t = G.tile_base + (x >> 3) + (int64_t)G.TX * ((y >> 3) + (int64_t)G.TY * (z >> 3));
    const int64_t g = t * TV + (x & 7) + 8 * (y & 7) + 64 * (z & 7);
    int h[4];
    unsigned b = 0;
    if (sink) ldcg4(P.h + g, h);
    if (source) b = __ldcg(reinterpret_cast<const unsigned*>(P.reach + g));
    if (sink) *sink = (h[0] < INF ? 1u : 0u) | (h[1] < INF ? 256u : 0u) | (h[2] < INF ? 65536u : 0u) | (h[3] < INF ? 1u << 24 : 0u);
    if (source) *source = b;  // bytes of 0 or 1
    return;
  }
  int64_t gk[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t t = G.tile_base + (x >> 3) + (int64_t)G.TX * ((y >> 3) + (int64_t)G.TY * (z >> 3));
    gk[k] = t * TV + (x & 7) + 8 * (y & 7) + 64 * (z & 7);
    if (v0 + k >= N) gk[k] = gk[0];
    if (++x == G.X) { x = 0; if (++y == G.Y) { y = 0; ++z; } }
  }
  unsigned a = 0, b = 0;
  int hv[4];
  unsigned char rv[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    hv[k] = sink ? __ldcg(P.h + gk[k]) : INF;
    rv[k] = source ? __ldcg(P.reach + gk[k]) : (unsigned char)0;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a |= (hv[k] < INF ? 1u : 0u) << (8 * k);
    b |= (rv[k] ? 1u : 0u) << (8 * k);
  }
  if (sink) *sink = a;
  if (source) *source = b;
}

// the bytes of `bits` (0 or 1 each) as mask / bg at out[v0 .. min(v0 + 4, N))
__device__ __forceinline__ void seg_store4(uint8_t* out, int64_t v0, int64_t N, unsigned bits, uint8_t mask,
                                           uint8_t bg) {
  unsigned w = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) w |= (unsigned)(((bits >> (8 * k)) & 1u) ? mask : bg) << (8 * k);
  uint8_t* p = out + v0;
  if (v0 + 4 <= N && ((reinterpret_cast<uintptr_t>(p) & 3u) == 0)) {
    *reinterpret_cast<unsigned*>(p) = w;
  } else {
    for (int k = 0; k < 4 && v0 + k < N; ++k) p[k] = (uint8_t)(w >> (8 * k));
  }
}

// Both cut sets of an instance into src / snk (1/0 bytes, each may be null);
// CTA `cta` of `ctas`.
__device__ __forceinline__ void seg_instance(const DevPool& P, int inst, uint8_t* src, uint8_t* snk, int cta, int ctas) {
  const InstGeo G = P.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
#pragma unroll 4
  for (int64_t v0 = 4 * ((int64_t)cta * blockDim.x + threadIdx.x); v0 < N; v0 += 4 * (int64_t)ctas * blockDim.x) {
    unsigned a = 0, b = 0;
    seg_gather4(P, G, v0, N, snk ? &a : nullptr, src ? &b : nullptr);
    if (src) seg_store4(src, v0, N, b, 1, 0);
    if (snk) seg_store4(snk, v0, N, a, 1, 0);
  }
}

// ---------------------------------------------------------------------------
// BFS seeding, first step: bfs_init_tile_w (a warp per tile).
// Second BFS seeding step, one thread per tile: queue every tile that is not
// all seeds and holds a seed or touches a seed on a neighbour's face.
__device__ __forceinline__ bool bfs_seed_tile(const DevPool& P, const int t) {
  bool q = false;
  if (t < P.T) {
    const int f = __ldcg(P.tflag + t);
    if (!(f & (TF_ALL_SEED | TF_DEAD))) {
      q = (f & TF_HAS_SEED) != 0;
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        const int nt = __ldcg(P.nbr + d * P.T + t);
        if (nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T) && ((__ldcg(P.tflag + nt) >> (1 + (d ^ 1))) & 1))
          q = true;  // dead tiles have no seed bits
      }
    }
  }
  return q;
}

__device__ __forceinline__ void bfs_queue_tile(const DevPool& P, const int t, const uint32_t id0, int32_t* list0,
                                               int32_t* cnt0) {
  const bool q = bfs_seed_tile(P, t);
  if (q) P.stamp_bfs[t] = id0;
  warp_append(P, q, t, list0, cnt0);
}

// faces that a changed half row lies on, as bits (end: its voxel on the x face changed)
__device__ __forceinline__ unsigned row_faces(int half, int y, int z, bool end) {
  return (end ? 1u << (half ? PX : MX) : 0u) | (y == 7 ? 1u << PY : 0u) | (y == 0 ? 1u << MY : 0u) |
         (z == 7 ? 1u << PZ : 0u) | (z == 0 ? 1u << MZ : 0u);
}

// One BFS visit: relax h(v) = min(h(v), 1 + h(u)) over residual edges v->u
// until the tile is stable; re-queue face neighbours whose halo changed.  What
// changed, and whether an excess voxel reaches the sink, is read off the heights
// once the relaxation has ended, and two steps share a barrier: a step is bound
// by its own chain of latencies, and a round by the visit with the most steps
// (about 20 where the mean is 5).  All relabels of a 256^3 solve: 0.83 -> 0.69
// ms, of a 150x140x96 segmentation 4.4 -> 3.8 (flags set as heights drop, a
// barrier per step).  The caller synchronises the group before S is used again;
// returns 1 for a visited tile.
__device__ __forceinline__ int bfs_tile(const DevPool& P, const TileGroup<GROUP> tg, const int t, BfsShared& S,
                                        const uint32_t id_next, int32_t* list_next, int32_t* cnt_next) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return 0;  // uniform over the group
  const int q = tg.q, half = q & 1, y = (q >> 1) & 7, z = q >> 4;
  const int row = hrow(y, z) + 4 * half;
  const int64_t g = (int64_t)t * TV + 4 * q;
  const int dead = __ldcg(P.tflag + t) & TF_DEAD;
  int h[4];
  ldcg4(P.h + g, h);
  const unsigned m = __ldcg(reinterpret_cast<const unsigned*>(P.rmask + g));
  bool far = far16(h[0]) || far16(h[1]) || far16(h[2]) || far16(h[3]);
  const int hx = load_halo_heights(P, t, q, S.h, nullptr, S.g, far);
  if (dead) return 0;  // uniform over the group; nothing can change
  const int nb = q >= 32 && q < 38 ? __ldcg(P.nbr + (q - 32) * P.T + t) : -1;  // face neighbour, for the re-queue
  unsigned d2[2] = {pack16(h[0], h[1]), pack16(h[2], h[3])};
  *reinterpret_cast<uint2*>(S.g + row) = make_uint2(d2[0], d2[1]);
  st4(S.h + row, h);
  if (q == 0) S.flags = 0;
  far = tg.any(far);
  bool changed, end;  // a voxel of the row dropped, and the one on the tile's x face
  if (!far) {
    const unsigned w0 = d2[0], w1 = d2[1];
    unsigned c[6][2];
#pragma unroll
    for (int d = 0; d < 6; ++d)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        c[d][j] = (((m >> (16 * j + d)) & 1u) ? 1u : (unsigned)CLOSED16) |
                  (((m >> (16 * j + 8 + d)) & 1u) ? 1u << 16 : (unsigned)CLOSED16 << 16);
    const unsigned hx2 = pack16(hx, 0);
    for (int it = 0; it < 1024; ++it) {  // converges in < 512 steps (path length in a tile)
      bool ch = relax_row16(S.g, row, half, hx2, d2, c);
      __syncwarp();
      ch = relax_row16(S.g, row, half, hx2, d2, c) || ch;
      if (!tg.any(ch)) break;
    }
    changed = d2[0] != w0 || d2[1] != w1;
    end = half ? ((d2[1] ^ w1) >> 16) != 0 : ((d2[0] ^ w0) & 0xffffu) != 0;
    unpack16(d2[0], h[0], h[1]);
    unpack16(d2[1], h[2], h[3]);
  } else {
    const int4 was = make_int4(h[0], h[1], h[2], h[3]);
    int c[6][4];
#pragma unroll
    for (int d = 0; d < 6; ++d)
#pragma unroll
      for (int k = 0; k < 4; ++k) c[d][k] = ((m >> (8 * k + d)) & 1u) ? 1 : CLOSED;
    for (int it = 0; it < 1024; ++it) {
      const bool ch = relax_row(S.h, row, half, hx, h, c);
      if (!tg.any(ch)) break;
    }
    changed = h[0] != was.x || h[1] != was.y || h[2] != was.z || h[3] != was.w;
    end = half ? h[3] != was.w : h[0] != was.x;
  }
  // faces whose voxels changed (bits 0..5) and, in bit 6, an excess voxel that
  // reaches the sink
  unsigned flags = 0;
  if (changed) flags = row_faces(half, y, z, end);
  if (((m & 0x80u) && h[0] < INF) || ((m & 0x8000u) && h[1] < INF) || ((m & 0x800000u) && h[2] < INF) ||
      ((m & 0x80000000u) && h[3] < INF))
    flags |= 64u;
  flags = __reduce_or_sync(FULL, flags);
  if ((q & 31) == 0 && flags) atomicOr(&S.flags, flags);
  tg.sync();
  flags = S.flags;
  if (q >= 32 && q < 38 && ((flags >> (q - 32)) & 1u) && nb >= 0)
    queue_tile(P, P.stamp_bfs, nb, id_next, list_next, cnt_next);
  if (changed) st4(P.h + g, h);
  if (q == 0) P.act[t] = (uint8_t)((flags >> 6) & 1u);  // heights only drop in later visits: the last visit's value is final
  return 1;
}

// ---------------------------------------------------------------------------
// Incremental global relabel.  Heights are a valid labelling at all times
// (h <= d, the exact distance to the sink), and h(v) == d(v) exactly when v is
// supported: a sink-adjacent voxel at height 1 (rT > 0), or a voxel with a
// residual edge to a supported neighbour exactly one lower.  (Along a shortest
// path every step of a valid labelling drops by at most one, so h == d forces
// each step to drop by exactly one down to a seed at 1.)  Right after an exact
// relabel every finite voxel is supported; a sweep cycle can break support
// only inside the tiles it queued (their heights and out-residuals changed)
// and, through their face voxels, in the face neighbours of those tiles.  So
// the invalidation pass below visits those tiles, sets every unsupported
// voxel to INF and re-checks the neighbours of every voxel it drops; the
// voxels it leaves finite are exact, and the tile Bellman-Ford (bfs_tile)
// started from the tiles with dropped voxels recomputes the rest exactly.
// The heights that come out equal the full BFS's bit for bit.

// a tile's sweep stamps (both halves under exclusive sweeps) were written
// after id c0, i.e. the tile was queued during the current sweep cycle
__device__ __forceinline__ bool queued_since(const DevPool& P, int t, uint32_t c0, bool exclusive) {
  const uint32_t a = __ldcg(P.stamp_sw + t);
  const uint32_t b = exclusive ? __ldcg(P.stamp_sw + P.T + t) : 0u;
  return (int32_t)(a - c0) > 0 || (exclusive && (int32_t)(b - c0) > 0);
}

// Seed of the invalidation pass, one thread per tile: tiles queued during the
// cycle and their face neighbours.
__device__ __forceinline__ void inval_queue_tile(const DevPool& P, const int t, const uint32_t c0, const bool exclusive,
                                                 const uint32_t id0, int32_t* list0, int32_t* cnt0) {
  bool q = false;
  if (t < P.T) {
    q = queued_since(P, t, c0, exclusive);
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      const int nt = __ldcg(P.nbr + d * P.T + t);
      if (!q && nt >= 0 && CGC_IN_BOUNDS(P, nt, P.T)) q = queued_since(P, nt, c0, exclusive);
    }
    if (q && (__ldcg(P.tflag + t) & TF_DEAD)) q = false;  // all INF, nothing to check
  }
  if (q) P.stamp_bfs[t] = id0;
  warp_append(P, q, t, list0, cnt0);
}

// One invalidation visit: drop unsupported voxels of tile t to INF until the
// tile is stable (drops are monotone, so in-place updates are safe and the
// result is the largest supported set); re-queue the face neighbours of
// dropped face voxels, and list the tile once (stamp_inc) for the BFS rounds.
// The caller synchronises the group before S is used again.
__device__ __forceinline__ int inval_tile(const DevPool& P, const TileGroup<GROUP> tg, const int t, BfsShared& S,
                                          const uint32_t id_next, int32_t* list_next, int32_t* cnt_next,
                                          const uint32_t id_bfs, int32_t* list_bfs, int32_t* cnt_bfs) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return 0;  // uniform over the group
  const int q = tg.q, half = q & 1, y = (q >> 1) & 7, z = q >> 4;
  const int row = hrow(y, z) + 4 * half;
  const int64_t g = (int64_t)t * TV + 4 * q;
  int h[4];
  ldcg4(P.h + g, h);
  const unsigned m = __ldcg(reinterpret_cast<const unsigned*>(P.rmask + g));
  bool far = false;
  const int hx = load_halo_heights(P, t, q, S.h, nullptr, nullptr, far);
  const int nb = q >= 32 && q < 38 ? __ldcg(P.nbr + (q - 32) * P.T + t) : -1;  // face neighbour, for the re-queue
  st4(S.h + row, h);
  if (q == 0) S.flags = 0;
  tg.sync();
  unsigned drop = 0;  // bit k: voxel k was dropped
  for (int it = 0; it < 1024; ++it) {  // a drop per step climbs one height: < 512 steps in a tile
    const int4 yp = ld4(S.h + row + 8), ym = ld4(S.h + row - 8), zp = ld4(S.h + row + 80), zm = ld4(S.h + row - 80);
    const int xo = __shfl_xor_sync(FULL, half ? h[0] : h[3], 1);
    bool ch = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned mk = m >> (8 * k);
      const int hm = h[k] - 1;
      const int r = k < 3 ? h[k < 3 ? k + 1 : 3] : (half ? hx : xo);
      const int l = k > 0 ? h[k > 0 ? k - 1 : 0] : (half ? xo : hx);
      const bool sup = ((mk & 64u) && hm == 0) || ((mk & 1u) && r == hm) || ((mk & 2u) && l == hm) ||
                       ((mk & 4u) && at(yp, k) == hm) || ((mk & 8u) && at(ym, k) == hm) ||
                       ((mk & 16u) && at(zp, k) == hm) || ((mk & 32u) && at(zm, k) == hm);
      if (h[k] < INF && !sup) {
        h[k] = INF;
        ch = true;
        drop |= 1u << k;
      }
    }
    if (ch) st4(S.h + row, h);
    if (!tg.any(ch)) break;
  }
  unsigned flags = 0;  // faces that voxels were dropped on (bits 0..5), any drop (bit 6)
  if (drop) flags = 64u | row_faces(half, y, z, (drop >> (half ? 3 : 0)) & 1u);
  flags = __reduce_or_sync(FULL, flags);
  if ((q & 31) == 0 && flags) atomicOr(&S.flags, flags);
  tg.sync();
  flags = S.flags;
  if (q == 0 && (flags & 64u)) queue_tile(P, P.stamp_inc, t, id_bfs, list_bfs, cnt_bfs);
  if (q >= 32 && q < 38 && ((flags >> (q - 32)) & 1u) && nb >= 0)
    queue_tile(P, P.stamp_bfs, nb, id_next, list_next, cnt_next);
  if (drop) st4(P.h + g, h);
  return 1;
}

// ---------------------------------------------------------------------------
// Source-side reachability (canonical cut) after the maximum preflow:
// closure of {v : e(v) > 0} over residual edges, seeded by reach_init_tile_w
// (a warp per tile).  One warp visits a tile, with the reach set and the
// residual masks as bits: lane l owns the rows y = 2(l&3), +1 of plane z = l>>2
// (16 voxels, bit = 8 (y&1) + x), so a step of the closure is a few shifts and
// shuffles, without shared memory or barriers.
__device__ __forceinline__ unsigned byte_bits(unsigned w, int bit) {  // bit `bit` of each byte of w -> bits 0..3
  w = (w >> bit) & 0x01010101u;
  return (w * 0x01020408u) >> 24 & 15u;  // byte k -> bit k
}

__device__ __forceinline__ void reach_tile_w(const DevPool& P, const int t, const uint32_t id_next, int32_t* list_next,
                                             int32_t* cnt_next) {
  if (!CGC_IN_BOUNDS(P, t, P.T)) return;  // uniform over the warp
  const int lane = threadIdx.x & 31, j = lane & 3, z = lane >> 2;
  const int64_t g = (int64_t)t * TV + 16 * lane;
  const uint4 rc4 = __ldcg(reinterpret_cast<const uint4*>(P.reach + g));
  const uint4 m4 = __ldcg(reinterpret_cast<const uint4*>(P.rmask + g));
  const int nb = lane < 6 ? __ldcg(P.nbr + lane * P.T + t) : -1;
  int nt[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) nt[d] = __shfl_sync(FULL, nb, d);
  // flow of reachability into this lane's voxels through the tile's faces: a
  // reached voxel of the neighbour with a residual edge towards the tile
  unsigned in = 0;
  auto row_in = [&](int f, int src) {  // 8 voxels of a neighbour's row at src
    const int64_t ng = (int64_t)nt[f] * TV + src;
    const uint2 a = __ldcg(reinterpret_cast<const uint2*>(P.reach + ng));
    const uint2 b = __ldcg(reinterpret_cast<const uint2*>(P.rmask + ng));
    const int bit = f ^ 1;
    return byte_bits(a.x, 0) & byte_bits(b.x, bit) | (byte_bits(a.y, 0) & byte_bits(b.y, bit)) << 4;
  };
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (nt[d] >= 0 && !CGC_IN_BOUNDS(P, nt[d], P.T)) nt[d] = -1;
  if (nt[PY] >= 0 && j == 3) in |= row_in(PY, 64 * z) << 8;
  if (nt[MY] >= 0 && j == 0) in |= row_in(MY, 64 * z + 56);
  if (nt[PZ] >= 0 && z == 7) in |= row_in(PZ, 16 * j) | row_in(PZ, 16 * j + 8) << 8;
  if (nt[MZ] >= 0 && z == 0) in |= row_in(MZ, 448 + 16 * j) | row_in(MZ, 448 + 16 * j + 8) << 8;
#pragma unroll
  for (int s = 0; s < 2; ++s) {  // x faces: the voxel next to each row end
    if (nt[PX] >= 0) {
      const int64_t ng = (int64_t)nt[PX] * TV + 16 * lane + 8 * s;
      if (__ldcg(P.reach + ng) && ((__ldcg(P.rmask + ng) >> MX) & 1)) in |= 0x80u << (8 * s);
    }
    if (nt[MX] >= 0) {
      const int64_t ng = (int64_t)nt[MX] * TV + 16 * lane + 8 * s + 7;
      if (__ldcg(P.reach + ng) && ((__ldcg(P.rmask + ng) >> PX) & 1)) in |= 0x01u << (8 * s);
    }
  }
  auto bits16 = [](const uint4& w, int bit) {
    return byte_bits(w.x, bit) | byte_bits(w.y, bit) << 4 | byte_bits(w.z, bit) << 8 | byte_bits(w.w, bit) << 12;
  };
  const unsigned r0 = bits16(rc4, 0);
  unsigned M[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) M[d] = bits16(m4, d);
  unsigned r = r0 | in;
  for (int it = 0; it < 1024; ++it) {  // < 512 steps
    unsigned n = r | (r & M[PX] & 0x7f7fu) << 1;
    n |= (n & M[MX] & 0xfefeu) >> 1;
    const unsigned yp = n & M[PY], ym = n & M[MY];
    const unsigned yu = __shfl_up_sync(FULL, yp, 1), yd = __shfl_down_sync(FULL, ym, 1);
    const unsigned zu = __shfl_up_sync(FULL, n & M[PZ], 4), zd = __shfl_down_sync(FULL, n & M[MZ], 4);
    n |= (yp & 0xffu) << 8 | (ym >> 8 & 0xffu);
    if (j > 0) n |= yu >> 8 & 0xffu;
    if (j < 3) n |= (yd & 0xffu) << 8;
    if (z > 0) n |= zu;
    if (z < 7) n |= zd;
    const bool ch = n != r;
    r = n;
    if (!__any_sync(FULL, ch)) break;
  }
  const unsigned fresh = r & ~r0;
  unsigned faces = 0;
  if (fresh) {
    // only voxels with a residual edge through the face can reach the neighbour
    faces = ((fresh & M[PX] & 0x8080u) ? 1u << PX : 0u) | ((fresh & M[MX] & 0x0101u) ? 1u << MX : 0u) |
            ((j == 3 && (fresh & M[PY] & 0xff00u)) ? 1u << PY : 0u) | ((j == 0 && (fresh & M[MY] & 0xffu)) ? 1u << MY : 0u) |
            ((z == 7 && (fresh & M[PZ])) ? 1u << PZ : 0u) | ((z == 0 && (fresh & M[MZ])) ? 1u << MZ : 0u);
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned b = r >> (4 * k);
      w[k] = (b & 1u) | (b & 2u) << 7 | (b & 4u) << 14 | (b & 8u) << 21;
    }
    *reinterpret_cast<uint4*>(P.reach + g) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  faces = __reduce_or_sync(FULL, faces);
  if (lane < 6 && ((faces >> lane) & 1) && nb >= 0) queue_tile(P, P.stamp_bfs, nb, id_next, list_next, cnt_next);
}

}  // namespace cgc
