// Kernels and host driver of the grid push-relabel engine, plus the C ABI.
//
// The host driver replaces MinCut::compute / MinimalGraphCutComputation::run
// (include/cugip/advanced_operations/detail/graph_cut_implementation.hpp:122-198,
// 286-308): preflow initialisation, then {exact global relabel; K sweep pairs}
// until a global relabel finds no active voxel, then the cut sets.  With
// `persistent` (the default) the whole loop runs inside one cooperative
// launch whose phases are separated by a grid barrier with a bounded wait, so
// no host round trip happens per BFS level or push level (the reference
// synchronises and copies a counter back for every level,
// detail/graph_cut_relabeling.hpp:962-984, detail/graph_cut_push.hpp:395-459).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "cgc.h"
#include "cgc_internal.h"
#include "cgc_kernels.cuh"
#include "cgc_sched.cuh"
#include "cgc_warp.cuh"
#include "cgc_sync.cuh"
#include "cgc_pool.h"

namespace cgc {

static thread_local std::string g_last_error;
std::atomic<long long> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}
int ok() {
  g_last_error.clear();
  return CGC_OK;
}


// ===========================================================================
// kernels
// ===========================================================================

// Fused upload + preflow of a single instance whose 8 input planes are passed
// by value, so a queued solve reads exactly the planes of its own set_* calls
// (put_run).
__global__ void __launch_bounds__(128, 8) k_put_one(DevPool P, InputPlanes in, bool two_halves) {
  const int TX = P.geo[0].TX, rx = (TX + 3) / 4, row = blockIdx.x / rx;
  put_run(P, row * TX + 4 * (blockIdx.x - row * rx), in.p, two_halves);
}
__global__ void __launch_bounds__(256) k_seg_one(DevPool P, uint8_t* src, uint8_t* snk) {
  seg_instance(P, 0, src, snk, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(256) k_copy_two(int32_t* __restrict__ d0, const int32_t* __restrict__ s0,
                                                  int32_t* __restrict__ d1, const int32_t* __restrict__ s1, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    d0[i] = s0[i];
    d1[i] = s1[i];
  }
}

// Cut sets as mask / background bytes from the 1/0 bytes of one buffer
// (16 bytes per thread where src and dst allow it).
__global__ void k_mask_remap(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t n, uint8_t mask,
                             uint8_t bg) {
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (vec) {
    const int64_t n16 = n / 16;
    for (int64_t i = i0; i < n16; i += stride) {
      uint4 v = reinterpret_cast<const uint4*>(src)[i];
      unsigned* w = reinterpret_cast<unsigned*>(&v);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        unsigned o = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) o |= (unsigned)(((w[k] >> (8 * b)) & 1u) ? mask : bg) << (8 * b);
        w[k] = o;
      }
      reinterpret_cast<uint4*>(dst)[i] = v;
    }
    for (int64_t i = n16 * 16 + i0; i < n; i += stride) dst[i] = src[i] ? mask : bg;
  } else {
    for (int64_t i = i0; i < n; i += stride) dst[i] = src[i] ? mask : bg;
  }
}

// Host-driven schedule: one launch per sweep / BFS round; 512 threads (sweeps),
// a tile group (BFS) or a warp (reachability) per list entry.
__global__ void __launch_bounds__(WIDE) k_sweep_list(DevPool P, const int32_t* list, const int32_t* cnt, int L, int R) {
  __shared__ WideShared S;
  const auto tg = TileGroup<WIDE>::of_thread();
  const int n = *cnt;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int p = sweep_tile_wide<false>(P, tg, list[i], L, R, false, S, 0, nullptr, nullptr, 0, nullptr, nullptr,
                                         SweepExtra(), nullptr);
    if (tg.q == 0) {
      atomicAdd(P.stats + S_TILES_SWEPT, 1ull);
      atomicAdd(P.stats + S_PULSES, (unsigned long long)p);
    }
    tg.sync();
  }
}

__global__ void k_compact(DevPool P, int parity, int32_t* list, int32_t* cnt) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool pred = t < P.T && P.act[t] && P.tpar[t] == parity;
  warp_append(P, pred, t, list, cnt);
}

__global__ void __launch_bounds__(512) k_bfs_init(DevPool P, bool fresh) {
  const int nw = gridDim.x * (blockDim.x >> 5);
  for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < P.T; t += nw) bfs_init_tile_w(P, t, fresh);
}

__global__ void k_bfs_queue(DevPool P, uint32_t id0, int32_t* list0, int32_t* cnt0) {
  bfs_queue_tile(P, blockIdx.x * blockDim.x + threadIdx.x, id0, list0, cnt0);
}

__global__ void __launch_bounds__(GROUP) k_bfs_round(DevPool P, const int32_t* list, const int32_t* cnt, uint32_t id_next,
                                                     int32_t* list_next, int32_t* cnt_next) {
  __shared__ __align__(16) BfsShared S;
  const auto tg = TileGroup<GROUP>::of_thread();
  const int n = *cnt;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int v = bfs_tile(P, tg, list[i], S, id_next, list_next, cnt_next);
    if (tg.q == 0 && v) atomicAdd(P.stats + S_TILES_BFS, 1ull);
    tg.sync();
  }
}

__global__ void __launch_bounds__(512) k_reach_init(DevPool P, uint32_t id0, int32_t* list0, int32_t* cnt0) {
  const int nw = gridDim.x * (blockDim.x >> 5);
  for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < P.T; t += nw)
    reach_init_tile_w(P, t, id0, list0, cnt0);
}

__global__ void __launch_bounds__(GROUP) k_reach_round(DevPool P, const int32_t* list, const int32_t* cnt, uint32_t id_next,
                                                       int32_t* list_next, int32_t* cnt_next) {
  const int n = *cnt, nw = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw)
    reach_tile_w(P, list[i], id_next, list_next, cnt_next);
}

__device__ __forceinline__ int ld_cnt(const int32_t* p) { return *(volatile const int32_t*)p; }


// Learned-scheduler stage at the start of a relabel cycle: the features of
// every tile (zero for inactive ones; recorded when tracing), then the three
// convolution layers on the tensor cores, the last one with the head (budgets
// and priorities).  The active tiles are the entries of the cycle's first
// lists (la: na entries, lb: nb).  Four grid barriers.  Returns false when a
// barrier failed.
__device__ __forceinline__ bool sched_stage(const DevPool& P, const SolveParams& prm, int cycle, bool learned,
                                            bool tracing, const int32_t* la, int na, const int32_t* lb, int nb,
                                            uint32_t& bar_target) {
  const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int gw = b * (blockDim.x >> 5) + (tid >> 5), nw = G * (blockDim.x >> 5);
  // zeros for the inactive tiles, a thread per tile
  for (int t = b * blockDim.x + tid; t < P.T; t += G * blockDim.x) {
    const int64_t r = (int64_t)cycle * P.T + t;  // trace row
    if (tracing) { P.tpulses[r] = 0; P.tsink[r] = 0; }
    if (__ldcg(P.act + t)) continue;
    uint4* f = reinterpret_cast<uint4*>(P.sfeat + (int64_t)t * SCHED_C);
    f[0] = make_uint4(0, 0, 0, 0);
    f[1] = make_uint4(0, 0, 0, 0);
    if (tracing) {
      uint4* tf = reinterpret_cast<uint4*>(P.tfeat + r * SCHED_C);
      tf[0] = make_uint4(0, 0, 0, 0);
      tf[1] = make_uint4(0, 0, 0, 0);
    }
  }
  // features of the active tiles, a warp per list entry
  for (int i = gw; i < na + nb; i += nw) {
    const int t = __ldcg(i < na ? la + i : lb + (i - na));
    sched_features_warp(P, t, P.sfeat, tracing ? P.tfeat + ((int64_t)cycle * P.T + t) * SCHED_C : nullptr);
  }
  if (!grid_barrier(P.bar, bar_target, prm.limit_ns)) return false;
  if (!learned) return true;
  const PoolSpace sp{&P};
  for (int layer = 0; layer < 3; ++layer) {
    sched_layer(sp, layer, pool_io(P, layer), gw, nw, nullptr);
    if (!grid_barrier(P.bar, bar_target, prm.limit_ns)) return false;
  }
  return true;
}

// Shared memory of one tile group.
union TileShared {  // size a multiple of 16: the members are aligned
  SweepShared sw;
  BfsShared bfs;
};
// wide visits and warp visits use the groups' memory together
static_assert(sizeof(WideShared) <= GROUPS * sizeof(TileShared) &&
              GROUPS * GROUP / 32 * WREL_SMEM * sizeof(unsigned short) <= GROUPS * sizeof(TileShared) &&
              sizeof(TileShared) % 16 == 0 && GROUPS * GROUP == WIDE, "shared memory of the solve's visits");

// Bookkeeping of a CTA that one thread updates: kept out of the registers,
// which the visits need.
struct SolveBook {
  unsigned long long tmark, t_launch, ns_bfs, ns_sweep, ns_reach, ns_sched;  // CTA 0
  int ntrace;                                                               // CTA 0
  unsigned visits_sw[GROUPS], pulses[GROUPS], visits_bfs[GROUPS], visits_chk[GROUPS];
  int next[2 * GROUPS];  // for_entries
};

// a list entry, loaded ahead of the test that may discard it
__device__ __forceinline__ int ld_ahead(const int32_t* p) {
  int v;
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// The whole solve in one cooperative launch of one CTA per SM: its groups of
// 128 threads each visit a tile at a time, and a grid barrier has one arrival
// per SM.
__device__ __forceinline__ void solve_body(const DevPool& P, const SolveParams& prm, TileShared* groups) {
  __shared__ SolveBook book;
  const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const auto tg = TileGroup<GROUP>::of_thread();
  const int q = tg.q, grp = tid / GROUP;
  TileShared& S = groups[grp];
  // warps of the grid, for the passes that visit every tile with a warp
  const int gw = b * (int)(blockDim.x >> 5) + (tid >> 5), nw = G * (int)(blockDim.x >> 5);
  uint32_t bar_target = 0;
  auto sync = [&]() { return grid_barrier(P.bar, bar_target, prm.limit_ns); };
  if (tid < GROUPS) book.visits_sw[tid] = book.pulses[tid] = book.visits_bfs[tid] = book.visits_chk[tid] = 0;
  if (tid == 0) {
    book.tmark = book.t_launch = globaltimer_ns();
    book.ns_bfs = book.ns_sweep = book.ns_reach = book.ns_sched = 0;
    book.ntrace = 0;
  }
  auto list = [&](int k) { return P.lists + (int64_t)k * P.T; };  // 0..2: BFS rounds, 3..6: sweeps
  // Hands out the n entries of a round to the groups.  Group g of CTA b starts
  // with entry g * G + b, so the first G entries go to distinct SMs; later ones
  // come from the round's counter (C_TAKE0 + round % 3, the next round's slot
  // is cleared meanwhile) through an atomic issued when the current visit
  // starts and read when it ends, so visits of uneven cost spread over the
  // groups.  The barrier between visits also lets the next one reuse S.
  // t0: the group's first entry, if it has one.
  int round_no = 0;
  auto first_entry = [&](const int32_t* lst) {
    const int i = grp * G + b;
    return i < P.T ? ld_ahead(lst + i) : 0;
  };
  auto for_entries = [&](const int32_t* lst, int t0, int n, auto&& visit) {
    if (!CGC_IN_BOUNDS(P, n, P.T + 1)) n = P.T;  // a list holds at most T entries
    int32_t* take = P.cnt + C_TAKE0 + round_no % 3;
    if (b == 0 && tid == 0) P.cnt[C_TAKE0 + (round_no + 1) % 3] = 0;
    ++round_no;
    const int first = G * GROUPS;
    int i = grp * G + b, j = 2 * grp;
    while (i < n) {
      int nx = 0;
      if (q == 0 && n > first) nx = atomicAdd(take, 1);
      visit(t0);
      if (n <= first) break;
      if (q == 0) book.next[j] = first + nx;
      tg.sync();
      i = book.next[j];
      j ^= 1;
      if (i < n) t0 = __ldcg(lst + i);
    }
  };
  int32_t* const bc = P.cnt + C_BFS0;
  int32_t* const sc = P.cnt + C_SW0;
  uint32_t bfs_id = 1;
  int s = 0;        // sweep index; sweep s uses list 3 + (s & 3) and stamp id s + 1
  int sweeps = 0, rounds = 0, relabels = 0, traced = 0, spare = 0;
  // block 0 records one phase step (after the barrier that ended it)
  auto record = [&](unsigned long long kind, long long index, int tiles) {
    if (b == 0 && tid == 0 && P.trace && book.ntrace < TRACE_CAP) {
      const int i = book.ntrace++;
      P.trace[2 * i] = (kind << 56) | ((unsigned long long)(index & 0xffffffffll) << 24) | (unsigned)(tiles & 0xffffff);
      P.trace[2 * i + 1] = globaltimer_ns() - book.t_launch;
    }
  };
  auto lap = [&](unsigned long long& acc) {
    if (b == 0 && tid == 0) {
      const uint64_t now = globaltimer_ns();
      acc += now - book.tmark;
      book.tmark = now;
    }
  };
  // Tile rounds of one relabel pass: round 0 visits the entries of list0
  // (count *cnt0), round k > 0 the tiles round k - 1 queued in list k % 3
  // (bc[1], bc[2] zero on entry).  inval: invalidation visits, otherwise BFS
  // visits.  False when a grid barrier gave up.
  auto relabel_rounds = [&](const int32_t* list0, int32_t* cnt0, bool inval) -> bool {
    int k = 0;
    for (;;) {
      const int32_t* lst = k == 0 ? list0 : list(k % 3);
      const int t0 = first_entry(lst);
      const int n = ld_cnt(k == 0 ? cnt0 : bc + k % 3);
      if (n == 0) break;
      if (b == 0 && tid == 0) bc[(k + 2) % 3] = 0;
      // More tiles than groups: a warp per tile; else the groups' shorter steps
      // win (relabels of a 150x140x96 segmentation with a warp from more than 1,
      // 2, 3, 4 tiles per SM on: 4.19, 4.09, 4.03, 3.89 ms; of a batch of 160^3:
      // 1.69, 1.68, 1.67, 1.61.  Without warp visits the segmentation's solve
      // took 10.3 ms, with them 9.1).
      if (n > GROUPS * G) {
        const int nn = CGC_IN_BOUNDS(P, n, P.T + 1) ? n : P.T;
        int32_t* take = P.cnt + C_TAKE0 + round_no % 3;  // handed out as in for_entries
        if (b == 0 && tid == 0) P.cnt[C_TAKE0 + (round_no + 1) % 3] = 0;
        ++round_no;
        unsigned short* const g = reinterpret_cast<unsigned short*>(groups) + (tid >> 5) * WREL_SMEM;
        int32_t* const ln = list((k + 1) % 3);
        int32_t* const cn = bc + (k + 1) % 3;
        int visits = 0;
        for (int i = (tid >> 5) * G + b; i < nn;) {
          int nx = 0;
          if ((tid & 31) == 0) nx = atomicAdd(take, 1);
          const int t = __ldcg(lst + i);
          visits += inval ? relabel_tile_w<true>(P, t, g, bfs_id + k + 1, ln, cn, (uint32_t)(relabels + 1), list(3), P.cnt + C_INC)
                          : relabel_tile_w<false>(P, t, g, bfs_id + k + 1, ln, cn, 0u, nullptr, nullptr);
          i = nw + __shfl_sync(FULL, nx, 0);
        }
        if ((tid & 31) == 0) atomicAdd(inval ? &book.visits_chk[grp] : &book.visits_bfs[grp], (unsigned)visits);
      } else if (inval) {
        for_entries(lst, t0, n, [&](int t) {
          const int v = inval_tile(P, tg, t, S.bfs, bfs_id + k + 1, list((k + 1) % 3), bc + (k + 1) % 3,
                                   (uint32_t)(relabels + 1), list(3), P.cnt + C_INC);
          if (q == 0) book.visits_chk[grp] += v;
        });
      } else {
        for_entries(lst, t0, n, [&](int t) {
          const int v = bfs_tile(P, tg, t, S.bfs, bfs_id + k + 1, list((k + 1) % 3), bc + (k + 1) % 3);
          if (q == 0) book.visits_bfs[grp] += v;
        });
      }
      ++k;
      if (!sync()) return false;
      record(TR_BFS_ROUND, rounds + k, n);
    }
    bfs_id += k + 1;
    rounds += k;
    return true;
  };
  uint32_t c0 = 0;  // sweep stamps above c0 were written during the current cycle
  for (;;) {
    // ------------------------------------------------ exact global relabel
    // The first relabel of a solve is a full BFS from the sink; later ones
    // are incremental when the pool has the stamps for it.
    const bool inc = prm.incremental && relabels > 0 && P.stamp_inc != nullptr;
    if (b == 0 && tid == 0) {
      bc[0] = bc[1] = bc[2] = 0;
      sc[0] = sc[1] = sc[2] = sc[3] = 0;
      P.cnt[C_SINKT0] = P.cnt[C_SINKT0 + 1] = P.cnt[C_SINKT0 + 2] = 0;
      P.cnt[C_TAKE0] = P.cnt[C_TAKE0 + 1] = P.cnt[C_TAKE0 + 2] = 0;
      P.cnt[C_INC] = P.cnt[C_ACT] = 0;
    }
    round_no = 0;
    if (!sync()) return;
    if (!inc) {
      for (int t = gw; t < P.T; t += nw) bfs_init_tile_w(P, t, relabels == 0);  // a warp per tile
      if (!sync()) return;
      for (int t0 = b * blockDim.x; t0 < P.T; t0 += G * blockDim.x) bfs_queue_tile(P, t0 + tid, bfs_id, list(0), bc + 0);
      if (!sync()) return;
      if (!relabel_rounds(list(0), bc + 0, false)) return;
    } else {
      // invalidation from the tiles the last cycle queued, then BFS rounds
      // from the tiles with dropped voxels (listed in list 3, free until the
      // sweep lists are rebuilt below)
      for (int t0 = b * blockDim.x; t0 < P.T; t0 += G * blockDim.x)
        inval_queue_tile(P, t0 + tid, c0, prm.exclusive != 0, bfs_id, list(0), bc + 0);
      if (!sync()) return;
      if (!relabel_rounds(list(0), bc + 0, true)) return;
      if (b == 0 && tid == 0) bc[0] = bc[1] = bc[2] = 0;
      if (!sync()) return;
      if (!relabel_rounds(list(3), P.cnt + C_INC, false)) return;
    }
    ++relabels;
    lap(book.ns_bfs);
    // ------------------------------------------------ active tiles -> parity lists
    s += 2;  // fresh stamp ids for the lists built here
    c0 = (uint32_t)s;
    for (int t0 = b * blockDim.x + (tid & ~31); t0 < P.T; t0 += G * blockDim.x) {  // warp-aggregated appends
      const int t = t0 + (tid & 31);
      const bool a = t < P.T && __ldcg(P.act + t);
      const int par = a ? __ldcg(P.tpar + t) : 0;
      const unsigned acts = __ballot_sync(FULL, a);
      if ((tid & 31) == 0 && acts) atomicAdd(P.cnt + C_ACT, __popc(acts));
      if (prm.exclusive) {  // one list: the whole active set is queued for sweep s
        if (a) P.stamp_sw[(int64_t)(s & 1) * P.T + t] = (uint32_t)(s + 1);
        warp_append(P, a, t, list(3 + (s & 3)), sc + (s & 3));
      } else {              // one list per parity, for sweeps s and s + 1
        if (a) P.stamp_sw[t] = (uint32_t)(s + par + 1);
        warp_append(P, a && par == 0, t, list(3 + (s & 3)), sc + (s & 3));
        warp_append(P, a && par == 1, t, list(3 + ((s + 1) & 3)), sc + ((s + 1) & 3));
      }
    }
    if (!sync()) return;
    // From a counter of its own: the lists' counters grow as soon as the first
    // CTA sweeps, and a CTA that read them late would choose another cycle length
    // or scheduler stage than the others, and meet other grid barriers.
    const int nact = ld_cnt(P.cnt + C_ACT);
    record(TR_RELABEL_DONE, relabels, nact);
    if (b == 0 && tid == 0 && P.trace && book.ntrace < TRACE_CAP) {  // flow at this relabel (after the barrier)
      unsigned long long f = 0;
      for (int i = 0; i < P.ninst; ++i) f += __ldcg(P.flow + i);
      const int i = book.ntrace++;
      P.trace[2 * i] = ((unsigned long long)TR_FLOW << 56) | ((unsigned long long)relabels << 24);
      P.trace[2 * i + 1] = f;
    }
    if (nact == 0) break;
    // Sweep pairs of this cycle.  Where a sweep costs more than a relabel -- more
    // than 16 active tiles per SM -- a cycle ends after 4 pairs at the latest,
    // unless the caller asked for an exact number (then dense_K = K), since by then most tiles hold excess that a relabel finds cut off from the
    // sink: 405x377x362 8.9 -> 8.0 ms, 512x512x128 tubes 3.6 -> 3.3, 256^3 3.13
    // -> 3.05, segmentation of 150x140x96 9.1 -> 8.9 (K = 8).  2 pairs are better
    // on balls (7.6 ms) and worse on the segmentation (10.0 ms), whose relabels
    // take long; lower limits on the tiles cost small grids 10 %.
    const int K = nact > 16 * G ? prm.dense_K : prm.K;
    // The limit on sweeps is checked before a cycle, so full cycles run up to
    // 2 K - 1 sweeps past it; a solve with shorter ones may run as many.
    if (sweeps >= prm.max_sweeps + spare) {
      if (b == 0 && tid == 0) raise_error(P, CGC_ERR_NOT_CONVERGED);
      break;
    }
    if (K < prm.K) spare = 2 * prm.K - 1;
    // ------------------------------------------------ learned scheduler
    const int cycle = relabels - 1;
    const bool tracing = prm.trace_cycles > cycle;
    if (tracing) traced = cycle + 1;
    // Priorities (deferral) only pay off while active tiles outnumber what
    // runs at a time: with fewer, a sweep lasts one tile visit whatever the
    // order.  Budgets can still shorten that visit, so learned = 3 runs the
    // stage in every cycle, with each tile's budget capped at the schedule's L
    // (a budget may only end a visit early).
    const bool throughput = nact > 2 * G * GROUPS;
    const bool learned = prm.learned && (throughput || prm.learned == 3);
    if (learned || tracing) {
      if (!sched_stage(P, prm, cycle, learned, tracing, list(3 + (s & 3)), ld_cnt(sc + (s & 3)), list(3 + ((s + 1) & 3)),
                       prm.exclusive ? 0 : ld_cnt(sc + ((s + 1) & 3)), bar_target))
        return;
      lap(book.ns_sched);
    }
    // ------------------------------------------------ sweeps
    int idle = 0;  // consecutive sweeps in which no tile delivered flow to the sink
    for (int j = 0; j < 2 * K; ++j, ++s) {
      const int32_t* const lst = list(3 + (s & 3));
      const int t0 = first_entry(lst), tw = b < P.T ? ld_ahead(lst + b) : 0;
      const int n = ld_cnt(sc + (s & 3));
      if (n == 0 && (prm.exclusive || ld_cnt(sc + ((s + 1) & 3)) == 0)) break;
      if (b == 0 && tid == 0) {
        sc[(s + 3) & 3] = 0;
        P.cnt[C_SINKT0 + (s + 1) % 3] = 0;
      }
      // Parity sweeps: sweep s uses stamp id s + 1; a visited tile queues the
      // tiles it pushed into for sweep s + 1 and itself, of the same parity,
      // for sweep s + 2.  Exclusive sweeps: every queued tile runs unless it
      // has the other parity than s and a face neighbour is queued for sweep
      // s, so the tiles that run form an independent set (no two share a
      // face) and the halo heights and cross-face pushes are exact as under
      // the parity schedule; everything is queued for sweep s + 1, with the
      // stamps in half (s+1)&1 of stamp_sw, so half s&1 -- this sweep's list --
      // does not change during the sweep.
      auto sweep_visit = [&](const auto vg, auto& sh, int t) {
        uint32_t* const stamp_q = prm.exclusive ? P.stamp_sw + (int64_t)((s + 1) & 1) * P.T : P.stamp_sw;
        const int sn = s + 1, ss = prm.exclusive ? s + 1 : s + 2;  // the sweeps the neighbours and the tile queue for
        // the learned scheduler defers low-priority tiles during the first half
        // of the cycle; every active tile is swept in the second half
        if (learned && throughput && prm.learned != 2 && j < K && !__ldcg(P.sprio + t)) {
          if (vg.q == 0) queue_tile(P, stamp_q, t, (uint32_t)(ss + 1), list(3 + (ss & 3)), sc + (ss & 3));
          return;
        }
        if (prm.exclusive && (int)__ldcg(P.tpar + t) != (s & 1)) {  // uniform over the group
          bool queued_nb = false;
          if (vg.q < 6) {
            const int nb = __ldcg(P.nbr + vg.q * P.T + t);
            queued_nb = nb >= 0 && __ldcg(P.stamp_sw + (int64_t)(s & 1) * P.T + nb) == (uint32_t)(s + 1);
          }
          if (vg.any(queued_nb)) {  // wait one sweep
            if (vg.q == 0) queue_tile(P, stamp_q, t, (uint32_t)(sn + 1), list(3 + (sn & 3)), sc + (sn & 3));
            return;
          }
        }
        const int L = !learned ? prm.L
                      : prm.learned == 3 ? min((int)__ldcg(P.sbudget + t), prm.L) : (int)__ldcg(P.sbudget + t);
        SweepExtra ex;
        if (prm.stall > 0) ex.sink_tiles = P.cnt + C_SINKT0 + s % 3;
        if (tracing) {
          ex.tr_pulses = P.tpulses + (int64_t)cycle * P.T;
          ex.tr_sink = P.tsink + (int64_t)cycle * P.T;
        }
        int np;
        if constexpr (decltype(vg)::width == WIDE)
          np = sweep_tile_wide<true>(P, vg, t, L, prm.R, j == 0, sh, (uint32_t)(sn + 1), list(3 + (sn & 3)), sc + (sn & 3),
                                     (uint32_t)(ss + 1), list(3 + (ss & 3)), sc + (ss & 3), ex, stamp_q);
        else
          np = sweep_tile(P, vg, t, L, prm.R, j == 0, sh, (uint32_t)(sn + 1), list(3 + (sn & 3)), sc + (sn & 3),
                                (uint32_t)(ss + 1), list(3 + (ss & 3)), sc + (ss & 3), ex, stamp_q);
        if (vg.q == 0) {
          ++book.visits_sw[grp];
          book.pulses[grp] += (unsigned)np;
        }
      };
      // At most one tile per SM: 512 threads per visit, which shortens a visit's
      // own chain (kernel times with groups alone and so: 128^3 1.03 and 0.94 ms,
      // 640x480 0.47 and 0.44, segmentation 8.45 and 8.34; the 160^3 batch 5.64
      // and 5.86).  With two tiles per SM, one after the other, it gains nothing
      // over two groups side by side (128^3 0.97, 256^3 2.94 -> 3.07, batch 6.16).
      if (n <= G) {
        const auto wide = TileGroup<WIDE>::of_thread();
        if (tid < WIDE && b < n) sweep_visit(wide, *reinterpret_cast<WideShared*>(groups), tw);
      } else {
        for_entries(lst, t0, n, [&](int t) { sweep_visit(tg, S.sw, t); });
      }
      ++sweeps;
      if (!sync()) return;
      record(TR_SWEEP, sweeps, n);
      // Early relabel: after stall consecutive non-empty sweeps of each parity
      // delivered no flow to the sink.  Empty sweeps do not count, so every
      // cycle performs at least one push or relabel; labels never decrease
      // (an exact relabel only raises valid labels), so the solve still ends.
      if (prm.stall > 0 && n > 0) idle = ld_cnt(P.cnt + C_SINKT0 + s % 3) ? 0 : idle + 1;
      if (prm.stall > 0 && idle >= 2 * prm.stall) { ++s; break; }
    }
    lap(book.ns_sweep);
  }
  lap(book.ns_bfs);
  // ------------------------------------------------ source-side reachability
  if (b == 0 && tid == 0) bc[0] = bc[1] = bc[2] = 0;
  if (!sync()) return;
  for (int t = gw; t < P.T; t += nw) reach_init_tile_w(P, t, bfs_id, list(0), bc + 0);
  if (!sync()) return;
  for (int k = 0;;) {
    const int n = ld_cnt(bc + k % 3);
    if (n == 0) break;
    if (b == 0 && tid == 0) bc[(k + 2) % 3] = 0;
    for (int i = (tid >> 5) * G + b; i < n; i += nw)  // a warp per tile
      reach_tile_w(P, __ldcg(list(k % 3) + i), bfs_id + k + 1, list((k + 1) % 3), bc + (k + 1) % 3);
    ++k;
    if (!sync()) return;
    record(TR_REACH_ROUND, k, n);
  }
  if (q == 0) {
    atomicAdd(P.stats + S_TILES_SWEPT, (unsigned long long)book.visits_sw[grp]);
    atomicAdd(P.stats + S_PULSES, (unsigned long long)book.pulses[grp]);
    atomicAdd(P.stats + S_TILES_BFS, (unsigned long long)book.visits_bfs[grp]);
    atomicAdd(P.stats + S_TILES_CHECK, (unsigned long long)book.visits_chk[grp]);
  }
  if (b == 0 && tid == 0) {
    lap(book.ns_reach);
    P.stats[S_SWEEPS] = (unsigned long long)sweeps;
    P.stats[S_RELABELS] = (unsigned long long)relabels;
    P.stats[S_ROUNDS] = (unsigned long long)rounds;
    P.stats[S_NS_BFS] = book.ns_bfs;
    P.stats[S_NS_SWEEP] = book.ns_sweep;
    P.stats[S_NS_REACH] = book.ns_reach;
    P.stats[S_TRACE_N] = (unsigned long long)book.ntrace;
    P.stats[S_TRACE_CYC] = (unsigned long long)traced;
    P.stats[S_NS_SCHED] = book.ns_sched;
  }
}

// Cooperative launches of this library on one device run one after another.
// Each waits on the device (an event, no host synchronisation) for the
// previous one to end: two grid-barrier kernels in flight on different
// streams could each hold part of the SMs and wait for their missing CTAs,
// until their bounded barriers gave up.  Launches into a stream under capture
// are not ordered (a CUDA graph is replayed on its own).
static std::mutex g_coop_mu;
static cudaEvent_t g_coop_last[64] = {};

int coop_launch_ordered(int device, cudaStream_t stream, const std::function<int()>& launch) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CGC_CUDA(cudaStreamIsCapturing(stream, &cs));
  if (cs != cudaStreamCaptureStatusNone || device < 0 || device >= 64) return launch();
  std::lock_guard<std::mutex> lock(g_coop_mu);
  cudaEvent_t& last = g_coop_last[device];
  if (!last) CGC_CUDA(cudaEventCreateWithFlags(&last, cudaEventDisableTiming));
  CGC_CUDA(cudaStreamWaitEvent(stream, last, 0));  // a no-op before the first record
  if (int rc = launch()) return rc;
  CGC_CUDA(cudaEventRecord(last, stream));
  return CGC_OK;
}

// One CTA of GROUPS tile groups per SM, 128 registers per thread.  Five groups
// (96 registers) and eight (64) spill in the sweep: 256^3 balls 3.9 -> 4.2 and
// 4.8 ms, 48-instance batch 5.9 -> 6.4 and 7.2 ms; only the tubes, all short
// visits, gain 3 % (5.06 -> 4.90 ms at L = 4, R = 2).
extern __shared__ __align__(16) unsigned char solve_smem[];
__global__ void __launch_bounds__(GROUPS * GROUP, 1) k_solve(DevPool P, SolveParams prm) {
  solve_body(P, prm, reinterpret_cast<TileShared*>(solve_smem));
}

int launch_solve(const DevPool& d, const SolveParams& prm, int device, int sms, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.stream = stream;
  cfg.gridDim = dim3(sms);
  cfg.blockDim = dim3(GROUPS * GROUP);
  cfg.dynamicSmemBytes = GROUPS * sizeof(TileShared);
  // a property of the function on the current device, set before its first launch there
  static std::atomic<bool> done[64] = {};
  if (device < 0 || device >= 64 || !done[device].load(std::memory_order_acquire)) {
    CGC_CUDA(cudaFuncSetAttribute(k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes));
    if (device >= 0 && device < 64) done[device].store(true, std::memory_order_release);
  }
  int rc = coop_launch_ordered(device, stream, [&]() -> int {
    CGC_CUDA(cudaLaunchKernelEx(&cfg, k_solve, d, prm));
    return CGC_OK;
  });
  if (rc) return rc;
  note_launch();
  return ok();
}

// One cut set of an instance after a device-resident solve, any mask and
// background (linear layout).
__global__ void __launch_bounds__(256) k_segments_lin(DevPool P, int inst, int which, uint8_t* out, uint8_t mask,
                                                      uint8_t bg) {
  const InstGeo G = P.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  for (int64_t v0 = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); v0 < N;
       v0 += 4 * (int64_t)gridDim.x * blockDim.x) {
    unsigned bits = 0;
    if (which == CGC_SEG_SINK_REACH) seg_gather4(P, G, v0, N, &bits, nullptr);
    else seg_gather4(P, G, v0, N, nullptr, &bits);
    seg_store4(out, v0, N, bits, mask, bg);
  }
}

__global__ void k_unpermute(DevPool P, int inst, const int32_t* plane, int32_t* out) {
  const InstGeo G = P.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < N; v += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(v % G.X), y = (int)((v / G.X) % G.Y), z = (int)(v / ((int64_t)G.X * G.Y));
    const int64_t t = G.tile_base + (x >> 3) + G.TX * ((y >> 3) + G.TY * (z >> 3));
    out[v] = plane[t * TV + (x & 7) + 8 * (y & 7) + 64 * (z & 7)];
  }
}

// ===========================================================================
// host side
// ===========================================================================

static std::mutex g_mem_mu;
static cudaMemPool_t g_mem_pool[64] = {};
static cudaStream_t g_mem_stream[64] = {};
static bool g_mem_tried[64] = {};

int dev_alloc(int device, void** p, size_t bytes) {
  constexpr size_t kLargest = (size_t)128 << 20;
  constexpr unsigned long long kKept = 256ull << 20;
  if (bytes <= kLargest && device >= 0 && device < 64) {
    std::lock_guard<std::mutex> lock(g_mem_mu);
    if (!g_mem_tried[device]) {
      g_mem_tried[device] = true;
      int has = 0;
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      unsigned long long kept = kKept;
      if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, device) == cudaSuccess && has &&
          cudaMemPoolCreate(&g_mem_pool[device], &props) == cudaSuccess) {
        if (cudaMemPoolSetAttribute(g_mem_pool[device], cudaMemPoolAttrReleaseThreshold, &kept) != cudaSuccess ||
            cudaStreamCreateWithFlags(&g_mem_stream[device], cudaStreamNonBlocking) != cudaSuccess) {
          cudaMemPoolDestroy(g_mem_pool[device]);
          g_mem_pool[device] = nullptr;
        }
      }
      cudaGetLastError();
    }
    if (g_mem_pool[device]) {
      // allocated on a stream of its own and waited for, so any stream may use it
      if (cudaMallocFromPoolAsync(p, bytes, g_mem_pool[device], g_mem_stream[device]) == cudaSuccess) {
        CGC_CUDA(cudaStreamSynchronize(g_mem_stream[device]));
        return CGC_OK;
      }
      cudaGetLastError();
    }
  }
  CGC_CUDA(cudaMalloc(p, bytes));
  return CGC_OK;
}

bool wait_for_device(int device) {
  int cur = 0;
  const bool other = cudaGetDevice(&cur) == cudaSuccess && cur != device && cudaSetDevice(device) == cudaSuccess;
  void* q = nullptr;
  const bool done = cudaMalloc(&q, 1) == cudaSuccess && cudaFree(q) == cudaSuccess;
  if (other) cudaSetDevice(cur);
  cudaGetLastError();
  return done;
}

bool Pool::idle() {
  bool told = !untracked;
  for (cudaEvent_t e : {used, ev[1]})  // no wait for one that was never recorded
    if (e && cudaEventSynchronize(e) != cudaSuccess) {
      cudaGetLastError();
      told = false;
    }
  return told || wait_for_device(device);
}

void Pool::note_use() {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (!used || cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone ||
      cudaEventRecord(used, stream) != cudaSuccess) {
    cudaGetLastError();
    untracked = true;
  }
}

static std::mutex g_pin_mu;
static char* g_pin = nullptr;
static uint64_t g_pin_used = 0;
constexpr size_t kPinSlot = 1024, kPinSlots = 64;

void* pinned_take(size_t bytes) {
  void* p = nullptr;
  if (bytes <= kPinSlot) {
    std::lock_guard<std::mutex> lock(g_pin_mu);
    if (!g_pin && cudaMallocHost(&p, kPinSlot * kPinSlots) == cudaSuccess) g_pin = (char*)p;
    if (g_pin && ~g_pin_used) {
      const int i = __builtin_ctzll(~g_pin_used);
      g_pin_used |= 1ull << i;
      return g_pin + i * kPinSlot;
    }
  }
  return cudaMallocHost(&p, bytes) == cudaSuccess ? p : nullptr;
}

void pinned_give(void* p) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lock(g_pin_mu);
    const char* c = (const char*)p;
    if (g_pin && c >= g_pin && c < g_pin + kPinSlot * kPinSlots) {
      g_pin_used &= ~(1ull << ((c - g_pin) / kPinSlot));
      return;
    }
  }
  cudaFreeHost(p);
}

static int device_error(int err, long long bound_at, const char* where) {
  if (err == 0) return CGC_OK;
#ifdef CGC_BOUNDS_CHECK
  if (err == CGC_ERR_ARG)
    return fail(err, std::string(where) + ": index out of range (bounds-checked build): " + std::to_string(bound_at) +
                         ", or a negative capacity");
#endif
  (void)bound_at;
  const char* what = err == CGC_ERR_OVERFLOW ? "capacities may overflow int32 excess/residuals (or a capacity points outside the grid)"
                   : err == CGC_ERR_ARG ? "negative capacity"
                   : err == CGC_ERR_TIMEOUT ? "a device-side wait timed out"
                   : err == CGC_ERR_NOT_CONVERGED ? "max_sweeps reached before convergence"
                   : "device error";
  return fail(err, std::string(where) + ": " + what);
}

int queue_back(Pool& p, cudaStream_t stream) {
  CGC_CUDA(cudaMemcpyAsync(p.pinned_cnt + 64, p.back_dev, p.back_bytes, cudaMemcpyDeviceToHost, stream));
  return CGC_OK;
}

int check_device_error(Pool& p, const char* where) {
  if (int rc = queue_back(p, p.stream)) return rc;
  CGC_CUDA(cudaStreamSynchronize(p.stream));
  return device_error((int)(p.back()[S_NSTATS] >> 32), (long long)p.back()[S_BOUND_AT], where);
}

int read_back(Pool& p, const char* where) {
  const unsigned long long* stats = p.back();
  if (int rc = device_error((int)(stats[S_NSTATS] >> 32), (long long)stats[S_BOUND_AT], where)) return rc;
  std::memcpy(p.flows.data(), stats + S_NSTATS + 1, (size_t)p.ninst * 8);
  std::memset(&p.st, 0, sizeof(p.st));
  for (int64_t f : p.flows) p.st.flow += f;
  p.st.sweeps = (int64_t)stats[S_SWEEPS];
  p.st.global_relabels = (int64_t)stats[S_RELABELS];
  p.st.bfs_rounds = (int64_t)stats[S_ROUNDS];
  p.st.tiles_swept = (int64_t)stats[S_TILES_SWEPT];
  p.st.tiles_relabelled = (int64_t)stats[S_TILES_BFS];
  p.st.tiles_checked = (int64_t)stats[S_TILES_CHECK];
  p.st.pulses = (int64_t)stats[S_PULSES];
  p.st.bfs_ms = 1e-6 * (double)stats[S_NS_BFS];
  p.st.sweep_ms = 1e-6 * (double)stats[S_NS_SWEEP];
  p.st.reach_ms = 1e-6 * (double)stats[S_NS_REACH];
  p.st.sched_ms = 1e-6 * (double)stats[S_NS_SCHED];
  return CGC_OK;
}

int pool_create(int32_t count, const int32_t* ext, void* stream, Pool** out) {
  if (!out || count <= 0 || !ext) return fail(CGC_ERR_ARG, "create: bad arguments");
  std::unique_ptr<Pool> p(new (std::nothrow) Pool());
  if (!p) return fail(CGC_ERR_OOM, "create: host allocation");
  CGC_CUDA(cudaGetDevice(&p->device));
  p->stream = (cudaStream_t)stream;
  p->ninst = count;
  int64_t T = 0;
  for (int i = 0; i < count; ++i) {
    const int32_t X = ext[3 * i], Y = ext[3 * i + 1], Z = ext[3 * i + 2];
    if (X <= 0 || Y <= 0 || Z <= 0) return fail(CGC_ERR_ARG, "create: extents must be positive");
    InstGeo G{};
    G.X = X; G.Y = Y; G.Z = Z;
    G.TX = (X + 7) / 8; G.TY = (Y + 7) / 8; G.TZ = (Z + 7) / 8;
    G.tile_base = (int32_t)T;
    const int64_t n = (int64_t)X * Y * Z;
    if (n + 1 >= (int64_t)INF) return fail(CGC_ERR_ARG, "create: instance too large for int32 heights");
    G.hdead = (int32_t)(n + 1);  // a distance to the sink is at most n (a path through every voxel)
    T += (int64_t)G.TX * G.TY * G.TZ;
    if (T > (int64_t)1 << 30) return fail(CGC_ERR_ARG, "create: too many tiles");
    p->maxN = std::max(p->maxN, n);
    p->geo.push_back(G);
  }
  p->T = (int32_t)T;
  p->Np = T * TV;
  p->uploaded.assign(count, 0u);
  p->flows.assign(count, 0);

  // one device allocation for all state (planes first, 256-byte aligned pieces)
  const int64_t Np = p->Np;
  auto al = [](int64_t b) { return (b + 255) & ~(int64_t)255; };
  int64_t off = 0;
  const int64_t o_e = off; off += al(Np * 4);
  const int64_t o_h = off; off += al(Np * 4);
  const int64_t o_rT = off; off += al(Np * 4);
  const int64_t o_r = off; off += al(6 * Np * 4);
  const int64_t o_rm = off; off += al(Np);
  const int64_t o_rc = off; off += al(Np);
  const int64_t o_nbr = off; off += al(6 * T * 4);
  const int64_t o_ti = off; off += al(T * 4);
  const int64_t o_tp = off; off += al(T);
  const int64_t o_run = off; off += al(T * 4);
  const int64_t o_act = off; off += al(T);
  const int64_t o_tf = off; off += al(T * 2);
  const int64_t o_sb = off; off += al(T * 4);
  const int64_t o_ss = off; off += al(2 * T * 4);
  const int64_t o_si = off; off += al(T * 4);
  const int64_t o_li = off; off += al(7 * T * 4);
  const int64_t o_cnt = off; off += al(C_NCOUNTERS * 4);
  const int64_t o_geo = off; off += al((int64_t)count * sizeof(InstGeo));
  // read back together: statistics, barrier count and error word, flows
  const int64_t o_st = off, o_bar = off + S_NSTATS * 8, o_fl = o_bar + 8;
  p->back_bytes = (size_t)(o_fl + (int64_t)count * 8 - o_st);
  off += al((int64_t)p->back_bytes);
  const int64_t o_tr = off; off += al(2 * TRACE_CAP * 8);
  if (int rc = dev_alloc(p->device, &p->dbuf, off)) return rc;
  p->untracked = true;  // until the wait below
  p->back_dev = (char*)p->dbuf + o_st;
  CGC_CUDA(cudaMemsetAsync(p->dbuf, 0, off, p->stream));
  char* base = (char*)p->dbuf;
  DevPool& d = p->dp;
  d.T = p->T; d.ninst = count; d.Np = Np;
  d.e = (int32_t*)(base + o_e); d.h = (int32_t*)(base + o_h); d.rT = (int32_t*)(base + o_rT);
  d.r = (int32_t*)(base + o_r); d.rmask = (uint8_t*)(base + o_rm); d.reach = (uint8_t*)(base + o_rc);
  d.nbr = (int32_t*)(base + o_nbr); d.tinst = (int32_t*)(base + o_ti); d.tpar = (uint8_t*)(base + o_tp);
  d.act = (uint8_t*)(base + o_act); d.tflag = (uint16_t*)(base + o_tf); d.stamp_bfs = (uint32_t*)(base + o_sb); d.stamp_sw = (uint32_t*)(base + o_ss);
  d.stamp_inc = (uint32_t*)(base + o_si);
  d.lists = (int32_t*)(base + o_li); d.cnt = (int32_t*)(base + o_cnt);
  d.flow = (unsigned long long*)(base + o_fl); d.geo = (InstGeo*)(base + o_geo);
  d.stats = (unsigned long long*)(base + o_st); d.bar = (uint32_t*)(base + o_bar); d.err = (int32_t*)(d.bar + 1);
  d.trace = (unsigned long long*)(base + o_tr);

  d.runs = (int32_t*)(base + o_run);

  // tile tables
  std::vector<int32_t> nbr(6 * (size_t)T, -1), ti((size_t)T), runs;
  std::vector<uint8_t> tp((size_t)T);
  for (int i = 0; i < count; ++i) {
    const InstGeo& G = p->geo[i];
    for (int tz = 0; tz < G.TZ; ++tz)
      for (int ty = 0; ty < G.TY; ++ty)
        for (int tx = 0; tx < G.TX; ++tx) {
          const int64_t t = G.tile_base + tx + (int64_t)G.TX * (ty + (int64_t)G.TY * tz);
          ti[t] = i;
          if (tx % 4 == 0) runs.push_back((int32_t)t);
          tp[t] = (uint8_t)((tx + ty + tz) & 1);
          auto id = [&](int a, int b2, int c) -> int32_t {
            if (a < 0 || b2 < 0 || c < 0 || a >= G.TX || b2 >= G.TY || c >= G.TZ) return -1;
            return (int32_t)(G.tile_base + a + (int64_t)G.TX * (b2 + (int64_t)G.TY * c));
          };
          nbr[PX * T + t] = id(tx + 1, ty, tz); nbr[MX * T + t] = id(tx - 1, ty, tz);
          nbr[PY * T + t] = id(tx, ty + 1, tz); nbr[MY * T + t] = id(tx, ty - 1, tz);
          nbr[PZ * T + t] = id(tx, ty, tz + 1); nbr[MZ * T + t] = id(tx, ty, tz - 1);
        }
  }
  CGC_CUDA(cudaMemcpyAsync((void*)d.nbr, nbr.data(), nbr.size() * 4, cudaMemcpyHostToDevice, p->stream));
  d.nruns = (int32_t)runs.size();
  CGC_CUDA(cudaMemcpyAsync((void*)d.runs, runs.data(), runs.size() * 4, cudaMemcpyHostToDevice, p->stream));
  CGC_CUDA(cudaMemcpyAsync((void*)d.tinst, ti.data(), ti.size() * 4, cudaMemcpyHostToDevice, p->stream));
  CGC_CUDA(cudaMemcpyAsync((void*)d.tpar, tp.data(), tp.size(), cudaMemcpyHostToDevice, p->stream));
  CGC_CUDA(cudaMemcpyAsync((void*)d.geo, p->geo.data(), p->geo.size() * sizeof(InstGeo), cudaMemcpyHostToDevice, p->stream));
  p->voff.resize(count);
  for (int i = 0; i < count; ++i) {  // offsets of multiples of 4: 16-byte aligned plane rows
    p->voff[i] = p->sumN;
    p->sumN += ((int64_t)p->geo[i].X * p->geo[i].Y * p->geo[i].Z + 3) & ~(int64_t)3;
  }
  p->host_in.assign(8 * (size_t)count, nullptr);
  p->pinned_cnt = (int32_t*)pinned_take(64 * 4 + p->back_bytes);
  if (!p->pinned_cnt) return fail(CGC_ERR_OOM, "create: pinned host memory");
  for (cudaEvent_t* e : {&p->inputs_read, &p->used}) CGC_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  for (auto& e : p->ev) CGC_CUDA(cudaEventCreate(&e));

  CGC_CUDA(cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, p->device));
  int occ2 = 0;
  CGC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, k_sweep_list, WIDE, 0));
  p->sweep_blocks = std::max(1, occ2) * p->sms;
  CGC_CUDA(cudaStreamSynchronize(p->stream));
  p->untracked = false;
  *out = p.release();
  return ok();
}

// Inputs of the set_* calls go into linear device planes (one copy per
// plane, no kernel); the fused upload kernel of the next solve reads them.
// Host uploads run on a copy stream of their own, after the upload kernel of
// the last enqueued solve has read the planes (event inputs_read), and the
// setter returns once the host array has been read: the reference's setters
// copy at call time too (graph_cut.hpp:284-285, 298-299).  Device-pointer
// setters copy device to device on the solve stream.
// The same allocation holds the cut sets of the solve that will read them and
// the device table of their addresses.
static int ensure_lin(Pool& p, bool bwd, bool host) {
  if (!p.lin) {
    const size_t in = 5 * (size_t)p.sumN * 4, seg = (2 * (size_t)p.sumN + 255) & ~(size_t)255;
    const size_t tab = 2 * (size_t)p.ninst * sizeof(uint8_t*);
    if (int rc = dev_alloc(p.device, &p.lin, ((in + 255) & ~(size_t)255) + seg + tab)) return rc;
    p.segbuf = (uint8_t*)p.lin + ((in + 255) & ~(size_t)255);
    p.d_segtab = (uint8_t**)(p.segbuf + seg);
    std::vector<uint8_t*> addr(2 * (size_t)p.ninst);
    for (int i = 0; i < p.ninst; ++i) {
      addr[2 * i] = p.segbuf + p.voff[i];               // source side
      addr[2 * i + 1] = p.segbuf + p.sumN + p.voff[i];  // sink side
    }
    // pageable source: staged before the call returns
    CGC_CUDA(cudaMemcpyAsync(p.d_segtab, addr.data(), tab, cudaMemcpyHostToDevice, p.stream));
  }
  if (bwd && !p.lin_bwd)
    if (int rc = dev_alloc(p.device, &p.lin_bwd, 3 * (size_t)p.sumN * 4)) return rc;
  if (host && !p.copy_stream) CGC_CUDA(cudaStreamCreateWithFlags(&p.copy_stream, cudaStreamNonBlocking));
  return CGC_OK;
}

static int copy_plane(Pool& p, int32_t* dst, const int32_t* src, int64_t N, bool host) {
  if (host) {
    CGC_CUDA(cudaStreamWaitEvent(p.copy_stream, p.inputs_read, 0));  // no-op before the first record
    CGC_CUDA(cudaMemcpyAsync(dst, src, N * 4, cudaMemcpyHostToDevice, p.copy_stream));
  } else {
    CGC_CUDA(cudaMemcpyAsync(dst, src, N * 4, cudaMemcpyDeviceToDevice, p.stream));
  }
  return CGC_OK;
}

// Whether a kernel on `device` may read `bytes` at p where a copy command would:
// ordinary memory of that device, aligned, and all of it inside one allocation.
// Copy commands also take other devices' memory, managed and pinned memory and
// any alignment, and they answer an invalid range with an error.
static bool kernel_may_read(const void* p, size_t bytes, int device) {
  using Query = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Query query = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    const bool ok = cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &found) == cudaSuccess &&
                    found == cudaDriverEntryPointSuccess;
    if (!ok) cudaGetLastError();
    return ok ? reinterpret_cast<Query>(f) : nullptr;
  }();
  if (!query || (reinterpret_cast<uintptr_t>(p) & 3)) return false;
  CUmemorytype type = (CUmemorytype)0;
  unsigned managed = 1;
  int ordinal = -1;
  CUdeviceptr start = 0;
  size_t size = 0;
  CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* to[] = {&type, &managed, &ordinal, &start, &size};
  const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(p);
  return query(5, what, to, at) == CUDA_SUCCESS && type == CU_MEMORYTYPE_DEVICE && !managed && ordinal == device &&
         start != 0 && at - start <= size && size - (at - start) >= bytes;
}

// Two planes device to device on the solve stream, by one kernel where it may
// read them and they are small: the eight planes of directed n-links take 25 us
// at 64^3 by kernels and 47 by copy commands (whole solve of 24x20x12: 287 and
// 309 us).  At 128^3 (33 and 50 us) that is 2 % of the solve and at 200^3 (93 and
// 133) less, so above 2^18 voxels the copy commands, which take any memory, stay.
static int copy_two(Pool& p, int32_t* d0, const int32_t* s0, int32_t* d1, const int32_t* s1, int64_t N, bool host) {
  if (!host && N <= (1 << 18) && kernel_may_read(s0, (size_t)N * 4, p.device) && kernel_may_read(s1, (size_t)N * 4, p.device)) {
    k_copy_two<<<(unsigned)((N + 1023) / 1024), 256, 0, p.stream>>>(d0, s0, d1, s1, N);
    note_launch();
    CGC_CUDA(cudaGetLastError());
    return CGC_OK;
  }
  if (int rc = copy_plane(p, d0, s0, N, host)) return rc;
  return copy_plane(p, d1, s1, N, host);
}

int pool_put_tlinks(Pool& p, int inst, const int32_t* capS, const int32_t* capT, bool host) {
  if (inst < 0 || inst >= p.ninst || !capS || !capT) return fail(CGC_ERR_ARG, "set_tlinks: bad arguments");
  const InstGeo& G = p.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  NoteUse note(p);
  note.waited = host && p.lin;  // host planes are waited for, the table that comes with `lin` is not
  if (int rc = ensure_lin(p, false, host)) return rc;
  int32_t* s = p.lin + p.voff[inst];
  int32_t* c = p.lin + p.sumN + p.voff[inst];
  if (int rc = copy_two(p, s, capS, c, capT, N, host)) return rc;
  if (host) CGC_CUDA(cudaStreamSynchronize(p.copy_stream));
  p.host_in[8 * (size_t)inst] = s;
  p.host_in[8 * (size_t)inst + 1] = c;
  p.uploaded[inst] |= 1u;
  p.solved = false;
  p.seg_valid = false;
  return ok();
}

int pool_put_nlinks(Pool& p, int inst, int axis, const int32_t* fwd, const int32_t* bwd, bool host) {
  if (inst < 0 || inst >= p.ninst || axis < 0 || axis > 2 || !fwd || !bwd)
    return fail(CGC_ERR_ARG, "set_nlinks: bad arguments");
  const InstGeo& G = p.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  const bool same = bwd == fwd;  // symmetric weights: one plane
  NoteUse note(p);
  note.waited = host && p.lin;
  if (int rc = ensure_lin(p, !same, host)) return rc;
  int32_t* f = p.lin + (2 + axis) * p.sumN + p.voff[inst];
  int32_t* b = same ? f : p.lin_bwd + axis * p.sumN + p.voff[inst];
  if (int rc = same ? copy_plane(p, f, fwd, N, host) : copy_two(p, f, fwd, b, bwd, N, host)) return rc;
  if (host) CGC_CUDA(cudaStreamSynchronize(p.copy_stream));
  p.host_in[8 * (size_t)inst + 2 + axis] = f;
  p.host_in[8 * (size_t)inst + 5 + axis] = b;
  p.uploaded[inst] |= 2u << axis;
  p.solved = false;
  p.seg_valid = false;
  return ok();
}

cgc_options resolve_options(const cgc_options* o) {
  cgc_options r{};
  r.struct_size = sizeof(cgc_options);
  r.local_pulses = 4;
  r.sweeps_per_relabel = 8;
  r.wait_limit_us = 20 * 1000 * 1000;
  r.max_sweeps = 1 << 17;
  r.persistent = 1;
  r.region_relabels = 2;
  r.stall_sweeps = 0;
  r.ctas_per_sm = 2;
  r.relabel = 2;
  if (o) {
    if (o->local_pulses > 0) r.local_pulses = std::min(o->local_pulses, 64);
    if (o->sweeps_per_relabel) r.sweeps_per_relabel = (int)std::min<int64_t>(std::abs((int64_t)o->sweeps_per_relabel), 1 << 24);
    if (o->wait_limit_us > 0) r.wait_limit_us = o->wait_limit_us;
    if (o->max_sweeps > 0) r.max_sweeps = o->max_sweeps;
    if (o->persistent) r.persistent = o->persistent;
    if (o->region_relabels) r.region_relabels = o->region_relabels < 0 ? 0 : std::min(o->region_relabels, 16);
    if (o->stall_sweeps) r.stall_sweeps = o->stall_sweeps < 0 ? 0 : o->stall_sweeps;
    if (o->ctas_per_sm >= 2 && o->ctas_per_sm <= 4) r.ctas_per_sm = o->ctas_per_sm;
    r.bfs_warp_min = o->bfs_warp_min > 0 ? o->bfs_warp_min : 0;
    r.exclusive = o->exclusive > 0 ? 1 : 0;
    if (o->relabel == 1 || o->relabel == 2) r.relabel = o->relabel;
    r.learned = (o->learned == 2 || o->learned == 3) ? o->learned : (o->learned > 0 ? 1 : 0);
    r.trace_cycles = o->trace_cycles > 0 ? std::min(o->trace_cycles, 64) : 0;
  }
  return r;
}

uint64_t wait_limit_ns(const cgc_options& o) {
  return (uint64_t)(o.wait_limit_us > 0 ? o.wait_limit_us : 20 * 1000 * 1000) * 1000ull;
}

// Parameters of the persistent solve kernel from resolved options and the
// caller's (may be null).
SolveParams solve_params(const cgc_options& o, const cgc_options* given) {
  SolveParams prm;
  prm.L = o.local_pulses;
  prm.R = o.region_relabels;
  prm.K = o.sweeps_per_relabel;
  prm.dense_K = given && given->sweeps_per_relabel < 0 ? prm.K : std::min(prm.K, 4);
  prm.stall = o.stall_sweeps;
  prm.learned = o.learned;
  prm.trace_cycles = o.trace_cycles > 0 ? o.trace_cycles : 0;
  prm.max_sweeps = (int64_t)o.max_sweeps;
  prm.limit_ns = wait_limit_ns(o);
  prm.exclusive = o.exclusive ? 1 : 0;
  prm.incremental = o.relabel == 2 ? 1 : 0;
  return prm;
}

// host-driven BFS (or reachability) pass; returns rounds executed
template <bool REACH>
static int host_bfs(Pool& p, uint32_t& id, int64_t& rounds) {
  DevPool& d = p.dp;
  int32_t* bl[3] = {d.lists, d.lists + d.T, d.lists + 2 * d.T};
  CGC_CUDA(cudaMemsetAsync(d.cnt + C_BFS0, 0, 3 * 4, p.stream));
  const int gi = std::min<int>(d.T, p.sms * 8);
  if (REACH) { k_reach_init<<<gi, 512, 0, p.stream>>>(d, id, bl[0], d.cnt + C_BFS0); note_launch(); }
  else {
    k_bfs_init<<<gi, 512, 0, p.stream>>>(d, rounds == 0); note_launch();
    k_bfs_queue<<<(d.T + 255) / 256, 256, 0, p.stream>>>(d, id, bl[0], d.cnt + C_BFS0); note_launch();
  }
  CGC_CUDA(cudaGetLastError());
  for (int k = 0;; ++k) {
    CGC_CUDA(cudaMemcpyAsync(p.pinned_cnt, d.cnt + C_BFS0 + k % 3, 4, cudaMemcpyDeviceToHost, p.stream));
    CGC_CUDA(cudaStreamSynchronize(p.stream));
    const int n = p.pinned_cnt[0];
    if (n == 0) { id += k + 1; break; }
    CGC_CUDA(cudaMemsetAsync(d.cnt + C_BFS0 + (k + 1) % 3, 0, 4, p.stream));
    const int gb = std::min(n, p.sweep_blocks);
    if (REACH) { k_reach_round<<<gb, GROUP, 0, p.stream>>>(d, bl[k % 3], d.cnt + C_BFS0 + k % 3, id + k + 1, bl[(k + 1) % 3], d.cnt + C_BFS0 + (k + 1) % 3); note_launch(); }
    else { k_bfs_round<<<gb, GROUP, 0, p.stream>>>(d, bl[k % 3], d.cnt + C_BFS0 + k % 3, id + k + 1, bl[(k + 1) % 3], d.cnt + C_BFS0 + (k + 1) % 3); note_launch(); }
    CGC_CUDA(cudaGetLastError());
    ++rounds;
  }
  return CGC_OK;
}

// Enqueues one solve of the set_* inputs on p.stream: fused upload and
// preflow, the solve, and both cut sets of every instance into segbuf.  With
// the persistent solve (the default) nothing synchronises the host, so the
// next grid's host uploads can run while this one solves; the host-driven
// schedule (persistent = -1) runs its loop here.
int pool_solve_async(Pool& p, const cgc_options* opts) {
  if (p.pending) return fail(CGC_ERR_STATE, "maxflow: the previous solve of this handle was not waited for");
  const cgc_options o = resolve_options(opts);
  DevPool& d = p.dp;
  for (int i = 0; i < p.ninst; ++i)
    if (!(p.uploaded[i] & 1u)) return fail(CGC_ERR_STATE, "maxflow: set_tlinks was not called since the last solve");
  // axes not set since the last solve have zero capacity
  std::vector<const int32_t*> in = p.host_in;
  for (int i = 0; i < p.ninst; ++i)
    for (int a = 0; a < 3; ++a)
      if (!(p.uploaded[i] & (2u << a))) in[8 * (size_t)i + 2 + a] = in[8 * (size_t)i + 5 + a] = nullptr;
  const SolveParams prm = solve_params(o, opts);
  NoteUse note(p);
  if (o.persistent > 0 && (prm.learned || prm.trace_cycles))  // buffers and weights before anything is queued
    if (int rc = ensure_sched(p, prm.learned != 0, prm.trace_cycles)) return rc;
  if (p.ninst > 1) {
    if (!p.d_host_in)
      if (int rc = dev_alloc(p.device, &p.d_host_in, 8 * (size_t)p.ninst * sizeof(int32_t*))) return rc;
    // pageable source: the table is staged before the call returns
    CGC_CUDA(cudaMemcpyAsync(p.d_host_in, in.data(), in.size() * sizeof(int32_t*), cudaMemcpyHostToDevice, p.stream));
  }
  p.launches0 = g_launches.load();
  CGC_CUDA(cudaEventRecord(p.ev[0], p.stream));
  CGC_CUDA(cudaMemsetAsync(p.back_dev, 0, p.back_bytes, p.stream));  // statistics, barrier, error word, flows
  if (p.ninst == 1) {
    InputPlanes ip;
    for (int k = 0; k < 8; ++k) ip.p[k] = in[k];
    k_put_one<<<d.nruns, 128, 0, p.stream>>>(d, ip, true);
  } else {
    k_put_all<<<d.nruns, 128, 0, p.stream>>>(d, p.d_host_in);
  }
  note_launch();
  CGC_CUDA(cudaGetLastError());
  CGC_CUDA(cudaEventRecord(p.inputs_read, p.stream));  // the setters may overwrite the planes from here on
  // the inputs are consumed: another solve needs new set_* calls
  for (auto& u : p.uploaded) u = 0;
  p.solved = false;
  p.seg_valid = false;
  p.pending = true;
  p.pending_persistent = o.persistent;

  int rc = CGC_OK;
  if (o.persistent > 0) {
    CGC_CUDA(cudaEventRecord(p.ev[2], p.stream));
    rc = launch_solve(d, prm, p.device, p.sms, p.stream);
    CGC_CUDA(cudaEventRecord(p.ev[3], p.stream));
  } else {
    // the host loop reads counters back every round; a preparation error
    // (overflowing capacities) stops it before it starts
    rc = check_device_error(p, "maxflow");
    CGC_CUDA(cudaEventRecord(p.ev[2], p.stream));
    int64_t sweeps = 0, relabels = 0, rounds = 0;
    uint32_t id = 1;
    int32_t* sl = d.lists + 3 * d.T;
    while (!rc) {
      rc = host_bfs<false>(p, id, rounds);
      if (rc) break;
      ++relabels;
      CGC_CUDA(cudaMemsetAsync(d.cnt + C_SW0, 0, 8, p.stream));
      k_compact<<<(d.T + 255) / 256, 256, 0, p.stream>>>(d, 0, sl, d.cnt + C_SW0); note_launch();
      k_compact<<<(d.T + 255) / 256, 256, 0, p.stream>>>(d, 1, sl + d.T, d.cnt + C_SW0 + 1); note_launch();
      CGC_CUDA(cudaMemcpyAsync(p.pinned_cnt, d.cnt + C_SW0, 8, cudaMemcpyDeviceToHost, p.stream));
      CGC_CUDA(cudaStreamSynchronize(p.stream));
      if (p.pinned_cnt[0] + p.pinned_cnt[1] == 0) break;
      if (sweeps >= o.max_sweeps) { rc = fail(CGC_ERR_NOT_CONVERGED, "maxflow: max_sweeps reached"); break; }
      for (int j = 0; j < 2 * o.sweeps_per_relabel; ++j) {
        const int par = j & 1;
        if (j > 0) {
          CGC_CUDA(cudaMemsetAsync(d.cnt + C_SW0 + par, 0, 4, p.stream));
          k_compact<<<(d.T + 255) / 256, 256, 0, p.stream>>>(d, par, sl + par * d.T, d.cnt + C_SW0 + par); note_launch();
        }
        k_sweep_list<<<p.sweep_blocks, WIDE, 0, p.stream>>>(d, sl + par * d.T, d.cnt + C_SW0 + par, o.local_pulses, o.region_relabels); note_launch();
        CGC_CUDA(cudaGetLastError());
        ++sweeps;
      }
    }
    if (!rc) rc = host_bfs<true>(p, id, rounds);
    CGC_CUDA(cudaEventRecord(p.ev[3], p.stream));
    p.host_counts[0] = sweeps;
    p.host_counts[1] = relabels;
    p.host_counts[2] = rounds;
  }
  if (!rc) {
    const unsigned gx = (unsigned)std::min<int64_t>(std::max<int64_t>((p.maxN + 8191) / 8192, 1), 4096);
    k_seg_all<<<dim3(gx, (unsigned)std::min(p.ninst, 65535)), 256, 0, p.stream>>>(d, p.d_segtab);
    note_launch();
    CGC_CUDA(cudaGetLastError());
  }
  if (!rc) rc = queue_back(p, p.stream);
  CGC_CUDA(cudaEventRecord(p.ev[1], p.stream));
  if (rc) {
    // nothing to wait for: leave the stream idle and report now
    cudaStreamSynchronize(p.stream);
    p.pending = false;
    return rc;
  }
  note.waited = true;  // ev[1] marks the end
  return ok();
}

// Waits for the solve enqueued by pool_solve_async; reports device errors and
// reads the flows and statistics.
int pool_solve_wait(Pool& p) {
  if (!p.pending) return fail(CGC_ERR_STATE, "wait: no solve was enqueued");
  p.pending = false;
  CGC_CUDA(cudaEventSynchronize(p.ev[1]));
  if (int rc = read_back(p, "maxflow")) return rc;
  float ms = 0.f, kms = 0.f;
  cudaEventElapsedTime(&ms, p.ev[0], p.ev[1]);
  cudaEventElapsedTime(&kms, p.ev[2], p.ev[3]);
  if (p.pending_persistent <= 0) {
    p.st.sweeps = p.host_counts[0];
    p.st.global_relabels = p.host_counts[1];
    p.st.bfs_rounds = p.host_counts[2];
  }
  p.st.solve_ms = ms;
  p.st.kernel_ms = kms;
  p.st.launches = g_launches.load() - p.launches0;
  p.solved = true;
  p.seg_valid = true;
  return ok();
}

int pool_solve(Pool& p, const cgc_options* opts) {
  if (int rc = pool_solve_async(p, opts)) return rc;
  return pool_solve_wait(p);
}

int pool_segments(Pool& p, int inst, int which, uint8_t* out, uint8_t mask, uint8_t bg, bool host) {
  if (inst < 0 || inst >= p.ninst || !out || (which != CGC_SEG_SINK_REACH && which != CGC_SEG_SOURCE_MIN))
    return fail(CGC_ERR_ARG, "get_segments: bad arguments");
  if (p.pending) return fail(CGC_ERR_STATE, "get_segments: wait for the solve first");
  if (!p.solved) return fail(CGC_ERR_STATE, "get_segments: call maxflow first");
  const InstGeo& G = p.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  NoteUse note(p);
  if ((host || !p.seg_valid || mask != 1 || bg != 0) && !p.segtmp)
    if (int rc = dev_alloc(p.device, &p.segtmp, p.maxN)) return rc;
  const unsigned blocks = (unsigned)std::min<int64_t>(std::max<int64_t>((N + 4095) / 4096, 1), 8 * (int64_t)p.sms);
  const uint8_t* src = nullptr;  // device bytes to copy to `out` as they are
  if (p.seg_valid) {
    // the host-path solve wrote both sets as 1/0 bytes
    const uint8_t* set = p.segbuf + (which == CGC_SEG_SOURCE_MIN ? 0 : p.sumN) + p.voff[inst];
    if (mask == 1 && bg == 0) {
      src = set;
    } else {
      uint8_t* dst = host ? p.segtmp : out;
      k_mask_remap<<<blocks, 256, 0, p.stream>>>(set, dst, N, mask, bg); note_launch();
      src = host ? p.segtmp : nullptr;
    }
  } else {
    // after a device-resident solve: from the solver state
    uint8_t* dst = host ? p.segtmp : out;
    k_segments_lin<<<blocks, 256, 0, p.stream>>>(p.dp, inst, which, dst, mask, bg); note_launch();
    src = host ? p.segtmp : nullptr;
  }
  CGC_CUDA(cudaGetLastError());
  if (src) CGC_CUDA(cudaMemcpyAsync(out, src, N, host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, p.stream));
  CGC_CUDA(cudaStreamSynchronize(p.stream));
  note.waited = true;
  return ok();
}

int pool_residuals(Pool& p, int inst, int32_t* const res[6], int32_t* resT, int32_t* excess) {
  if (inst < 0 || inst >= p.ninst) return fail(CGC_ERR_ARG, "get_residuals: bad instance");
  if (p.pending) return fail(CGC_ERR_STATE, "get_residuals: wait for the solve first");
  if (!p.solved) return fail(CGC_ERR_STATE, "get_residuals: call maxflow first");
  const InstGeo& G = p.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  NoteUse note(p);
  if (!p.resid)
    if (int rc = dev_alloc(p.device, &p.resid, (size_t)p.maxN * 4)) return rc;
  const int blocks = (int)std::min<int64_t>((N + 255) / 256, 65535);
  auto one = [&](const int32_t* plane, int32_t* out) -> int {
    if (!out) return CGC_OK;
    k_unpermute<<<blocks, 256, 0, p.stream>>>(p.dp, inst, plane, p.resid); note_launch();
    CGC_CUDA(cudaGetLastError());
    CGC_CUDA(cudaMemcpyAsync(out, p.resid, N * 4, cudaMemcpyDeviceToHost, p.stream));
    CGC_CUDA(cudaStreamSynchronize(p.stream));
    return CGC_OK;
  };
  int rc;
  if (res)
    for (int d = 0; d < 6; ++d)
      if ((rc = one(p.dp.r + d * p.Np, res[d]))) return rc;
  if ((rc = one(p.dp.rT, resT))) return rc;
  if ((rc = one(p.dp.e, excess))) return rc;
  note.waited = true;
  return ok();
}

// Distance labels of the last solve in linear order (INT32_MIN where the
// sink cannot be reached).
int pool_labels(Pool& p, int inst, int32_t* labels) {
  if (inst < 0 || inst >= p.ninst || !labels) return fail(CGC_ERR_ARG, "get_labels: bad arguments");
  if (p.pending) return fail(CGC_ERR_STATE, "get_labels: wait for the solve first");
  if (!p.solved) return fail(CGC_ERR_STATE, "get_labels: call maxflow first");
  const InstGeo& G = p.geo[inst];
  const int64_t N = (int64_t)G.X * G.Y * G.Z;
  NoteUse note(p);
  if (!p.resid)
    if (int rc = dev_alloc(p.device, &p.resid, (size_t)p.maxN * 4)) return rc;
  k_unpermute<<<(int)std::min<int64_t>((N + 255) / 256, 65535), 256, 0, p.stream>>>(p.dp, inst, p.dp.h, p.resid);
  note_launch();
  CGC_CUDA(cudaGetLastError());
  CGC_CUDA(cudaMemcpyAsync(labels, p.resid, N * 4, cudaMemcpyDeviceToHost, p.stream));
  CGC_CUDA(cudaStreamSynchronize(p.stream));
  note.waited = true;
  for (int64_t v = 0; v < N; ++v)
    if (labels[v] >= INF) labels[v] = INT32_MIN;
  return ok();
}

int pool_trace(Pool& p, int64_t* out, int32_t cap, int32_t* count) {
  if (!p.solved) return fail(CGC_ERR_STATE, "trace: call maxflow first");
  unsigned long long n = 0;
  CGC_CUDA(cudaMemcpy(&n, p.dp.stats + S_TRACE_N, 8, cudaMemcpyDeviceToHost));
  *count = (int32_t)n;
  if (out && cap > 0) {
    const int64_t m = std::min<int64_t>((int64_t)n, cap);
    CGC_CUDA(cudaMemcpy(out, p.dp.trace, (size_t)m * 16, cudaMemcpyDeviceToHost));
  }
  return ok();
}

}  // namespace cgc

// ===========================================================================
// C ABI
// ===========================================================================
using cgc::Pool;

struct cgc_grid { Pool* p; };
struct cgc_batch { Pool* p; };

extern "C" {

const char* cgc_last_error(void) { return cgc::g_last_error.c_str(); }
const char* cgc_version(void) { return "cgc 0.1 (sm_100a)"; }
int64_t cgc_launch_count(void) { return (int64_t)cgc::g_launches.load(); }

int cgc_init(int device) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) return cgc::fail(CGC_ERR_NO_DEVICE, "cgc_init: no CUDA device");
  if (device < 0 || device >= n) return cgc::fail(CGC_ERR_ARG, "cgc_init: bad device index");
  CGC_CUDA(cudaSetDevice(device));
  CGC_CUDA(cudaFree(nullptr));
  return cgc::ok();
}

int cgc_grid_create(int32_t X, int32_t Y, int32_t Z, void* stream, cgc_grid** out) {
  if (!out) return cgc::fail(CGC_ERR_ARG, "cgc_grid_create: null output");
  int32_t ext[3] = {X, Y, Z};
  Pool* p = nullptr;
  int rc = cgc::pool_create(1, ext, stream, &p);
  if (rc) return rc;
  *out = new cgc_grid{p};
  return cgc::ok();
}
int cgc_grid_destroy(cgc_grid* g) {
  if (!g) return cgc::ok();
  delete g->p;
  delete g;
  return cgc::ok();
}
int cgc_grid_set_tlinks(cgc_grid* g, const int32_t* capS, const int32_t* capT) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_put_tlinks(*g->p, 0, capS, capT, true);
}
int cgc_grid_set_nlinks(cgc_grid* g, int axis, const int32_t* fwd, const int32_t* bwd) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_put_nlinks(*g->p, 0, axis, fwd, bwd, true);
}
int cgc_grid_set_tlinks_device(cgc_grid* g, const int32_t* capS, const int32_t* capT) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_put_tlinks(*g->p, 0, capS, capT, false);
}
int cgc_grid_set_nlinks_device(cgc_grid* g, int axis, const int32_t* fwd, const int32_t* bwd) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_put_nlinks(*g->p, 0, axis, fwd, bwd, false);
}
int cgc_grid_maxflow(cgc_grid* g, const cgc_options* opts, int64_t* flow) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  int rc = cgc::pool_solve(*g->p, opts);
  if (rc) return rc;
  if (flow) *flow = g->p->flows[0];
  return cgc::ok();
}
int cgc_grid_maxflow_async(cgc_grid* g, const cgc_options* opts) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_solve_async(*g->p, opts);
}
int cgc_grid_wait(cgc_grid* g, int64_t* flow) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  int rc = cgc::pool_solve_wait(*g->p);
  if (rc) return rc;
  if (flow) *flow = g->p->flows[0];
  return cgc::ok();
}
int cgc_grid_get_segments(cgc_grid* g, int which, uint8_t* out, uint8_t mask, uint8_t background) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_segments(*g->p, 0, which, out, mask, background, true);
}
int cgc_grid_get_segments_device(cgc_grid* g, int which, uint8_t* out, uint8_t mask, uint8_t background) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_segments(*g->p, 0, which, out, mask, background, false);
}
int cgc_grid_get_labels(cgc_grid* g, int32_t* labels) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_labels(*g->p, 0, labels);
}
int cgc_grid_get_residuals(cgc_grid* g, int32_t* const res[6], int32_t* resT, int32_t* excess) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "null grid");
  return cgc::pool_residuals(*g->p, 0, res, resT, excess);
}
int cgc_grid_trace(cgc_grid* g, int64_t* out, int32_t cap, int32_t* count) {
  if (!g || !count) return cgc::fail(CGC_ERR_ARG, "null argument");
  return cgc::pool_trace(*g->p, out, cap, count);
}
int cgc_batch_trace(cgc_batch* b, int64_t* out, int32_t cap, int32_t* count) {
  if (!b || !count) return cgc::fail(CGC_ERR_ARG, "null argument");
  return cgc::pool_trace(*b->p, out, cap, count);
}
int cgc_grid_sched_trace(cgc_grid* g, uint16_t* feat, uint8_t* pulses, uint8_t* sink, int32_t max_cycles,
                         int32_t* cycles) {
  if (!g || !cycles) return cgc::fail(CGC_ERR_ARG, "null argument");
  return cgc::pool_sched_trace(*g->p, feat, pulses, sink, max_cycles, cycles);
}
int cgc_grid_stats(cgc_grid* g, cgc_stats* out) {
  if (!g || !out) return cgc::fail(CGC_ERR_ARG, "null argument");
  *out = g->p->st;
  return cgc::ok();
}

int cgc_batch_create(int32_t count, const int32_t* extents, void* stream, cgc_batch** out) {
  if (!out) return cgc::fail(CGC_ERR_ARG, "cgc_batch_create: null output");
  Pool* p = nullptr;
  int rc = cgc::pool_create(count, extents, stream, &p);
  if (rc) return rc;
  *out = new cgc_batch{p};
  return cgc::ok();
}
int cgc_batch_destroy(cgc_batch* b) {
  if (!b) return cgc::ok();
  delete b->p;
  delete b;
  return cgc::ok();
}
int cgc_batch_set_tlinks(cgc_batch* b, int32_t i, const int32_t* capS, const int32_t* capT) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_put_tlinks(*b->p, i, capS, capT, true);
}
int cgc_batch_set_nlinks(cgc_batch* b, int32_t i, int axis, const int32_t* fwd, const int32_t* bwd) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_put_nlinks(*b->p, i, axis, fwd, bwd, true);
}
int cgc_batch_maxflow(cgc_batch* b, const cgc_options* opts, int64_t* flows) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  int rc = cgc::pool_solve(*b->p, opts);
  if (rc) return rc;
  if (flows) std::memcpy(flows, b->p->flows.data(), b->p->flows.size() * 8);
  return cgc::ok();
}
int cgc_batch_get_segments(cgc_batch* b, int32_t i, int which, uint8_t* out, uint8_t mask, uint8_t background) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_segments(*b->p, i, which, out, mask, background, true);
}
int cgc_batch_stats(cgc_batch* b, cgc_stats* out) {
  if (!b || !out) return cgc::fail(CGC_ERR_ARG, "null argument");
  *out = b->p->st;
  return cgc::ok();
}

}  // extern "C"
