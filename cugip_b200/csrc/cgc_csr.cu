// Generic (non-grid) graphs: exact push-relabel over a CSR residual graph.
//
// The reference solves every graph through one CSR layout
// (include/cugip/advanced_operations/graph_cut.hpp:239-290: neighbour lists,
// one residual pair per undirected edge) with a level-synchronous BFS
// relabel and per-level pushes (detail/graph_cut_relabeling.hpp:1004-1029,
// detail/graph_cut_push.hpp:461-482).  Grids go to the tile engine; this file
// handles every other edge list with the same options, statuses and cut
// semantics:
//   * CSR built on the device: per-vertex degree count, exclusive scan,
//     atomic scatter of the two arcs of every edge with reverse-arc links.
//     The original arc capacities are kept, so a graph can be solved again.
//   * one cooperative launch per solve, 4 to 16 lanes per vertex: exact global
//     relabel (BFS from the vertices with a sink residual over reverse residual
//     arcs, heights set by CAS), then up to K synchronous pulses over a
//     deduplicated active-vertex list: a push step with fixed labels (a vertex pushes along arcs to
//     neighbours one level lower; excess and reverse residuals of the
//     neighbour by atomics) and a relabel step (1 + the lowest residual
//     neighbour; labels only grow, so concurrent relabels keep them valid).
//     The solve ends when an exact relabel leaves no active vertex.
//   * int32 capacities, int64 flow, t-links cancelled up front (min(capS,
//     capT) flows straight through), pushes to the sink capped by its residual.
//   * cuts: sink side = vertices with a finite height after the last exact
//     relabel (the reference's fill_segments, graph_cut.hpp:304-333); source
//     side = residual closure of the vertices that hold excess.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "cgc.h"
#include "cgc_arcs.h"
#include "cgc_internal.h"
#include "cgc_pool.h"
#include "cgc_sync.cuh"

namespace cgc {
namespace {

constexpr int CSR_THREADS = 1024;  // solve: one CTA per SM
constexpr int SCAN_BLOCK = 1024;

enum CsrStat { CS_PULSES = 0, CS_RELABELS, CS_LEVELS, CS_PUSHES, CS_BFS_VISITS, CS_NS_BFS, CS_NS_PUSH, CS_NS_REACH, CS_N = 16 };
enum CsrCounter { CC_BFS0 = 0, CC_PULSE0 = 3, CC_N = 8 };

struct CsrDev {
  int32_t n;
  int64_t arcs;
  int32_t hdead;             // heights >= hdead cannot reach the sink (n + 1)
  const int32_t* row;        // n + 1: first arc of each vertex
  const int32_t* to;         // arcs: head vertex
  const int32_t* rev;        // arcs: index of the reverse arc
  int32_t* res;              // arcs: residual capacity
  const int32_t* res0;       // arcs: capacity
  const int32_t* capS;       // n
  const int32_t* capT;       // n
  int32_t* e;                // n: excess
  int32_t* h;                // n: height
  int32_t* rT;               // n: sink residual
  int32_t* reach;            // n: source side
  uint32_t* stamp;           // n: last list the vertex was queued for
  int32_t* list;             // 2n: two vertex lists
  int2* front;               // 2n: two BFS frontiers (arc ranges of their vertices)
  int32_t* cnt;              // CC_N counters
  unsigned long long* flow;  // 1
  unsigned long long* stats; // CS_N
  int32_t* err;
  uint32_t* bar;             // 2
};

struct CsrParams {
  int K;                 // pulses between exact relabels
  int64_t max_pulses;    // safety cap
  uint64_t limit_ns;     // bounded barrier waits
};

__device__ __forceinline__ int ldv(const int32_t* p) { return *(volatile const int32_t*)p; }

// loaded ahead of the test that may discard it
__device__ __forceinline__ int ld_early(const int32_t* p) {
  int v;
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int2 ld_early(const int2* p) {
  int2 v;
  asm volatile("ld.global.cg.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// warp-aggregated append (all lanes of the warp call it)
template <typename T>
__device__ __forceinline__ void csr_append(bool pred, T item, T* list, int32_t* cnt) {
  const unsigned mask = __ballot_sync(0xffffffffu, pred);
  if (!mask) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(cnt, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) list[base + __popc(mask & ((1u << lane) - 1))] = item;
}

// ---------------------------------------------------------------- CSR build
__global__ void k_csr_degree(int64_t m, const int32_t* __restrict__ a, const int32_t* __restrict__ b, int32_t* deg) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const int u = a[i], v = b[i];
    if (u == v) continue;  // a self loop carries no flow
    atomicAdd(deg + u, 1);
    atomicAdd(deg + v, 1);
  }
}

// exclusive scan, pass 1: each block scans SCAN_BLOCK entries
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_block(const int32_t* in, int32_t* out, int32_t* bsum, int n) {
  __shared__ int32_t ws[SCAN_BLOCK / 32];
  const int64_t i = blockIdx.x * (int64_t)SCAN_BLOCK + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int v = i < n ? in[i] : 0;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = ws[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    ws[lane] = s;
  }
  __syncthreads();
  const int incl = x + (w > 0 ? ws[w - 1] : 0);
  if (i < n) out[i] = incl - v;
  if (threadIdx.x == SCAN_BLOCK - 1) bsum[blockIdx.x] = incl;
}

// pass 2: exclusive scan of the block sums by one block; total into *total
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_sums(int32_t* bsum, int nb, int32_t* total) {
  __shared__ int32_t ws[SCAN_BLOCK / 32];
  __shared__ int32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < nb; base += SCAN_BLOCK) {
    const int i = base + threadIdx.x;
    const int v = i < nb ? bsum[i] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = ws[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      ws[lane] = s;
    }
    __syncthreads();
    const int incl = x + (w > 0 ? ws[w - 1] : 0);
    const int c = carry;
    if (i < nb) bsum[i] = c + incl - v;
    __syncthreads();
    if (threadIdx.x == SCAN_BLOCK - 1) carry = c + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// pass 3: add the block offsets
__global__ void k_scan_add(int32_t* out, const int32_t* bsum, int n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] += bsum[i / SCAN_BLOCK];
}

__global__ void k_csr_scatter(int64_t m, const int32_t* __restrict__ a, const int32_t* __restrict__ b,
                              const int32_t* __restrict__ fwd, const int32_t* __restrict__ bwd, const int32_t* row,
                              int32_t* cur, int32_t* to, int32_t* rev, int32_t* res0) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const int u = a[i], v = b[i];
    if (u == v) continue;
    const int pu = row[u] + atomicAdd(cur + u, 1);
    const int pv = row[v] + atomicAdd(cur + v, 1);
    to[pu] = v; rev[pu] = pv; res0[pu] = fwd[i];
    to[pv] = u; rev[pv] = pu; res0[pv] = bwd[i];
  }
}

// ---------------------------------------------------------------- solve
__global__ void k_csr_prepare(CsrDev D) {
  const int64_t nt = (int64_t)gridDim.x * blockDim.x, gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t a = gt; a < D.arcs; a += nt) D.res[a] = D.res0[a];
  long long through = 0;
  for (int64_t v = gt; v < D.n; v += nt) {
    const int s = D.capS[v], t = D.capT[v], mn = min(s, t);
    D.e[v] = s - mn;
    D.rT[v] = t - mn;
    D.h[v] = 0;
    D.stamp[v] = 0;
    through += mn;
    // Excess and residuals stay int32: the excess is at most the source
    // excess plus every capacity into v, a residual at most the two
    // capacities of its edge.
    long long inflow = s - mn;
    bool bad = false;
    const int a1 = D.row[v + 1];
    for (int a = D.row[v]; a < a1; ++a) {
      const long long back = D.res0[D.rev[a]];
      inflow += back;
      if (back + D.res0[a] > 2147483647ll) bad = true;
    }
    if (bad || inflow > 2147483647ll) atomicCAS(D.err, 0, CGC_ERR_OVERFLOW);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) through += __shfl_down_sync(0xffffffffu, through, o);
  if ((threadIdx.x & 31) == 0 && through) atomicAdd(D.flow, (unsigned long long)through);
}

// W lanes work on a vertex: they read its arcs W at a time, so a vertex costs
// a few dependent memory round trips instead of one chain per arc.  A round of
// the BFS or a pulse is bound by those round trips (about 0.3 us each) and by
// the grid barrier (one CTA per SM, one arrival each), not by bytes.  A thread
// per vertex and a loop over its arcs took 15 us per BFS round and 32 us per
// pulse on the layered graph of 100 x 1024 vertices, this takes 4 and 10 (solve
// 13.7 -> 3.9 ms); random graph of 200 k vertices, 800 k edges: 5.6 -> 2.1 ms.
// W is 16, 8 or 4 by the average degree (graph_create).
// Spreading a short list's vertices over all SMs was not faster (BFS 2.9 -> 3.0 ms).
template <int W>
__global__ void __launch_bounds__(CSR_THREADS, 1) k_csr_solve(CsrDev D, CsrParams prm) {
  constexpr unsigned FULL = 0xffffffffu;
  const int n = D.n;
  const int lane = threadIdx.x & 31;
  const int sub = threadIdx.x & (W - 1);       // lane of the vertex
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const int slot = gt / W, slots = nt / W;     // vertices of a list: slot, slot + slots, ...
  const int wslot = (gt - lane) / W;           // the warp's first slot: loops over a list are uniform over a warp
  int32_t* const L[2] = {D.list, D.list + n};
  int32_t* const cb = D.cnt + CC_BFS0;    // 3 rotating counters of the BFS frontiers
  int32_t* const cp = D.cnt + CC_PULSE0;  // 3 rotating counters of the pulse lists
  const bool lead = gt == 0;
  uint32_t sid = 0;
  int pulses = 0, relabels = 0, levels = 0;
  long long flow = 0;  // delivered to the sink by this thread
  unsigned long long ns_bfs = 0, ns_push = 0, ns_reach = 0;
  uint64_t tmark = sync_globaltimer_ns();
  auto lap = [&](unsigned long long& acc) {
    if (!lead) return;
    const uint64_t now = sync_globaltimer_ns();
    acc += now - tmark;
    tmark = now;
  };
  uint32_t bar_target = 0;
  auto sync = [&]() { return grid_barrier(D.bar, bar_target, prm.limit_ns); };
  // Frontier BFS.  A frontier holds the arc ranges of its vertices, loaded
  // while the vertex is claimed, so the next round starts with the arcs.
  // take(arc, head, k) says whether the arc's head joins the next frontier;
  // returns the number of rounds, -1 on a failed barrier.
  auto arcs_of = [&](int v) { return make_int2(__ldg(D.row + v), __ldg(D.row + v + 1)); };
  auto bfs = [&](auto&& take) -> int {
    int k = 0;
    for (;;) {
      const int2* lc = D.front + (k & 1) * (int64_t)n;
      int2* ln = D.front + ((k + 1) & 1) * (int64_t)n;
      int2 f = slot < n ? ld_early(lc + slot) : make_int2(0, 0);
      const int nf = ldv(cb + k % 3);
      if (nf == 0) return k;
      if (lead) cb[(k + 2) % 3] = 0;
      for (int i0 = wslot, i = slot; i0 < nf;) {
        ArcWalk<W> a;
        if (i < nf) a = ArcWalk<W>(f.x, f.y, sub);
        for (; __any_sync(FULL, a.on()); a.step()) {
          bool ok = a.on();
          int2 r = make_int2(0, 0);
          if (ok) {
            const int v = __ldg(D.to + a.at);
            r = arcs_of(v);
            ok = take(a.at, v, k);
          }
          csr_append(ok, r, ln, cb + (k + 1) % 3);
        }
        i0 += slots;
        i += slots;
        if (i < nf) f = __ldcg(lc + i);
      }
      ++k;
      if (!sync()) return -1;
    }
  };

  for (;;) {
    // ------------------------------------------------ exact global relabel
    if (lead) { cb[0] = cb[1] = cb[2] = 0; cp[0] = cp[1] = cp[2] = 0; }
    if (!sync()) return;
    for (int v = gt; v - lane < n; v += nt) {
      const bool seed = v < n && __ldcg(D.rT + v) > 0;
      if (v < n) D.h[v] = seed ? 1 : INF;
      csr_append(seed, seed ? arcs_of(v) : make_int2(0, 0), D.front, cb + 0);
    }
    if (!sync()) return;
    const int rounds = bfs([&](uint32_t a, int v, int k) {
      const int r = __ldcg(D.res + __ldg(D.rev + a));
      // the frontier of round k has height k + 1
      return ldv(D.h + v) == INF && r > 0 && atomicCAS(D.h + v, INF, k + 2) == INF;
    });
    if (rounds < 0) return;
    levels += rounds;
    ++relabels;
    lap(ns_bfs);
    // ------------------------------------------------ active vertices
    ++sid;
    for (int v = gt; v - lane < n; v += nt) {
      const bool act = v < n && __ldcg(D.e + v) > 0 && __ldcg(D.h + v) < INF;
      if (act) D.stamp[v] = sid;
      csr_append(act, v, L[0], cp + 0);
    }
    if (!sync()) return;
    if (ldv(cp + 0) == 0) break;
    if (pulses >= prm.max_pulses) {
      if (lead) atomicCAS(D.err, 0, CGC_ERR_NOT_CONVERGED);
      break;
    }
    // ------------------------------------------------ pulses
    for (int p = 0; p < prm.K; ++p) {
      const int32_t* lc = L[p & 1];
      int32_t* ln = L[(p + 1) & 1];
      int v = slot < n ? ld_early(lc + slot) : 0;
      const int ncur = ldv(cp + p % 3);
      if (ncur == 0) break;
      if (lead) cp[(p + 2) % 3] = 0;
      ++sid;
      int32_t* cn = cp + (p + 1) % 3;
      // push step: labels fixed; the vertex's lanes split its excess among the
      // admissible arcs by a saturating prefix sum
      for (int i0 = wslot, i = slot; i0 < ncur; i0 += slots, i += slots) {
        ArcWalk<W> a;
        int ev = 0, hv = INF, rt = 0;
        if (i < ncur) {
          if (i != slot) v = __ldcg(lc + i);
          a = ArcWalk<W>(__ldg(D.row + v), __ldg(D.row + v + 1), sub);
          hv = __ldcg(D.h + v);
          if (sub == 0) {
            ev = __ldcg(D.e + v);
            rt = __ldcg(D.rT + v);
          }
        }
        // One read for all lanes: neighbours add to the excess meanwhile, and the
        // lanes share out what is subtracted from it below.
        ev = __shfl_sync(FULL, ev, 0, W);
        rt = __shfl_sync(FULL, rt, 0, W);
        if (ev <= 0 || hv >= INF) { ev = 0; a.stop(); }
        const int e0 = ev;
        if (rt > 0 && hv == 1 && ev > 0) {
          const int dl = min(ev, rt);
          ev -= dl;
          if (sub == 0) {
            D.rT[v] = rt - dl;
            flow += dl;
          }
        }
        for (; __any_sync(FULL, a.on() && ev > 0); a.step()) {
          unsigned cap = 0;
          int r = 0, u = 0, rv = 0;
          if (a.on() && ev > 0) {
            r = __ldcg(D.res + a.at);
            u = __ldg(D.to + a.at);
            rv = __ldg(D.rev + a.at);
            if (r > 0 && __ldcg(D.h + u) == hv - 1) cap = (unsigned)min(r, ev);
          }
          unsigned s = cap;
#pragma unroll
          for (int o = 1; o < W; o <<= 1) {
            const unsigned x = __shfl_up_sync(FULL, s, o, W);
            if (sub >= o) s = min(s + x, (unsigned)ev);
          }
          unsigned below = __shfl_up_sync(FULL, s, 1, W);
          if (sub == 0) below = 0;
          const int dl = (int)(s - below);
          ev -= (int)__shfl_sync(FULL, s, W - 1, W);
          bool fresh = false;
          if (dl > 0) {
            D.res[a.at] = r - dl;  // only v writes this arc in this step
            atomicAdd(D.res + rv, dl);
            atomicAdd(D.e + u, dl);
            fresh = atomicExch(D.stamp + u, sid) != sid;
          }
          csr_append(fresh, u, ln, cn);
        }
        if (sub == 0 && ev != e0) atomicSub(D.e + v, e0 - ev);
        csr_append(sub == 0 && ev > 0 && atomicExch(D.stamp + v, sid) != sid, v, ln, cn);
      }
      if (!sync()) return;
      // relabel step: an active vertex moves to one above its lowest residual
      // neighbour (which is its own height while it has an admissible arc);
      // labels only grow, so concurrent relabels keep them valid
      v = slot < n ? ld_early(ln + slot) : 0;
      const int nn = ldv(cn);
      for (int i0 = wslot, i = slot; i0 < nn; i0 += slots, i += slots) {
        ArcWalk<W> a;
        int hv = INF, mn = INF;
        if (i < nn) {
          if (i != slot) v = __ldcg(ln + i);
          a = ArcWalk<W>(__ldg(D.row + v), __ldg(D.row + v + 1), sub);
          const int ev = __ldcg(D.e + v), rt = __ldcg(D.rT + v);
          hv = __ldcg(D.h + v);
          if (ev <= 0 || (rt > 0 && hv == 1)) hv = INF;
          if (rt > 0) mn = 0;
        }
        if (hv >= INF) a.stop();
        for (; __any_sync(FULL, a.on()); a.step()) {
          if (a.on()) {
            const int r = __ldcg(D.res + a.at);
            const int hu = ldv(D.h + __ldg(D.to + a.at));
            if (r > 0) mn = min(mn, hu);
          }
        }
#pragma unroll
        for (int o = 1; o < W; o <<= 1) mn = min(mn, __shfl_xor_sync(FULL, mn, o));
        if (sub == 0 && hv < INF && mn >= hv) {
          const int hn = mn >= INF || mn + 1 >= D.hdead ? INF : mn + 1;
          D.h[v] = hn;
        }
      }
      ++pulses;
      if (!sync()) return;
    }
    lap(ns_push);
  }
  lap(ns_bfs);
  // ------------------------------------------------ source side: residual
  // closure of the vertices that hold excess
  if (lead) { cb[0] = cb[1] = cb[2] = 0; }
  if (!sync()) return;
  for (int v = gt; v - lane < n; v += nt) {
    const bool seed = v < n && __ldcg(D.e + v) > 0;
    if (v < n) D.reach[v] = seed ? 1 : 0;
    csr_append(seed, seed ? arcs_of(v) : make_int2(0, 0), D.front, cb + 0);
  }
  if (!sync()) return;
  const int rrounds = bfs([&](uint32_t a, int v, int) {
    const int r = __ldcg(D.res + a);
    return ldv(D.reach + v) == 0 && r > 0 && atomicCAS(D.reach + v, 0, 1) == 0;
  });
  if (rrounds < 0) return;
  lap(ns_reach);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) flow += __shfl_down_sync(FULL, flow, o);
  if (lane == 0 && flow) atomicAdd(D.flow, (unsigned long long)flow);
  if (lead) {
    D.stats[CS_PULSES] = (unsigned long long)pulses;
    D.stats[CS_RELABELS] = (unsigned long long)relabels;
    D.stats[CS_LEVELS] = (unsigned long long)levels;
    D.stats[CS_NS_BFS] = ns_bfs;
    D.stats[CS_NS_PUSH] = ns_push;
    D.stats[CS_NS_REACH] = ns_reach;
  }
}

__global__ void k_csr_segments(CsrDev D, int which, uint8_t* out, uint8_t mask, uint8_t bg) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < D.n; v += (int64_t)gridDim.x * blockDim.x) {
    const bool in = which == CGC_SEG_SOURCE_MIN ? D.reach[v] != 0 : D.h[v] < INF;
    out[v] = in ? mask : bg;
  }
}

int grid_blocks(int64_t work, int threads) { return (int)std::max<int64_t>(1, std::min<int64_t>((work + threads - 1) / threads, 1 << 16)); }

}  // namespace
}  // namespace cgc

struct cgc_graph {
  int device = 0;
  cudaStream_t stream = nullptr;
  int32_t n = 0;
  int64_t m = 0;
  void* dbuf = nullptr;
  uint8_t* seg = nullptr;
  cgc::CsrDev d{};
  int coop_blocks = 0;
  int lanes = 8;  // lanes per vertex in the solve
  bool tlinks = false, solved = false;
  bool untracked = false;  // a call failed before it had waited for what it queued
  cgc_stats st{};
};

namespace {

using cgc::fail;
using cgc::ok;

// Around calls that queue work: marks the graph where one returns before it
// has waited.
struct Queued {
  cgc_graph* g;
  bool waited = false;
  explicit Queued(cgc_graph* graph) : g(graph) {}
  Queued(const Queued&) = delete;
  ~Queued() { if (!waited) g->untracked = true; }
};

void graph_free(cgc_graph* g) {
  if (!g) return;
  // every call that succeeded has waited for its work; a block that something
  // may still be using is not handed out again
  if (g->dbuf && (!g->untracked || cgc::wait_for_device(g->device))) cgc::dev_free(g->dbuf);
  delete g;
}

int graph_create(int32_t n, int64_t m, const int32_t* a, const int32_t* b, const int32_t* cab, const int32_t* cba,
                 void* stream, cgc_graph** out) {
  using namespace cgc;
  if (!out) return fail(CGC_ERR_ARG, "cgc_graph_create: null output");
  *out = nullptr;
  if (n <= 0 || m < 0 || (m > 0 && (!a || !b || !cab || !cba)))
    return fail(CGC_ERR_ARG, "cgc_graph_create: bad arguments");
  int64_t loops = 0;
  for (int64_t i = 0; i < m; ++i) {
    if (a[i] < 0 || a[i] >= n || b[i] < 0 || b[i] >= n)
      return fail(CGC_ERR_ARG, "cgc_graph_create: edge " + std::to_string(i) + " has a vertex outside [0, n)");
    if (cab[i] < 0 || cba[i] < 0)
      return fail(CGC_ERR_ARG, "cgc_graph_create: negative capacity on edge " + std::to_string(i));
    loops += a[i] == b[i];
  }
  const int64_t arcs = 2 * (m - loops);
  if (arcs > 2147483647ll || n > 2147483646) return fail(CGC_ERR_ARG, "cgc_graph_create: graph too large for int32 arc ids");
  cgc_graph* g = new (std::nothrow) cgc_graph();
  if (!g) return fail(CGC_ERR_OOM, "cgc_graph_create: host allocation");
  g->n = n;
  g->m = m;
  g->stream = (cudaStream_t)stream;
  int rc = [&]() -> int {
    CGC_CUDA(cudaGetDevice(&g->device));
    auto al = [](int64_t bytes) { return (bytes + 255) & ~(int64_t)255; };
    const int nb = (int)((n + SCAN_BLOCK - 1) / SCAN_BLOCK);
    int64_t off = 0;
    const int64_t o_row = off; off += al(((int64_t)n + 1) * 4);
    const int64_t o_to = off; off += al(arcs * 4);
    const int64_t o_rev = off; off += al(arcs * 4);
    const int64_t o_res = off; off += al(arcs * 4);
    const int64_t o_res0 = off; off += al(arcs * 4);
    const int64_t o_cs = off; off += al((int64_t)n * 4);
    const int64_t o_ct = off; off += al((int64_t)n * 4);
    const int64_t o_e = off; off += al((int64_t)n * 4);
    const int64_t o_h = off; off += al((int64_t)n * 4);
    const int64_t o_rt = off; off += al((int64_t)n * 4);
    const int64_t o_rc = off; off += al((int64_t)n * 4);
    const int64_t o_st = off; off += al((int64_t)n * 4);
    const int64_t o_li = off; off += al(2 * (int64_t)n * 4);
    const int64_t o_fr = off; off += al(2 * (int64_t)n * 8);
    const int64_t o_cnt = off; off += al(CC_N * 4);
    const int64_t o_fl = off; off += al(8);
    const int64_t o_sta = off; off += al(CS_N * 8);
    const int64_t o_bar = off; off += al(8);
    const int64_t o_seg = off; off += al(n);
    const int64_t o_bs = off; off += al((int64_t)nb * 4);
    if (int rc2 = dev_alloc(g->device, &g->dbuf, off)) return rc2;
    Queued queued(g);
    CGC_CUDA(cudaMemsetAsync(g->dbuf, 0, off, g->stream));
    char* base = (char*)g->dbuf;
    CsrDev& d = g->d;
    d.n = n;
    d.arcs = arcs;
    d.hdead = (int32_t)std::min<int64_t>((int64_t)n + 1, INF);
    d.row = (int32_t*)(base + o_row);
    d.to = (int32_t*)(base + o_to);
    d.rev = (int32_t*)(base + o_rev);
    d.res = (int32_t*)(base + o_res);
    d.res0 = (int32_t*)(base + o_res0);
    d.capS = (int32_t*)(base + o_cs);
    d.capT = (int32_t*)(base + o_ct);
    d.e = (int32_t*)(base + o_e);
    d.h = (int32_t*)(base + o_h);
    d.rT = (int32_t*)(base + o_rt);
    d.reach = (int32_t*)(base + o_rc);
    d.stamp = (uint32_t*)(base + o_st);
    d.list = (int32_t*)(base + o_li);
    d.front = (int2*)(base + o_fr);
    d.cnt = (int32_t*)(base + o_cnt);
    d.flow = (unsigned long long*)(base + o_fl);
    d.stats = (unsigned long long*)(base + o_sta);
    d.bar = (uint32_t*)(base + o_bar);
    d.err = (int32_t*)(d.bar + 1);
    g->seg = (uint8_t*)(base + o_seg);
    int32_t* bsum = (int32_t*)(base + o_bs);
    if (m > 0) {
      // edges to the device, then degrees -> row offsets -> arcs
      int32_t* stage = nullptr;
      if (int rc2 = dev_alloc(g->device, &stage, 4 * m * 4)) return rc2;
      int rc2 = [&]() -> int {
        CGC_CUDA(cudaMemcpyAsync(stage, a, m * 4, cudaMemcpyHostToDevice, g->stream));
        CGC_CUDA(cudaMemcpyAsync(stage + m, b, m * 4, cudaMemcpyHostToDevice, g->stream));
        CGC_CUDA(cudaMemcpyAsync(stage + 2 * m, cab, m * 4, cudaMemcpyHostToDevice, g->stream));
        CGC_CUDA(cudaMemcpyAsync(stage + 3 * m, cba, m * 4, cudaMemcpyHostToDevice, g->stream));
        int32_t* deg = d.reach;   // scratch until the first solve
        int32_t* cur = (int32_t*)d.stamp;
        const int eb = grid_blocks(m, 256);
        k_csr_degree<<<eb, 256, 0, g->stream>>>(m, stage, stage + m, deg); note_launch();
        k_scan_block<<<nb, SCAN_BLOCK, 0, g->stream>>>(deg, (int32_t*)d.row, bsum, n); note_launch();
        k_scan_sums<<<1, SCAN_BLOCK, 0, g->stream>>>(bsum, nb, (int32_t*)d.row + n); note_launch();
        k_scan_add<<<grid_blocks(n, 256), 256, 0, g->stream>>>((int32_t*)d.row, bsum, n); note_launch();
        k_csr_scatter<<<eb, 256, 0, g->stream>>>(m, stage, stage + m, stage + 2 * m, stage + 3 * m, d.row, cur,
                                                 (int32_t*)d.to, (int32_t*)d.rev, (int32_t*)d.res0); note_launch();
        CGC_CUDA(cudaGetLastError());
        CGC_CUDA(cudaMemsetAsync(deg, 0, (size_t)n * 4, g->stream));
        CGC_CUDA(cudaMemsetAsync(cur, 0, (size_t)n * 4, g->stream));
        CGC_CUDA(cudaStreamSynchronize(g->stream));
        return CGC_OK;
      }();
      if (!rc2 || wait_for_device(g->device)) dev_free(stage);
      if (rc2) return rc2;
    }
    int sms = 0;
    CGC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
    // Lanes per vertex by its average number of arcs, so that few idle and a
    // vertex takes few steps (kernel ms with 4, 8 and 16 lanes on random graphs of
    // average degree 2: 1.90 2.06 2.51, 4: 4.64 4.52 5.22, 6: 3.40 3.15 3.43,
    // 8: 2.02 1.85 1.93, 12: 2.04 1.79 1.74, 16: 2.63 2.12 1.94, 48: 1.84 1.23 0.93;
    // layered 100x1024, degree 16: 6.2 4.6 3.9).  Enough CTAs to cover the
    // vertices, at most one per SM.
    const int64_t degree = arcs / n;
    g->lanes = degree >= 12 ? 16 : degree >= 6 ? 8 : 4;
    g->coop_blocks = std::max(1, std::min(sms, grid_blocks((int64_t)n * g->lanes, CSR_THREADS)));
    CGC_CUDA(cudaStreamSynchronize(g->stream));
    queued.waited = true;
    return CGC_OK;
  }();
  if (rc) {
    graph_free(g);
    return rc;
  }
  *out = g;
  return ok();
}

int graph_maxflow(cgc_graph* g, const cgc_options* opts, int64_t* flow) {
  using namespace cgc;
  if (!g) return fail(CGC_ERR_ARG, "cgc_graph_maxflow: null graph");
  if (!g->tlinks) return fail(CGC_ERR_STATE, "cgc_graph_maxflow: set the terminal capacities first");
  const cgc_options o = resolve_options(opts);
  CsrParams prm;
  prm.K = std::max(1, 2 * o.sweeps_per_relabel);
  prm.max_pulses = (int64_t)o.max_sweeps;
  prm.limit_ns = wait_limit_ns(o);
  const long long launches0 = g_launches.load();
  CsrDev& d = g->d;
  cudaEvent_t ev[4] = {};
  for (auto& e : ev) CGC_CUDA(cudaEventCreate(&e));
  auto destroy = [&]() {
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
  };
  Queued queued(g);
  int rc = [&]() -> int {
    CGC_CUDA(cudaEventRecord(ev[0], g->stream));
    CGC_CUDA(cudaMemsetAsync(d.flow, 0, 8, g->stream));
    CGC_CUDA(cudaMemsetAsync(d.stats, 0, CS_N * 8, g->stream));
    CGC_CUDA(cudaMemsetAsync(d.bar, 0, 8, g->stream));  // and the error word
    CGC_CUDA(cudaMemsetAsync(d.cnt, 0, CC_N * 4, g->stream));
    k_csr_prepare<<<grid_blocks(std::max<int64_t>(d.arcs, d.n), 256), 256, 0, g->stream>>>(d); note_launch();
    CGC_CUDA(cudaGetLastError());
    CGC_CUDA(cudaEventRecord(ev[1], g->stream));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = g->stream;
    cfg.gridDim = dim3(g->coop_blocks);
    cfg.blockDim = dim3(CSR_THREADS);
    if (int rc2 = coop_launch_ordered(g->device, g->stream, [&]() -> int {
          CGC_CUDA(cudaLaunchKernelEx(
              &cfg, g->lanes == 16 ? k_csr_solve<16> : g->lanes == 8 ? k_csr_solve<8> : k_csr_solve<4>, d, prm));
          return CGC_OK;
        }))
      return rc2;
    note_launch();
    CGC_CUDA(cudaEventRecord(ev[2], g->stream));
    CGC_CUDA(cudaEventRecord(ev[3], g->stream));
    CGC_CUDA(cudaEventSynchronize(ev[3]));
    queued.waited = true;
    int32_t err = 0;
    CGC_CUDA(cudaMemcpy(&err, d.err, 4, cudaMemcpyDeviceToHost));
    if (err == CGC_ERR_TIMEOUT) return fail(CGC_ERR_TIMEOUT, "cgc_graph_maxflow: a grid barrier timed out");
    if (err == CGC_ERR_NOT_CONVERGED) return fail(CGC_ERR_NOT_CONVERGED, "cgc_graph_maxflow: pulse cap reached");
    if (err == CGC_ERR_OVERFLOW)
      return fail(CGC_ERR_OVERFLOW, "cgc_graph_maxflow: capacities may overflow int32 excess or residuals");
    if (err) return fail(err, "cgc_graph_maxflow: device error");
    unsigned long long f = 0, stats[CS_N];
    CGC_CUDA(cudaMemcpy(&f, d.flow, 8, cudaMemcpyDeviceToHost));
    CGC_CUDA(cudaMemcpy(stats, d.stats, sizeof(stats), cudaMemcpyDeviceToHost));
    float ms = 0.f, kms = 0.f;
    cudaEventElapsedTime(&ms, ev[0], ev[3]);
    cudaEventElapsedTime(&kms, ev[1], ev[2]);
    std::memset(&g->st, 0, sizeof(g->st));
    g->st.flow = (int64_t)f;
    g->st.sweeps = (int64_t)stats[CS_PULSES];
    g->st.global_relabels = (int64_t)stats[CS_RELABELS];
    g->st.bfs_rounds = (int64_t)stats[CS_LEVELS];
    g->st.pulses = (int64_t)stats[CS_PULSES];
    g->st.solve_ms = ms;
    g->st.kernel_ms = kms;
    g->st.launches = g_launches.load() - launches0;
    g->st.bfs_ms = 1e-6 * (double)stats[CS_NS_BFS];
    g->st.sweep_ms = 1e-6 * (double)stats[CS_NS_PUSH];
    g->st.reach_ms = 1e-6 * (double)stats[CS_NS_REACH];
    if (flow) *flow = (int64_t)f;
    g->solved = true;
    return CGC_OK;
  }();
  destroy();
  return rc ? rc : ok();
}

}  // namespace

extern "C" {

int cgc_graph_create(int32_t n, int64_t m, const int32_t* a, const int32_t* b, const int32_t* cap_ab,
                     const int32_t* cap_ba, void* stream, cgc_graph** out) {
  return graph_create(n, m, a, b, cap_ab, cap_ba, stream, out);
}

int cgc_graph_destroy(cgc_graph* g) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "cgc_graph_destroy: null graph");
  graph_free(g);
  return cgc::ok();
}

int cgc_graph_set_tlinks(cgc_graph* g, const int32_t* capS, const int32_t* capT) {
  if (!g || !capS || !capT) return cgc::fail(CGC_ERR_ARG, "cgc_graph_set_tlinks: bad arguments");
  for (int32_t v = 0; v < g->n; ++v)
    if (capS[v] < 0 || capT[v] < 0)
      return cgc::fail(CGC_ERR_ARG, "cgc_graph_set_tlinks: negative capacity at vertex " + std::to_string(v));
  Queued queued(g);
  CGC_CUDA(cudaMemcpyAsync((void*)g->d.capS, capS, (size_t)g->n * 4, cudaMemcpyHostToDevice, g->stream));
  CGC_CUDA(cudaMemcpyAsync((void*)g->d.capT, capT, (size_t)g->n * 4, cudaMemcpyHostToDevice, g->stream));
  CGC_CUDA(cudaStreamSynchronize(g->stream));
  queued.waited = true;
  g->tlinks = true;
  return cgc::ok();
}

int cgc_graph_maxflow(cgc_graph* g, const cgc_options* opts, int64_t* flow) { return graph_maxflow(g, opts, flow); }

int cgc_graph_get_segments(cgc_graph* g, int which, uint8_t* out, uint8_t mask, uint8_t background) {
  if (!g || !out || (which != CGC_SEG_SINK_REACH && which != CGC_SEG_SOURCE_MIN))
    return cgc::fail(CGC_ERR_ARG, "cgc_graph_get_segments: bad arguments");
  if (!g->solved) return cgc::fail(CGC_ERR_STATE, "cgc_graph_get_segments: call maxflow first");
  Queued queued(g);
  cgc::k_csr_segments<<<cgc::grid_blocks(g->n, 256), 256, 0, g->stream>>>(g->d, which, g->seg, mask, background);
  cgc::note_launch();
  CGC_CUDA(cudaGetLastError());
  CGC_CUDA(cudaMemcpyAsync(out, g->seg, (size_t)g->n, cudaMemcpyDeviceToHost, g->stream));
  CGC_CUDA(cudaStreamSynchronize(g->stream));
  queued.waited = true;
  return cgc::ok();
}

int cgc_graph_get_state(cgc_graph* g, int32_t* labels, int32_t* excess) {
  if (!g) return cgc::fail(CGC_ERR_ARG, "cgc_graph_get_state: null graph");
  if (!g->solved) return cgc::fail(CGC_ERR_STATE, "cgc_graph_get_state: call maxflow first");
  Queued queued(g);
  if (labels) CGC_CUDA(cudaMemcpyAsync(labels, g->d.h, (size_t)g->n * 4, cudaMemcpyDeviceToHost, g->stream));
  if (excess) CGC_CUDA(cudaMemcpyAsync(excess, g->d.e, (size_t)g->n * 4, cudaMemcpyDeviceToHost, g->stream));
  CGC_CUDA(cudaStreamSynchronize(g->stream));
  queued.waited = true;
  if (labels)
    for (int32_t v = 0; v < g->n; ++v)
      if (labels[v] >= cgc::INF) labels[v] = INT32_MIN;
  return cgc::ok();
}

int cgc_graph_stats(cgc_graph* g, cgc_stats* st) {
  if (!g || !st) return cgc::fail(CGC_ERR_ARG, "cgc_graph_stats: bad arguments");
  *st = g->st;
  return cgc::ok();
}

}  // extern "C"
