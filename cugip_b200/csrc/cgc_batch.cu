// Device-resident batch path: many grid instances whose capacities already
// sit in device memory are uploaded, solved and written back by a fixed
// sequence of 3 kernels and 2 memory operations with no host synchronisation
// -- one pointer-table upload and preflow kernel for all instances, one
// persistent cooperative solve, one pointer-table output kernel -- which
// is captured once into a CUDA graph and replayed per batch.
//
// The reference solves one graph per Graph object with a host round trip per
// BFS level and per push level (detail/graph_cut_relabeling.hpp:962-984,
// detail/graph_cut_push.hpp:395-459); it has no batch path.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "cgc.h"
#include "cgc_kernels.cuh"
#include "cgc_pool.h"

namespace cgc {

// Upload of every instance from its bound device inputs (8 pointers per
// instance: capS, capT, fwd x/y/z, bwd x/y/z; a null n-link pointer is zero),
// fused with the preflow initialisation (put_run, cgc_kernels.cuh).
__global__ void __launch_bounds__(128, 8) k_put_all(DevPool P, const int32_t* const* __restrict__ in) {
  const int t0 = P.runs[blockIdx.x];
  put_run(P, t0, in + 8 * (int64_t)P.tinst[t0], true);
}

// Both cut sets of every instance into its bound device outputs (1/0 bytes),
// in linear voxel order: grid row blockIdx.y takes instances blockIdx.y,
// blockIdx.y + gridDim.y, ... (one each unless there are more than 65535),
// and its CTAs stride over an instance four voxels per thread
// (seg_gather4 / seg_store4).
__global__ void __launch_bounds__(256) k_seg_all(DevPool P, uint8_t* const* __restrict__ out) {
  for (int inst = blockIdx.y; inst < P.ninst; inst += gridDim.y) {
    uint8_t* src = out[2 * inst];
    uint8_t* snk = out[2 * inst + 1];
    if (src || snk) seg_instance(P, inst, src, snk, blockIdx.x, gridDim.x);
  }
}

// `bytes` of a table to the device.  A copy of pageable memory may end after
// cudaMemcpy returns, and the solve's stream may not be ordered behind it, so
// its end is waited for.
static int copy_table(Pool& p, void* dst, const void* src, size_t bytes) {
  cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
  if (e != cudaSuccess) p.untracked = true;
  CGC_CUDA(e);
  return CGC_OK;
}

// The device tables start with null pointers: outputs need not be bound for
// every instance, and the blocks hold whatever their last handle left there.
static int ensure_tables(Pool& p) {
  if (!p.d_out) {
    p.in_ptrs.assign(8 * (size_t)p.ninst, nullptr);
    p.out_ptrs.assign(2 * (size_t)p.ninst, nullptr);
    const size_t in = sizeof(int32_t*) * p.in_ptrs.size(), out = sizeof(uint8_t*) * p.out_ptrs.size();
    if (!p.d_in) {
      if (int rc = dev_alloc(p.device, &p.d_in, in)) return rc;
    }
    if (int rc = copy_table(p, p.d_in, p.in_ptrs.data(), in)) return rc;
    uint8_t** d_out = nullptr;
    if (int rc = dev_alloc(p.device, &d_out, out)) return rc;
    if (int rc = copy_table(p, d_out, p.out_ptrs.data(), out)) {
      if (p.idle()) dev_free(d_out);
      return rc;
    }
    p.d_out = d_out;  // both tables are there
  }
  return CGC_OK;
}

int pool_bind_inputs(Pool& p, int inst, const int32_t* capS, const int32_t* capT, const int32_t* const fwd[3],
                     const int32_t* const bwd[3]) {
  if (inst < 0 || inst >= p.ninst || !capS || !capT) return fail(CGC_ERR_ARG, "bind_inputs: bad arguments");
  int rc = ensure_tables(p);
  if (rc) return rc;
  const int32_t** ip = p.in_ptrs.data() + 8 * (size_t)inst;
  ip[0] = capS;
  ip[1] = capT;
  for (int a = 0; a < 3; ++a) {
    ip[2 + a] = fwd ? fwd[a] : nullptr;
    ip[5 + a] = bwd ? bwd[a] : (fwd ? fwd[a] : nullptr);
  }
  if ((rc = copy_table(p, p.d_in + 8 * (size_t)inst, ip, 8 * sizeof(int32_t*)))) return rc;
  return ok();
}

int pool_bind_outputs(Pool& p, int inst, uint8_t* source_side, uint8_t* sink_side) {
  if (inst < 0 || inst >= p.ninst) return fail(CGC_ERR_ARG, "bind_outputs: bad instance");
  int rc = ensure_tables(p);
  if (rc) return rc;
  p.out_ptrs[2 * (size_t)inst] = source_side;
  p.out_ptrs[2 * (size_t)inst + 1] = sink_side;
  if ((rc = copy_table(p, p.d_out + 2 * (size_t)inst, p.out_ptrs.data() + 2 * (size_t)inst, 2 * sizeof(uint8_t*))))
    return rc;
  return ok();
}

// Enqueues one batched solve on `stream` without synchronising the host.
int pool_enqueue(Pool& p, const cgc_options* opts, int64_t* flows_dev, cudaStream_t stream) {
  if (!p.d_out) return fail(CGC_ERR_STATE, "enqueue: no device inputs bound");
  if (p.pending) return fail(CGC_ERR_STATE, "enqueue: a host-path solve of this handle was not waited for");
  for (int i = 0; i < p.ninst; ++i)
    if (!p.in_ptrs[8 * (size_t)i]) return fail(CGC_ERR_STATE, "enqueue: instance without bound inputs");
  const cgc_options o = resolve_options(opts);
  if (o.learned > 0 || o.trace_cycles > 0) {  // buffers and weights before anything is queued
    int rc = ensure_sched(p, o.learned > 0, o.trace_cycles);
    if (rc) return rc;
  }
  DevPool& d = p.dp;
  NoteUse note(p);
  note.waited = stream != p.stream;  // the handle's own capture queues nothing
  CGC_CUDA(cudaMemsetAsync(p.back_dev, 0, p.back_bytes, stream));  // statistics, barrier, error word, flows
  k_put_all<<<d.nruns, 128, 0, stream>>>(d, p.d_in);
  note_launch();
  const SolveParams prm = solve_params(o, opts);
  if (int rc = launch_solve(d, prm, p.device, p.sms, stream)) return rc;
  bool any_out = false;
  for (uint8_t* q : p.out_ptrs) any_out = any_out || q;
  if (any_out) {
    const unsigned gx = (unsigned)std::min<int64_t>(std::max<int64_t>((p.maxN + 8191) / 8192, 1), 4096);
    k_seg_all<<<dim3(gx, (unsigned)std::min(p.ninst, 65535)), 256, 0, stream>>>(d, p.d_out);
    note_launch();
  }
  if (flows_dev) CGC_CUDA(cudaMemcpyAsync(flows_dev, d.flow, (size_t)p.ninst * 8, cudaMemcpyDeviceToDevice, stream));
  CGC_CUDA(cudaGetLastError());
  for (auto& u : p.uploaded) u = 0;
  p.solved = true;
  p.seg_valid = false;
  return ok();
}

// Waits for the last enqueued or replayed batch; reports device errors and
// refreshes flows and statistics.
int pool_wait(Pool& p, cudaStream_t stream) {
  NoteUse note(p);
  if (int rc = queue_back(p, stream)) return rc;
  CGC_CUDA(cudaStreamSynchronize(stream));
  note.waited = true;
  if (int rc = read_back(p, "batch")) return rc;
  return ok();
}

int pool_graph_create(Pool& p, const cgc_options* opts, int64_t* flows_dev) {
  if (p.graph_exec) { cudaGraphExecDestroy(p.graph_exec); p.graph_exec = nullptr; }
  if (p.graph) { cudaGraphDestroy(p.graph); p.graph = nullptr; }
  if (!p.cap_stream) CGC_CUDA(cudaStreamCreateWithFlags(&p.cap_stream, cudaStreamNonBlocking));
  {
    const cgc_options o = resolve_options(opts);
    if (o.learned > 0 || o.trace_cycles > 0) {  // allocations and weight uploads stay outside the capture
      int rc = ensure_sched(p, o.learned > 0, o.trace_cycles);
      if (rc) return rc;
    }
  }
  CGC_CUDA(cudaStreamBeginCapture(p.cap_stream, cudaStreamCaptureModeThreadLocal));
  const long long before = g_launches.load();
  int rc = pool_enqueue(p, opts, flows_dev, p.cap_stream);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(p.cap_stream, &g);
  g_launches.store(before);  // capture does not launch anything
  if (rc) { if (g) cudaGraphDestroy(g); return rc; }
  if (e != cudaSuccess) return fail(CGC_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
  p.graph = g;
  CGC_CUDA(cudaGraphInstantiate(&p.graph_exec, p.graph, 0));
  size_t nodes = 0;
  CGC_CUDA(cudaGraphGetNodes(p.graph, nullptr, &nodes));
  p.graph_kernels = 0;
  std::vector<cudaGraphNode_t> all(nodes);
  CGC_CUDA(cudaGraphGetNodes(p.graph, all.data(), &nodes));
  for (auto nd : all) {
    cudaGraphNodeType ty;
    CGC_CUDA(cudaGraphNodeGetType(nd, &ty));
    if (ty == cudaGraphNodeTypeKernel) ++p.graph_kernels;
  }
  return ok();
}

int pool_graph_launch(Pool& p) {
  if (!p.graph_exec) return fail(CGC_ERR_STATE, "graph_launch: no graph (call cgc_batch_graph_create)");
  if (p.pending) return fail(CGC_ERR_STATE, "graph_launch: a host-path solve of this handle was not waited for");
  NoteUse note(p);
  CGC_CUDA(cudaGraphLaunch(p.graph_exec, p.stream));
  for (int i = 0; i < p.graph_kernels; ++i) note_launch();
  for (auto& u : p.uploaded) u = 0;
  p.solved = true;
  p.seg_valid = false;
  return ok();
}

}  // namespace cgc

struct cgc_batch { cgc::Pool* p; };

extern "C" {

int cgc_batch_bind_inputs(cgc_batch* b, int32_t i, const int32_t* capS, const int32_t* capT,
                          const int32_t* const fwd[3], const int32_t* const bwd[3]) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_bind_inputs(*b->p, i, capS, capT, fwd, bwd);
}
int cgc_batch_bind_outputs(cgc_batch* b, int32_t i, uint8_t* source_side, uint8_t* sink_side) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_bind_outputs(*b->p, i, source_side, sink_side);
}
int cgc_batch_enqueue(cgc_batch* b, const cgc_options* opts, int64_t* flows_dev) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_enqueue(*b->p, opts, flows_dev, b->p->stream);
}
int cgc_batch_graph_create(cgc_batch* b, const cgc_options* opts, int64_t* flows_dev) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_graph_create(*b->p, opts, flows_dev);
}
int cgc_batch_graph_launch(cgc_batch* b) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  return cgc::pool_graph_launch(*b->p);
}
int cgc_batch_wait(cgc_batch* b, int64_t* flows) {
  if (!b) return cgc::fail(CGC_ERR_ARG, "null batch");
  int rc = cgc::pool_wait(*b->p, b->p->stream);
  if (rc) return rc;
  if (flows) std::memcpy(flows, b->p->flows.data(), b->p->flows.size() * 8);
  return cgc::ok();
}

}  // extern "C"
