// frontier.cu -- launches of the single-launch frontier loop.
#include "frontier.cuh"

#include <algorithm>
#include <mutex>

#include "kernels_frontier.cuh"

namespace kites_internal {

// Segments of rows above kSeg edges: at most one short one per such row.
static uint64_t frontier_segments(const kites_graph *g) { return 2 * (g->m / kSeg) + 1; }

size_t frontier_bytes(const kites_graph *g, size_t *queues) {
  *queues = (sizeof(frontier_ctl) + 255) / 256 * 256;
  return *queues + 2 * frontier_segments(g) * 8 + 4 * g->n * 4 + 3 * g->nwords * 4;
}

namespace {

// The grid waits for its own CTAs, one on every SM, so two such kernels must
// not each hold a part of the chip: engines of other threads wait here.  (The
// kernel fills the chip; side by side they would only take turns.)
std::mutex &device_lock(int device) {
  static std::mutex locks[64];
  return locks[device & 63];
}

template <int OP, typename OffT>
int launch(kites_graph *g, int seed, uint32_t source, frontier_result *out, float *ms) {
  kites_engine *eng = g->eng;
  cudaStream_t s = eng->stream;
  size_t queues;
  frontier_bytes(g, &queues);
  frontier_args<OffT> a{};
  a.outR = (const OffT *)g->outR;
  a.outC = g->outC;
  a.R = (const OffT *)g->R;
  a.C = g->C;
  a.outE = g->outE;
  a.out_deg = g->out_deg;
  a.V = (uint32_t *)g->V;
  a.n = g->n;
  a.m = g->m;
  a.big[0] = (uint2 *)((char *)g->fr_mem + queues);
  a.big[1] = a.big[0] + frontier_segments(g);
  a.q[0] = (uint32_t *)(a.big[1] + frontier_segments(g));
  a.q[1] = a.q[0] + g->n;
  a.far[0] = a.q[1] + g->n;
  a.far[1] = a.far[0] + g->n;
  a.bits = a.far[1] + g->n;
  a.nwords = g->nwords;
  a.frontier = g->bitmaps;
  a.source = source;
  a.seed = seed;
  a.polls = eng->wait_polls;
  a.ctl = (frontier_ctl *)g->fr_mem;
  // The kernel writes its result to the engine's pinned scratch, behind the
  // run counters other loops read back there.
  frontier_result *res = (frontier_result *)((char *)eng->pinned + 2048);
  a.out = res;
  const size_t smem = sizeof(frontier_smem);
  KITES_CUDA_TRY(cudaFuncSetAttribute(k_frontier_run<OP, OffT>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const uint64_t want = (g->n + g->m) / kFrItems + 1;
  const unsigned grid = (unsigned)std::min<uint64_t>(want, eng->sm_count);
  std::lock_guard<std::mutex> hold(device_lock(eng->device));
  KITES_CUDA_TRY(cudaMemsetAsync(a.ctl, 0, sizeof(frontier_ctl), s));
  KITES_CUDA_TRY(cudaEventRecord(eng->ev0, s));
  void *args[] = {&a};
  KITES_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_frontier_run<OP, OffT>, dim3(grid),
                                             dim3(kFrThreads), args, smem, s));
  KITES_CUDA_TRY(cudaEventRecord(eng->ev1, s));
  KITES_CUDA_TRY(cudaStreamSynchronize(s));
  *out = *res;
  KITES_CUDA_TRY(cudaEventElapsedTime(ms, eng->ev0, eng->ev1));
  return KITES_OK;
}

template <typename OffT>
int launch_op(kites_graph *g, int op, int seed, uint32_t source, frontier_result *out,
              float *ms) {
  switch (op) {
    case OP_SSSP: return launch<OP_SSSP, OffT>(g, seed, source, out, ms);
    case OP_BFS: return launch<OP_BFS, OffT>(g, seed, source, out, ms);
    default: return launch<OP_CC, OffT>(g, seed, source, out, ms);
  }
}

}  // namespace

int launch_frontier(kites_graph *g, int op, int seed, uint32_t source, frontier_result *out,
                    float *ms) {
  return g->off64 ? launch_op<uint64_t>(g, op, seed, source, out, ms)
                  : launch_op<uint32_t>(g, op, seed, source, out, ms);
}

}  // namespace kites_internal
