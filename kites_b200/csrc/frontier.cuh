// frontier.cuh -- what the host side needs of the single-launch frontier loop
// (kernels_frontier.cuh, compiled in frontier.cu).
#pragma once
#include "engine.cuh"

namespace kites_internal {

constexpr uint32_t kSeg = 256;   // out-edges of one queue entry, at most

// A caller's state is taken (kSeedFinite) while its finite vertices have about
// this many out-edges at the most, by a sample: they are walked twice, for the
// check and as the first iteration, however few of them the caller's frontier
// needs.  From settled values with 100 frontier bits a call took 58 us at 0.10 M
// out-edges, 94 at 1.6 M and 284 at 16.6 M (R-MAT); pulling the frontier's rows
// takes the per-iteration loop 80 us whatever the size.  A state that the sample
// in init() finds too large costs a launch and a wait, about 27 us.
constexpr uint32_t kGivenEdges = 1u << 20;

// How the run starts.
enum : int {
  kSeedSource = 0,   // V = INF but 0 at `source`
  kSeedFinite = 1,   // the caller's V and frontier: every vertex below INF is
                     // queued, after a check that they are few enough and that
                     // the out-edges whose target is outside the frontier are
                     // already satisfied
  kSeedZeros = 2,    // V is set up; the vertices at 0 are queued
  kSeedLabels = 3    // V[v] = v, every vertex queued
};

// Result of a run, written to pinned host memory.
struct frontier_result {
  unsigned long long iterations, active, relaxed, updated;
  uint32_t violated, error;
};

// Bytes of the buffers a run on g works in: the control block, then from
// *queues on two queues of row segments (8 bytes each), two of vertices (n
// words), two far lists (n words) and three bitmaps (g->nwords words).
size_t frontier_bytes(const kites_graph *g, size_t *queues);

// Enqueues the run on the engine's stream (g->fr_mem holds the buffers) and
// waits for it; *ms is its device time.
int launch_frontier(kites_graph *g, int op, int seed, uint32_t source, frontier_result *out,
                    float *ms);

}  // namespace kites_internal
