// frontier.cuh -- what the host side needs of the single-launch frontier loop
// (kernels_frontier.cuh, compiled in frontier.cu).
#pragma once
#include "engine.cuh"

namespace kites_internal {

constexpr uint32_t kSeg = 256;   // out-edges of one queue entry, at most

// How the run starts.
enum : int {
  kSeedSource = 0,   // V = INF but 0 at `source`
  kSeedFinite = 1,   // the caller's V and frontier: every vertex below INF is
                     // queued, after a check that the out-edges whose target is
                     // outside the frontier are already satisfied
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
