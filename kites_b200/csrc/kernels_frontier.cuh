// kernels_frontier.cuh -- the single-launch frontier loop of the plain
// strategy: one cooperative kernel runs a whole SSSP, BFS or min-label run,
// from the initial values to the fixed point.
//
// What bounded the loop it replaces: six kernels an iteration (three gated
// pulls, the activation, the clear and the check), 20-25 us of launches and
// bitmap scans however small the frontier, and pulls over every in-edge of
// every activated row, when only the in-edges from the changed set can lower
// it.  Here the changed set is a queue whose out-edges are relaxed with
// atomicMin, an iteration ends with one grid barrier, and the only edges read
// are those of changed vertices.
//
// An iteration.  A warp takes a batch of queue entries, lays their out-edges
// over its lanes (a row start found from one ballot and one OR a window) and
// tests several a lane against V; the few that would lower V are collected
// per warp and applied together, so that the atomics, the queue bits and the
// appends run with full warps.  Rows above kSeg edges are queued by segment,
// which spreads a hub over the grid.  Two shapes: short iterations (up to
// kShort out-edges), where a step is a chain of dependent L2 accesses and a
// warp does one small batch; wide ones, bound by the 1 gather/clk an SM
// issues (148 x 1.9 GHz = 270 G gathers/s measured for random 4-byte reads),
// where warps draw batches from a ticket counter and keep the next window's
// edges loading under the current one's gathers.
//
// Order of work (near and far lists as in Davidson et al., "Work-efficient
// parallel GPU methods for single-source shortest paths", 2014; the bottom-up
// BFS step is that of Beamer et al., "Direction-optimizing breadth-first
// search", 2012).  With weights, candidates at or above a threshold are put
// aside (the far list) until everything below it has settled; the threshold
// then moves by a step that follows the work: small iterations double it (an
// iteration costs its latency whatever it holds), large ones halve it (less
// is relaxed twice).  Any order reaches the same fixed point.
//
// Exactness.  Between iterations every edge (u, v) either has u in the queue
// or on the far list or satisfies V[v] <= comp(V[u], w): a lowered u is queued
// by the thread that lowered it first, values only fall, and V[u] is read when
// the entry is processed.  The initial state must satisfy the same (the
// callers' seeds do; kSeedFinite is checked).  Needs comp(INF) = INF, so the
// wrap-around add does not come here.
//
// Whole calls, per-iteration loop -> this kernel (one B200, PLAIN): R-MAT
// 7,115 vertices and 103,689 edges 501 -> 199 us (kites_process, values to and
// from the host); R-MAT 2^22 vertices, 2^26 edges SSSP 2.49 -> 1.01 ms (4.22
// with another source); grid 512 x 512 22.9 -> 5.9 ms; BFS on 60,013 vertices
// and 983,040 edges 379 -> 107 us; min labels of a symmetrised R-MAT of 2^20
// vertices and 2^25 edges 720 -> 281 us; 64 R-MAT graphs in one run (768,000
// vertices, 12.3 M edges) 1.61 -> 0.72 ms.
#pragma once
#include "common.cuh"
#include "frontier.cuh"
#include "grid_wait.h"

namespace kites_internal {

constexpr int kFrThreads = 512;               // one CTA per SM, 128 registers a thread
constexpr int kFrWarps = kFrThreads / 32;
constexpr uint32_t kShort = 160u << 10;       // out-edges of a short iteration, at most
// BFS turns bottom-up when the frontier has more than a third of the out-edges
// not walked yet, and more than a short iteration's.  A third, a quarter, an
// eighth and a twentieth took 399, 416, 448 and 518 us on R-MAT of 2^22 vertices
// and 2^26 edges, 482, 480, 566 and 567 on an Erdos-Renyi graph of that size
// (549 and 680 us with pushes only).
constexpr uint32_t kBottomShare = 3;
constexpr uint32_t kLongRow = 1024;           // in-edges one warp looks through, at most
constexpr int kShortFlight = 2, kWideFlight = 8;  // edges in flight per lane
constexpr int kShortCand = 2, kWideCand = 4;      // candidates a lane applies together
constexpr uint32_t kCandRoom = 32 * (kWideCand + kWideFlight);
constexpr uint32_t kFlush = 128;              // queue entries a warp appends together
constexpr uint32_t kFarFlush = 96;
constexpr uint32_t kBatchEdges = 1024;        // out-edges of a wide batch, about
constexpr uint64_t kFrItems = 512;            // vertices + out-edges that earn a CTA
constexpr uint64_t kSplitEdges = 16u << 20;   // see split_pays()
constexpr uint32_t kWideLow = 768u << 10, kWideHigh = 4u << 20;

// Counters of one step: the queues it consumes and the tickets taken from
// them.  A slot is filled during one step, read during the next and cleared
// during the one after, so no CTA ever reads what another may already be
// changing.
struct frontier_slot {
  uint32_t qn, bn;               // whole rows, segments of long rows
  uint32_t ticket, bticket;
  unsigned long long edges;      // out-edges of both queues
  unsigned long long row_edges;  // out-edges of the whole rows
  uint32_t minv, pad;            // smallest value a split kept
};

// Device state of one run (zeroed by the host before the launch).  far_n is a
// ring like the slots: a split reads far_n[far_c], leaves its count in the
// next one and clears the one after that.
struct frontier_ctl {
  grid_word barrier;
  uint32_t violated, pad;
  frontier_slot slot[3];
  uint32_t far_n[3], finite;           // finite: in a sample of the caller's values
  unsigned long long wsum;             // sampled weights
  unsigned long long active, relaxed, updated;
};

template <typename OffT>
struct frontier_args {
  const OffT *R, *outR;   // in- and out-rows
  const uint32_t *C;
  const uint32_t *outC, *outE, *out_deg;
  uint32_t *V;
  uint64_t n, m;
  uint2 *big[2];          // segments of rows above kSeg: (vertex, segment)
  uint32_t *q[2];         // other queued vertices
  uint32_t *far[2];       // vertices put aside
  uint32_t *bits;         // [queued, parity 0 | parity 1 | far], nwords each
  uint64_t nwords;
  uint32_t *frontier;     // the graph's frontier and changed bitmaps, 4 * nwords
                          // words: empty after the run (kSeedFinite: the first
                          // nwords are the caller's frontier)
  uint32_t source;
  int seed;
  uint32_t polls;         // looks at the barrier before a CTA gives up
  frontier_ctl *ctl;
  frontier_result *out;
};

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ grid_word ld_acquire_u64(const grid_word *p) {
  grid_word v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add(grid_word *p, grid_word x) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}

// Sum over the warp: one REDUX while the lanes' values are small.
__device__ __forceinline__ unsigned long long warp_sum_fast(unsigned long long x) {
  if (!__any_sync(kFull, x >> 26)) return __reduce_add_sync(kFull, (uint32_t)x);
  return warp_sum_u64(x);
}

struct frontier_smem {
  uint2 cand[kFrWarps][kCandRoom];
  uint32_t near[kFrWarps][kFlush + 32];
  uint32_t far[kFrWarps][kFarFlush + 32];
};

template <int OP, typename OffT>
struct frontier_run {
  static constexpr bool kW = op_reads_weights<OP>();
  const frontier_args<OffT> &a;
  frontier_smem &sm;
  const uint32_t lane, wib;
  // Uniform over the grid.
  uint32_t ring = 0;      // slot[ring] is consumed, the one after it filled
  grid_word met = 0;      // grid barriers passed
  uint32_t qp = 0;        // q[qp], big[qp] are consumed, queued bits parity qp
  uint32_t fc = 0;        // far list in use
  uint32_t far_c = 0;     // its count: ctl->far_n[far_c]
  uint32_t thr = kInf, delta = kInf, bucket_rounds = 0, rounds = 0;
  unsigned long long bucket_edges = 0, spent = 0;
  // Per warp: entries in its buffers.
  uint32_t n_cand = 0, n_near = 0, n_far = 0;
  // Per lane: out-edges queued for the next step, and those of whole rows.
  unsigned long long next_edges = 0, next_row_edges = 0, n_relaxed = 0;
  uint32_t n_active = 0, n_updated = 0, min_keep = kInf;

  __device__ frontier_run(const frontier_args<OffT> &args, char *s)
      : a(args), sm(*reinterpret_cast<frontier_smem *>(s)), lane(lane_id()),
        wib(threadIdx.x >> 5) {}

  __device__ uint32_t *queued(uint32_t p) const { return a.bits + (uint64_t)p * a.nwords; }
  __device__ uint32_t *far_bits() const { return a.bits + 2 * a.nwords; }
  static __device__ uint32_t ring_after(uint32_t i) { return i == 2u ? 0u : i + 1u; }
  __device__ uint32_t far_next() const { return ring_after(far_c); }
  __device__ frontier_slot *cur() const { return &a.ctl->slot[ring]; }
  __device__ frontier_slot *next() const { return &a.ctl->slot[ring_after(ring)]; }

  // Called by warp 0 after a CTA barrier: arrives and waits for the grid.
  // False when the wait ran out or another CTA gave up.
  __device__ bool meet() {
    ++met;
    bool failed = false;
    if (lane == 0) {
      red_release_add(&a.ctl->barrier, 1u);
      uint32_t spins = 0;
      grid_word seen;
      while (!grid_met(seen = ld_acquire_u64(&a.ctl->barrier), met, gridDim.x)) {
        if (++spins > 64u) __nanosleep(spins > 4096u ? 256 : 32);
        if (spins > a.polls) {
          seen = atomicOr(&a.ctl->barrier, kGridGaveUp) | kGridGaveUp;
          break;
        }
      }
      failed = grid_failed(seen);
    }
    return !__any_sync(kFull, failed);
  }

  // ---- appends (called by whole warps) ------------------------------------

  // Appends the newest `near` and `far` staged entries (the rest stay where
  // they are); the far ones to list buf, counted in far_n[cnt].
  __device__ void flush(uint32_t near, uint32_t far, uint32_t buf, uint32_t cnt) {
    __syncwarp();
    // Both counters' round trips at once.
    uint32_t qb = 0, fb = 0;
    if (lane == 0) {
      if (near) qb = atomicAdd(&next()->qn, near);
      if (far) fb = atomicAdd(&a.ctl->far_n[cnt], far);
    }
    qb = __shfl_sync(kFull, qb, 0);
    fb = __shfl_sync(kFull, fb, 0);
    n_near -= near;
    n_far -= far;
    for (uint32_t i = lane; i < near; i += 32) a.q[qp ^ 1u][qb + i] = sm.near[wib][n_near + i];
    for (uint32_t i = lane; i < far; i += 32) a.far[buf][fb + i] = sm.far[wib][n_far + i];
    __syncwarp();
  }
  // Queues rows of deg > kSeg edges by segment.
  __device__ void push_big(bool on, uint32_t v, uint32_t deg) {
    uint32_t big = __ballot_sync(kFull, on);
    if (!big) return;
    const uint32_t segs = on ? deg / kSeg + (deg % kSeg ? 1u : 0u) : 0u;
    const uint32_t incl = warp_inclusive_scan(segs);
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&next()->bn, incl);
    base = __shfl_sync(kFull, base, 31) + incl - segs;
    while (big) {
      const uint32_t src = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bv = __shfl_sync(kFull, v, src), bs = __shfl_sync(kFull, segs, src),
                     at = __shfl_sync(kFull, base, src);
      for (uint32_t i = lane; i < bs; i += 32) a.big[qp ^ 1u][at + i] = make_uint2(bv, i);
    }
  }
  // Queues v (deg out-edges, its bit already set) where `near`, puts it on the
  // far list where `far`.
  __device__ void push(bool near, bool far, uint32_t v, uint32_t deg, uint32_t buf,
                       uint32_t cnt) {
    near = near && deg != 0;
    const bool one = near && deg <= kSeg;
    if (near) next_edges += deg;
    if (one) next_row_edges += deg;
    const uint32_t before = (1u << lane) - 1u;
    const uint32_t ones = __ballot_sync(kFull, one);
    if (one) sm.near[wib][n_near + __popc(ones & before)] = v;
    n_near += __popc(ones);
    push_big(near && !one, v, deg);
    if (kW) {
      const uint32_t fars = __ballot_sync(kFull, far);
      if (far) sm.far[wib][n_far + __popc(fars & before)] = v;
      n_far += __popc(fars);
    }
    if (n_near >= kFlush || n_far >= kFarFlush) flush(n_near, n_far, buf, cnt);
  }

  // Ends a step: what the warps still hold is flushed, the CTA's sums go to
  // the next slot, the grid meets, and the next slot is read back into *sl.
  __device__ bool end_step(uint32_t far_buf, uint32_t far_cnt, frontier_slot *sl,
                           uint32_t *far_count) {
    __shared__ unsigned long long s_edges[kFrWarps], s_rows[kFrWarps];
    __shared__ uint32_t s_min[kFrWarps], s_ok;
    if (n_near | n_far) flush(n_near, n_far, far_buf, far_cnt);
    const unsigned long long e = warp_sum_fast(next_edges), r = warp_sum_fast(next_row_edges);
    const uint32_t mn = __reduce_min_sync(kFull, min_keep);
    next_edges = next_row_edges = 0;
    min_keep = kInf;
    if (lane == 0) {
      s_edges[wib] = e;
      s_rows[wib] = r;
      s_min[wib] = mn;
    }
    __syncthreads();
    if (wib == 0) {
      const bool in = lane < (uint32_t)kFrWarps;
      const uint32_t l = in ? lane : 0u;
      const unsigned long long sum = warp_sum_fast(in ? s_edges[l] : 0ull),
                               rows = warp_sum_fast(in ? s_rows[l] : 0ull);
      const uint32_t smin = __reduce_min_sync(kFull, s_min[l]);
      if (lane == 0) {
        if (sum) atomicAdd(&next()->edges, sum);
        if (rows) atomicAdd(&next()->row_edges, rows);
        if (smin != kInf) atomicMin(&next()->minv, smin);
        if (blockIdx.x == 0) {
          // The slot of the previous step: nobody reads it any more.
          frontier_slot *old = &a.ctl->slot[ring_after(ring_after(ring))];
          old->qn = old->bn = old->ticket = old->bticket = 0;
          old->edges = old->row_edges = 0;
          old->minv = kInf;
        }
      }
      __syncwarp();
      const bool ok = meet();
      if (lane < sizeof(frontier_slot) / 4)
        reinterpret_cast<uint32_t *>(sl)[lane] =
            __ldcg(reinterpret_cast<const uint32_t *>(next()) + lane);
      if (lane == 31) *far_count = __ldcg(&a.ctl->far_n[far_cnt]);
      if (lane == 0) s_ok = ok;
    } else {
      ++met;
    }
    __syncthreads();
    ring = ring_after(ring);
    return s_ok != 0u;
  }

  // ---- an iteration ---------------------------------------------------------

  // Applies the warp's newest candidates, kPer a lane, while more than `keep`
  // are left.
  template <int kPer>
  __device__ void apply(uint32_t keep) {
    while (n_cand > keep) {
      __syncwarp();
      const uint32_t take = min(n_cand, 32u * kPer);
      uint32_t v[kPer], nd[kPer], old[kPer], deg[kPer];
      n_cand -= take;
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const uint32_t i = lane + 32 * k;
        nd[k] = kInf;
        old[k] = deg[k] = 0;
        v[k] = 0;
        if (i < take) {
          const uint2 c = sm.cand[wib][n_cand + i];
          v[k] = c.x;
          nd[k] = c.y;
          old[k] = atomicMin(a.V + v[k], nd[k]);
        }
      }
      // The bit decides who queues a vertex, and only that lane looks up its
      // degree.
      bool near[kPer], far[kPer];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const bool low = nd[k] < old[k];
        near[k] = low && nd[k] < thr;
        far[k] = low && !near[k];
        if (low) {
          n_updated += 1;
          const uint32_t bit = 1u << (v[k] & 31u);
          uint32_t *set = near[k] ? queued(qp ^ 1u) : far_bits();
          // (a short iteration looks without waiting for the bit)
          if (kPer <= kShortCand) deg[k] = near[k] ? a.out_deg[v[k]] : 0u;
          if (atomicOr(set + (v[k] >> 5), bit) & bit) near[k] = far[k] = false;
        }
      }
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (kPer > kShortCand) deg[k] = near[k] ? a.out_deg[v[k]] : 0u;
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (__any_sync(kFull, near[k] || far[k]))
          push(near[k], far[k], v[k], deg[k], fc, far_c);
      __syncwarp();
    }
  }

  // One batch: lane l holds row part [b, b + cnt) of a vertex at value d
  // (cnt = 0 past the batch's end).
  template <bool kCheck, int kFlight, int kPer>
  __device__ void relax_batch(OffT b, uint32_t cnt, uint32_t d) {
    const uint32_t incl = warp_inclusive_scan(cnt);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t ex = incl - cnt;
    const OffT off = b - (OffT)ex;      // edge of position i: off + i
    const bool valid = cnt != 0;        // a prefix of the lanes
    const uint32_t upto = kFull >> (31u - lane);
    if (!kCheck && lane == 0) n_relaxed += total;
    uint32_t c[kFlight], w[kFlight], du[kFlight], cn[kFlight], wn[kFlight], dn[kFlight];
    // Lane i of a 32-edge window finds its row from the row starts that fall
    // into the window (one ballot, one OR over the warp).
    auto load = [&](uint32_t t0, uint32_t (&lc)[kFlight], uint32_t (&lw)[kFlight],
                    uint32_t (&ld)[kFlight]) {
#pragma unroll
      for (int k = 0; k < kFlight; ++k) {
        const uint32_t p0 = t0 + k * 32, i = p0 + lane;
        lc[k] = kInf;
        ld[k] = kInf;
        lw[k] = 0;
        if (p0 >= total) continue;   // whole warps
        const uint32_t before = __popc(__ballot_sync(kFull, valid && ex < p0));
        const uint32_t at = ex - p0;
        const uint32_t heads = __reduce_or_sync(kFull, valid && at < 32u ? 1u << at : 0u);
        const uint32_t j = (before + __popc(heads & upto) - 1u) & 31u;
        const OffT e = __shfl_sync(kFull, off, j) + (OffT)i;
        ld[k] = __shfl_sync(kFull, d, j);
        if (i < total) {
          lc[k] = __ldcs(a.outC + e);
          if (kW) lw[k] = __ldcs(a.outE + e);
        }
      }
    };
    if (total) load(0, c, w, du);
    for (uint32_t t0 = 0; t0 < total; t0 += 32 * kFlight) {
      uint32_t pv[kFlight];
      // A stale V (this SM's L1) only ever reads too high: the atomicMin
      // decides.
#pragma unroll
      for (int k = 0; k < kFlight; ++k) pv[k] = c[k] != kInf ? a.V[c[k]] : 0u;
      if (t0 + 32 * kFlight < total) load(t0 + 32 * kFlight, cn, wn, dn);
#pragma unroll
      for (int k = 0; k < kFlight; ++k) {
        const uint32_t nd = nbr_comp<OP>(du[k], w[k]);
        const bool low = nd < pv[k];
        if constexpr (kCheck) {
          if (low && !((a.frontier[c[k] >> 5] >> (c[k] & 31u)) & 1u)) a.ctl->violated = 1u;
        } else {
          const uint32_t m = __ballot_sync(kFull, low);
          if (m) {
            if (low)
              sm.cand[wib][n_cand + __popc(m & ((1u << lane) - 1u))] = make_uint2(c[k], nd);
            n_cand += __popc(m);
          }
        }
        c[k] = cn[k];
        w[k] = wn[k];
        du[k] = dn[k];
      }
      if (!kCheck && n_cand >= 32u * kPer) apply<kPer>(32u * kPer - 1u);
    }
  }

  // Lane's part of entry i of the segments (kBig) or the whole rows.
  template <bool kBig, bool kCheck>
  __device__ void take(uint32_t i, OffT *b, uint32_t *cnt, uint32_t *d) {
    uint32_t u, seg = 0;
    if (kBig) {
      const uint2 en = __ldcg(a.big[qp] + i);
      u = en.x;
      seg = en.y;
    } else {
      u = __ldcg(a.q[qp] + i);
    }
    *d = __ldcg(a.V + u);
    const OffT r0 = a.outR[u], r1 = a.outR[u + 1];
    *b = r0 + (OffT)seg * kSeg;
    const OffT left = r1 - *b;
    *cnt = left < (OffT)kSeg ? (uint32_t)left : kSeg;
    if (!kCheck && seg == 0u) {
      atomicAnd(queued(qp) + (u >> 5), ~(1u << (u & 31u)));
      n_active += 1;
    }
  }

  // log2 of the whole rows that hold about `edges` out-edges, at most a lane
  // each.
  __device__ uint32_t rows_of(const frontier_slot &sl, uint32_t edges) const {
    const float rows = (float)edges * (float)sl.qn / fmaxf((float)sl.row_edges, 1.f);
    return 31u - __clz((uint32_t)fminf(fmaxf(rows, 1.f), 32.f));
  }

  // A short iteration: every warp takes at most a segment or some rows with
  // two windows of out-edges, all at once.  (Letting a warp go on with the
  // vertices it queued itself before the grid meets relaxed so much out of
  // order that R-MAT of 7,115 vertices took 323 us against 208 and the 512 x
  // 512 grid gained nothing.)
  __device__ void short_push(const frontier_slot &sl) {
    const uint32_t log = rows_of(sl, 64 * kShortFlight);
    const uint32_t rows = 1u << log, jobs = sl.bn + ((sl.qn + rows - 1u) >> log);
    // Neighbouring jobs go to different SMs.
    for (uint32_t job = wib * gridDim.x + blockIdx.x; job < jobs; job += gridDim.x * kFrWarps) {
      uint32_t cnt = 0, d = kInf;
      OffT b = 0;
      if (job < sl.bn) {
        if (lane == 0) take<true, false>(job, &b, &cnt, &d);
      } else {
        const uint32_t i = ((job - sl.bn) << log) + lane;
        if (lane < rows && i < sl.qn) take<false, false>(i, &b, &cnt, &d);
      }
      relax_batch<false, kShortFlight, kShortCand>(b, cnt, d);
    }
    apply<kShortCand>(0);
  }

  // A wide iteration's walk over one queue.  kCheck only looks for an
  // unsatisfied edge whose target is outside the caller's frontier.
  template <bool kBig, bool kCheck>
  __device__ void walk(uint32_t count, uint32_t *ticket, uint32_t batch, uint32_t taken) {
    const uint32_t warps = gridDim.x * kFrWarps;
    // Neighbouring batches go to different SMs; the first `taken` warps have
    // segments to do and come last.
    const uint32_t gw = wib * gridDim.x + blockIdx.x;
    uint64_t base = (uint64_t)(gw >= taken ? gw - taken : gw + warps - taken) * batch;
    const uint64_t first = (uint64_t)warps * batch;
    while (base < count) {
      uint32_t after = 0;
      if (lane == 0 && first < count) after = atomicAdd(ticket, batch);
      uint32_t cnt = 0, d = kInf;
      OffT b = 0;
      if (lane < batch && base + lane < count)
        take<kBig, kCheck>((uint32_t)base + lane, &b, &cnt, &d);
      relax_batch<kCheck, kWideFlight, kWideCand>(b, cnt, d);
      if (first >= count) break;
      base = first + __shfl_sync(kFull, after, 0);
    }
  }
  template <bool kCheck>
  __device__ void wide_push(const frontier_slot &sl) {
    const uint32_t warps = gridDim.x * kFrWarps;
    // Rows a batch: kBatchEdges' worth, fewer where that leaves warps without.
    uint32_t log = rows_of(sl, kBatchEdges);
    while (log && (uint64_t)warps << log > sl.qn) --log;
    walk<true, kCheck>(sl.bn, &cur()->bticket, sl.bn > 8 * warps ? 4u : 1u, 0);
    walk<false, kCheck>(sl.qn, &cur()->ticket, 1u << log, min(sl.bn, warps));
    if (!kCheck) apply<kWideCand>(0);
  }

  // All CTAs meet inside a step.
  __device__ bool mid_sync() {
    __shared__ uint32_t s_go;
    __syncthreads();
    if (wib == 0) {
      const bool ok = meet();
      if (lane == 0) s_go = ok;
    } else {
      ++met;
    }
    __syncthreads();
    return s_go != 0u;
  }

  // BFS with the frontier at `level`: instead of relaxing its out-edges, every
  // vertex not reached yet looks for an in-neighbour at `level`.  Where the
  // frontier holds much of what is left to explore, most rows end at one of
  // their first edges.  A lane looks at its vertex's first kProbe in-edges,
  // the warp at a row's rest; what is longer than kLongRow is left to the
  // whole grid by segment (in big[qp], which this step does not read).
  // V is read past L1: a stale value would hide a parent.
  __device__ bool bottom_up(uint32_t level) {
    constexpr uint32_t kProbe = 8, kWindows = 4;
    const uint64_t stride = (uint64_t)gridDim.x * kFrThreads;
    const uint64_t t0 = (uint64_t)blockIdx.x * kFrThreads + threadIdx.x;
    for (uint64_t w = t0; w < a.nwords; w += stride) queued(qp)[w] = 0u;
    // Whether one of in-edges [r, e) comes from `level` (whole warps).
    auto scan = [&](OffT r, OffT e) {
      for (OffT i = r; i < e; i += 32 * kWindows) {
        bool hit = false;
#pragma unroll
        for (uint32_t k = 0; k < kWindows; ++k) {
          const OffT j = i + (OffT)(k * 32 + lane);
          if (j < e) hit |= __ldcg(a.V + a.C[j]) == level;
        }
        if (lane == 0) n_relaxed += min((unsigned long long)(e - i), 32ull * kWindows);
        if (__any_sync(kFull, hit)) return true;
      }
      return false;
    };
    for (uint64_t v0 = t0 & ~31ull; v0 < a.n; v0 += stride) {
      const uint64_t v = v0 + lane;
      OffT r = 0, e = 0;
      if (v < a.n && __ldcg(a.V + v) == kInf) {
        r = a.R[v];
        e = a.R[v + 1];
      }
      if (!__any_sync(kFull, r < e)) continue;
      bool hit = false;
      for (uint32_t p = 0; p < kProbe; p += 4) {
        uint32_t u[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          u[k] = !hit && r + (OffT)k < e ? a.C[r + (OffT)k] : kInf;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          if (u[k] == kInf) continue;
          hit |= __ldcg(a.V + u[k]) == level;
          n_relaxed += 1;
        }
        if (!hit) r = e - r > (OffT)4 ? r + (OffT)4 : e;
      }
      const bool more = !hit && r < e;
      uint32_t rest = __ballot_sync(kFull, more && e - r <= (OffT)kLongRow);
      while (rest) {
        const uint32_t src = __ffs(rest) - 1;
        rest &= rest - 1;
        const bool found = scan(__shfl_sync(kFull, r, src), __shfl_sync(kFull, e, src));
        if (lane == src) hit = found;
      }
      for (uint32_t far = __ballot_sync(kFull, more && e - r > (OffT)kLongRow); far;
           far &= far - 1) {
        const uint32_t src = __ffs(far) - 1;
        const OffT len = __shfl_sync(kFull, e - r, src);
        const uint32_t segs = (uint32_t)((len + (OffT)(kLongRow - 1)) / (OffT)kLongRow);
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&cur()->bticket, segs);
        at = __shfl_sync(kFull, at, 0);
        for (uint32_t i = lane; i < segs; i += 32)
          a.big[qp][at + i] = make_uint2((uint32_t)(v0 + src), i);
      }
      uint32_t deg = 0;
      if (hit) {
        a.V[v] = level + 1u;
        deg = a.out_deg[v];
        n_updated += 1;
      }
      if (__any_sync(kFull, hit)) push(hit, false, (uint32_t)v, deg, fc, far_c);
    }
    if (!mid_sync()) return false;
    const uint32_t segs = __ldcg(&cur()->bticket);
    for (uint32_t i = wib * gridDim.x + blockIdx.x; i < segs; i += gridDim.x * kFrWarps) {
      const uint2 en = __ldcg(a.big[qp] + i);
      // One lane looks: other CTAs may be lowering the word, and the warp has to
      // take one way with the votes behind it.
      const uint32_t now = lane == 0 ? __ldcg(a.V + en.x) : 0u;
      if (__shfl_sync(kFull, now, 0) != kInf) continue;
      const OffT r = a.R[en.x] + (OffT)kProbe + (OffT)en.y * kLongRow, e = a.R[en.x + 1];
      if (!scan(r, e - r > (OffT)kLongRow ? r + (OffT)kLongRow : e)) continue;
      bool mine = false;
      if (lane == 0) mine = atomicMin(a.V + en.x, level + 1u) == kInf;
      if (lane == 0 && mine) n_updated += 1;
      push(mine, false, en.x, a.out_deg[en.x], fc, far_c);
    }
    return true;
  }

  // Queues every vertex for which on(v).
  template <class Pred>
  __device__ void seed_all(Pred on) {
    const uint64_t stride = (uint64_t)gridDim.x * kFrThreads;
    for (uint64_t v0 = ((uint64_t)blockIdx.x * kFrThreads + threadIdx.x) & ~31ull; v0 < a.n;
         v0 += stride) {
      const uint64_t v = v0 + lane;
      const bool take = v < a.n && on((uint32_t)v);
      const uint32_t deg = take ? a.out_deg[v] : 0u;
      const uint32_t bits = __ballot_sync(kFull, deg != 0);
      if (!bits) continue;
      if (lane == 0) queued(qp ^ 1u)[v0 >> 5] = bits;
      push(deg != 0, false, (uint32_t)v, deg, fc, far_c);
    }
  }

  // Moves the far entries below the new threshold into the queue; entries
  // below the old one were queued when they fell there.
  __device__ void split(uint32_t count, uint32_t old_thr) {
    const uint64_t stride = (uint64_t)gridDim.x * kFrThreads;
    for (uint64_t i0 = ((uint64_t)blockIdx.x * kFrThreads + threadIdx.x) & ~31ull; i0 < count;
         i0 += stride) {
      const uint64_t i = i0 + lane;
      uint32_t v = 0, d = 0, deg = 0;
      bool near = false, keep = false;
      if (i < count) {
        v = __ldcg(a.far[fc] + i);
        d = __ldcg(a.V + v);
        keep = d >= thr;
        near = !keep && d >= old_thr;
        if (!keep) atomicAnd(far_bits() + (v >> 5), ~(1u << (v & 31u)));
        if (near) {
          deg = a.out_deg[v];
          if (deg) atomicOr(queued(qp ^ 1u) + (v >> 5), 1u << (v & 31u));
        }
        if (keep) min_keep = min(min_keep, d);
      }
      push(near, keep, v, deg, fc ^ 1u, far_next());
    }
  }

  // Whether a weighted run is ordered by threshold: it relaxes less and takes
  // more iterations for it, so it pays where there is much to relax.  Unordered
  // -> ordered, means of 2-4 sources: Erdos-Renyi 16 edges a vertex, 2^24 edges
  // 1.04 -> 0.72 ms, 2^26 3.56 -> 1.60; R-MAT 2^24 0.54 -> 0.53, 2^26 1.45 -> 1.41;
  // smaller ones lose (R-MAT 2^20 0.18 -> 0.22, 2^23 0.41 -> 0.45; Erdos-Renyi 2^20
  // 0.25 -> 0.29).  Graphs with few edges a vertex are deep, and each wave that
  // arrives late relaxes again all that lies behind it: 2^21 vertices and 2^23
  // edges 0.93 -> 0.68, grids of 9 M vertices 126 -> 77, 4.2 M 44 -> 36, 1.05 M
  // 14.5 -> 13.1; the small ones among them lose a little (grid of 2^18 vertices
  // 5.9 -> 6.3, 2^18 vertices and 2^20 edges 0.27 -> 0.35).
  __device__ bool split_pays() const { return a.m >= kSplitEdges || a.m < 8 * a.n; }
  __device__ uint32_t step_up(uint32_t t) const { return t > kInf - delta ? kInf : t + delta; }
  // The threshold's step, from the mean iteration since its last move: an
  // iteration costs its latency up to some 10^5 edges and its edges beyond
  // some 10^6.  The few iterations in which a run grows out of its source say
  // nothing yet.
  __device__ void adapt() {
    if (delta != kInf && bucket_rounds) {
      const unsigned long long mean = bucket_edges / bucket_rounds;
      if (mean > kWideHigh) {
        if (delta > 1) delta >>= 1;
      } else if (mean < kWideLow && (bucket_rounds > 3 || spent > a.m / 4)) {
        delta = delta > kInf / 4 ? kInf / 2 : delta * 2;
      }
    }
    bucket_edges = 0;
    bucket_rounds = 0;
  }

  // ---- the run ---------------------------------------------------------------

  // First values, empty bitmaps, a sample of the weights.
  __device__ void init() {
    const uint64_t stride = (uint64_t)gridDim.x * kFrThreads;
    const uint64_t t0 = (uint64_t)blockIdx.x * kFrThreads + threadIdx.x;
    if (a.seed == kSeedSource) {
      // n is a multiple of 128.
      const uint64_t sv = a.source >> 2;
      for (uint64_t i = t0; i < a.n / 4; i += stride) {
        uint4 x = make_uint4(kInf, kInf, kInf, kInf);
        if (i == sv)
          (a.source & 2u ? (a.source & 1u ? x.w : x.z) : (a.source & 1u ? x.y : x.x)) = 0u;
        reinterpret_cast<uint4 *>(a.V)[i] = x;
      }
      // The queue of one (its bit, only a mark against a second append, may
      // stay clear).
      if (blockIdx.x == 0 && wib == 0)
        push(lane == 0, false, a.source, a.out_deg[a.source], fc, far_c);
    } else if (a.seed == kSeedLabels) {
      // Any in-neighbour's id is a label that reaches v; rows are sorted as a
      // rule, so the first is the least.
      for (uint64_t v = t0; v < a.n; v += stride) {
        const OffT r = a.R[v];
        const uint32_t id = (uint32_t)v;
        a.V[v] = r < a.R[v + 1] ? min(id, a.C[r]) : id;
      }
    }
    for (uint64_t w = t0; w < 3 * a.nwords; w += stride) a.bits[w] = 0u;
    if (a.seed != kSeedFinite)
      for (uint64_t w = t0; w < 4 * a.nwords; w += stride) a.frontier[w] = 0u;
    if (kW && threadIdx.x < 32) {
      // 32 weights a CTA, spread evenly over the edges.
      const uint64_t at =
          ((uint64_t)blockIdx.x * 32 + lane) * a.m / ((uint64_t)gridDim.x * 32);
      unsigned long long wt = at < a.m ? a.outE[at] : 0u;
      wt = warp_sum_u64(wt);
      if (lane == 0 && wt) atomicAdd(&a.ctl->wsum, wt);
    }
    if (a.seed == kSeedFinite && a.m > kGivenEdges && threadIdx.x < 32) {
      // 32 vertices a CTA, to leave a state with too many finite ones at once.
      const uint64_t at =
          ((uint64_t)blockIdx.x * 32 + lane) * a.n / ((uint64_t)gridDim.x * 32);
      const uint32_t some = __popc(__ballot_sync(kFull, a.V[at] != kInf));
      if (lane == 0 && some) atomicAdd(&a.ctl->finite, some);
    }
    if (blockIdx.x == 0 && threadIdx.x < 3) a.ctl->slot[threadIdx.x].minv = kInf;
  }

  // Sums the lanes' counts into ctl; CTA 0 writes the result.
  __device__ void finish(bool violated, bool gave_up) {
    __shared__ unsigned long long s_sum[3][kFrWarps];
    const unsigned long long x = warp_sum_fast(n_active), y = warp_sum_fast(n_relaxed),
                             z = warp_sum_fast(n_updated);
    __syncthreads();
    if (lane == 0) {
      s_sum[0][wib] = x;
      s_sum[1][wib] = y;
      s_sum[2][wib] = z;
    }
    __syncthreads();
    if (wib != 0) return;
    const bool in = lane < (uint32_t)kFrWarps;
    const uint32_t l = in ? lane : 0u;
    const unsigned long long sx = warp_sum_u64(in ? s_sum[0][l] : 0ull),
                             sy = warp_sum_u64(in ? s_sum[1][l] : 0ull),
                             sz = warp_sum_u64(in ? s_sum[2][l] : 0ull);
    if (lane == 0) {
      if (sx) atomicAdd(&a.ctl->active, sx);
      if (sy) atomicAdd(&a.ctl->relaxed, sy);
      if (sz) atomicAdd(&a.ctl->updated, sz);
    }
    __syncwarp();
    // A CTA that gave up left its flag in the barrier's word, where every later
    // meeting finds it, so CTA 0 needs no word of its own to tell the host.
    if (!gave_up) gave_up = !meet();
    if (blockIdx.x == 0 && lane == 0) {
      a.out->iterations = rounds;
      a.out->active = __ldcg(&a.ctl->active);
      a.out->relaxed = __ldcg(&a.ctl->relaxed);
      a.out->updated = __ldcg(&a.ctl->updated);
      a.out->violated = violated ? 1u : 0u;
      a.out->error = gave_up ? kErrWait : 0u;
    }
  }

  __device__ void run() {
    __shared__ frontier_slot s_slot;
    __shared__ uint32_t s_far;
    auto end = [&](uint32_t buf, uint32_t cnt) { return end_step(buf, cnt, &s_slot, &s_far); };
    // Step 0: everything in place, the single source queued.
    init();
    if (!end(fc, far_c)) return finish(false, true);
    if (kW && a.m && split_pays()) {
      const unsigned long long mean =
          __ldcg(&a.ctl->wsum) / ((unsigned long long)gridDim.x * 32u);
      const unsigned long long d = 4ull * mean * a.n / a.m;
      delta = d < 1 ? 1u : d > kInf / 2 ? kInf / 2 : (uint32_t)d;
      thr = delta;
    }
    if (a.seed == kSeedFinite && a.m > kGivenEdges &&
        __ldcg(&a.ctl->finite) * a.m / (gridDim.x * 32ull) > kGivenEdges)
      return finish(true, false);
    // Step 1 queues what other runs start from.
    if (a.seed == kSeedZeros) {
      seed_all([&](uint32_t v) { return __ldcg(a.V + v) == 0u; });
    } else if (a.seed == kSeedFinite) {
      seed_all([&](uint32_t v) { return __ldcg(a.V + v) != kInf; });
    } else if (a.seed == kSeedLabels) {
      // The label of a vertex's label reaches it too (whichever values the
      // others have got by now).  On R-MAT most labels are final after this,
      // and the iteration over every edge lowers few: 467 -> 281 us for the
      // symmetrised graph of 2^20 vertices and 2^25 edges.
      seed_all([&](uint32_t v) {
        const uint32_t l = __ldcg(a.V + v), ll = __ldcg(a.V + l);
        if (ll < l) atomicMin(a.V + v, ll);
        return true;
      });
    }
    if (a.seed != kSeedSource && !end(fc, far_c)) return finish(false, true);
    qp ^= 1u;
    if (a.seed == kSeedFinite) {
      // The caller's state: an out-edge of a finite vertex that its target
      // does not satisfy must lead into the caller's frontier, else the
      // iteration of process() would not relax it and the host runs that.
      const frontier_slot sl = s_slot;
      if (sl.edges > 4 * kGivenEdges) return finish(true, false);   // the sample missed
      wide_push<true>(sl);
      if (blockIdx.x == 0 && threadIdx.x == 0) {   // the queues stay, under the next slot
        frontier_slot *c = next();
        c->qn = sl.qn;
        c->bn = sl.bn;
        c->edges = sl.edges;
        c->row_edges = sl.row_edges;
      }
      if (!end(fc, far_c)) return finish(false, true);
      if (ld_acquire_u32(&a.ctl->violated)) return finish(true, false);
      const uint64_t stride = (uint64_t)gridDim.x * kFrThreads;
      for (uint64_t w = (uint64_t)blockIdx.x * kFrThreads + threadIdx.x; w < a.nwords; w += stride)
        a.frontier[w] = 0u;
    }
    for (;;) {
      const frontier_slot &sl = s_slot;
      if (sl.edges == 0) {
        // Nothing queued, so the far list's count stands still.
        const uint32_t count = s_far;
        if (count == 0) break;
        adapt();
        const uint32_t old_thr = thr;
        thr = step_up(sl.minv != kInf ? max(sl.minv, thr) : thr);
        split(count, old_thr);
        if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->far_n[far_c ? far_c - 1u : 2u] = 0;
        far_c = far_next();
        if (!end(fc ^ 1u, far_c)) return finish(false, true);
        fc ^= 1u;
      } else {
        ++rounds;
        ++bucket_rounds;
        bucket_edges += sl.edges;
        spent += sl.edges;
        if (OP == OP_BFS && a.seed != kSeedFinite && sl.edges > kShort &&
            sl.edges > (a.m + sl.edges - spent) / kBottomShare) {
          if (!bottom_up(rounds - 1u)) return finish(false, true);
        } else if (sl.edges <= kShort) {
          short_push(sl);
        } else {
          wide_push<false>(sl);
        }
        if (!end(fc, far_c)) return finish(false, true);
      }
      qp ^= 1u;
    }
    finish(false, false);
  }
};

template <int OP, typename OffT>
__global__ void __launch_bounds__(kFrThreads, 1)
    k_frontier_run(const __grid_constant__ frontier_args<OffT> a) {
  extern __shared__ __align__(16) char fr_smem[];
  frontier_run<OP, OffT> r(a, fr_smem);
  r.run();
}

}  // namespace kites_internal
