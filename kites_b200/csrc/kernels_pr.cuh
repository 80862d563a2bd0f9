// kernels_pr.cuh -- FP32 PageRank, one Jacobi step at a time:
// y[v] = sum_{u->v} x[u] with x[u] = PR(u) / outdeg(u), then
// PR(v) = (1-d)/n + d y[v].
//
// A step is bound by its gathers of x (the SMs issue about 270 G random
// 4-byte reads/s; the 8 streamed bytes an edge take a third of that time at
// HBM speed), so the work is laid out by edge: a warp takes kPrChunk
// consecutive edges, 256 at a time, eight a lane, all eight gathers of a lane
// in flight.  A row lying inside one lane is summed there; rows crossing lanes
// meet over the warp, rows crossing windows in the warp's carry.  A finished
// row becomes its next x at once; only the rows that cross chunks go through
// y, added there atomically and finished by k_pr_join.  R-MAT of 2^21 vertices
// and 2^25 edges, 20 steps: 4.26 ms for the row-chunk walk this replaces (211
// us a step with one window of 32 edges in flight a warp, 9 us for its
// separate update), 2.71 ms here (136 us a step, 247 G gathers/s).  The
// relative error against 64 bits is no larger: 8.8e-8 here and 9.5e-8 there,
// means of four graphs of that size; single runs of either lie between 7e-8 and
// 1.2e-7, as the order of the atomics has it.
#pragma once
#include "kernels_sweep.cuh"

namespace kites_internal {

constexpr uint64_t kPrChunk = 2048;   // edges of a warp's chunk
constexpr int kPrMinBlocks = 5;

template <typename OffT>
struct pr_args {
  const OffT *R;
  const uint32_t *C;
  const uint32_t *rowid;    // row of every edge
  uint64_t m, n_real;
  const float *x;           // this step's x
  float *x_next;
  float *y;                 // partial sums of rows that cross chunks, else 0
  const float *inv_out;
  float *pr;                // last step: the ranks, else null
  float base, damping;
};

template <typename OffT>
__device__ __forceinline__ void pr_finish(const pr_args<OffT> &a, uint32_t row, float sum) {
  if (row >= a.n_real) return;
  const float r = a.base + a.damping * sum;
  a.x_next[row] = r * a.inv_out[row];
  if (a.pr) a.pr[row] = r;
}

// Sum of `p` over this lane's run of equal owners, valid at the run's head;
// *last receives the run's last lane.
__device__ __forceinline__ float run_sum_to_head(float p, uint32_t owner, bool *head,
                                                 uint32_t *last) {
  const uint32_t rm = run_mask(owner, head);
  const uint32_t end = 31u - __clz(rm);
  const uint32_t lane = lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const float q = __shfl_down_sync(kFull, p, d);
    if (lane + d <= end) p += q;
  }
  *last = end;
  return p;
}

template <typename OffT>
__global__ void __launch_bounds__(kSweepThreads, kPrMinBlocks) k_pr_pull(pr_args<OffT> a) {
  const uint32_t lane = lane_id();
  const uint64_t warps = (uint64_t)gridDim.x * (kSweepThreads / 32);
  for (uint64_t begin = (((uint64_t)blockIdx.x * kSweepThreads + threadIdx.x) >> 5) * kPrChunk;
       begin < a.m; begin += warps * kPrChunk) {
    const uint64_t end = min(begin + kPrChunk, a.m);
    // A first row that started in the previous chunk is shared with it.
    const uint32_t before = begin ? a.rowid[begin - 1] : kNoRow;
    const uint32_t shared_row = before == a.rowid[begin] ? before : kNoRow;
    auto done = [&](uint32_t row, float sum) {
      if (row == shared_row) atomicAdd(a.y + row, sum);
      else pr_finish(a, row, sum);
    };
    uint32_t c_row = kNoRow;   // the row the previous window ended in
    float c_sum = 0.f;
    for (uint64_t w0 = begin; w0 < end; w0 += kWindowEdges) {
      const uint64_t e0 = w0 + (uint64_t)lane * kEdgesPerThread;
      uint32_t row[kEdgesPerThread], src[kEdgesPerThread];
      float val[kEdgesPerThread];
      load_edges8(a.rowid, a.C, e0, end, row, src);
#pragma unroll
      for (int k = 0; k < kEdgesPerThread; ++k) val[k] = row[k] != kNoRow ? a.x[src[k]] : 0.f;
      // Runs of equal row along the lane's edges: its first, its last, and
      // those between, which are whole rows.
      float p = val[0], first = 0.f;
      bool many = false;
#pragma unroll
      for (int k = 1; k < kEdgesPerThread; ++k) {
        const bool same = row[k] == row[k - 1];
        if (!same) {
          if (!many) first = p;
          else pr_finish(a, row[k - 1], p);
          many = true;
        }
        p = same ? p + val[k] : val[k];
      }
      const uint32_t f_row = row[0], l_row = many ? row[kEdgesPerThread - 1] : kNoRow;
      if (!many) first = p;
      // Lanes in one row: the run's sum at its head, with the last row of the
      // lane before it when that is the same one.
      bool head;
      uint32_t last;
      float sum = run_sum_to_head(first, f_row, &head, &last);
      const uint32_t up_row = __shfl_up_sync(kFull, l_row, 1);
      const float up_sum = __shfl_up_sync(kFull, p, 1);
      const uint32_t down_row = __shfl_down_sync(kFull, f_row, 1);
      const bool lane31_many = __shfl_sync(kFull, many ? 1u : 0u, 31) != 0u;
      const bool open = last == 31u && !lane31_many;   // goes on in the next window
      if (lane == 0) {
        if (c_row == f_row) sum += c_sum;
        else if (c_row != kNoRow) done(c_row, c_sum);
      } else if (head && up_row == f_row) {
        sum += up_sum;
      }
      if (head && !open && f_row != kNoRow) done(f_row, sum);
      if (many && lane < 31u && l_row != kNoRow && l_row != down_row) pr_finish(a, l_row, p);
      // The carry: lane 31's last row, or the run that reaches it.
      const uint32_t open_head = __ballot_sync(kFull, head && open);
      if (open_head) {
        const uint32_t h = __ffs(open_head) - 1;
        c_row = __shfl_sync(kFull, f_row, h);
        c_sum = __shfl_sync(kFull, sum, h);
      } else {
        c_row = __shfl_sync(kFull, l_row, 31);
        c_sum = __shfl_sync(kFull, p, 31);
      }
    }
    if (lane == 0 && c_row != kNoRow) {
      if (end < a.m && a.rowid[end] == c_row) atomicAdd(a.y + c_row, c_sum);
      else done(c_row, c_sum);
    }
  }
}

// Finishes the rows that cross chunks, each by the chunk it ends in.
template <typename OffT>
__global__ void k_pr_join(pr_args<OffT> a) {
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x + 1; c * kPrChunk < a.m;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t begin = c * kPrChunk;
    const uint32_t row = a.rowid[begin];
    if (a.rowid[begin - 1] != row || (uint64_t)a.R[row + 1] > begin + kPrChunk) continue;
    const float sum = a.y[row];
    a.y[row] = 0.f;
    pr_finish(a, row, sum);
  }
}

// First step's x and what no step writes: the second buffer's rows without
// in-edges (base / outdeg from the first step on) and their ranks.
template <typename OffT>
__global__ void k_pr_init(pr_args<OffT> a, const uint32_t *__restrict__ out_deg, uint64_t n,
                          uint32_t iterations, float *__restrict__ inv_out,
                          float *__restrict__ x0, float *__restrict__ x1,
                          float *__restrict__ pr) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = out_deg[v];
    const float inv = d ? 1.0f / (float)d : 0.0f;
    const bool real = v < a.n_real;
    const float r = real ? 1.0f / (float)a.n_real : 0.0f;
    // A row of zero in-edges: base + damping * 0.
    const float r1 = real ? a.base + a.damping * 0.0f : 0.0f;
    inv_out[v] = inv;
    x0[v] = r * inv;
    x1[v] = r1 * inv;
    a.y[v] = 0.0f;
    pr[v] = iterations && real ? r1 : r;
  }
}

// After the first step: the first buffer's rows without in-edges.
template <typename OffT>
__global__ void k_pr_empty(pr_args<OffT> a, float *__restrict__ x0) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < a.n_real;
       v += (uint64_t)gridDim.x * blockDim.x)
    if (a.R[v] == a.R[v + 1]) x0[v] = (a.base + a.damping * 0.0f) * a.inv_out[v];
}

}  // namespace kites_internal
