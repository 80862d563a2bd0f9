// kernels_build.cuh -- kernels of graph construction: edge keys, what a sorted
// key list says (sources, rows, row ends), the row of every edge, and the
// transposition's unpacking.  All are streams of a few bytes an edge, four or
// eight edges a thread with 16-byte accesses; what they replace searched a row
// per edge (588 us for 2^24 edges against 42 us here), counted degrees with one
// atomic per edge (398 us; row ends cost nothing beside the stream that finds
// them) and gathered the transposed rows and weights at random (406 us; they
// now travel with the sort).  With keys of 2 log2(n) bits (five radix passes
// instead of seven at 2^20 vertices) and device input read in place, an edge
// list of 2^24 edges built and answered one SSSP in 2.35 ms against 3.72.
#pragma once
#include "kernels.cuh"

namespace kites_internal {

constexpr int kBuildPer = 4;   // edges per thread

// keys[i] = dst << bits | src; any endpoint >= n sets *bad.  kVec: src and dst
// are 16-byte aligned.
template <typename KeyT, bool kVec>
__global__ void __launch_bounds__(256)
    k_edge_keys(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint64_t m,
                uint64_t n, int bits, KeyT *__restrict__ keys, uint32_t *bad) {
  const uint64_t i0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * kBuildPer;
  if (i0 >= m) return;
  uint32_t s[kBuildPer], d[kBuildPer];
  const uint32_t cnt = (uint32_t)min((uint64_t)kBuildPer, m - i0);
  if (kVec && cnt == kBuildPer) {
    const uint4 a = __ldcs(reinterpret_cast<const uint4 *>(src + i0));
    const uint4 b = __ldcs(reinterpret_cast<const uint4 *>(dst + i0));
    s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
    d[0] = b.x; d[1] = b.y; d[2] = b.z; d[3] = b.w;
  } else {
#pragma unroll
    for (uint32_t k = 0; k < kBuildPer; ++k) {
      s[k] = k < cnt ? src[i0 + k] : 0u;
      d[k] = k < cnt ? dst[i0 + k] : 0u;
    }
  }
  uint32_t top = 0;
#pragma unroll
  for (uint32_t k = 0; k < kBuildPer; ++k) {
    top = max(top, max(s[k], d[k]));
    if (k < cnt) keys[i0 + k] = (KeyT)d[k] << bits | (KeyT)s[k];
  }
  if (top >= n) atomicOr(bad, 1u);
}

// first[r] and last[r] (one past) of every row r among m sorted row numbers;
// rows that do not occur keep what they hold (0).
__device__ __forceinline__ void mark_ends(uint64_t i, uint64_t m, uint32_t row, uint32_t before,
                                          uint32_t *first, uint32_t *last) {
  if (i == 0 || before != row) {
    first[row] = (uint32_t)i;
    if (i) last[before] = (uint32_t)i;
  }
  if (i + 1 == m) last[row] = (uint32_t)m;
}

// Sorted keys -> C, the row of every edge, the rows' ends.
template <typename KeyT>
__global__ void __launch_bounds__(256)
    k_split_keys(const KeyT *__restrict__ keys, uint64_t m, int bits, uint32_t *__restrict__ C,
                 uint32_t *__restrict__ rowid, uint32_t *__restrict__ first,
                 uint32_t *__restrict__ last) {
  const uint64_t i0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * kBuildPer;
  if (i0 >= m) return;
  const KeyT mask = ((KeyT)1 << bits) - 1;
  uint32_t before = i0 ? (uint32_t)(keys[i0 - 1] >> bits) : 0u;
  uint32_t c[kBuildPer], r[kBuildPer];
  const uint32_t cnt = (uint32_t)min((uint64_t)kBuildPer, m - i0);
#pragma unroll
  for (uint32_t k = 0; k < kBuildPer; ++k) {
    const KeyT key = k < cnt ? keys[i0 + k] : 0;
    c[k] = (uint32_t)(key & mask);
    r[k] = (uint32_t)(key >> bits);
    if (k < cnt) {
      mark_ends(i0 + k, m, r[k], before, first, last);
      before = r[k];
    }
  }
  if (cnt == kBuildPer) {
    *reinterpret_cast<uint4 *>(C + i0) = make_uint4(c[0], c[1], c[2], c[3]);
    *reinterpret_cast<uint4 *>(rowid + i0) = make_uint4(r[0], r[1], r[2], r[3]);
  } else {
    for (uint32_t k = 0; k < cnt; ++k) {
      C[i0 + k] = c[k];
      rowid[i0 + k] = r[k];
    }
  }
}

// Row lengths from their ends, as OffT for the scan (and as uint32 if deg).
template <typename OffT>
__global__ void k_row_lengths(const uint32_t *__restrict__ first, const uint32_t *__restrict__ last,
                              uint64_t n, OffT *__restrict__ wide, uint32_t *__restrict__ deg) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = last[i] - first[i];
    wide[i] = (OffT)d;
    if (deg) deg[i] = d;
  }
}

// The row of every edge: one search for a thread's first edge, then along the
// row ends (again a search where many rows are empty).
template <typename OffT>
__global__ void __launch_bounds__(256)
    k_row_of_edge(const OffT *__restrict__ R, uint64_t n_rows, uint64_t n_edges,
                  uint32_t *__restrict__ row) {
  constexpr int kPer = 8;
  const uint64_t e0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * kPer;
  if (e0 >= n_edges) return;
  // Largest r in [lo, n_rows) with R[r] <= e.
  auto search = [&](uint64_t lo, uint64_t e) {
    uint64_t hi = n_rows;
    while (hi - lo > 1) {
      const uint64_t mid = (lo + hi) >> 1;
      if ((uint64_t)R[mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
  };
  uint64_t r = search(0, e0), end = (uint64_t)R[r + 1];
  uint32_t out[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const uint64_t e = e0 + k;
    if (e < n_edges && e >= end) {
      for (int step = 0; step < 4 && e >= end; ++step) end = (uint64_t)R[++r + 1];
      if (e >= end) {
        r = search(r, e);
        end = (uint64_t)R[r + 1];
      }
    }
    out[k] = (uint32_t)r;
  }
  if (e0 + kPer <= n_edges) {
    uint4 *to = reinterpret_cast<uint4 *>(row + e0);
    to[0] = make_uint4(out[0], out[1], out[2], out[3]);
    to[1] = make_uint4(out[4], out[5], out[6], out[7]);
  } else {
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (e0 + k < n_edges) row[e0 + k] = out[k];
  }
}

// The transposition's payload (row << 32 | weight), and its keys (C) unless
// keys is null.  All arrays are 16-byte aligned.
__global__ void __launch_bounds__(256)
    k_pack_edges(const uint32_t *__restrict__ row, const uint32_t *__restrict__ C,
                 const uint32_t *__restrict__ E, uint64_t m, uint32_t *__restrict__ keys,
                 uint64_t *__restrict__ pay) {
  const uint64_t i0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * kBuildPer;
  if (i0 + kBuildPer <= m) {
    const uint4 r = *reinterpret_cast<const uint4 *>(row + i0);
    const uint4 w = *reinterpret_cast<const uint4 *>(E + i0);
    if (keys) *reinterpret_cast<uint4 *>(keys + i0) = *reinterpret_cast<const uint4 *>(C + i0);
    ulonglong2 *to = reinterpret_cast<ulonglong2 *>(pay + i0);
    to[0] = make_ulonglong2((uint64_t)r.x << 32 | w.x, (uint64_t)r.y << 32 | w.y);
    to[1] = make_ulonglong2((uint64_t)r.z << 32 | w.z, (uint64_t)r.w << 32 | w.w);
    return;
  }
  for (uint64_t i = i0; i < m; ++i) {
    if (keys) keys[i] = C[i];
    pay[i] = (uint64_t)row[i] << 32 | E[i];
  }
}

// Adds a 64-bit mix of every edge's number and weight to *sum, so that a weight
// changed in place shows.  A stream of 4 bytes an edge.
__global__ void __launch_bounds__(256)
    k_weight_sum(const uint32_t *__restrict__ E, uint64_t m, unsigned long long *sum) {
  unsigned long long x = 0;
  const uint64_t stride = (uint64_t)gridDim.x * 256;
  auto mix = [](uint64_t e, uint32_t w) {   // SplitMix64's finaliser (Steele et al. 2014)
    uint64_t z = (e << 32 ^ e >> 32) + w + 0x9E3779B97F4A7C15ull;
    z = (z ^ z >> 30) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ z >> 27) * 0x94D049BB133111EBull;
    return z ^ z >> 31;
  };
  const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  for (uint64_t i = t; i < m / 4; i += stride) {
    const uint4 w = __ldcs(reinterpret_cast<const uint4 *>(E) + i);
    x += mix(4 * i, w.x) + mix(4 * i + 1, w.y) + mix(4 * i + 2, w.z) + mix(4 * i + 3, w.w);
  }
  for (uint64_t e = m / 4 * 4 + t; e < m; e += stride) x += mix(e, E[e]);
  x = warp_sum_u64(x);
  if (lane_id() == 0 && x) atomicAdd(sum, x);
}

// Edges sorted by source -> outC, outE (PayT: row << 32 | weight, or the row
// alone and weights of 1) and the sources' row ends.
template <typename PayT>
__global__ void __launch_bounds__(256)
    k_unpack_edges(const uint32_t *__restrict__ key, const PayT *__restrict__ pay, uint64_t m,
                   uint32_t *__restrict__ outC, uint32_t *__restrict__ outE,
                   uint32_t *__restrict__ first, uint32_t *__restrict__ last) {
  const uint64_t i0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * kBuildPer;
  if (i0 >= m) return;
  uint32_t before = i0 ? key[i0 - 1] : 0u;
  uint32_t c[kBuildPer], w[kBuildPer];
  const uint32_t cnt = (uint32_t)min((uint64_t)kBuildPer, m - i0);
#pragma unroll
  for (uint32_t k = 0; k < kBuildPer; ++k) {
    if (k >= cnt) break;
    const PayT p = pay[i0 + k];
    c[k] = sizeof(PayT) == 8 ? (uint32_t)((uint64_t)p >> 32) : (uint32_t)p;
    w[k] = sizeof(PayT) == 8 ? (uint32_t)p : 1u;
    mark_ends(i0 + k, m, key[i0 + k], before, first, last);
    before = key[i0 + k];
  }
  if (cnt == kBuildPer) {
    *reinterpret_cast<uint4 *>(outC + i0) = make_uint4(c[0], c[1], c[2], c[3]);
    *reinterpret_cast<uint4 *>(outE + i0) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    for (uint32_t k = 0; k < cnt; ++k) {
      outC[i0 + k] = c[k];
      outE[i0 + k] = w[k];
    }
  }
}

}  // namespace kites_internal
