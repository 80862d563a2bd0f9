// grid_wait.h -- the word on which the CTAs of one kernel meet, for the kernel
// and for host tests of its arithmetic.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define KITES_HD __host__ __device__ __forceinline__
#else
#define KITES_HD inline
#endif

namespace kites_internal {

// Arrivals since the launch.  They are never taken back, so that a meeting is
// one addition and one wait; bit 63 says that a CTA gave up waiting.  One CTA
// on each of 148 SMs adds 148 a meeting, and a run has a meeting or more per
// level of the graph: 31 bits would be full after 14.5 M levels, which a path
// of 2^24 vertices has, 63 bits outlast any run.
using grid_word = unsigned long long;
constexpr grid_word kGridGaveUp = 1ull << 63;

// Whether a CTA's wait for its `met`-th meeting (counted from 1) is over.
KITES_HD bool grid_met(grid_word seen, grid_word met, uint32_t ctas) {
  return seen >= met * ctas;
}
KITES_HD bool grid_failed(grid_word seen) { return (seen & kGridGaveUp) != 0; }

}  // namespace kites_internal
