// Grid of an operation straight between the buffers of ranks on one GPU; plain C++, so that it is tested without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>

namespace Al {
namespace internal {
namespace device {

struct LocalGrid {
  unsigned x, y;   ///< CTAs of a job, jobs at a time
};

/**
 * `jobs` jobs of up to `tiles` tiles of one warp each: one warp per tile, or at most max_ctas CTAs in all (0: no limit), fewer jobs at
 * a time than there are where these are fewer.
 */
inline LocalGrid local_grid(size_t tiles, int jobs, int max_ctas, int threads) {
  const size_t per = (size_t)threads / 32, want = std::max<size_t>(1, (tiles + per - 1) / per);
  const int y = max_ctas > 0 ? std::min(jobs, max_ctas) : jobs;
  return {(unsigned)std::min<size_t>(want, max_ctas > 0 ? (size_t)(max_ctas / y) : size_t{0x7fffffff}), (unsigned)y};
}

}  // namespace device
}  // namespace internal
}  // namespace Al
