// Which token goes where: the stable order by destination rank and the count per destination, for every local rank in one
// launch.  A general sort and a histogram per rank took several launches and a host synchronisation each, which is what
// bounded a dispatch: dispatch and combine of 4 x 4099 tokens of width 2048, 891 us with them, 196 us with this kernel.
// There are at most kMaxRanks destinations, so a counting sort with warp votes does it in two passes over the
// destinations: a token's place is the tokens of smaller destinations, those of the same destination in earlier warps'
// segments and those before it in the own segment.
//
// One block per rank: what bounds it is latency.  A warp has the destinations of eight rows under way at once and the segments' counts are
// scanned by warps (one row after the other, and one thread for the scan: 8.3 us for 4 x 4099 tokens, now 7.1; 262144
// tokens to two ranks 245, now 186).  With all ranks in this process the counts go to pinned host memory, which the host polls, instead
// of through a copy that it waits for: dispatch and combine of 4 x 4099 tokens 89.3 -> 77.7 us.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "common.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kWarps = 32;
constexpr int kRows = 8;   // rows of 32 tokens whose destinations a warp has under way at once

__global__ void __launch_bounds__(32 * kWarps) route_kernel(const __grid_constant__ RouteParams P) {
  const int r = (int)blockIdx.x, p = P.p;
  const long long* dest = P.dest[r];
  const size_t n = P.n[r];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a warp's segment is a whole number of rows of 32 tokens
  const size_t rows = (n + 31) / 32, per = (rows + kWarps - 1) / kWarps;
  const size_t lo = warp * per, hi = lo + per < rows ? lo + per : rows;
  __shared__ unsigned long long count[kMaxRanks][kWarps];   // tokens per destination and segment, then first places
  __shared__ unsigned long long total[kMaxRanks];
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();

  // Destinations of kRows rows at once (-1 behind the last token); the first ones stay in registers for the second pass.
  auto fetch = [&](int* d, size_t row) {
    long long v[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const size_t t = (row + i) * 32 + lane;
      v[i] = row + i < hi && t < n ? dest[t] : -1;
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const bool token = row + i < hi && (row + i) * 32 + lane < n;
      d[i] = v[i] >= 0 && v[i] < p ? (int)v[i] : (token ? p : -1);   // p: none of the ranks
    }
  };
  int kept[kRows];
  fetch(kept, lo);
  unsigned long long mine = 0;   // lane d counts destination d
  bool wrong = false;
  auto tally = [&](const int* d) {
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      wrong |= d[i] == p;
      for (int k = 0; k < p; ++k) {
        const unsigned votes = __ballot_sync(0xffffffffu, d[i] == k);
        if ((int)lane == k) mine += __popc(votes);
      }
    }
  };
  tally(kept);
  for (size_t row = lo + kRows; row < hi; row += kRows) {
    int d[kRows];
    fetch(d, row);
    tally(d);
  }
  if (lane < p) count[lane][warp] = mine;
  if (wrong) bad = 1;
  __syncthreads();
  // warp k scans destination k's segments
  unsigned long long before = 0;
  if ((int)warp < p) {
    const unsigned long long c = count[warp][lane];
    unsigned long long sum = c;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, sum, o);
      if ((int)lane >= o) sum += up;
    }
    before = sum - c;
    if (lane == 31) total[warp] = sum;
  }
  __syncthreads();
  if ((int)warp < p) {
    unsigned long long first = 0;
    for (int k = 0; k < (int)warp; ++k) first += total[k];
    count[warp][lane] = first + before;
  }
  if ((int)threadIdx.x < p) {
    const long long c = bad ? -1 : (long long)total[threadIdx.x];
    P.counts[(size_t)r * p + threadIdx.x] = c;
    if (P.host_counts) P.host_counts[(size_t)r * p + threadIdx.x] = c;
  }
  if (P.host_counts && warp == 0) {   // the host reads on while the places are still being written
    __threadfence_system();
    __syncwarp();
    if (lane == 0) st_release_sys((uint64_t*)P.host_flags + r, P.host_seq);
  }
  __syncthreads();
  if (bad) return;
  unsigned long long next = lane < p ? count[lane][warp] : 0;
  auto place = [&](const int* d, size_t row) {
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      if (row + i >= hi) break;
      const unsigned same = __match_any_sync(0xffffffffu, d[i]);
      const unsigned long long first = __shfl_sync(0xffffffffu, next, d[i] < 0 ? 0 : d[i]);
      if (d[i] >= 0) P.order[r][first + __popc(same & ((1u << lane) - 1))] = (long long)((row + i) * 32 + lane);
      for (int k = 0; k < p; ++k) {
        const unsigned votes = __ballot_sync(0xffffffffu, d[i] == k);
        if ((int)lane == k) next += __popc(votes);
      }
    }
  };
  place(kept, lo);
  for (size_t row = lo + kRows; row < hi; row += kRows) {
    int d[kRows];
    fetch(d, row);
    place(d, row);
  }
}

}  // namespace

void launch_route(const RouteParams& P, int local_ranks, cudaStream_t stream) {
  route_kernel<<<local_ranks, 32 * kWarps, 0, stream>>>(P);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
