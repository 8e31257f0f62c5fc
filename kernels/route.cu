// Which token goes where: the stable order by destination rank and the count per destination, for every local rank in one
// launch.  A general sort and a histogram per rank took several launches and a host synchronisation each, which is what
// bounded a dispatch: dispatch and combine of 4 x 4099 tokens of width 2048, 891 us with them, 196 us with this kernel.
// There are at most kMaxRanks destinations, so a counting sort with warp votes does it in two passes over the
// destinations: a token's place is the tokens of smaller destinations, those of the same destination in earlier warps'
// segments and those before it in the own segment.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "common.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kWarps = 32;

__global__ void __launch_bounds__(32 * kWarps) route_kernel(const __grid_constant__ RouteParams P) {
  const int r = (int)blockIdx.x, p = P.p;
  const long long* dest = P.dest[r];
  const size_t n = P.n[r];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a warp's segment is a whole number of rows of 32 tokens
  const size_t rows = (n + 31) / 32, per = (rows + kWarps - 1) / kWarps;
  const size_t lo = warp * per, hi = lo + per < rows ? lo + per : rows;
  __shared__ unsigned long long count[kMaxRanks][kWarps];   // tokens per destination and segment, then first places
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();

  unsigned long long mine = 0;   // lane d counts destination d
  bool wrong = false;
  for (size_t row = lo; row < hi; ++row) {
    const size_t t = row * 32 + lane;
    const long long d = t < n ? dest[t] : -1;
    wrong |= t < n && (d < 0 || d >= p);
    for (int k = 0; k < p; ++k) {
      const unsigned votes = __ballot_sync(0xffffffffu, d == k);
      if ((int)lane == k) mine += __popc(votes);
    }
  }
  if (lane < p) count[lane][warp] = mine;
  if (wrong) bad = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long at = 0;
    for (int k = 0; k < p; ++k) {
      const unsigned long long first = at;
      for (int w = 0; w < kWarps; ++w) {
        const unsigned long long c = count[k][w];
        count[k][w] = at;
        at += c;
      }
      P.counts[(size_t)r * p + k] = bad ? -1 : (long long)(at - first);
    }
  }
  __syncthreads();
  if (bad) return;
  unsigned long long next = lane < p ? count[lane][warp] : 0;
  for (size_t row = lo; row < hi; ++row) {
    const size_t t = row * 32 + lane;
    const long long d = t < n ? dest[t] : -1;
    for (int k = 0; k < p; ++k) {
      const unsigned votes = __ballot_sync(0xffffffffu, d == k);
      const unsigned long long first = __shfl_sync(0xffffffffu, next, k);
      if (d == k) P.order[r][first + __popc(votes & ((1u << lane) - 1))] = (long long)t;
      if ((int)lane == k) next += __popc(votes);
    }
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
