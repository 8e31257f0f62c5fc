// Data movement straight between the buffers of ranks that all live on this GPU: allgather and alltoall.
//
// What bounds them is HBM: every byte is read once and written once (allgather: once per rank), where the staging protocol and the
// mailboxes move it twice and make CTAs wait for each other.  Nothing waits here, so the launches are ordinary ones; the host has
// checked that no byte is written that another thread still has to read (src/device_comm.cpp).
//
// Layout: warps are independent workers that take tiles of up to 2 KiB (four 16-byte loads per thread under way before the first
// store; 2 x 512 threads per SM keep 64 KB under way) from the list of jobs in turn, so that any mix of sizes fills the GPU.
// Tiles begin on 16-byte boundaries of the destination; sources on other addresses modulo 16 are shifted into place.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "local_reduce.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kLoads = 4;   // per thread, before the first store
constexpr unsigned kTile = 32 * 16 * kLoads;

/** group_copy() of one warp to several destinations with the same address modulo 16: `at(d)` of every d in `to`. */
template <typename At>
__device__ __forceinline__ void warp_fanout(unsigned to, unsigned phase, At at, const char* src, size_t n, unsigned lane) {
  size_t head = (0 - phase) & 15;
  if (head > n) head = n;
  const size_t nv = (n - head) >> 4, done = head + (nv << 4);
  auto bytes = [&](size_t k) {
    const char v = src[k];
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
      if (to >> d & 1) at(d)[k] = v;
  };
  if (lane < head) bytes(lane);
  const WordSource s(src + head, false);
  auto store = [&](size_t i, const uint4& v) {
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
      if (to >> d & 1) ((uint4*)(at(d) + head))[i] = v;
  };
  if (s.sh == 0) batched_units<kLoads, Rest::row>(nv, lane, 32, [&](size_t i) { return s.base[i]; }, store);
  else batched_units<kLoads / 2, Rest::spread>(nv, lane, 32, [&](size_t i) { return s.shifted(i); }, store);
  if (lane < n - done) bytes(done + lane);
}

/** FAN: every job has the destinations fan[d] + its offset, else the one destination dst. */
template <bool FAN>
__global__ void __launch_bounds__(kLocalThreads, 2) local_copy_kernel(const __grid_constant__ LocalCopyParams P) {
  if (any_poisoned(P.flags, P.p)) return;
  const unsigned lane = threadIdx.x & 31;
  const unsigned nwarps = gridDim.x * (blockDim.x >> 5), total = P.first[P.jobs];
  int j = 0;
  for (unsigned t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < total; t += nwarps) {
    while (t >= P.first[j + 1]) ++j;
    const unsigned per_row = (P.first[j + 1] - P.first[j]) / P.rows;
    const unsigned row = (t - P.first[j]) / per_row, k = (t - P.first[j]) - row * per_row;
    const char* src = P.src[j] + row * P.src_stride;
    char* dst = P.dst[j] + row * P.dst_stride;   // (FAN: an offset)
    const unsigned phase = (unsigned)(((uintptr_t)dst + (FAN ? (uintptr_t)P.fan[0] : 0)) & 15);
    size_t lo = (size_t)k * P.tile, hi = lo + P.tile - phase;
    if (k) lo -= phase;
    if (hi > P.bytes[j]) hi = P.bytes[j];
    if (lo >= hi) continue;
    if constexpr (FAN) {
      warp_fanout(P.to[j], k ? 0 : phase, [&](int d) { return P.fan[d] + ((size_t)dst + lo); }, src + lo, hi - lo, lane);
    } else {
      group_copy<kLoads, Rest::row>(dst + lo, src + lo, hi - lo, false, lane, 32);
    }
  }
}

}  // namespace

void launch_local_copy(LocalCopyParams& P, int max_ctas, int threads, cudaStream_t stream) {
  size_t total = 0;
  for (int j = 0; j < P.jobs; ++j) total += P.bytes[j] * P.rows;
  // Small exchanges are cut finer, so that every warp of the GPU gets some; rows of whole tiles keep the divisions above exact.
  const size_t warps = (size_t)max_ctas * (size_t)(threads / 32);
  P.tile = 512;
  while (P.tile < kTile && total / P.tile > 2 * warps) P.tile *= 2;
  while (total / P.tile > (size_t{1} << 30)) P.tile *= 2;
  unsigned n = 0;
  for (int j = 0; j < P.jobs; ++j) {
    P.first[j] = n;
    n += (unsigned)((P.bytes[j] + 15 + P.tile - 1) / P.tile) * P.rows;
  }
  P.first[P.jobs] = n;
  if (n == 0) return;
  const unsigned per = (unsigned)threads / 32;
  const unsigned ctas = std::max(1u, std::min((unsigned)max_ctas, (n + per - 1) / per));
  if (P.fans) local_copy_kernel<true><<<ctas, (unsigned)threads, 0, stream>>>(P);
  else local_copy_kernel<false><<<ctas, (unsigned)threads, 0, stream>>>(P);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
