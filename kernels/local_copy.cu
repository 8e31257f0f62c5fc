// Data movement straight between the buffers of ranks that all live on this GPU: allgather and alltoall.
//
// What bounds them is HBM: every byte is read once and written once (allgather: once per rank), where the staging protocol and the
// mailboxes move it twice and make CTAs wait for each other.  Nothing waits here, so the launches are ordinary ones; the host has
// checked that no byte is written that another thread still has to read (src/device_comm.cpp).
//
// Layout: a warp takes a tile of up to 2 KiB (four 16-byte loads per thread under way before the first store; two per thread where each
// goes to several destinations) of the list of jobs, so that any mix of sizes fills the GPU.  Tiles begin on 16-byte
// boundaries of the destination; sources on other addresses modulo 16 are shifted into place.  The grid has a warp for every tile
// unless the caller's budget of CTAs is less than the GPU: CTAs that come and go keep to one stretch of each buffer at a time, those of
// one wave that walk the tiles drift apart.  One wave of 2 CTAs per SM / a warp per tile, us: 4 x 25 MB from buffer to buffer 37.7 / 32.4,
// allgather of 8 x 2 MiB 32.8 / 26.5, of 4 x 64 MiB 245 / 204 (6.6 TB/s).
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "local_reduce.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kLoads = 4, kFanLoads = 2;   // per thread, before the first store

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
  if (s.sh == 0) batched_units<kFanLoads, Rest::row>(nv, lane, 32, [&](size_t i) { return s.base[i]; }, store);
  else batched_units<kFanLoads, Rest::spread>(nv, lane, 32, [&](size_t i) { return s.shifted(i); }, store);
  if (lane < n - done) bytes(done + lane);
}

/**
 * FAN: every job has the destinations fan[d] + its offset, else the one destination dst.  WORDS: everything but the lengths is a whole
 * number of 16-byte words.  blockIdx.y is the job; its warps take one tile of one of its rows each.
 */
template <bool FAN, bool WORDS>
__global__ void __launch_bounds__(kLocalThreads, 2) local_copy_kernel(const __grid_constant__ LocalCopyParams P) {
  constexpr int U = FAN ? kFanLoads : kLoads;
  const uint64_t failed = status_word(P.flags, P.p);
  const unsigned lane = threadIdx.x & 31, j = blockIdx.y;
  const size_t bytes = P.bytes[j];
  const unsigned per_row = (unsigned)((bytes + 15 + P.tile - 1) / P.tile), total = per_row * P.rows;
  const unsigned nwarps = gridDim.x * (blockDim.x >> 5);
  for (unsigned t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < total; t += nwarps) {
    const unsigned row = P.rows == 1 ? 0 : t / per_row, k = t - row * per_row;
    const char* src = P.src[j] + row * P.src_stride;
    char* dst = P.dst[j] + row * P.dst_stride;   // (FAN: an offset)
    if constexpr (WORDS) {
      // A tile is at most 32 * U words; the bytes behind the last whole word go with the last tile.
      const size_t words = bytes / 16, end = min(words, (size_t)(k + 1) * (P.tile / 16)), w0 = (size_t)k * (P.tile / 16) + lane;
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (w0 + 32 * u < end) v[u] = load_now((const uint4*)src + w0 + 32 * u);
      if (__any_sync(0xffffffffu, failed != 0)) return;
      auto put = [&](char* to) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (w0 + 32 * u < end) ((uint4*)to)[w0 + 32 * u] = v[u];
        if (k == per_row - 1 && lane < bytes % 16) to[words * 16 + lane] = src[words * 16 + lane];
      };
      if constexpr (FAN) {
#pragma unroll
        for (int d = 0; d < kMaxRanks; ++d)
          if (P.to[j] >> d & 1) put(P.fan[d] + (size_t)dst);
      } else {
        put(dst);
      }
    } else {
      if (__any_sync(0xffffffffu, failed != 0)) return;
      const unsigned phase = (unsigned)(((uintptr_t)dst + (FAN ? (uintptr_t)P.fan[0] : 0)) & 15);
      size_t lo = (size_t)k * P.tile, hi = lo + P.tile - phase;
      if (k) lo -= phase;
      if (hi > bytes) hi = bytes;
      if (lo >= hi) continue;
      if constexpr (FAN) warp_fanout(P.to[j], k ? 0 : phase, [&](int d) { return P.fan[d] + ((size_t)dst + lo); }, src + lo, hi - lo, lane);
      else group_copy<kLoads, Rest::row>(dst + lo, src + lo, hi - lo, false, lane, 32);
    }
  }
}

}  // namespace

void launch_local_copy(LocalCopyParams& P, int max_ctas, int sm_count, int threads, cudaStream_t stream) {
  size_t total = 0, longest = 0;
  bool words = P.src_stride % 16 == 0 && P.dst_stride % 16 == 0;
  for (int r = 0; P.fans && r < P.p; ++r) words = words && (uintptr_t)P.fan[r] % 16 == 0;
  for (int j = 0; j < P.jobs; ++j) {
    total += P.bytes[j] * P.rows;
    longest = std::max(longest, P.bytes[j]);
    words = words && (uintptr_t)P.src[j] % 16 == 0 && (uintptr_t)P.dst[j] % 16 == 0;
  }
  if (longest == 0) return;
  // As much to a warp as leaves 16 of them to an SM.
  const size_t most = 32 * 16 * (P.fans ? kFanLoads : kLoads);
  size_t tile = 512;
  while (tile < most && total / (2 * tile) >= (size_t)sm_count * 16) tile *= 2;
  while (!words && longest / tile * P.rows > (size_t{1} << 30)) tile *= 2;
  const size_t most_tiles = (longest + 15 + tile - 1) / tile * P.rows;
  if (most_tiles >= (size_t{1} << 32)) throw_al_exception("internal error: a copy of ", longest, " bytes in one piece");
  P.tile = (unsigned)tile;
  const LocalGrid g = local_grid(most_tiles, P.jobs, max_ctas, threads);
  auto launch = [&](const LocalCopyParams& Q) {
    const dim3 grid(g.x, (unsigned)Q.jobs);
    if (Q.fans && words) local_copy_kernel<true, true><<<grid, (unsigned)threads, 0, stream>>>(Q);
    else if (Q.fans) local_copy_kernel<true, false><<<grid, (unsigned)threads, 0, stream>>>(Q);
    else if (words) local_copy_kernel<false, true><<<grid, (unsigned)threads, 0, stream>>>(Q);
    else local_copy_kernel<false, false><<<grid, (unsigned)threads, 0, stream>>>(Q);
    AL_CHECK_CUDA(cudaGetLastError());
  };
  if ((int)g.y == P.jobs) return launch(P);
  // Fewer CTAs than jobs: some at a time.  (A loop over the jobs in the kernel costs all launches 8 registers, and with them a CTA per SM.)
  for (int from = 0; from < P.jobs; from += (int)g.y) {
    LocalCopyParams Q = P;
    Q.jobs = std::min(P.jobs - from, (int)g.y);
    std::copy_n(P.src + from, Q.jobs, Q.src);
    std::copy_n(P.dst + from, Q.jobs, Q.dst);
    std::copy_n(P.bytes + from, Q.jobs, Q.bytes);
    std::copy_n(P.to + from, Q.jobs, Q.to);
    launch(Q);
  }
}

}  // namespace device
}  // namespace internal
}  // namespace Al
