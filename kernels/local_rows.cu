// Row exchanges of ranks that all live on this GPU: every row from tensor to tensor (the pack and the unpack of sequence <-> head
// transpositions and of expert dispatch / combine included), where the staging protocol moves it through memory once more.
//
// What bounds them is HBM.  A warp takes 2 KiB at a time: several rows where they are short, a part
// of one where it is long, four 16-byte loads per thread under way before the first store, whose row indexes were fetched together
// just before.  An exchange that is too small to give every warp 2 KiB is dealt in pieces of 512 bytes.
// Measured, one B200, device time through staging / here, us: transposition of 8 x 1024 x 32 x 128 bf16 (67 MB, 1 KiB rows) 69.7 / 23.6, dispatch of
// 4 x 4099 tokens of 4 KiB 52.1 / 23.8 and combine 52.1 / 21.3 (20.5 at the copy rate), 2 x 16 rows of 512 bytes 13.9 / 2.3.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "local_reduce.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

/** The last entry of first[0 .. n) that is at most t (of equal ones the last). */
__device__ __forceinline__ int place_of(const unsigned* first, int n, unsigned t) {
  int j = 0;
#pragma unroll
  for (int s = kMaxRanks * kMaxRanks / 2; s > 0; s >>= 1)
    if (j + s < n && t >= first[j + s]) j += s;
  return j;
}

constexpr int kLoads = 4;                        // per thread, before the first store
constexpr size_t kTile = 32 * 16 * kLoads;       // bytes that a warp takes at a time

/**
 * WORDS: everything lies on 16-byte boundaries; a warp then takes 32 * U words at a time, of several rows where they are short
 * (`group` rows; a row's `per_row` > 1 parts where it is long).  Else one row at a time.
 */
template <bool WORDS, int U, bool EVEN>
__global__ void __launch_bounds__(kLocalThreads, 2) local_rows_kernel(const __grid_constant__ LocalRowsParams P) {
  const uint64_t failed = status_word(P.flags, P.p);
  const unsigned lane = threadIdx.x & 31;
  const unsigned nwarps = gridDim.x * (blockDim.x >> 5), end = EVEN ? P.first[blockIdx.y + 1] : P.first[P.p * P.p];
  const unsigned wpr = (unsigned)(P.row_bytes / 16);   // words per row
  for (unsigned t = (EVEN ? P.first[blockIdx.y] : 0) + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < end; t += nwarps) {
    const int q = EVEN ? (int)blockIdx.y : place_of(P.first, P.p * P.p, t);
    const int s = q / P.p, d = q - s * P.p;
    const RowTable &S = P.tab[s], &D = P.tab[d];
    const char* src = (const char*)P.send[s] + S.send_peer_off[d];
    char* dst = (char*)P.recv[d] + D.recv_peer_off[s];
    const long long* sidx = P.send_idx[s];
    const long long* ridx = P.recv_idx[d];
    const size_t s0 = S.send_first[d], d0 = D.recv_first[s], rows = S.send_rows[d];
    auto from = [&](size_t k) { return src + (sidx ? (size_t)sidx[s0 + k] : s0 + k) * P.send_row_stride; };
    auto to = [&](size_t k) { return dst + (ridx ? (size_t)ridx[d0 + k] : d0 + k) * P.recv_row_stride; };
    const unsigned unit = t - P.first[q];
    if constexpr (WORDS) {
      const unsigned part = unit % P.per_row;
      const size_t k0 = (size_t)(unit / P.per_row) * P.group;
      const unsigned words = P.per_row > 1 ? wpr : (unsigned)(rows - k0 < P.group ? rows - k0 : P.group) * wpr;
      const unsigned w0 = part * (32 * U) + lane;
      uint4 v[U];
      uint4* at[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const unsigned w = w0 + 32 * i;
        if (w < words) {
          const unsigned r = P.per_row > 1 ? 0 : w / wpr, c = w - r * wpr;
          at[i] = (uint4*)to(k0 + r) + c;
          v[i] = load_now((const uint4*)from(k0 + r) + c);
        }
      }
      if (__any_sync(0xffffffffu, failed != 0)) return;
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (w0 + 32 * i < words) *at[i] = v[i];
    } else {
      if (__any_sync(0xffffffffu, failed != 0)) return;
      group_copy<kLoads, Rest::row>(to(unit), from(unit), P.row_bytes, false, lane, 32);
    }
  }
}

}  // namespace

void launch_local_rows(LocalRowsParams& P, int max_ctas, int sm_count, int threads, cudaStream_t stream) {
  const int p = P.p;
  bool words = P.row_bytes % 16 == 0 && P.send_row_stride % 16 == 0 && P.recv_row_stride % 16 == 0;
  size_t rows = 0;
  for (int s = 0; s < p; ++s) {
    words = words && (uintptr_t)P.send[s] % 16 == 0 && (uintptr_t)P.recv[s] % 16 == 0;
    for (int d = 0; d < p; ++d) {
      rows += P.tab[s].send_rows[d];
      words = words && P.tab[s].send_peer_off[d] % 16 == 0 && P.tab[s].recv_peer_off[d] % 16 == 0;
    }
  }
  const size_t warps = max_ctas > 0 ? (size_t)max_ctas * (size_t)(threads / 32) : (size_t)sm_count * 2 * kLocalThreads / 32;
  const bool small = rows * P.row_bytes / kTile < warps;   // one load per thread then, so that more warps get some
  const unsigned unit = small ? 32 : 32 * kLoads;                 // words of 16 bytes
  P.group = P.per_row = 1;
  if (words) {
    const size_t wpr = P.row_bytes / 16;
    if (wpr < unit) P.group = unit / (unsigned)wpr;
    else P.per_row = (unsigned)((wpr + unit - 1) / unit);
  }
  unsigned n = 0;
  for (int s = 0; s < p; ++s)
    for (int d = 0; d < p; ++d) {
      P.first[s * p + d] = n;
      n += (unsigned)((P.tab[s].send_rows[d] + P.group - 1) / P.group) * P.per_row;
    }
  P.first[p * p] = n;
  if (n == 0) return;
  // Pairs of about the same size: each has its part of the grid, and every warp one unit (transposition of 8 x 1024 x 32 x 128 there and back
  // 47.2 us, 48.7 with one wave that walks them; dispatch and combine of uneven pairs 23.8 and 21.3 in one wave, 26.2 and 24.4 with a
  // warp per unit that looks its pair up).
  unsigned most = 0;
  for (int q = 0; q < p * p; ++q) most = std::max(most, P.first[q + 1] - P.first[q]);
  auto run = [&](auto kernel, dim3 grid) { kernel<<<grid, (unsigned)threads, 0, stream>>>(P); };
  const LocalGrid even = local_grid(most, p * p, max_ctas, threads);
  if ((size_t)most * (size_t)(p * p) <= (size_t)n + n / 4 && even.y == (unsigned)(p * p)) {
    const dim3 grid(even.x, even.y);
    if (!words) run(local_rows_kernel<false, 1, true>, grid);
    else if (small) run(local_rows_kernel<true, 1, true>, grid);
    else run(local_rows_kernel<true, kLoads, true>, grid);
  } else {
    const dim3 grid(local_grid(n, 1, max_ctas > 0 ? max_ctas : sm_count * (1024 / threads), threads).x);
    if (!words) run(local_rows_kernel<false, 1, false>, grid);
    else if (small) run(local_rows_kernel<true, 1, false>, grid);
    else run(local_rows_kernel<true, kLoads, false>, grid);
  }
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
