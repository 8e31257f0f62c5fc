// Row exchanges of ranks that all live on this GPU: every row from tensor to tensor (the pack and the unpack of sequence <-> head
// transpositions and of expert dispatch / combine included), where the staging protocol moves it through memory once more.
//
// What bounds them is HBM.  One wave of warps walks the exchange; each takes 2 KiB at a time: several rows where they are short, a part
// of one where it is long, four 16-byte loads per thread under way before the first store, whose row indexes were fetched together
// just before.  An exchange that is too small to give every warp 2 KiB is dealt in pieces of 512 bytes.
// Measured, one B200, device time through staging / here, us: transposition of 8 x 1024 x 32 x 128 bf16 (67 MB, 1 KiB rows) 69.7 / 24.4, dispatch of
// 4 x 4099 tokens of 4 KiB 52.1 / 23.8 and combine 52.1 / 21.3 (20.5 at the copy rate), 2 x 16 rows of 512 bytes 13.9 / 2.3.  (A warp per piece
// as in local_copy.cu: 57.6 for the first there and back, 27.8, 26.4: the tables of a pair of ranks are looked up once per piece.)
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
template <bool WORDS, int U>
__global__ void __launch_bounds__(kLocalThreads, 2) local_rows_kernel(const __grid_constant__ LocalRowsParams P) {
  if (__any_sync(0xffffffffu, status_word(P.flags, P.p) != 0)) return;
  const unsigned lane = threadIdx.x & 31;
  const unsigned nwarps = gridDim.x * (blockDim.x >> 5), total = P.first[P.p * P.p];
  const unsigned wpr = (unsigned)(P.row_bytes / 16);   // words per row
  for (unsigned t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < total; t += nwarps) {
    const int q = place_of(P.first, P.p * P.p, t);
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
          v[i] = ((const uint4*)from(k0 + r))[c];
        }
      }
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (w0 + 32 * i < words) *at[i] = v[i];
    } else {
      group_copy<kLoads, Rest::row>(to(unit), from(unit), P.row_bytes, false, lane, 32);
    }
  }
}

}  // namespace

void launch_local_rows(LocalRowsParams& P, int max_ctas, int threads, cudaStream_t stream) {
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
  const size_t warps = max_ctas > 0 ? (size_t)max_ctas * (size_t)(threads / 32) : kLocalWarps;
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
  const unsigned ctas = local_grid(n, max_ctas > 0 ? max_ctas : 148 * (1024 / threads), threads);
  if (!words) local_rows_kernel<false, 1><<<ctas, (unsigned)threads, 0, stream>>>(P);
  else if (small) local_rows_kernel<true, 1><<<ctas, (unsigned)threads, 0, stream>>>(P);
  else local_rows_kernel<true, kLoads><<<ctas, (unsigned)threads, 0, stream>>>(P);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
