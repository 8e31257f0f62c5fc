// Reductions straight between the buffers of ranks that all live on this GPU: one pass reads every rank's contribution and
// writes every rank's result.
//
// What bounds it is HBM: p vectors in and p (allreduce) or one (reduce_scatter) out, where the staging protocol moves every byte
// twice more and makes all CTAs wait for each other twice.  Nothing waits here, so the launch is an ordinary one.  The host
// has checked that no byte is written that another thread still has to read (`local_buffers_apart`, src/device_comm.cpp).
//
// Layout: a warp owns U rows of 32 consecutive 16-byte words of the result and has the words of all ranks under way before it folds
// the first one (eight loads per thread: 1 word of up to eight ranks, 2 of four, 4 of two; 2 x 512 threads of 64 registers per SM keep
// 128 KB under way, more than twice what HBM3e at about 1 us wants).  Contributions are folded in rank order, in the
// type and with the roundings of the staged kernels, so that a call's result does not depend on the route.  Contributions that
// lie on another address modulo 16 than the result (slices of an odd number of elements) are read as aligned words and
// shifted into place; the second word of each comes out of L1.
//
// Measured, one B200, device time through staging (loops or bulk copies, whichever was faster) / here, us: gradient bucket of 4 x 26 MB
// fp32 103 / 34.3, 8 x 12 MB fp32 with a bf16 type between ranks 95.3 / 31.6, reduce_scatter of 8 x 16 MiB bf16 86.9 / 24.4, of 4 x 256 MiB
// 506 / 187 (7.2 TB/s, nearly all reads).  With one wave of 2 CTAs per SM that walks the vector instead of a warp per piece: 38.2, 36.5,
// 28.6, 206.
#pragma once
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "datamove.cuh"
#include "local_grid.hpp"

namespace Al {
namespace internal {
namespace device {

constexpr int kLocalThreads = 512;   // of a CTA at most

/**
 * Has an earlier operation of the communicator failed?  A lane's word of the ranks' status words, to be looked at with
 * __any_sync() behind the first loads of data, which this one's latency then overlaps.  Earlier kernels wrote it, so it may come out of
 * L1: every warp of the grid asks, and past L1 all of them meet in a few sectors of L2 (allgather of 4 x 64 MiB 222 us).
 */
__device__ __forceinline__ uint64_t status_word(uint64_t* const* flags, int p) {
  const unsigned lane = threadIdx.x & 31;
  uint64_t v = 0;
  if (lane < (unsigned)p)
    asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(flag_slot(flags[lane], FlagLayout::off_status, 0)) : "memory");
  return v;
}

/** A load that stays where it is written (past L1: nothing here is read twice). */
__device__ __forceinline__ uint4 load_now(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

/** T: the buffers' type, W: the type that crosses the links between GPUs (contributions, and in two phases the result, are rounded to it). */
template <typename T, typename W, typename Red, int R, int U, bool SHIFT>
__global__ void __launch_bounds__(kLocalThreads, 2) local_reduce_kernel(const __grid_constant__ LocalReduceParams P, Red red) {
  using A = typename Elem<T>::Acc;
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr bool kRounds = !std::is_same<T, W>::value;
  const int p = P.p;
  const uint64_t failed = status_word(P.flags, p);
  const size_t job = blockIdx.y;   // reduce_scatter: the rank whose slice this is
  const size_t from = P.scatter ? job * P.count : 0;
  const unsigned outs = P.scatter ? 1u << job : (1u << p) - 1;
  auto src = [&](int r) { return (const T*)P.src[r] + from; };
  auto in = [&](T v) -> A {
    if constexpr (kRounds) return acc_cast<A>(Elem<W>::up(Elem<W>::down(Elem<T>::up(v))));
    else return Elem<T>::up(v);
  };
  auto out = [&](A a) -> T {
    a = finish_acc(a, P.scale, P.int_div);
    if constexpr (kRounds)
      if (P.round_result) a = acc_cast<A>(Elem<W>::up(Elem<W>::down(a)));
    return Elem<T>::down(a);
  };
  // elements up to the first 16-byte boundary of the results (the same in all of them)
  size_t head = ((0 - (uintptr_t)P.dst[job]) & 15) / sizeof(T);
  if (head > P.count) head = P.count;
  const size_t nvec = (P.count - head) / VEC, done = head + nvec * VEC;
  union Pack { uint4 u; T e[VEC]; };
  const unsigned lane = threadIdx.x & 31;
  const size_t warp = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), nwarps = (size_t)gridDim.x * (blockDim.x >> 5);
  auto load = [&](int r, size_t v) {
    if constexpr (SHIFT) {
      const WordSource s((const char*)(src(r) + head), false);
      return s.sh == 0 ? s.base[v] : s.shifted(v);
    } else {
      return load_now((const uint4*)(src(r) + head) + v);
    }
  };
  for (size_t first = warp * (32 * U); first < nvec; first += nwarps * (32 * U)) {
    const size_t v0 = first + lane;
    Pack w[R][U];
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < p) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < nvec) w[r][u].u = load(r, v0 + 32 * u);
      }
    if (__any_sync(0xffffffffu, failed != 0)) return;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v0 + 32 * u < nvec) {
        Pack o;
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          A acc = in(w[0][u].e[k]);
#pragma unroll
          for (int r = 1; r < R; ++r)
            if (r < p) acc = red(acc, in(w[r][u].e[k]));
          o.e[k] = out(acc);
        }
#pragma unroll
        for (int d = 0; d < kMaxRanks; ++d)
          if (outs >> d & 1) ((uint4*)((T*)P.dst[d] + head))[v0 + 32 * u] = o.u;
      }
  }
  // the elements before the first and behind the last whole word
  if (warp == nwarps - 1 && !__any_sync(0xffffffffu, failed != 0)) {
    const size_t i = lane < head ? lane : done + (lane - head);
    if (i < P.count) {
      A acc = in(src(0)[i]);
#pragma unroll
      for (int r = 1; r < kMaxRanks; ++r)
        if (r < p) acc = red(acc, in(src(r)[i]));
      const T o = out(acc);
#pragma unroll
      for (int d = 0; d < kMaxRanks; ++d)
        if (outs >> d & 1) ((T*)P.dst[d])[i] = o;
    }
  }
}

template <typename T, typename W, typename Red, int R, int U, bool SHIFT>
void local_reduce_run(const LocalReduceParams& P, Red red, int max_ctas, int threads, cudaStream_t stream) {
  const int jobs = P.scatter ? P.p : 1;
  const size_t words = P.count * sizeof(T) / 16 + 1;
  const LocalGrid grid = local_grid((words + 32 * U - 1) / (32 * U), jobs, max_ctas, threads);
  if ((int)grid.y != jobs) throw_al_exception("internal error: fewer CTAs than ranks");   // (a budget is some CTAs for every rank)
  local_reduce_kernel<T, W, Red, R, U, SHIFT><<<dim3(grid.x, grid.y), (unsigned)threads, 0, stream>>>(P, red);
  AL_CHECK_CUDA(cudaGetLastError());
}

/** SHIFT where a contribution lies on another address modulo 16 than the result. */
template <typename T, typename W, typename Red>
void local_reduce_launch(const LocalReduceParams& P, Red red, int max_ctas, int threads, cudaStream_t stream) {
  bool shifted = false;
  for (int job = 0; job < (P.scatter ? P.p : 1); ++job)
    for (int r = 0; r < P.p; ++r)
      shifted = shifted || (((uintptr_t)P.src[r] + (P.scatter ? (size_t)job * P.count * sizeof(T) : 0)) ^ (uintptr_t)P.dst[job]) % 16 != 0;
  if (shifted) {
    if (P.p == 2) return local_reduce_run<T, W, Red, 2, 2, true>(P, red, max_ctas, threads, stream);
    if (P.p <= 4) return local_reduce_run<T, W, Red, 4, 1, true>(P, red, max_ctas, threads, stream);
    return local_reduce_run<T, W, Red, 8, 1, true>(P, red, max_ctas, threads, stream);
  }
  if (P.p == 2) return local_reduce_run<T, W, Red, 2, 4, false>(P, red, max_ctas, threads, stream);
  if (P.p <= 4) return local_reduce_run<T, W, Red, 4, 2, false>(P, red, max_ctas, threads, stream);
  return local_reduce_run<T, W, Red, 8, 1, false>(P, red, max_ctas, threads, stream);
}

// One per file so that the instantiations compile in parallel; false: not compiled for this operator.
bool local_reduce_f32(const LocalReduceParams& P, DType wire, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream);
bool local_reduce_16bit(const LocalReduceParams& P, DType dt, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream);
bool local_reduce_wide(const LocalReduceParams& P, DType dt, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream);

}  // namespace device
}  // namespace internal
}  // namespace Al
