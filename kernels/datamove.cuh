// CTA-wide copy, convert and multi-source reduce loops used by the collective
// kernels.  Reads of staging memory (local or a peer's) bypass L1 (ld.cg), so a
// line cached during an earlier operation can never be served stale.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace Al {
namespace internal {
namespace device {

// ---------------------------------------------------------------------------
// element traits: accumulator type and conversions
// ---------------------------------------------------------------------------
template <typename T> struct Elem { using Acc = T; static __device__ __forceinline__ Acc up(T v) { return v; } static __device__ __forceinline__ T down(Acc a) { return a; } };
template <> struct Elem<__half> {
  using Acc = float;
  static __device__ __forceinline__ float up(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half down(float a) { return __float2half_rn(a); }
};
template <> struct Elem<__nv_bfloat16> {
  using Acc = float;
  static __device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 down(float a) { return __float2bfloat16_rn(a); }
};

/** Convert between accumulator types (float <-> float only in practice). */
template <typename To, typename From>
__device__ __forceinline__ To acc_cast(From v) { return (To)v; }

// ---------------------------------------------------------------------------
// reduction functors on accumulator values
// ---------------------------------------------------------------------------
struct RedSum { template <typename A> __device__ __forceinline__ A operator()(A a, A b) const { return a + b; } };
struct RedMin { template <typename A> __device__ __forceinline__ A operator()(A a, A b) const { return b < a ? b : a; } };
struct RedMax { template <typename A> __device__ __forceinline__ A operator()(A a, A b) const { return a < b ? b : a; } };
struct RedNone { template <typename A> __device__ __forceinline__ A operator()(A a, A) const { return a; } };

template <typename A, bool IsInt = std::is_integral<A>::value>
struct BitOps {
  static __device__ __forceinline__ A apply(int, A a, A) { return a; }
};
template <typename A>
struct BitOps<A, true> {
  static __device__ __forceinline__ A apply(int op, A a, A b) {
    switch ((ReductionOperator)op) {
      case ReductionOperator::bor: return (A)(a | b);
      case ReductionOperator::band: return (A)(a & b);
      case ReductionOperator::bxor: return (A)(a ^ b);
      default: return a;
    }
  }
};

/** Operator chosen at run time (integer types and the less common operators). */
struct RedRuntime {
  int op;
  template <typename A>
  __device__ __forceinline__ A operator()(A a, A b) const {
    switch ((ReductionOperator)op) {
      case ReductionOperator::sum:
      case ReductionOperator::avg: return a + b;
      case ReductionOperator::prod: return a * b;
      case ReductionOperator::min: return b < a ? b : a;
      case ReductionOperator::max: return a < b ? b : a;
      case ReductionOperator::lor: return (A)((a != A(0)) || (b != A(0)));
      case ReductionOperator::land: return (A)((a != A(0)) && (b != A(0)));
      case ReductionOperator::lxor: return (A)((a != A(0)) != (b != A(0)));
      default: return BitOps<A>::apply(op, a, b);
    }
  }
};

// ---------------------------------------------------------------------------
// work split
// ---------------------------------------------------------------------------
/** Sub-range [lo, hi) of [0, len) owned by part `i` of `n`, boundaries multiples of `align`. */
__device__ __forceinline__ void split_range(size_t len, unsigned i, unsigned n, size_t align, size_t& lo, size_t& hi) {
  size_t per = (len + n - 1) / n;
  per = (per + align - 1) / align * align;
  lo = per * i;
  if (lo > len) lo = len;
  hi = lo + per;
  if (hi > len) hi = len;
}

__device__ __forceinline__ size_t clamp_len(size_t count, size_t lo, size_t cap) {
  if (count <= lo) return 0;
  const size_t r = count - lo;
  return r < cap ? r : cap;
}

// ---------------------------------------------------------------------------
// copies
// ---------------------------------------------------------------------------
// What bounds the loops below is the number of bytes in flight: the staged kernel runs 512 threads per SM (its
// register count allows one CTA), so with 4 x 16 bytes per thread 148 SMs keep 4.8 MB under way where HBM3e at
// about 0.8 us of latency wants 6 MB.  Eight loads per thread cover that in kernels that only copy (halo exchange of
// 8 MiB planes on one GPU 31.4 -> 27.6 us, ring pass of 4 x 25 MB 103.5 -> 90.5 us).  In an instantiation with folding loops the
// copies keep four: with eight, and an end of a round under predicates, they spilled 0.5 to 1.4 KB per thread, and what no
// other kernel takes over got slower.  Four loads before that / eight / now, us, all ranks on one GPU: allreduce max of 4 x 8 MiB
// fp32 87 / 105 / 66, sum of 4 x 64 MiB 589 / 705 / 439, of 8 x 8 MiB int32 426 / 371 / 228, of 8 x 8 MiB int8 1737 / 463 / 242,
// reduce max of 8 x 8 MiB 163 / 224 / 95, bcast of 4 x 64 MiB 224 / 260 / 216.  (Conversions were done one element at a time before:
// allreduce of 8 x 8 MiB fp32 with an fp16 wire 267 / 173 / 148 us.)  Loops that are not inlined, or two CTAs of 64 registers, spill
// inside the loop and were slower.  Buffers whose addresses differ modulo 16 (rows or slices of an odd number of
// elements) are read as aligned 16-byte words and shifted into place, so that they move in 16-byte stores too instead
// of in units of the common alignment.
constexpr int kUnroll = 8;

/** 16-byte source words at any byte address: word i is bytes [16 i, 16 i + 16) of `src`.  An unaligned word is put
 *  together from the two aligned words around it; both hold at least one byte of it, so nothing outside the 16-byte
 *  granules that the caller's bytes occupy is touched. */
struct WordSource {
  const uint4* base;
  unsigned sh;    ///< bytes that `src` lies above `base`
  bool staging;   ///< read past L1 (staging memory changes under a running kernel)

  __device__ __forceinline__ WordSource(const char* src, bool is_staging)
      : base((const uint4*)((uintptr_t)src & ~(uintptr_t)15)), sh((unsigned)((uintptr_t)src & 15)), staging(is_staging) {}
  __device__ __forceinline__ uint4 raw(size_t i) const { return staging ? __ldcg(base + i) : base[i]; }
  __device__ __forceinline__ uint4 shifted(size_t i) const {
    const uint4 a = raw(i), b = raw(i + 1);
    const unsigned q = sh >> 2, bits = (sh & 3) * 8;
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t x[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const uint32_t lo = q & 1 ? w[k + 1] : w[k];
      const uint32_t hi = q & 1 ? w[k + 3 < 8 ? k + 3 : 7] : w[k + 2];
      x[k] = q & 2 ? hi : lo;
    }
    return uint4{__funnelshift_r(x[0], x[1], bits), __funnelshift_r(x[1], x[2], bits), __funnelshift_r(x[2], x[3], bits),
                 __funnelshift_r(x[3], x[4], bits)};
  }
};

/** What batched_units() does with the units that are less than a round. */
enum class Rest {
  spread,    ///< over all warps: half of U loads at once, half of that, then singly (fewest registers)
  together,  ///< a warp's rows as in a full round, all at once under predicates (least latency; kernels with many such loops spill over it)
  row        ///< together, for a group that is one warp
};

/** For every i in [0, units): store(i, load(i)), U independent loads per thread before the first store.  In a full round a
 *  warp takes U rows of 32 consecutive units, so that its accesses differ by constants and share one address register. */
template <int U, Rest REST = Rest::spread, typename Load, typename Store>
__device__ __forceinline__ void batched_units(size_t units, unsigned lane, unsigned nlanes, Load load, Store store) {
  const unsigned warps = nlanes >> 5;   // (of a group that is no multiple of 32 threads the last few stay idle)
  if ((lane >> 5) >= warps) return;
  const size_t step = (size_t)warps * 32;
  uint4 v[U];
  auto batch = [&](size_t i, size_t apart, auto n) __attribute__((always_inline)) {
#pragma unroll
    for (int k = 0; k < decltype(n)::value; ++k) v[k] = load(i + k * apart);
#pragma unroll
    for (int k = 0; k < decltype(n)::value; ++k) store(i + k * apart, v[k]);
  };
  const size_t first = (size_t)(lane >> 5) * (32 * U) + (lane & 31);
  if constexpr (REST == Rest::together) {
    for (size_t i = first; i < units; i += U * step) {
      if (i + 32 * (U - 1) < units) {
        batch(i, 32, std::integral_constant<int, U>());
      } else {
        const unsigned left = (unsigned)((units - i + 31) >> 5);
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (k < left) v[k] = load(i + 32 * k);
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (k < left) store(i + 32 * k, v[k]);
      }
    }
  } else {
    size_t done = 0;
    for (; done + U * step <= units; done += U * step) batch(done + first, 32, std::integral_constant<int, U>());
    size_t i = done + lane;
    if constexpr (REST == Rest::row) {
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (i + k * step < units) v[k] = load(i + k * step);
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (i + k * step < units) store(i + k * step, v[k]);
      return;
    }
    auto some = [&](auto n) __attribute__((always_inline)) {
      constexpr int N = decltype(n)::value;
      if constexpr (N >= 2) {
        if (i + (N - 1) * step < units) {
          batch(i, step, n);
          i += N * step;
        }
      }
    };
    some(std::integral_constant<int, U / 2>());
    some(std::integral_constant<int, U / 4>());
#pragma unroll 1
    for (; i < units; i += step) store(i, load(i));
  }
}

/** Copy `nbytes` with `nlanes` cooperating threads (this thread is `lane`), whatever the two alignments. */
template <int U = kUnroll, Rest REST = U == kUnroll ? Rest::together : Rest::spread>
__device__ __forceinline__ void group_copy(char* dst, const char* src, size_t nbytes, bool src_is_staging,
                                           unsigned lane, unsigned nlanes) {
  if (nbytes == 0) return;
  size_t head = (0 - (uintptr_t)dst) & 15;  // bytes up to the first 16-byte boundary of the destination
  if (head > nbytes) head = nbytes;
  const size_t nv = (nbytes - head) >> 4, done = head + (nv << 4);
  for (size_t k = lane; k < head; k += nlanes) dst[k] = src_is_staging ? __ldcg(src + k) : src[k];
  uint4* d = (uint4*)(dst + head);
  const WordSource s(src + head, src_is_staging);
  auto store = [&](size_t i, const uint4& v) { d[i] = v; };
  if (s.sh == 0) {
    if (src_is_staging) batched_units<U, REST>(nv, lane, nlanes, [&](size_t i) { return __ldcg(s.base + i); }, store);
    else batched_units<U, REST>(nv, lane, nlanes, [&](size_t i) { return s.base[i]; }, store);
  } else {
    batched_units<U / 4, REST>(nv, lane, nlanes, [&](size_t i) { return s.shifted(i); }, store);
  }
  for (size_t k = done + lane; k < nbytes; k += nlanes) dst[k] = src_is_staging ? __ldcg(src + k) : src[k];
}

/** Copy with all threads of the CTA.  (Kernels that are held to 64 registers and spill with eight loads pass U = 4; the three
 *  NVLS kernels take 55 to 63 registers then and spill nothing.) */
template <int U = kUnroll>
__device__ __forceinline__ void cta_copy(char* dst, const char* src, size_t nbytes, bool src_is_staging) {
  group_copy<U>(dst, src, nbytes, src_is_staging, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------------------
// publish: one local source, several (possibly remote) destinations
// ---------------------------------------------------------------------------
/**
 * Store `nbytes` read once from local `src` to dst(d) of every rank d whose bit is set in `ranks` (peer-mapped
 * memory: plain stores over NVLink, which do not stall the issuing thread the way remote loads do).  Every
 * dst(d) is 16-byte aligned; `dst` is called with compile-time ranks.
 */
template <typename Dst>
__device__ __forceinline__ void cta_fanout(unsigned ranks, Dst dst, const char* src, size_t nbytes) {
  if (nbytes == 0) return;
  const size_t nv = nbytes >> 4, done = nv << 4;
  const WordSource s(src, false);
  auto store = [&](size_t i, const uint4& v) {
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
      if (ranks >> d & 1) ((uint4*)dst(d))[i] = v;
  };
  if (s.sh == 0) batched_units<kUnroll / 2>(nv, threadIdx.x, blockDim.x, [&](size_t i) { return s.base[i]; }, store);
  else batched_units<kUnroll / 4>(nv, threadIdx.x, blockDim.x, [&](size_t i) { return s.shifted(i); }, store);
  if (threadIdx.x < nbytes - done) {
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
      if (ranks >> d & 1) ((char*)dst(d))[done + threadIdx.x] = src[done + threadIdx.x];
  }
}

/** 16 bytes of wire elements converted from consecutive user elements: one or two 16-byte loads per vector. */
template <typename Ti, typename Tw>
struct Converter {
  static constexpr int VEC = 16 / (int)sizeof(Tw);
  static constexpr int in_bytes = VEC * (int)sizeof(Ti);
  struct alignas(in_bytes < 16 ? in_bytes : 16) In { Ti e[VEC]; };
  union Out { uint4 u; Tw e[VEC]; };
  static __device__ __forceinline__ Tw one(Ti v) {
    using Ai = typename Elem<Ti>::Acc;
    using Aw = typename Elem<Tw>::Acc;
    return Elem<Tw>::down(acc_cast<Aw, Ai>(Elem<Ti>::up(v)));
  }
  static __device__ __forceinline__ bool aligned(const Ti* src) { return (uintptr_t)src % alignof(In) == 0; }
  static __device__ __forceinline__ uint4 word(const Ti* src, size_t i) { return convert(((const In*)src)[i]); }
  /** The same out of staging memory (past L1). */
  static __device__ __forceinline__ uint4 word_staged(const Ti* src, size_t i) {
    using L = std::conditional_t<(in_bytes >= 16), uint4, std::conditional_t<in_bytes == 8, uint2, uint32_t>>;
    union { In a; L l[in_bytes / sizeof(L)]; } x;
#pragma unroll
    for (int k = 0; k < (int)(in_bytes / sizeof(L)); ++k) x.l[k] = __ldcg((const L*)src + i * (in_bytes / sizeof(L)) + k);
    return convert(x.a);
  }
  static __device__ __forceinline__ uint4 convert(const In& a) {
    Out o;
#pragma unroll
    for (int k = 0; k < VEC; ++k) o.e[k] = one(a.e[k]);
    return o.u;
  }
};

/** Single destination (16-byte aligned), a subset of the CTA's threads: used to serve all peers of a small message at once. */
template <typename Ti, typename Tw, int U = kUnroll>
__device__ __forceinline__ void group_publish(char* dst, const Ti* src, size_t n, unsigned lane, unsigned nlanes) {
  if constexpr (std::is_same<Ti, Tw>::value) {
    group_copy<U, Rest::spread>(dst, (const char*)src, n * sizeof(Ti), false, lane, nlanes);
  } else {
    using C = Converter<Ti, Tw>;
    const size_t nv = C::aligned(src) ? n / C::VEC : 0;
    batched_units<2>(nv, lane, nlanes, [&](size_t i) { return C::word(src, i); }, [&](size_t i, const uint4& v) { ((uint4*)dst)[i] = v; });
    for (size_t i = nv * C::VEC + lane; i < n; i += nlanes) ((Tw*)dst)[i] = C::one(src[i]);
  }
}

/** Publish n elements of user type Ti as wire type Tw to dst(d) of every rank d in `ranks` (cast fused in). */
template <typename Ti, typename Tw, typename Dst>
__device__ __forceinline__ void cta_publish(unsigned ranks, Dst dst, const Ti* src, size_t n) {
  if constexpr (std::is_same<Ti, Tw>::value) {
    cta_fanout(ranks, dst, (const char*)src, n * sizeof(Ti));
  } else {
    using C = Converter<Ti, Tw>;
    const size_t nv = C::aligned(src) ? n / C::VEC : 0;
    batched_units<4>(nv, threadIdx.x, blockDim.x, [&](size_t i) { return C::word(src, i); }, [&](size_t i, const uint4& v) {
#pragma unroll
      for (int d = 0; d < kMaxRanks; ++d)
        if (ranks >> d & 1) ((uint4*)dst(d))[i] = v;
    });
    for (size_t i = nv * C::VEC + threadIdx.x; i < n; i += blockDim.x) {
      const Tw v = C::one(src[i]);
#pragma unroll
      for (int d = 0; d < kMaxRanks; ++d)
        if (ranks >> d & 1) ((Tw*)dst(d))[i] = v;
    }
  }
}

/** Copy n staged elements (16-byte aligned) of type Tw out as To. */
template <typename Tw, typename To>
__device__ __forceinline__ void cta_expand(To* dst, const Tw* src, size_t n) {
  using C = Converter<Tw, To>;
  const size_t nv = (uintptr_t)dst % 16 == 0 ? n / C::VEC : 0;
  batched_units<4>(nv, threadIdx.x, blockDim.x, [&](size_t i) { return C::word_staged(src, i); },
                   [&](size_t i, const uint4& v) { ((uint4*)dst)[i] = v; });
  for (size_t i = nv * C::VEC + threadIdx.x; i < n; i += blockDim.x) dst[i] = C::one(__ldcg(src + i));
}

// ---------------------------------------------------------------------------
// multi-source reduction
// ---------------------------------------------------------------------------
template <typename A>
__device__ __forceinline__ A finish_acc(A a, double scale, int int_div) {
  if constexpr (std::is_integral<A>::value) {
    return int_div > 1 ? (A)(a / (A)int_div) : a;
  } else {
    return scale != 1.0 ? (A)(a * (A)scale) : a;
  }
}

/**
 * out[i] = finish(red(src(0)[i], src(1)[i], ..., src(p-1)[i])) for i in [0, n), written to dst(d) for every
 * rank d in `ranks` (several destinations are used when a reduced slice is pushed to every peer).  src(r) gives
 * the first Tw element of rank r's contribution, dst(d) the first To element of a destination; both are called with
 * compile-time ranks.  Contributions are folded in rank order so every rank computes
 * bit-identical results.  A destination may alias one of the sources.  Where an address is not 16-byte aligned
 * everything is read element by element.  PAIR: vectors that a thread reads at once of up to four ranks.
 */
template <typename Tw, typename To, int PAIR = 2, typename Red, typename Src, typename Dst>
__device__ __forceinline__ void reduce_to(unsigned ranks, Dst dst, Src src, int p, size_t n, Red red, double scale, int int_div) {
  using Aw = typename Elem<Tw>::Acc;
  using Ao = typename Elem<To>::Acc;
  constexpr int VEC = 16 / (int)sizeof(Tw);
  constexpr size_t out_bytes = (size_t)VEC * sizeof(To);
  constexpr size_t out_align = out_bytes < 16 ? out_bytes : 16;
  bool aligned = true;
#pragma unroll
  for (int d = 0; d < kMaxRanks; ++d) aligned = aligned && (!(ranks >> d & 1) || (uintptr_t)dst(d) % out_align == 0);
#pragma unroll
  for (int r = 0; r < kMaxRanks; ++r) aligned = aligned && (r >= p || (uintptr_t)src(r) % 16 == 0);
  const size_t nvec = aligned ? n / VEC : 0;
  union InPack { uint4 u; Tw e[VEC]; };
  union OutPack { uint4 u[(out_bytes + 15) / 16]; To e[VEC]; };

  auto store = [&](size_t v, const OutPack& o) {
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d) {
      if (ranks >> d & 1) {
        To* out = dst(d);
        if constexpr (out_bytes >= 16) {
#pragma unroll
          for (int q = 0; q < (int)(out_bytes / 16); ++q) ((uint4*)out)[v * (out_bytes / 16) + q] = o.u[q];
        } else if constexpr (out_bytes == 8) {
          ((uint2*)out)[v] = *(const uint2*)&o.u[0];
        } else {
          ((uint32_t*)out)[v] = *(const uint32_t*)&o.u[0];
        }
      }
    }
  };

  // Every rank's words are under way before the first one is folded (eight 16-byte loads per thread: two vectors of up
  // to four ranks, one of up to eight): one memory latency per round instead of one per rank.
  const size_t stride = blockDim.x;
  auto rounds = [&](auto most, auto vecs) __attribute__((always_inline)) {
    constexpr int R = decltype(most)::value, U = decltype(vecs)::value;
    for (size_t v = (size_t)(threadIdx.x >> 5) * (32 * U) + (threadIdx.x & 31); v < nvec; v += stride * U) {
      InPack in[R][U];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r < p) {
          const uint4* s = (const uint4*)src(r) + v;
          in[r][0].u = __ldcg(s);
          if constexpr (U == 2) in[r][1].u = v + 32 < nvec ? __ldcg(s + 32) : uint4{0, 0, 0, 0};
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        Aw acc[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = Elem<Tw>::up(in[0][u].e[k]);
#pragma unroll
        for (int r = 1; r < R; ++r)
          if (r < p) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) acc[k] = red(acc[k], Elem<Tw>::up(in[r][u].e[k]));
          }
        OutPack o;
#pragma unroll
        for (int k = 0; k < VEC; ++k) o.e[k] = Elem<To>::down(acc_cast<Ao, Aw>(finish_acc(acc[k], scale, int_div)));
        if (u == 0 || v + 32 * u < nvec) store(v + 32 * u, o);
      }
    }
  };
  if (p <= kMaxRanks / 2) rounds(std::integral_constant<int, kMaxRanks / 2>(), std::integral_constant<int, PAIR>());
  else rounds(std::integral_constant<int, kMaxRanks>(), std::integral_constant<int, 1>());
  // scalar remainder (and the whole range when an address is not aligned for vector accesses)
  for (size_t i = nvec * VEC + threadIdx.x; i < n; i += stride) {
    Aw acc = Aw();
#pragma unroll
    for (int r = 0; r < kMaxRanks; ++r) {
      if (r < p) {
        const Aw x = Elem<Tw>::up(__ldcg((const Tw*)src(r) + i));
        acc = r == 0 ? x : red(acc, x);
      }
    }
    const To out = Elem<To>::down(acc_cast<Ao, Aw>(finish_acc(acc, scale, int_div)));
#pragma unroll
    for (int d = 0; d < kMaxRanks; ++d)
      if (ranks >> d & 1) dst(d)[i] = out;
  }
}

/** One destination, contributions at bases[r] + byte_off. */
template <typename Tw, typename To, int PAIR = 2, typename Red>
__device__ __forceinline__ void cta_reduce(To* out, char* const* bases, size_t byte_off, int p, size_t n, Red red, double scale,
                                           int int_div) {
  reduce_to<Tw, To, PAIR>(1u, [&](int) { return out; }, [&](int r) { return bases[r] + byte_off; }, p, n, red, scale, int_div);
}

}  // namespace device
}  // namespace internal
}  // namespace Al
