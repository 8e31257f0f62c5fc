// Max pooling of channels-last 16-bit activations and its backward.
//
// Both are bound by memory: the input is read (forward) or its gradient written (backward) once.  A thread owns 8
// channels of one pixel; forward leaves the winner's place in its window as one byte (the framework's own operation
// leaves eight bytes), and backward gathers - each input pixel asks the few windows that cover it - so that nothing is
// zeroed first and nothing is added atomically.
//
// Windows of 3 every 2 pixels with a border of 1 (what residual networks pool with) have kernels of their own: what the loops below wait
// for is one load after the other, so forward has its nine loads under way at once, and backward gives a thread two by two
// pixels, which four windows cover, instead of asking one, two, two and four windows for the four of them.  256 x 64 x 112 x 112
// bf16, loops / now, us: forward 250 / 127 (342 with the nine compared one channel at a time in fp32), backward 443 / 135; 86 at the copy rate.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kThreads = 256;

template <typename T>
union Pack8 {
  uint4 u;
  T e[8];
};
union Bytes8 {
  uint2 u;
  unsigned char e[8];
};

template <typename T>
__global__ void __launch_bounds__(kThreads) maxpool_forward_kernel(const T* __restrict__ x, T* __restrict__ y, unsigned char* __restrict__ place,
                                                                   const PoolShape s, unsigned total) {
  const unsigned i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= total) return;
  const unsigned cols = (unsigned)s.c / 8;
  const unsigned pixel = i / cols, col = i - pixel * cols;
  const unsigned row = pixel / (unsigned)s.ow;
  const int ow = (int)(pixel - row * (unsigned)s.ow);
  const size_t n = row / (unsigned)s.oh;
  const int oh = (int)(row % (unsigned)s.oh);
  const int h0 = oh * s.stride - s.pad, w0 = ow * s.stride - s.pad;
  Pack8<T> best;
  Bytes8 at;
  bool first = true;
  for (int ky = 0; ky < s.k; ++ky) {
    const int h = h0 + ky;
    if (h < 0 || h >= s.h) continue;
    for (int kx = 0; kx < s.k; ++kx) {
      const int w = w0 + kx;
      if (w < 0 || w >= s.w) continue;
      Pack8<T> v;
      v.u = ((const uint4*)x)[((n * s.h + h) * s.w + w) * cols + col];
      const unsigned char k = (unsigned char)(ky * s.k + kx);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float a = Elem<T>::up(v.e[e]), b = Elem<T>::up(best.e[e]);
        if (first || a > b || a != a) {   // the first of equals; a NaN wins
          best.e[e] = v.e[e];
          at.e[e] = k;
        }
      }
      first = false;
    }
  }
  ((uint4*)y)[i] = best.u;
  ((uint2*)place)[i] = at.u;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) maxpool_backward_kernel(const T* __restrict__ dy, const unsigned char* __restrict__ place,
                                                                    T* __restrict__ dx, const PoolShape s, unsigned total) {
  const unsigned i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= total) return;
  const unsigned cols = (unsigned)s.c / 8;
  const unsigned pixel = i / cols, col = i - pixel * cols;
  const unsigned row = pixel / (unsigned)s.w;
  const int w = (int)(pixel - row * (unsigned)s.w) + s.pad;
  const size_t n = row / (unsigned)s.h;
  const int h = (int)(row % (unsigned)s.h) + s.pad;
  // windows [lo, hi] start at most k - 1 before this pixel and not behind it
  const int h_hi = min(h / s.stride, s.oh - 1), h_lo = h < s.k ? 0 : (h - s.k) / s.stride + 1;
  const int w_hi = min(w / s.stride, s.ow - 1), w_lo = w < s.k ? 0 : (w - s.k) / s.stride + 1;
  float sum[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) sum[e] = 0.f;
  for (int oh = h_lo; oh <= h_hi; ++oh)
    for (int ow = w_lo; ow <= w_hi; ++ow) {
      const size_t o = ((n * s.oh + oh) * s.ow + ow) * cols + col;
      const unsigned char k = (unsigned char)((h - oh * s.stride) * s.k + (w - ow * s.stride));
      Bytes8 at;
      Pack8<T> g;
      at.u = ((const uint2*)place)[o];
      g.u = ((const uint4*)dy)[o];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (at.e[e] == k) sum[e] += Elem<T>::up(g.e[e]);
    }
  Pack8<T> out;
#pragma unroll
  for (int e = 0; e < 8; ++e) out.e[e] = Elem<T>::down(sum[e]);
  ((uint4*)dx)[i] = out.u;
}

/** Two elements at once: their larger ones (NaN if one is), and 0xffff where they are equal. */
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b, __nv_bfloat16) {
  const __nv_bfloat162 m = __hmax2_nan(*(const __nv_bfloat162*)&a, *(const __nv_bfloat162*)&b);
  return *(const uint32_t*)&m;
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b, __half) {
  const __half2 m = __hmax2_nan(*(const __half2*)&a, *(const __half2*)&b);
  return *(const uint32_t*)&m;
}
__device__ __forceinline__ uint32_t equal2(uint32_t a, uint32_t b, __nv_bfloat16) { return __heq2_mask(*(const __nv_bfloat162*)&a, *(const __nv_bfloat162*)&b); }
__device__ __forceinline__ uint32_t equal2(uint32_t a, uint32_t b, __half) { return __heq2_mask(*(const __half2*)&a, *(const __half2*)&b); }
template <typename T> constexpr uint32_t kLowest2 = std::is_same<T, __half>::value ? 0xfc00fc00u : 0xff80ff80u;   // minus infinity, twice

/** A thread has eight channels of one result: the largest of nine, then the first pixel that equals it, two channels to an instruction. */
template <typename T>
__global__ void __launch_bounds__(kThreads) maxpool3_forward_kernel(const T* __restrict__ x, T* __restrict__ y, unsigned char* __restrict__ place,
                                                                    const PoolShape s, unsigned total) {
  const unsigned i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= total) return;
  const unsigned cols = (unsigned)s.c / 8;
  const unsigned pixel = i / cols, col = i - pixel * cols;
  const unsigned row = pixel / (unsigned)s.ow;
  const int w0 = 2 * (int)(pixel - row * (unsigned)s.ow) - 1, h0 = 2 * (int)(row % (unsigned)s.oh) - 1;
  const uint4* image = (const uint4*)x + (size_t)(row / (unsigned)s.oh) * s.h * s.w * cols + col;
  union Words { uint4 u; uint32_t w[4]; };
  Words v[9];
  bool in[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int h = h0 + k / 3, w = w0 + k % 3;
    in[k] = (unsigned)h < (unsigned)s.h && (unsigned)w < (unsigned)s.w;
    v[k].u = uint4{kLowest2<T>, kLowest2<T>, kLowest2<T>, kLowest2<T>};
    if (in[k]) v[k].u = image[(ptrdiff_t)(h * s.w + w) * cols];
  }
  Words best;
  uint32_t at[4];
  bool settled = true;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t top = v[0].w[q];
#pragma unroll
    for (int k = 1; k < 9; ++k) top = max2(top, v[k].w[q], T());
    uint32_t found = 0;
    at[q] = best.w[q] = 0;
#pragma unroll
    for (int k = 8; k >= 0; --k) {   // backwards, so that the first of equals stays
      const uint32_t m = in[k] ? equal2(v[k].w[q], top, T()) : 0u;
      at[q] = (at[q] & ~m) | ((k * 0x10001u) & m);
      best.w[q] = (best.w[q] & ~m) | (v[k].w[q] & m);
      found |= m;
    }
    settled = settled && found == 0xffffffffu;
  }
  uint2 where = uint2{__byte_perm(at[0], at[1], 0x6420), __byte_perm(at[2], at[3], 0x6420)};
  if (!settled) {   // there is a NaN: it wins, the last one of several
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      uint32_t value = best.w[e / 2] >> (e % 2 * 16) & 0xffffu, k_at = (e < 4 ? where.x : where.y) >> (e % 4 * 8) & 0xffu;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const uint32_t bits = v[k].w[e / 2] >> (e % 2 * 16) & 0xffffu;
        if (in[k] && (bits & 0x7fffu) > (kLowest2<T> & 0x7fffu)) {
          value = bits;
          k_at = (uint32_t)k;
        }
      }
      best.w[e / 2] = (best.w[e / 2] & ~(0xffffu << (e % 2 * 16))) | value << (e % 2 * 16);
      uint32_t& half = e < 4 ? where.x : where.y;
      half = (half & ~(0xffu << (e % 4 * 8))) | k_at << (e % 4 * 8);
    }
  }
  ((uint4*)y)[i] = best.u;
  ((uint2*)place)[i] = where;
}

/** A thread has the pixels (2 i, 2 j) to (2 i + 1, 2 j + 1): the even ones lie in the middle of a window, the odd ones between two. */
template <typename T>
__global__ void __launch_bounds__(kThreads) maxpool3_backward_kernel(const T* __restrict__ dy, const unsigned char* __restrict__ place,
                                                                     T* __restrict__ dx, const PoolShape s, unsigned total) {
  const unsigned t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= total) return;
  const unsigned cols = (unsigned)s.c / 8, bw = (unsigned)(s.w + 1) / 2, bh = (unsigned)(s.h + 1) / 2;
  const unsigned block = t / cols, col = t - block * cols;
  const unsigned row = block / bw;
  const int j = (int)(block - row * bw), i = (int)(row % bh);
  const size_t n = row / bh;
  Bytes8 at[4];
  Pack8<T> g[4];
  bool in[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {   // window (i + q / 2, j + q % 2)
    const int oh = i + q / 2, ow = j + q % 2;
    in[q] = oh < s.oh && ow < s.ow;
    if (in[q]) {
      const size_t o = ((n * s.oh + oh) * s.ow + ow) * cols + col;
      at[q].u = ((const uint2*)place)[o];
      g[q].u = ((const uint4*)dy)[o];
    }
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int h = 2 * i + a, w = 2 * j + b;
      if (h >= s.h || w >= s.w) continue;
      Pack8<T> out;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int ky = a + 1 - 2 * (q / 2), kx = b + 1 - 2 * (q % 2);   // the pixel's place in the window
          if (ky < 0 || kx < 0) continue;
          if (in[q] && at[q].e[e] == ky * 3 + kx) sum += Elem<T>::up(g[q].e[e]);
        }
        out.e[e] = Elem<T>::down(sum);
      }
      ((uint4*)dx)[((n * s.h + h) * s.w + w) * cols + col] = out.u;
    }
}

bool three_by_two(const PoolShape& s) { return s.k == 3 && s.stride == 2 && s.pad == 1; }

void check_shape(const PoolShape& s) {
  if (s.c % 8 != 0 || s.k < 1 || s.k > 15 || s.stride < 1 || s.pad < 0 || 2 * s.pad > s.k || s.n < 1 || s.oh < 1 || s.ow < 1 ||
      (s.oh - 1) * s.stride - s.pad >= s.h || (s.ow - 1) * s.stride - s.pad >= s.w)
    throw_al_exception("max pooling: unsupported shape");
}

/** Threads of a launch; the kernels count them in 32 bits (64-bit divisions doubled their time). */
unsigned threads_of(size_t total) {
  if (total > 0xffffff00u) throw_al_exception("max pooling: more than 2^35 elements");
  return (unsigned)total;
}
unsigned blocks_of(unsigned total) { return (total + kThreads - 1) / kThreads; }

template <typename T>
void forward(const void* x, void* y, unsigned char* place, const PoolShape& s, cudaStream_t stream) {
  const unsigned total = threads_of((size_t)s.n * s.oh * s.ow * (s.c / 8));
  const auto kernel = three_by_two(s) ? maxpool3_forward_kernel<T> : maxpool_forward_kernel<T>;
  kernel<<<blocks_of(total), kThreads, 0, stream>>>((const T*)x, (T*)y, place, s, total);
  AL_CHECK_CUDA(cudaGetLastError());
}
template <typename T>
void backward(const void* dy, const unsigned char* place, void* dx, const PoolShape& s, cudaStream_t stream) {
  const bool by_four = three_by_two(s);
  const unsigned total = threads_of(by_four ? (size_t)s.n * ((s.h + 1) / 2) * ((s.w + 1) / 2) * (s.c / 8) : (size_t)s.n * s.h * s.w * (s.c / 8));
  const auto kernel = by_four ? maxpool3_backward_kernel<T> : maxpool_backward_kernel<T>;
  kernel<<<blocks_of(total), kThreads, 0, stream>>>((const T*)dy, place, (T*)dx, s, total);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace

void launch_maxpool_forward(const void* x, void* y, unsigned char* place, const PoolShape& s, DType dt, cudaStream_t stream) {
  check_shape(s);
  if (dt == DType::bf16) return forward<__nv_bfloat16>(x, y, place, s, stream);
  if (dt == DType::f16) return forward<__half>(x, y, place, s, stream);
  throw_al_exception("max pooling: unsupported datatype ", dtype_name(dt));
}
void launch_maxpool_backward(const void* dy, const unsigned char* place, void* dx, const PoolShape& s, DType dt, cudaStream_t stream) {
  check_shape(s);
  if (dt == DType::bf16) return backward<__nv_bfloat16>(dy, place, dx, s, stream);
  if (dt == DType::f16) return backward<__half>(dy, place, dx, s, stream);
  throw_al_exception("max pooling: unsupported datatype ", dtype_name(dt));
}

}  // namespace device
}  // namespace internal
}  // namespace Al
