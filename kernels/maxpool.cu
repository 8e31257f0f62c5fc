// Max pooling of channels-last 16-bit activations and its backward.
//
// Both are bound by memory: the input is read (forward) or its gradient written (backward) once.  A thread owns 8
// channels of one pixel; forward leaves the winner's place in its window as one byte (the framework's own operation
// leaves eight bytes), and backward gathers - each input pixel asks the few windows that cover it - so that nothing is
// zeroed first and nothing is added atomically.
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
  maxpool_forward_kernel<T><<<blocks_of(total), kThreads, 0, stream>>>((const T*)x, (T*)y, place, s, total);
  AL_CHECK_CUDA(cudaGetLastError());
}
template <typename T>
void backward(const void* dy, const unsigned char* place, void* dx, const PoolShape& s, cudaStream_t stream) {
  const unsigned total = threads_of((size_t)s.n * s.h * s.w * (s.c / 8));
  maxpool_backward_kernel<T><<<blocks_of(total), kThreads, 0, stream>>>((const T*)dy, place, (T*)dx, s, total);
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
