// Input of a network's first convolution (7 x 7 every two pixels, border 3, three channels) laid out for tensor cores, and the weight's
// gradient back in the weight's layout.
//
// The library convolves three channels on its legacy tensor path alone, with an input that it pads to four or eight
// channels first: 256 x 3 x 224 x 224 bf16 takes 1600 us forward and 911 us for the weight's gradient, of which memory would be 75 and 65.
// Here the pixels that a row of outputs sees are put side by side as channels: 8 columns x 3 channels of two input rows
// (48 channels, and 16 of zeros) make one pixel, and the convolution becomes one of 64 channels over four rows, which takes 261 and
// 168 us.  (48 channels 335 / 179, two by two pixels as 16 channels and 4 x 4 taps 516 / 588, the seven rows on their own 273 / 326.)
//
// What bounds the layout kernel is writing 128 bytes per pixel (422 MB in that case).  A CTA has eight input rows, a warp one of them: it
// reads each once, converts it into shared memory with its border, and the threads write 16 bytes of a pixel each, eight to a
// pixel.  (With two rows to a CTA the loads' latency was most of it: 141 us; now 93, 88 at the copy rate.)
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kThreads = 256;
constexpr int kSeen = 8, kIn = 3, kCh = 64;   // columns that an output sees (one more than it has taps), channels of an image, of a pixel here
constexpr int kRow = kSeen * kIn;             // values of one input row
constexpr int kPairs = 4;                     // row pairs of a CTA: as many rows as it has warps
static_assert(2 * kPairs == kThreads / 32, "a warp has one row");

/** Is one of two values infinite or NaN? */
template <typename T>
__device__ __forceinline__ bool not_finite2(uint32_t w) {
  constexpr uint32_t top = std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
  return (w & top) == top || (w >> 16 & top) == top;
}

/** watch (or nullptr): a word per CTA, whether the second row of one of its pairs has a value that is not finite (stem_repair_kernel). */
template <typename Ti, typename To>
__global__ void __launch_bounds__(kThreads) stem_gather_kernel(const __grid_constant__ StemShape s, const Ti* __restrict__ x, To* __restrict__ out,
                                                               const float* __restrict__ weight, To* __restrict__ packed, unsigned rows,
                                                               unsigned* __restrict__ watch) {
  auto as = [](Ti v) { return Elem<To>::down((float)Elem<Ti>::up(v)); };
  const To zero = Elem<To>::down(0.f);
  if (blockIdx.x >= rows) {   // the weight: [output][row pair][channel], zero where there is no tap
    const unsigned i = (blockIdx.x - rows) * kThreads + threadIdx.x;
    if (i >= (unsigned)s.oc * 4 * kCh) return;
    const int c = (int)(i % kCh), a = (int)(i / kCh) % 4, o = (int)(i / (4 * kCh));
    const int u = 2 * a + c / kRow, v = c % kRow / kIn, ch = c % kIn;
    packed[i] = c < 2 * kRow && u < 7 && v < 7 ? Elem<To>::down(weight[o * s.ws[0] + ch * s.ws[1] + u * s.ws[2] + v * s.ws[3]]) : zero;
    return;
  }
  extern __shared__ uint32_t smem[];   // 2 kPairs rows of (columns + border) x 3 values
  const int cols = 2 * s.ow + 6, groups = (s.oh + 3 + kPairs - 1) / kPairs;
  const int n = (int)(blockIdx.x / (unsigned)groups), r0 = (int)(blockIdx.x % (unsigned)groups) * kPairs;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    const int h = 2 * r0 + warp - 3;
    To* buf = (To*)smem + warp * cols * kIn;
    const Ti* line = x + (ptrdiff_t)n * s.xs[0] + (ptrdiff_t)h * s.xs[2];
    if (h < 0 || h >= s.h) {
      for (int i = lane; i < cols * kIn; i += 32) buf[i] = zero;
    } else {
      for (int i = lane; i < 3 * kIn; i += 32) buf[i] = zero;
      for (int i = (s.w + 3) * kIn + lane; i < cols * kIn; i += 32) buf[i] = zero;
      buf += 3 * kIn;
      const int run = s.w * kIn;
      if (s.xs[1] == 1 && s.xs[3] == kIn && sizeof(Ti) == 4 && (uintptr_t)line % 16 == 0) {   // channels-last: one run of values
        for (int i0 = 0; i0 < run / 4; i0 += 4 * 32) {
          float4 v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (i0 + k * 32 + lane < run / 4) v[k] = ((const float4*)line)[i0 + k * 32 + lane];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int i = i0 + k * 32 + lane;
            if (i < run / 4) {
              buf[4 * i] = Elem<To>::down(v[k].x);
              buf[4 * i + 1] = Elem<To>::down(v[k].y);
              buf[4 * i + 2] = Elem<To>::down(v[k].z);
              buf[4 * i + 3] = Elem<To>::down(v[k].w);
            }
          }
        }
        for (int i = run / 4 * 4 + lane; i < run; i += 32) buf[i] = as(line[i]);
      } else {
        for (int w0 = 0; w0 < s.w; w0 += 4 * 32) {   // any strides: the channels of four pixels under way at once
          Ti v[4][kIn];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int ch = 0; ch < kIn; ++ch)
              if (w0 + k * 32 + lane < s.w) v[k][ch] = line[(ptrdiff_t)(w0 + k * 32 + lane) * s.xs[3] + ch * s.xs[1]];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int ch = 0; ch < kIn; ++ch)
              if (w0 + k * 32 + lane < s.w) buf[(w0 + k * 32 + lane) * kIn + ch] = as(v[k][ch]);
        }
      }
    }
  }
  __syncthreads();
  if (watch) {
    bool odd = false;
    const unsigned words = (unsigned)cols * kIn / 2;
    for (unsigned i = threadIdx.x; i < kPairs * words; i += kThreads) odd |= not_finite2<To>(smem[(2 * (i / words) + 1) * words + i % words]);
    odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) watch[blockIdx.x] = odd;
  }
  // a pixel's 24 values of a row begin 6 values behind its neighbour's: on 4 bytes, not on 16.  The last three are of the column behind its
  // window: zeros here, so that the weight's zeros there meet nothing that is not finite.
  const int pixels = min(kPairs, s.oh + 3 - r0) * s.ow, k = threadIdx.x % (kCh / 8);
  uint4* dst = (uint4*)out + ((size_t)n * (s.oh + 3) + r0) * s.ow * (kCh / 8);
  int j = threadIdx.x / (kCh / 8) % s.ow, pair = threadIdx.x / (kCh / 8) / s.ow;
  for (int i = threadIdx.x / (kCh / 8); i < pixels; i += kThreads / (kCh / 8)) {
    uint4 v = uint4{0, 0, 0, 0};
    if (k < 6) {
      const uint32_t* p = smem + (((2 * pair + k / 3) * cols + 2 * j) * kIn + (k % 3) * 8) / 2;
      v = uint4{p[0], p[1], p[2], p[3]};
      if (k % 3 == 2) v = uint4{v.x, v.y, v.z & 0xffffu, 0};
    }
    dst[(size_t)i * (kCh / 8) + k] = v;
    for (j += kThreads / (kCh / 8); j >= s.ow; j -= s.ow) ++pair;
  }
}

/**
 * Results whose window ends beside a value that is not finite.  The second row of a result's last pair lies below its window; the weight is zero
 * there, but that row is in the window of the next result, so its values have to be in the layout, and zero times infinity is NaN.
 * Those results are computed again without that row, a warp per pixel.  Images are finite nearly always: then the launch
 * reads a word per eight rows of them and is gone.
 */
template <typename T>
__global__ void __launch_bounds__(kThreads) stem_repair_kernel(const __grid_constant__ StemShape s, const T* __restrict__ seen, const T* __restrict__ packed,
                                                               const unsigned* __restrict__ watch, unsigned rows, T* __restrict__ y) {
  __shared__ unsigned found[kThreads];
  const unsigned from = blockIdx.x * kThreads;
  found[threadIdx.x] = from + threadIdx.x < rows ? watch[from + threadIdx.x] : 0;
  if (!__syncthreads_or(found[threadIdx.x])) return;
  const int groups = (s.oh + 3 + kPairs - 1) / kPairs, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned t = 0; t < kThreads; ++t) {
    if (!found[t]) continue;
    const int n = (int)((from + t) / (unsigned)groups), r0 = (int)((from + t) % (unsigned)groups) * kPairs;
    const int pixels = min(kPairs, s.oh + 3 - r0) * s.ow;
    for (int i = warp; i < pixels; i += kThreads / 32) {
      const int oh = r0 + i / s.ow - 3, ow = i % s.ow;
      if (oh < 0) continue;
      const T* first = seen + (((size_t)n * (s.oh + 3) + oh) * s.ow + ow) * kCh;   // of four pairs of rows, s.ow pixels apart
      const size_t step = (size_t)s.ow * kCh;
      const bool odd = lane < 7 * kIn && not_finite2<T>(((const uint16_t*)first)[3 * step + kRow + lane]);
      if (!__any_sync(0xffffffffu, odd)) continue;
      for (int o = lane; o < s.oc; o += 32) {
        float sum = 0.f;
        for (int u = 0; u < 7; ++u)
          for (int c = 0; c < 7 * kIn; ++c)
            sum = fmaf(Elem<T>::up(first[u / 2 * step + u % 2 * kRow + c]), Elem<T>::up(packed[(o * 4 + u / 2) * kCh + u % 2 * kRow + c]), sum);
        y[(size_t)n * s.ws[0] + (size_t)o * s.ws[1] + (size_t)oh * s.ws[2] + (size_t)ow * s.ws[3]] = Elem<T>::down(sum);
      }
    }
  }
}

/** grad[o][ch][u][v] out of the gradient of the packed weight. */
template <typename T>
__global__ void __launch_bounds__(kThreads) stem_scatter_kernel(const __grid_constant__ StemShape s, const T* __restrict__ packed, float* __restrict__ grad) {
  const unsigned i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= (unsigned)s.oc * kIn * 49) return;
  const int v = (int)(i % 7), u = (int)(i / 7) % 7, ch = (int)(i / 49) % kIn, o = (int)(i / (49 * kIn));
  grad[o * s.ws[0] + ch * s.ws[1] + u * s.ws[2] + v * s.ws[3]] = (float)Elem<T>::up(packed[(o * 4 + u / 2) * kCh + u % 2 * kRow + v * kIn + ch]);
}

void check(const StemShape& s) {
  if (s.n < 1 || s.h < 1 || s.w < 1 || s.oc < 1 || s.oh != (s.h - 1) / 2 + 1 || s.ow != (s.w - 1) / 2 + 1 ||
      (size_t)s.n * (size_t)(s.oh + 3) > 0x70000000u || s.w > 700 || s.oc > 1 << 16)
    throw_al_exception("first convolution: unsupported shape");
}

unsigned gather_rows(const StemShape& s) { return (unsigned)(s.n * ((s.oh + 3 + kPairs - 1) / kPairs)); }

template <typename Ti, typename To>
void gather(const StemShape& s, const void* x, void* out, const float* weight, void* packed, unsigned* watch, cudaStream_t stream) {
  const unsigned rows = gather_rows(s), more = (unsigned)((s.oc * 4 * kCh + kThreads - 1) / kThreads);
  const size_t smem = (size_t)2 * kPairs * (2 * s.ow + 6) * kIn * sizeof(To);   // (a whole number of 4-byte words: a row is 6 (ow + 3) values)
  stem_gather_kernel<Ti, To><<<rows + more, kThreads, smem, stream>>>(s, (const Ti*)x, (To*)out, weight, (To*)packed, rows, watch);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace

size_t stem_watch_words(const StemShape& s) {
  check(s);
  return gather_rows(s);
}

void launch_stem_gather(const StemShape& s, const void* x, DType in, void* out, const float* weight, void* packed, DType dt, unsigned* watch,
                        cudaStream_t stream) {
  using bf = __nv_bfloat16;
  check(s);
  if (in == DType::f32 && dt == DType::bf16) return gather<float, bf>(s, x, out, weight, packed, watch, stream);
  if (in == DType::f32 && dt == DType::f16) return gather<float, __half>(s, x, out, weight, packed, watch, stream);
  if (in == DType::bf16 && dt == DType::bf16) return gather<bf, bf>(s, x, out, weight, packed, watch, stream);
  if (in == DType::f16 && dt == DType::f16) return gather<__half, __half>(s, x, out, weight, packed, watch, stream);
  throw_al_exception("first convolution: unsupported datatypes ", dtype_name(in), ", ", dtype_name(dt));
}

void launch_stem_repair(const StemShape& s, const void* seen, const void* packed, const unsigned* watch, void* y, DType dt, cudaStream_t stream) {
  check(s);
  const unsigned rows = gather_rows(s), blocks = (rows + kThreads - 1) / kThreads;
  if (dt == DType::bf16) stem_repair_kernel<<<blocks, kThreads, 0, stream>>>(s, (const __nv_bfloat16*)seen, (const __nv_bfloat16*)packed, watch, rows, (__nv_bfloat16*)y);
  else if (dt == DType::f16) stem_repair_kernel<<<blocks, kThreads, 0, stream>>>(s, (const __half*)seen, (const __half*)packed, watch, rows, (__half*)y);
  else throw_al_exception("first convolution: unsupported datatype ", dtype_name(dt));
  AL_CHECK_CUDA(cudaGetLastError());
}

void launch_stem_scatter(const StemShape& s, const void* packed, float* grad, DType dt, cudaStream_t stream) {
  check(s);
  const unsigned blocks = (unsigned)((s.oc * kIn * 49 + kThreads - 1) / kThreads);
  if (dt == DType::bf16) stem_scatter_kernel<__nv_bfloat16><<<blocks, kThreads, 0, stream>>>(s, (const __nv_bfloat16*)packed, grad);
  else if (dt == DType::f16) stem_scatter_kernel<__half><<<blocks, kThreads, 0, stream>>>(s, (const __half*)packed, grad);
  else throw_al_exception("first convolution: unsupported datatype ", dtype_name(dt));
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
