// Stand-alone element-wise kernels: scale + dtype cast, fused momentum SGD over
// a flat parameter buffer, fill.  All are bandwidth bound; each thread moves
// 16 bytes per access and grids are sized in multiples of the SM count.
#include <algorithm>

#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kThreads = 256;

int grid_for(size_t work_items) {
  // persistent-style grid: 148 SMs x 8 CTAs of 256 threads covers the machine
  size_t blocks = (work_items + kThreads - 1) / kThreads;
  const size_t cap = 148 * 8;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  return (int)blocks;
}

template <typename Ti, typename To>
__global__ void __launch_bounds__(kThreads) scale_cast_kernel(To* __restrict__ out, const Ti* __restrict__ in,
                                                               size_t n, float scale) {
  constexpr int VEC = 16 / (sizeof(Ti) > sizeof(To) ? sizeof(Ti) : sizeof(To));  // widest side moves 16 B
  using Ai = typename Elem<Ti>::Acc;
  using Ao = typename Elem<To>::Acc;
  const bool aligned = ((uintptr_t)in % (VEC * sizeof(Ti)) == 0) && ((uintptr_t)out % (VEC * sizeof(To)) == 0);
  const size_t nvec = aligned ? n / VEC : 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  struct alignas(VEC * sizeof(Ti)) PI { Ti e[VEC]; };
  struct alignas(VEC * sizeof(To)) PO { To e[VEC]; };
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += stride) {
    PI a = ((const PI*)in)[v];
    PO o;
#pragma unroll
    for (int k = 0; k < VEC; ++k) o.e[k] = Elem<To>::down((Ao)((Ai)Elem<Ti>::up(a.e[k]) * (Ai)scale));
    ((PO*)out)[v] = o;
  }
  for (size_t i = nvec * VEC + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = Elem<To>::down((Ao)((Ai)Elem<Ti>::up(in[i]) * (Ai)scale));
}

template <typename Ti, typename To>
void run_scale_cast(void* out, const void* in, size_t n, double scale, cudaStream_t s) {
  if (n == 0) return;
  constexpr int VEC = 16 / (sizeof(Ti) > sizeof(To) ? sizeof(Ti) : sizeof(To));
  scale_cast_kernel<Ti, To><<<grid_for(n / VEC + 1), kThreads, 0, s>>>((To*)out, (const Ti*)in, n, (float)scale);
  AL_CHECK_CUDA(cudaGetLastError());
}

__global__ void __launch_bounds__(kThreads) scale_f64_kernel(double* out, const double* in, size_t n, double scale) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = in[i] * scale;
}

/**
 * Casts of several tensors: a CTA has 2048 elements of one of them, eight per thread.  A block's weights are small (4 K to 2.4 M elements), and a
 * launch each way for every one of them costs more than moving them.
 */
constexpr unsigned kCastTile = kThreads * 8;

template <typename Ti, typename To>
__global__ void __launch_bounds__(kThreads) cast_all_kernel(const __grid_constant__ CastTable t) {
  int k = 0;
#pragma unroll
  for (int s = CastTable::kMax / 2; s > 0; s >>= 1)
    if (k + s < t.count && blockIdx.x >= t.first[k + s]) k += s;
  const size_t i = (size_t)(blockIdx.x - t.first[k]) * kCastTile + (size_t)threadIdx.x * 8, n = t.n[k];
  const Ti* in = (const Ti*)t.in[k] + i;
  To* out = (To*)t.out[k] + i;
  auto one = [](Ti v) { return Elem<To>::down((float)Elem<Ti>::up(v)); };
  struct alignas(16) PI { Ti e[8]; };
  struct alignas(16) PO { To e[8]; };
  if (i + 8 <= n) {
    const PI a = *(const PI*)in;
    PO o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.e[e] = one(a.e[e]);
    *(PO*)out = o;
  } else {
    for (int e = 0; e < 8 && i + e < n; ++e) out[e] = one(in[e]);
  }
}

/** One element; the roundings are written out, so that every path to it gives the same bits. */
__device__ __forceinline__ void sgd_update(float& p, float& m, float g, float lr, float mu, float wd, float gscale, int first) {
  const float ge = fmaf(wd, p, g * gscale);
  m = first ? ge : fmaf(mu, m, ge);
  p = fmaf(-lr, m, p);
}

__global__ void __launch_bounds__(kThreads) sgd_momentum_kernel(float* __restrict__ param, float* __restrict__ mom,
                                                                 float* __restrict__ grad, size_t n, float lr,
                                                                 float mu, float wd, float gscale, int first,
                                                                 int zero_grad) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const bool aligned = (((uintptr_t)param | (uintptr_t)mom | (uintptr_t)grad) & 15) == 0;
  const size_t nvec = aligned ? n / 4 : 0;
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += stride) {
    float4 p = ((float4*)param)[v];
    float4 g = ((float4*)grad)[v];
    float4 m = first ? make_float4(0.f, 0.f, 0.f, 0.f) : ((float4*)mom)[v];
    float* pp = (float*)&p; float* gg = (float*)&g; float* mm = (float*)&m;
#pragma unroll
    for (int k = 0; k < 4; ++k) sgd_update(pp[k], mm[k], gg[k], lr, mu, wd, gscale, first);
    ((float4*)param)[v] = p;
    ((float4*)mom)[v] = m;
    if (zero_grad) ((float4*)grad)[v] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (size_t i = nvec * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    float p = param[i], m = first ? 0.f : mom[i];
    sgd_update(p, m, grad[i], lr, mu, wd, gscale, first);
    mom[i] = m;
    param[i] = p;
    if (zero_grad) grad[i] = 0.f;
  }
}

/**
 * Momentum SGD over tensors whose gradients lie where backward left them.  Adding each to the flat gradient first takes a launch and three
 * passes per tensor (161 of them, 340 us of a ResNet-50 step, and 0.8 ms of the host); here the optimizer reads the tensor and the
 * flat gradient (whatever the caller left there), and zeroes the latter: seven passes over the model, 97 us for 25.6 M parameters.
 * A CTA has a tile of 4096 elements of one tensor, 16 of them per thread under way at once in four arrays.
 */
constexpr unsigned kSgdTile = kThreads * 16;

__global__ void __launch_bounds__(kThreads) sgd_momentum_from_kernel(float* __restrict__ param, float* __restrict__ mom, float* __restrict__ flat,
                                                                      const __grid_constant__ GradTable t, float lr, float mu, float wd,
                                                                      float gscale, int first) {
  int k = 0;
#pragma unroll
  for (int s = GradTable::kMax / 2; s > 0; s >>= 1)
    if (k + s < t.n && blockIdx.x >= t.first[k + s]) k += s;
  const unsigned from = (blockIdx.x - t.first[k]) * kSgdTile, count = t.numel[k];
  const float* grad = t.grad[k];
  const size_t base = t.at[k];
  auto step = [&](float& p, float& m, float f, float g) { sgd_update(p, m, f + g, lr, mu, wd, gscale, first); };
  float4 p[4], m[4], f[4], g[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned i = from + (threadIdx.x + j * kThreads) * 4;
    if (i + 4 <= count) {
      p[j] = *(const float4*)(param + base + i);
      f[j] = *(const float4*)(flat + base + i);
      m[j] = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *(const float4*)(mom + base + i);
      g[j] = grad ? *(const float4*)(grad + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned i = from + (threadIdx.x + j * kThreads) * 4;
    if (i + 4 <= count) {
      step(p[j].x, m[j].x, f[j].x, g[j].x);
      step(p[j].y, m[j].y, f[j].y, g[j].y);
      step(p[j].z, m[j].z, f[j].z, g[j].z);
      step(p[j].w, m[j].w, f[j].w, g[j].w);
      *(float4*)(param + base + i) = p[j];
      *(float4*)(mom + base + i) = m[j];
      *(float4*)(flat + base + i) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      for (unsigned e = i; e < count && e < i + 4; ++e) {
        float pe = param[base + e], me = first ? 0.f : mom[base + e];
        step(pe, me, flat[base + e], grad ? grad[e] : 0.f);
        param[base + e] = pe;
        mom[base + e] = me;
        flat[base + e] = 0.f;
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads) fill_u32_kernel(uint32_t* out, size_t n, uint32_t value) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t nvec = (((uintptr_t)out & 15) == 0) ? n / 4 : 0;
  const uint4 v4 = make_uint4(value, value, value, value);
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += stride) ((uint4*)out)[v] = v4;
  for (size_t i = nvec * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = value;
}

}  // namespace

void launch_scale_cast(void* out, DType out_dt, const void* in, DType in_dt, size_t n, double scale,
                       cudaStream_t stream) {
  using bf = __nv_bfloat16;
  using hf = __half;
#define AL_SC(DI, DO, TI, TO) \
  if (in_dt == DType::DI && out_dt == DType::DO) return run_scale_cast<TI, TO>(out, in, n, scale, stream);
  AL_SC(f32, f32, float, float)
  AL_SC(f32, bf16, float, bf)
  AL_SC(f32, f16, float, hf)
  AL_SC(bf16, f32, bf, float)
  AL_SC(f16, f32, hf, float)
  AL_SC(bf16, bf16, bf, bf)
  AL_SC(f16, f16, hf, hf)
  AL_SC(bf16, f16, bf, hf)
  AL_SC(f16, bf16, hf, bf)
#undef AL_SC
  if (in_dt == DType::f64 && out_dt == DType::f64) {
    if (n == 0) return;
    scale_f64_kernel<<<grid_for(n), kThreads, 0, stream>>>((double*)out, (const double*)in, n, scale);
    AL_CHECK_CUDA(cudaGetLastError());
    return;
  }
  throw_al_exception("scale_cast: unsupported type pair ", dtype_name(in_dt), " -> ", dtype_name(out_dt));
}

void launch_cast_all(void* const* out, DType out_dt, const void* const* in, DType in_dt, const size_t* n, int count, cudaStream_t stream) {
  using bf = __nv_bfloat16;
  void (*kernel)(const CastTable) = nullptr;
  if (in_dt == DType::f32 && out_dt == DType::bf16) kernel = cast_all_kernel<float, bf>;
  else if (in_dt == DType::f32 && out_dt == DType::f16) kernel = cast_all_kernel<float, __half>;
  else if (in_dt == DType::bf16 && out_dt == DType::f32) kernel = cast_all_kernel<bf, float>;
  else if (in_dt == DType::f16 && out_dt == DType::f32) kernel = cast_all_kernel<__half, float>;
  else throw_al_exception("cast_all: unsupported type pair ", dtype_name(in_dt), " -> ", dtype_name(out_dt));
  for (int from = 0; from < count; from += CastTable::kMax) {
    CastTable t;
    t.count = std::min(count - from, CastTable::kMax);
    size_t tiles = 0;
    for (int k = 0; k < t.count; ++k) {
      t.in[k] = in[from + k];
      t.out[k] = out[from + k];
      t.n[k] = n[from + k];
      if (((uintptr_t)t.in[k] | (uintptr_t)t.out[k]) % 16 != 0) throw_al_exception("cast_all: a tensor does not begin on 16 bytes");
      t.first[k] = (unsigned)tiles;
      tiles += (t.n[k] + kCastTile - 1) / kCastTile;
      if (tiles > 0x7fffffff) throw_al_exception("cast_all: too many elements");
    }
    t.first[t.count] = (unsigned)tiles;
    if (tiles == 0) continue;
    kernel<<<(unsigned)tiles, kThreads, 0, stream>>>(t);
    AL_CHECK_CUDA(cudaGetLastError());
  }
}

void launch_sgd_momentum(float* param, float* momentum, float* grad, size_t n, float lr, float mu,
                         float weight_decay, float grad_scale, int first_step, int zero_grad,
                         cudaStream_t stream) {
  if (n == 0) return;
  sgd_momentum_kernel<<<grid_for(n / 4 + 1), kThreads, 0, stream>>>(param, momentum, grad, n, lr, mu, weight_decay,
                                                                  grad_scale, first_step, zero_grad);
  AL_CHECK_CUDA(cudaGetLastError());
}

void launch_sgd_momentum_from(float* param, float* momentum, float* flat_grad, const float* const* grad, const size_t* at,
                              const size_t* numel, int n, float lr, float mu, float weight_decay, float grad_scale, int first_step,
                              cudaStream_t stream) {
  for (int from = 0; from < n; from += GradTable::kMax) {
    GradTable t;
    t.n = std::min(n - from, GradTable::kMax);
    unsigned tiles = 0;
    for (int k = 0; k < t.n; ++k) {
      const size_t count = numel[from + k];
      if (count > 0xffffff00u - kSgdTile || at[from + k] % 4 != 0 || (uintptr_t)grad[from + k] % 16 != 0)
        throw_al_exception("sgd: a gradient of ", count, " elements at ", at[from + k], " is not of the form that the kernel reads");
      t.grad[k] = grad[from + k];
      t.at[k] = at[from + k];
      t.numel[k] = (unsigned)count;
      t.first[k] = tiles;
      tiles += (unsigned)((count + kSgdTile - 1) / kSgdTile);
    }
    t.first[t.n] = tiles;
    if (tiles == 0) continue;
    sgd_momentum_from_kernel<<<tiles, kThreads, 0, stream>>>(param, momentum, flat_grad, t, lr, mu, weight_decay, grad_scale, first_step);
    AL_CHECK_CUDA(cudaGetLastError());
  }
}

void launch_fill_u32(uint32_t* out, size_t n, uint32_t value, cudaStream_t stream) {
  if (n == 0) return;
  fill_u32_kernel<<<grid_for(n / 4 + 1), kThreads, 0, stream>>>(out, n, value);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace device
}  // namespace internal
}  // namespace Al
