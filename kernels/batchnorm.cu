// Batch normalisation of channels-last activations in training, with the residual addition and the ReLU that follow
// it in the same pass, and its backward.
//
// What bounds it is memory: a ResNet-50 step at batch 256 in bf16 normalises 5.7 GB of convolution outputs.  Statistics
// have to be complete before the first output, so the least is two reads and one write forward, two reads of the
// gradient and of the input and one write backward.  A separate ReLU (and addition) costs a read and a write more
// forward and a read, a read and a write backward; here the ReLU leaves one bit per element, which backward reads instead of
// the output.
//
// Layout: x is M rows (N * H * W) of C channels.  A thread owns 8 consecutive channels (one 16-byte access per row) for
// the whole kernel, so that its accumulators and its channels' coefficients stay in registers; a warp covers 512
// consecutive bytes.  CTAs walk the rows in interleaved tiles and the second pass walks them backwards: what the first
// pass read last (up to the 126 MB L2) is what the second reads first.
// Statistics are a thread's sums of deviations, folded with the parallel update of mean and sum of squared deviations (Chan, Golub and
// LeVeque, "Updating formulae and a pairwise algorithm for computing sample variances", 1979), in fp32 and in a fixed order.
//
// Measured, one B200, ResNet-50 training step in bf16 with the modules / when these kernels were new (what came since has it at 20.0 and about
// 8 ms): batch 256 53.7 / 26.2 ms, batch 24 (bound by the host's launches: 1013 / 795 a step) 10.9 / 9.0 ms (repeats differ by up to 8 %).  Three CTAs per
// SM (80 registers, spills in the gradient kernels) took 27.8 ms.
// All 53 of a step, device time before / with sums of deviations, folds in parallel and launches behind the kernel before, us: batch 256 forward 4062 /
// 3799, backward 5419 / 5293; batch 24 795 / 732 and 829 / 723.  Folding in fp64 took 1.5 us more per fold; errors against 64 bits of values around one mean, over
// fourteen shapes, are 0.67 (means), 1.0 (variances), 0.89 and 0.99 (gradients of weight and bias) of what they were.
#include <algorithm>

#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kBnThreads = 256;
constexpr int kBnSms = 148;
constexpr int kBnPerSm = 2;        // CTAs per SM (no spills at up to 128 registers): 2 x 256 threads x 8 x 16 bytes = 64 KB under way per SM
constexpr int kBnRows = 4;         // rows a thread loads at once of each array
constexpr int kBnStatRows = 4, kBnStatPerSm = 4;   // the statistics, which read one array

/**
 * The kernels of a batch norm are launched while the kernel before them on the stream still runs and wait here for its end: their
 * launch then costs the stream nothing.  Everything that a kernel reads or writes comes behind this.
 */
__device__ __forceinline__ void after_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
void launch_behind(void (*kernel)(Params...), dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  AL_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
}

/** How M rows of C channels are cut. */
struct BnGrid {
  size_t rows;          // M
  int channels, cols;   // C, C / 8
  int lx;               // log2 of the columns of a CTA
  unsigned tiles;       // row tiles
  unsigned nblk, ntile_y;
  unsigned each, more;  // row tiles of every CTA, and how many CTAs have one more
  unsigned tile_rows, missing;  // rows of a tile, and how many the last one lacks
};

BnGrid bn_grid(size_t rows, int channels, int rows_per_thread, int per_sm) {
  BnGrid g;
  g.rows = rows;
  g.channels = channels;
  g.cols = channels / 8;
  g.lx = 0;
  while ((1 << g.lx) < g.cols && g.lx < 5) ++g.lx;
  g.ntile_y = (unsigned)((g.cols + (1 << g.lx) - 1) >> g.lx);
  const size_t tile = (size_t)(kBnThreads >> g.lx) * (size_t)rows_per_thread;
  g.tiles = (unsigned)((rows + tile - 1) / tile);
  // one wave: every SM gets per_sm CTAs, each of which walks its share of the tiles
  g.nblk = std::max(1u, std::min(g.tiles, (unsigned)(kBnSms * per_sm) / g.ntile_y));
  g.each = g.tiles / g.nblk;
  g.more = g.tiles % g.nblk;
  g.tile_rows = (unsigned)tile;
  g.missing = (unsigned)((size_t)g.tiles * tile - rows);
  return g;
}

/** Rows that CTA b of g.nblk reads (the last tile belongs to the last CTA that has one more, or else to the last CTA). */
__device__ __forceinline__ float rows_of(const BnGrid& g, unsigned b) {
  const unsigned last = (g.more ? g.more : g.nblk) - 1;
  return (float)((g.each + (b < g.more ? 1u : 0u)) * (size_t)g.tile_rows - (b == last ? g.missing : 0u));
}

template <typename T>
union Pack8 {
  uint4 u;
  T e[8];
};

template <typename T>
__device__ __forceinline__ float up(T v) { return Elem<T>::up(v); }

/** Where a thread stands: its column of 8 channels and its first row inside a tile. */
struct Place {
  int col, ty, TY;
  bool active;
  __device__ __forceinline__ explicit Place(const BnGrid& g) {
    const int tx = threadIdx.x & ((1 << g.lx) - 1);
    col = (int)(blockIdx.y << g.lx) + tx;
    ty = (int)threadIdx.x >> g.lx;
    TY = kBnThreads >> g.lx;
    active = col < g.cols;
  }
};

__device__ __forceinline__ void load8(float* v, const float* src, int col) {
  const float4 a = ((const float4*)src)[2 * col], b = ((const float4*)src)[2 * col + 1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
/**
 * part[b][c] = (mean, sum of squared deviations) of channel c over the rows of CTA b.  A thread sums the deviations of its rows from a
 * value near their mean, and their squares: four instructions per element, where updating the mean with every batch of
 * eight rows took seven, and few enough registers for twice the CTAs.  That value is the mean of the first kBnStatRows rows, and whenever there
 * are four times as many the mean of all so far: with the first rows' mean for good, 256 x 256 x 56 x 56 whose first eight rows of pixels lie a
 * thousand deviations off had errors of the variance of 9.8e-7, now 5.9e-8.  (All 53 forwards of a step 3652 -> 3705 us at batch 256, 815 -> 829 at 24; moved
 * at every doubling, behind the rows and not while they are loaded, 3730 and 843.)
 */
template <typename T>
__global__ void __launch_bounds__(kBnThreads, kBnStatPerSm) bn_stats_kernel(const T* __restrict__ x, float2* __restrict__ part, const BnGrid g) {
  constexpr int U = kBnStatRows;
  after_previous_kernel();
  const Place at(g);
  const size_t tile_rows = (size_t)at.TY * U;
  float ref[8], mean[8], m2[8], n = 0.f, move_at = 4.f * U;
#pragma unroll
  for (int k = 0; k < 8; ++k) ref[k] = mean[k] = m2[k] = 0.f;
  if (at.active) {
    const size_t step = (size_t)at.TY * g.cols;
    for (size_t t = blockIdx.x; t < g.tiles; t += g.nblk) {
      const size_t r0 = t * tile_rows + at.ty;
      const uint4* src = (const uint4*)x + r0 * g.cols + at.col;
      Pack8<T> v[U];
      int nb = 0;
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (r0 + (size_t)i * at.TY < g.rows) {
          v[i].u = src[i * step];
          nb = i + 1;
        }
      if (nb == 0) break;
      if (n >= move_at) {   // (while the rows just asked for are on their way)
        move_at = 4.f * n;
        const float inv = 1.f / n;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float to = fmaf(mean[k], inv, ref[k]), by = to - ref[k], rest = fmaf(-n, by, mean[k]);
          m2[k] = fmaf(-by, mean[k] + rest, m2[k]);
          mean[k] = rest;   // (what rounding left)
          ref[k] = to;
        }
      }
      if (n == 0.f) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
#pragma unroll
          for (int i = 0; i < U; ++i)
            if (i < nb) ref[k] += up(v[i].e[k]);
          ref[k] /= (float)nb;
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float s = 0.f, q = 0.f;   // of these rows: one addition to the long sums per round
#pragma unroll
        for (int i = 0; i < U; ++i)
          if (i < nb) {
            const float d = up(v[i].e[k]) - ref[k];
            s += d;
            q = fmaf(d, d, q);
          }
        mean[k] += s;
        m2[k] += q;
      }
      n += (float)nb;
    }
    if (n > 0.f) {
      const float inv = 1.f / n;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = mean[k] * inv;
        m2[k] = fmaf(-mean[k], d, m2[k]);
        m2[k] = m2[k] < 0.f ? 0.f : m2[k];   // a NaN stays one
        mean[k] = ref[k] + d;
      }
    }
  }
  // fold the CTA's rows of threads, one thread per channel
  __shared__ float s_mean[kBnThreads * 8], s_m2[kBnThreads * 8], s_n[kBnThreads];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    s_mean[k * kBnThreads + threadIdx.x] = mean[k];
    s_m2[k * kBnThreads + threadIdx.x] = m2[k];
  }
  s_n[threadIdx.x] = n;
  __syncthreads();
  const int TX = 1 << g.lx;
  const int k = (int)threadIdx.x >> g.lx, tx = threadIdx.x & (TX - 1);   // channel k of column tx
  const int col = (int)(blockIdx.y << g.lx) + tx;
  if (k < 8 && col < g.cols) {
    // four sums at a time: shorter chains, and less rounding than one
    float sum[4] = {}, total[4] = {}, q[4] = {};
    for (int y = 0; y < at.TY; y += 4)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float m = s_n[(y + j) * TX + tx];
        sum[j] = fmaf(m, s_mean[k * kBnThreads + (y + j) * TX + tx], sum[j]);
        total[j] += m;
      }
    const float m = ((sum[0] + sum[1]) + (sum[2] + sum[3])) / ((total[0] + total[1]) + (total[2] + total[3]));
    for (int y = 0; y < at.TY; y += 4)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = s_mean[k * kBnThreads + (y + j) * TX + tx] - m;
        q[j] += fmaf(s_n[(y + j) * TX + tx] * d, d, s_m2[k * kBnThreads + (y + j) * TX + tx]);
      }
    part[(size_t)blockIdx.x * g.channels + col * 8 + k] = make_float2(m, (q[0] + q[1]) + (q[2] + q[3]));
  }
}

/**
 * The partial results of 8 channels, folded by a CTA of (8, 128) threads: each has its share of them under way at once and in
 * registers after that.  (One CTA per 32 channels whose threads walked the partials in turn was most of a small batch norm's
 * time: 24 x 64 x 56 x 56 forward 17.6 us.)
 */
constexpr int kFinishRows = 128;
constexpr int kFinishEach = (kBnSms * kBnStatPerSm + kFinishRows - 1) / kFinishRows;   // partials that a thread has at most
static_assert(kBnStatPerSm >= kBnPerSm, "the statistics have the most partials");

__device__ __forceinline__ void load_partials(float2* p, const float2* __restrict__ part, const BnGrid& g, int c) {
#pragma unroll
  for (int i = 0; i < kFinishEach; ++i) {
    const unsigned b = threadIdx.y + i * kFinishRows;
    p[i] = b < g.nblk ? part[(size_t)b * g.channels + c] : make_float2(0.f, 0.f);
  }
}

/** Sums over the rows of threads for every column, of two values at once, broadcast to all rows; in pairs throughout. */
__device__ __forceinline__ float2 column_sums(float2 v, float2 (*s)[9], float2* total) {
#pragma unroll
  for (int o = 8; o <= 16; o *= 2) {   // a warp holds four rows
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if (threadIdx.y % 4 == 0) s[threadIdx.y / 4][threadIdx.x] = v;
  __syncthreads();
  const int t = threadIdx.y * 8 + threadIdx.x;
  if (t < 256) {   // warp w folds column w
    v = s[t % 32][t / 32];
#pragma unroll
    for (int o = 16; o > 0; o /= 2) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (t % 32 == 0) total[t / 32] = v;
  }
  __syncthreads();
  return total[threadIdx.x];
}

__global__ void __launch_bounds__(8 * kFinishRows) bn_stats_finish_kernel(const float2* __restrict__ part, float* __restrict__ save_mean,
                                                                          float* __restrict__ save_invstd, float* running_mean,
                                                                          float* running_var, long long* batches, float momentum,
                                                                          float eps, const BnGrid g) {
  __shared__ float2 s[kFinishRows / 4][9], total[2][8];
  after_previous_kernel();
  const int c = (int)(blockIdx.x * 8 + threadIdx.x);
  float2 p[kFinishEach];
  load_partials(p, part, g, c);
  // (what lies above n times the first partial's mean: short sums are as exact as their values are close.  Where that partial lies far
  // from the others, what rounding left of the mean is in the deviations from it, and is summed with their squares: in the case
  // above 1.5e-9 deviations instead of 5.3e-8.)
  const float n = (float)g.rows, inv = 1.f / n, near = part[c].x;
  float sum = 0.f, q = 0.f;
#pragma unroll
  for (int i = 0; i < kFinishEach; ++i) {
    const unsigned b = threadIdx.y + i * kFinishRows;
    if (b < g.nblk) sum = fmaf(rows_of(g, b), p[i].x - near, sum);
  }
  const float first = near + column_sums(make_float2(sum, 0.f), s, total[0]).x * inv;
  sum = 0.f;
#pragma unroll
  for (int i = 0; i < kFinishEach; ++i) {
    const unsigned b = threadIdx.y + i * kFinishRows;
    const float d = p[i].x - first;
    if (b < g.nblk) {
      sum = fmaf(rows_of(g, b), d, sum);
      q += fmaf(rows_of(g, b) * d, d, p[i].y);
    }
  }
  const float2 both = column_sums(make_float2(q, sum), s, total[1]);
  const float by = both.y * inv, mean = first + by;
  q = fmaf(-both.y, by, both.x);
  if (threadIdx.y == 0) {
    save_mean[c] = mean;
    save_invstd[c] = rsqrtf(q / n + eps);
    if (running_mean) running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mean;
    if (running_var) running_var[c] = (1.f - momentum) * running_var[c] + momentum * (q / (n - 1.f));
  }
  if (batches && blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) *batches += 1;
}

/** y = act((x - mean) * invstd * weight + bias (+ residual)); one bit per element says where the gradient passes the ReLU. */
template <typename T, bool RES, bool RELU>
__global__ void __launch_bounds__(kBnThreads, kBnPerSm)
    bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ res, T* __restrict__ y, unsigned char* __restrict__ mask,
                    const float* __restrict__ save_mean, const float* __restrict__ save_invstd, const float* __restrict__ weight,
                    const float* __restrict__ bias, const BnGrid g) {
  constexpr int U = kBnRows;
  after_previous_kernel();
  const Place at(g);
  if (!at.active) return;
  float mean[8], scale[8], shift[8];
  load8(mean, save_mean, at.col);
  load8(scale, save_invstd, at.col);
  load8(shift, weight, at.col);
#pragma unroll
  for (int k = 0; k < 8; ++k) scale[k] *= shift[k];
  load8(shift, bias, at.col);
  const size_t tile_rows = (size_t)at.TY * U, step = (size_t)at.TY * g.cols;
  for (size_t t = blockIdx.x; t < g.tiles; t += g.nblk) {
    const size_t r0 = (g.tiles - 1 - t) * tile_rows + at.ty;
    const size_t i0 = r0 * g.cols + at.col;
    Pack8<T> v[U], a[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (r0 + (size_t)i * at.TY < g.rows) {
        v[i].u = ((const uint4*)x)[i0 + i * step];
        if constexpr (RES) a[i].u = ((const uint4*)res)[i0 + i * step];
      }
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (r0 + (size_t)i * at.TY < g.rows) {
        unsigned bits = 0;
        Pack8<T> o;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float f = fmaf(up(v[i].e[k]) - mean[k], scale[k], shift[k]);
          if constexpr (RES) f += up(a[i].e[k]);
          if constexpr (RELU) f = f < 0.f ? 0.f : f;   // a NaN stays one
          o.e[k] = Elem<T>::down(f);
          if constexpr (RELU) bits |= (up(o.e[k]) <= 0.f ? 0u : 1u) << k;
        }
        ((uint4*)y)[i0 + i * step] = o.u;
        if constexpr (RELU) mask[i0 + i * step] = (unsigned char)bits;
      }
  }
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
/**
 * part[b][c] = (sum of g, sum of g * (x - mean)) over the rows of CTA b, g the gradient behind the ReLU.  SUM: the output was used
 * twice (a block's input goes to its first convolution and to its end); the two gradients are added here, rounded as the
 * framework's addition rounds them, and g is left in `sum`, which is the residual's gradient too: seven passes over the activation
 * instead of the nine of an addition on its own, sums of it, and both gradients out of it.
 */
template <typename T, bool RELU, bool SUM>
__global__ void __launch_bounds__(kBnThreads, kBnPerSm)
    bn_grad_sums_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ dy2, T* __restrict__ sum,
                        const unsigned char* __restrict__ mask, const float* __restrict__ save_mean, float2* __restrict__ part, const BnGrid g) {
  constexpr int U = kBnRows;
  after_previous_kernel();
  const Place at(g);
  float mean[8], s1[8], s2[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) s1[k] = s2[k] = 0.f;
  if (at.active) {
    load8(mean, save_mean, at.col);
    const size_t tile_rows = (size_t)at.TY * U, step = (size_t)at.TY * g.cols;
    for (size_t t = blockIdx.x; t < g.tiles; t += g.nblk) {
      const size_t r0 = t * tile_rows + at.ty;
      const size_t i0 = r0 * g.cols + at.col;
      Pack8<T> v[U], d[U], d2[SUM ? U : 1];
      unsigned bits[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const bool in = r0 + (size_t)i * at.TY < g.rows;
        d[i].u = in ? ((const uint4*)dy)[i0 + i * step] : uint4{0, 0, 0, 0};
        if constexpr (SUM)
          if (in) d2[i].u = ((const uint4*)dy2)[i0 + i * step];
        if (in) v[i].u = ((const uint4*)x)[i0 + i * step];
        bits[i] = in ? 0xffu : 0u;
        if constexpr (RELU) bits[i] = in ? mask[i0 + i * step] : 0u;
      }
      if constexpr (SUM) {
#pragma unroll
        for (int i = 0; i < U; ++i)
          if (r0 + (size_t)i * at.TY < g.rows) {
#pragma unroll
            for (int k = 0; k < 8; ++k) d[i].e[k] = Elem<T>::down(bits[i] >> k & 1 ? up(d[i].e[k]) + up(d2[i].e[k]) : 0.f);
            ((uint4*)sum)[i0 + i * step] = d[i].u;
          }
      }
#pragma unroll
      for (int i = 0; i < U; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (bits[i] >> k & 1) {
            const float gr = up(d[i].e[k]);
            s1[k] += gr;
            s2[k] = fmaf(gr, up(v[i].e[k]) - mean[k], s2[k]);
          }
    }
  }
  __shared__ float s_1[kBnThreads * 8], s_2[kBnThreads * 8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    s_1[k * kBnThreads + threadIdx.x] = s1[k];
    s_2[k * kBnThreads + threadIdx.x] = s2[k];
  }
  __syncthreads();
  const int TX = 1 << g.lx;
  const int k = (int)threadIdx.x >> g.lx, tx = threadIdx.x & (TX - 1);
  const int col = (int)(blockIdx.y << g.lx) + tx;
  if (k < 8 && col < g.cols) {
    float a[4] = {}, b[4] = {};
    for (int y = 0; y < at.TY; y += 4)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a[j] += s_1[k * kBnThreads + (y + j) * TX + tx];
        b[j] += s_2[k * kBnThreads + (y + j) * TX + tx];
      }
    part[(size_t)blockIdx.x * g.channels + col * 8 + k] = make_float2((a[0] + a[1]) + (a[2] + a[3]), (b[0] + b[1]) + (b[2] + b[3]));
  }
}

/** Gradients of weight and bias, and what the second pass subtracts: coef[c] = (mean of g, mean of g * xhat, over sigma). */
__global__ void __launch_bounds__(8 * kFinishRows) bn_grad_finish_kernel(const float2* __restrict__ part, const float* __restrict__ save_invstd,
                                                                         float* __restrict__ grad_weight, float* __restrict__ grad_bias,
                                                                         float2* __restrict__ coef, const BnGrid g) {
  __shared__ float2 s[kFinishRows / 4][9], total[1][8];
  after_previous_kernel();
  const int c = (int)(blockIdx.x * 8 + threadIdx.x);
  float2 p[kFinishEach];
  load_partials(p, part, g, c);
#pragma unroll
  for (int i = 1; i < kFinishEach; ++i) {
    p[0].x += p[i].x;
    p[0].y += p[i].y;
  }
  const float2 both = column_sums(p[0], s, total[0]);
  const float a = both.x, b = both.y;
  if (threadIdx.y == 0) {
    const float is = save_invstd[c], n = (float)g.rows;
    grad_weight[c] = b * is;
    grad_bias[c] = a;
    coef[c] = make_float2(a / n, b * is * is / n);
  }
}

/** dx = (g - mean(g) - (x - mean) * coef) * invstd * weight; the residual's gradient is g itself. */
template <typename T, bool RES, bool RELU>
__global__ void __launch_bounds__(kBnThreads, kBnPerSm)
    bn_grad_apply_kernel(const T* __restrict__ x, const T* __restrict__ dy, const unsigned char* __restrict__ mask, T* __restrict__ dx,
                         T* __restrict__ dres, const float* __restrict__ save_mean, const float* __restrict__ save_invstd,
                         const float* __restrict__ weight, const float2* __restrict__ coef, const BnGrid g) {
  constexpr int U = kBnRows;
  after_previous_kernel();
  const Place at(g);
  if (!at.active) return;
  float mean[8], scale[8], cx[8], c0[8];   // dx = g * scale + (x - mean) * cx + c0
  load8(mean, save_mean, at.col);
  load8(scale, save_invstd, at.col);
  load8(c0, weight, at.col);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    scale[k] *= c0[k];
    const float2 c = coef[at.col * 8 + k];
    cx[k] = -scale[k] * c.y;
    c0[k] = -scale[k] * c.x;
  }
  const size_t tile_rows = (size_t)at.TY * U, step = (size_t)at.TY * g.cols;
  for (size_t t = blockIdx.x; t < g.tiles; t += g.nblk) {
    const size_t r0 = (g.tiles - 1 - t) * tile_rows + at.ty;
    const size_t i0 = r0 * g.cols + at.col;
    Pack8<T> v[U], d[U];
    unsigned bits[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (r0 + (size_t)i * at.TY < g.rows) {
        d[i].u = ((const uint4*)dy)[i0 + i * step];
        v[i].u = ((const uint4*)x)[i0 + i * step];
        if constexpr (RELU) bits[i] = mask[i0 + i * step];
      }
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (r0 + (size_t)i * at.TY < g.rows) {
        Pack8<T> o, r;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          T gt = d[i].e[k];
          if constexpr (RELU) gt = bits[i] >> k & 1 ? gt : Elem<T>::down(0.f);
          r.e[k] = gt;
          o.e[k] = Elem<T>::down(fmaf(up(gt), scale[k], fmaf(up(v[i].e[k]) - mean[k], cx[k], c0[k])));
        }
        ((uint4*)dx)[i0 + i * step] = o.u;
        if constexpr (RES) ((uint4*)dres)[i0 + i * step] = r.u;
      }
  }
}

size_t bn_part_bytes(const BnGrid& g) { return (size_t)g.nblk * (size_t)g.channels * sizeof(float2); }

void bn_check(const BnGrid& g, size_t extra, size_t workspace_bytes) {
  if (g.channels % 8 != 0 || g.rows < 2) throw_al_exception("batch norm: the channel count must be a multiple of 8 and there must be two rows at least");
  if (bn_part_bytes(g) + extra > workspace_bytes) throw_al_exception("batch norm: the workspace is too small");
}

template <typename T>
void bn_forward(const BnForward& a, cudaStream_t stream) {
  const BnGrid s = bn_grid(a.rows, a.channels, kBnStatRows, kBnStatPerSm), g = bn_grid(a.rows, a.channels, kBnRows, kBnPerSm);
  bn_check(s, 0, a.workspace_bytes);
  float2* part = (float2*)a.workspace;
  launch_behind(bn_stats_kernel<T>, dim3(s.nblk, s.ntile_y), kBnThreads, stream, (const T*)a.x, part, s);
  launch_behind(bn_stats_finish_kernel, (unsigned)a.channels / 8, dim3(8, kFinishRows), stream, part, a.save_mean, a.save_invstd, a.running_mean,
                a.running_var, a.batches, a.momentum, a.eps, s);
  auto run = [&](auto kernel) {
    launch_behind(kernel, dim3(g.nblk, g.ntile_y), kBnThreads, stream, (const T*)a.x, (const T*)a.residual, (T*)a.y, a.mask, a.save_mean,
                  a.save_invstd, a.weight, a.bias, g);
  };
  if (a.residual && a.mask) run(bn_apply_kernel<T, true, true>);
  else if (a.residual) run(bn_apply_kernel<T, true, false>);
  else if (a.mask) run(bn_apply_kernel<T, false, true>);
  else run(bn_apply_kernel<T, false, false>);
  AL_CHECK_CUDA(cudaGetLastError());
}

template <typename T>
void bn_backward(const BnBackward& a, cudaStream_t stream) {
  const BnGrid g = bn_grid(a.rows, a.channels, kBnRows, kBnPerSm);
  bn_check(g, (size_t)a.channels * sizeof(float2), a.workspace_bytes);
  if (a.dy2 && !a.dres) throw_al_exception("batch norm: the sum of two gradients needs a place");
  float2* coef = (float2*)a.workspace;
  float2* part = coef + a.channels;
  const dim3 grid(g.nblk, g.ntile_y);
  const auto sums = a.dy2 ? (a.mask ? bn_grad_sums_kernel<T, true, true> : bn_grad_sums_kernel<T, false, true>)
                          : (a.mask ? bn_grad_sums_kernel<T, true, false> : bn_grad_sums_kernel<T, false, false>);
  launch_behind(sums, grid, kBnThreads, stream, (const T*)a.x, (const T*)a.dy, (const T*)a.dy2, (T*)a.dres, a.mask, a.save_mean, part, g);
  launch_behind(bn_grad_finish_kernel, (unsigned)a.channels / 8, dim3(8, kFinishRows), stream, part, a.save_invstd, a.grad_weight, a.grad_bias,
                coef, g);
  const void* dy = a.dy2 ? a.dres : a.dy;   // (the sum has passed the ReLU already)
  auto run = [&](auto kernel) {
    launch_behind(kernel, grid, kBnThreads, stream, (const T*)a.x, (const T*)dy, a.mask, (T*)a.dx, (T*)a.dres, a.save_mean, a.save_invstd,
                  a.weight, coef, g);
  };
  if (a.dy2) run(bn_grad_apply_kernel<T, false, false>);
  else if (a.dres && a.mask) run(bn_grad_apply_kernel<T, true, true>);
  else if (a.dres) run(bn_grad_apply_kernel<T, true, false>);
  else if (a.mask) run(bn_grad_apply_kernel<T, false, true>);
  else run(bn_grad_apply_kernel<T, false, false>);
  AL_CHECK_CUDA(cudaGetLastError());
}

}  // namespace

size_t bn_workspace_bytes(int channels) {
  // partial sums of one wave of CTAs, 256 channels each (or of one CTA per 256 channels), and the backward's coefficients
  return (size_t)kBnSms * std::max(kBnPerSm, kBnStatPerSm) * 256 * sizeof(float2) + 2 * sizeof(float2) * (size_t)channels;
}

void launch_bn_forward(const BnForward& a, DType dt, cudaStream_t stream) {
  if (dt == DType::bf16) return bn_forward<__nv_bfloat16>(a, stream);
  if (dt == DType::f16) return bn_forward<__half>(a, stream);
  throw_al_exception("batch norm: unsupported datatype ", dtype_name(dt));
}

void launch_bn_backward(const BnBackward& a, DType dt, cudaStream_t stream) {
  if (dt == DType::bf16) return bn_backward<__nv_bfloat16>(a, stream);
  if (dt == DType::f16) return bn_backward<__half>(a, stream);
  throw_al_exception("batch norm: unsupported datatype ", dtype_name(dt));
}

}  // namespace device
}  // namespace internal
}  // namespace Al
