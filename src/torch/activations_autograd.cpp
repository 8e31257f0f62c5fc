// Autograd of the fused batch norm (kernels/batchnorm.cu), of max pooling (kernels/maxpool.cu) and of a network's first convolution
// (kernels/stem.cu) for PyTorch, in native code: a small network's step is bound by
// the host, and 53 layers of a Python autograd function cost it 2 ms more than the three framework operations each
// replaces.  Registered under torch.ops.aluminum_b200; aluminum_b200/ops/activations.py decides when they are called.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include "al/al_c.h"
#include "al/base.hpp"
#include "comm_calls.hpp"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kArgs = 11;  // of forward()

int type_code(const Tensor& t) { return (int)(t.scalar_type() == at::kBFloat16 ? Al::DType::bf16 : Al::DType::f16); }

Tensor workspace(const Tensor& x, int64_t channels) { return at::empty({(int64_t)al_bn_workspace_bytes((int)channels)}, x.options().dtype(at::kByte)); }

/**
 * A saved tensor as the kernels read it.  Saved-tensor hooks give back the values but not always the layout (a copy to pinned
 * host memory and back drops channels-last); what has lost its layout or alignment is laid out again, anything else that
 * changed is an error before a kernel gets its address.
 */
Tensor restored(const Tensor& t, at::IntArrayRef sizes, at::ScalarType type, const Tensor& like, at::MemoryFormat format) {
  TORCH_CHECK(t.device() == like.device() && t.scalar_type() == type && t.sizes() == sizes,
              "a saved tensor came back with another device, type or shape");
  return t.is_contiguous(format) && (uintptr_t)t.data_ptr() % 16 == 0 ? t : t.clone(format);
}

/** `twice`: the output comes as two tensors on the same memory, whose gradients backward() adds where it reads them. */
struct BatchNormAct : public torch::autograd::Function<BatchNormAct> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias,
                               const std::optional<Tensor>& residual, const Tensor& running_mean, const Tensor& running_var,
                               const std::optional<Tensor>& batches, double momentum, double eps, bool relu, bool twice) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t c = x.size(1), rows = x.numel() / c;
    Tensor y = at::empty_like(x);
    Tensor mask = at::empty({relu ? rows * c / 8 : 0}, x.options().dtype(at::kByte));
    Tensor stats = at::empty({2, c}, weight.options());
    Tensor ws = workspace(x, c);
    float* at = stats.data_ptr<float>();
    TORCH_CHECK(al_bn_forward(type_code(x), x.data_ptr(), residual ? residual->data_ptr() : nullptr, y.data_ptr(),
                              relu ? mask.data_ptr<uint8_t>() : nullptr, weight.data_ptr<float>(), bias.data_ptr<float>(),
                              running_mean.data_ptr<float>(), running_var.data_ptr<float>(),
                              batches ? (long long*)batches->data_ptr<int64_t>() : nullptr, at, at + c, ws.data_ptr(), (size_t)ws.numel(),
                              (size_t)rows, (int)c, (float)momentum, (float)eps, c10::cuda::getCurrentCUDAStream().stream()) == 0,
                al_last_error());
    running_mean.unsafeGetTensorImpl()->bump_version();
    running_var.unsafeGetTensorImpl()->bump_version();
    if (batches) batches->unsafeGetTensorImpl()->bump_version();
    ctx->save_for_backward({x, weight, stats, mask});
    ctx->saved_data["relu"] = relu;
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["residual"] = residual.has_value() && residual->requires_grad();
    ctx->set_materialize_grads(false);
    if (twice) return {y, y.variable_data()};
    return {y};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list out(kArgs);
    Tensor dy = grads[0], dy2 = grads.size() > 1 ? grads[1] : Tensor();
    if (!dy.defined()) std::swap(dy, dy2);
    if (!dy.defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    Tensor x = saved[0], weight = saved[1], stats = saved[2], mask = saved[3];
    const bool relu = ctx->saved_data["relu"].toBool(), want_res = ctx->saved_data["residual"].toBool();
    const c10::cuda::CUDAGuard guard(dy.device());
    const int64_t c = x.size(1), rows = x.numel() / c;
    if (dy2.defined() && (at::GradMode::is_enabled() || dy.scalar_type() != x.scalar_type() || dy2.scalar_type() != x.scalar_type())) {
      dy = dy + dy2;
      dy2.reset();
    }
    if (at::GradMode::is_enabled() || dy.scalar_type() != x.scalar_type()) {
      // a graph of the backward is wanted: operations that have a derivative themselves
      if (relu) {
        const Tensor bits = mask.reshape({x.size(0), x.size(2), x.size(3), c / 8, 1}).bitwise_right_shift(at::arange(8, mask.options())).bitwise_and(1);
        const Tensor passes = bits.reshape({x.size(0), x.size(2), x.size(3), c}).permute({0, 3, 1, 2}).to(at::kBool);
        dy = at::where(passes, dy, at::zeros({}, dy.options()));   // (not a product: an infinite gradient that the ReLU stops is 0)
      }
      auto g = at::native_batch_norm_backward(dy, x, weight, {}, {}, stats[0], stats[1], true, ctx->saved_data["eps"].toDouble(), {true, true, true});
      out[0] = std::get<0>(g);
      out[1] = std::get<1>(g);
      out[2] = std::get<2>(g);
      if (want_res) out[3] = dy;
      return out;
    }
    auto laid_out = [](const Tensor& t) {
      return t.is_contiguous(at::MemoryFormat::ChannelsLast) && (uintptr_t)t.data_ptr() % 16 == 0 ? t : t.clone(at::MemoryFormat::ChannelsLast);
    };
    dy = laid_out(dy);
    if (dy2.defined()) dy2 = laid_out(dy2);
    x = restored(x, dy.sizes(), dy.scalar_type(), dy, at::MemoryFormat::ChannelsLast);
    weight = restored(weight, {c}, at::kFloat, dy, at::MemoryFormat::Contiguous);
    stats = restored(stats, {2, c}, at::kFloat, dy, at::MemoryFormat::Contiguous);
    mask = restored(mask, {relu ? rows * c / 8 : 0}, at::kByte, dy, at::MemoryFormat::Contiguous);
    Tensor dx = at::empty_like(x), dres, gw = at::empty_like(weight), gb = at::empty_like(weight);
    if (want_res || dy2.defined()) dres = at::empty_like(x);
    Tensor ws = workspace(x, c);
    float* at = stats.data_ptr<float>();
    void* const stream = c10::cuda::getCurrentCUDAStream().stream();
    const unsigned char* passes = relu ? mask.data_ptr<uint8_t>() : nullptr;
    const int rc = dy2.defined()
                       ? al_bn_backward_sum(type_code(x), x.data_ptr(), dy.data_ptr(), dy2.data_ptr(), passes, dx.data_ptr(), dres.data_ptr(),
                                            weight.data_ptr<float>(), at, at + c, gw.data_ptr<float>(), gb.data_ptr<float>(), ws.data_ptr(),
                                            (size_t)ws.numel(), (size_t)rows, (int)c, stream)
                       : al_bn_backward(type_code(x), x.data_ptr(), dy.data_ptr(), passes, dx.data_ptr(), want_res ? dres.data_ptr() : nullptr,
                                        weight.data_ptr<float>(), at, at + c, gw.data_ptr<float>(), gb.data_ptr<float>(), ws.data_ptr(),
                                        (size_t)ws.numel(), (size_t)rows, (int)c, stream);
    TORCH_CHECK(rc == 0, al_last_error());
    out[0] = dx;
    out[1] = gw;
    out[2] = gb;
    if (want_res) out[3] = dres;
    return out;
  }
};

Tensor batch_norm_act(const Tensor& x, const Tensor& weight, const Tensor& bias, const std::optional<Tensor>& residual,
                      const Tensor& running_mean, const Tensor& running_var, const std::optional<Tensor>& batches, double momentum,
                      double eps, bool relu) {
  return BatchNormAct::apply(x, weight, bias, residual, running_mean, running_var, batches, momentum, eps, relu, false)[0];
}

std::tuple<Tensor, Tensor> batch_norm_act_twice(const Tensor& x, const Tensor& weight, const Tensor& bias, const std::optional<Tensor>& residual,
                                                const Tensor& running_mean, const Tensor& running_var, const std::optional<Tensor>& batches,
                                                double momentum, double eps, bool relu) {
  const variable_list y = BatchNormAct::apply(x, weight, bias, residual, running_mean, running_var, batches, momentum, eps, relu, true);
  return {y[0], y[1]};
}

struct MaxPool : public torch::autograd::Function<MaxPool> {
  static std::array<int, 9> shape(const Tensor& x, int64_t k, int64_t stride, int64_t pad) {
    const int64_t h = x.size(2), w = x.size(3);
    return {(int)x.size(0), (int)h, (int)w, (int)x.size(1), (int)((h + 2 * pad - k) / stride + 1), (int)((w + 2 * pad - k) / stride + 1),
            (int)k, (int)stride, (int)pad};
  }

  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t k, int64_t stride, int64_t pad) {
    const c10::cuda::CUDAGuard guard(x.device());
    const auto s = shape(x, k, stride, pad);
    Tensor y = at::empty({s[0], s[3], s[4], s[5]}, x.options(), at::MemoryFormat::ChannelsLast);
    Tensor place = at::empty({s[0], s[4], s[5], s[3]}, x.options().dtype(at::kByte));
    TORCH_CHECK(al_maxpool_forward(type_code(x), x.data_ptr(), y.data_ptr(), place.data_ptr<uint8_t>(), s.data(),
                                   c10::cuda::getCurrentCUDAStream().stream()) == 0,
                al_last_error());
    ctx->save_for_backward({x, place});
    ctx->saved_data["k"] = k;
    ctx->saved_data["stride"] = stride;
    ctx->saved_data["pad"] = pad;
    ctx->set_materialize_grads(false);
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list out(4);
    if (!grads[0].defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];   // (only its shape matters here)
    Tensor place = saved[1], dy = grads[0];
    const int64_t k = ctx->saved_data["k"].toInt(), stride = ctx->saved_data["stride"].toInt(), pad = ctx->saved_data["pad"].toInt();
    const c10::cuda::CUDAGuard guard(dy.device());
    const auto s = shape(x, k, stride, pad);
    if (at::GradMode::is_enabled() || dy.scalar_type() != x.scalar_type()) {
      // a graph of the backward is wanted: the framework's own backward, with the places as its indices
      const auto wide = place.options().dtype(at::kLong);
      const Tensor p = place.to(at::kLong);
      const Tensor h = at::arange(s[4], wide).mul(stride).sub(pad).view({1, s[4], 1, 1}) + at::floor_divide(p, k);
      const Tensor w = at::arange(s[5], wide).mul(stride).sub(pad).view({1, 1, s[5], 1}) + at::remainder(p, k);
      out[0] = at::max_pool2d_with_indices_backward(dy, x, {k, k}, {stride, stride}, {pad, pad}, {1, 1}, false, (h * s[2] + w).permute({0, 3, 1, 2}));
      return out;
    }
    if (!dy.is_contiguous(at::MemoryFormat::ChannelsLast) || (uintptr_t)dy.data_ptr() % 16) dy = dy.clone(at::MemoryFormat::ChannelsLast);
    place = restored(place, {s[0], s[4], s[5], s[3]}, at::kByte, dy, at::MemoryFormat::Contiguous);
    Tensor dx = at::empty(x.sizes(), dy.options(), at::MemoryFormat::ChannelsLast);
    TORCH_CHECK(al_maxpool_backward(type_code(x), dy.data_ptr(), place.data_ptr<uint8_t>(), dx.data_ptr(), s.data(),
                                    c10::cuda::getCurrentCUDAStream().stream()) == 0,
                al_last_error());
    out[0] = dx;
    return out;
  }
};

Tensor max_pool(const Tensor& x, int64_t k, int64_t stride, int64_t pad) { return MaxPool::apply(x, k, stride, pad); }

/**
 * First convolution: images of three channels laid out as 64 channels (kernels/stem.cu) and convolved by the library over 4 x 1 taps.
 * No gradient of the images (ops/convolution.py sends what wants one to the module).
 */
struct StemConv : public torch::autograd::Function<StemConv> {
  struct Shape {
    std::array<int, 6> sizes;
    std::array<long long, 8> strides;
    Shape(at::IntArrayRef x, at::IntArrayRef x_strides, const Tensor& weight)
        : sizes{(int)x[0], (int)x[2], (int)x[3], (int)((x[2] - 1) / 2 + 1), (int)((x[3] - 1) / 2 + 1), (int)weight.size(0)} {
      for (int i = 0; i < 4; ++i) {
        strides[i] = x_strides[i];
        strides[4 + i] = weight.stride(i);
      }
    }
  };

  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, at::ScalarType type) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Shape s(x.sizes(), x.strides(), weight);
    const int64_t oc = weight.size(0);
    Tensor seen = at::empty({s.sizes[0], 64, s.sizes[3] + 3, s.sizes[4]}, x.options().dtype(type), at::MemoryFormat::ChannelsLast);
    Tensor packed = at::empty({oc, 64, 4, 1}, seen.options(), at::MemoryFormat::ChannelsLast);
    const int in = x.scalar_type() == at::kFloat ? (int)Al::DType::f32 : type_code(x);
    Tensor watch = at::empty({(int64_t)al_stem_watch_words(s.sizes.data())}, x.options().dtype(at::kInt));
    void* const stream = c10::cuda::getCurrentCUDAStream().stream();
    TORCH_CHECK(al_stem_gather_watched(in, x.data_ptr(), type_code(seen), seen.data_ptr(), weight.data_ptr<float>(), packed.data_ptr(),
                                       (unsigned*)watch.data_ptr<int>(), s.sizes.data(), s.strides.data(), stream) == 0,
                al_last_error());
    ctx->save_for_backward({seen, packed});
    ctx->saved_data["strides"] = weight.strides().vec();
    Tensor y = at::conv2d(seen, packed);
    const Shape result(x.sizes(), {0, 0, 0, 0}, y);   // (with y's strides)
    std::array<int, 6> sizes = result.sizes;
    sizes[5] = (int)oc;
    TORCH_CHECK(al_stem_repair(type_code(seen), seen.data_ptr(), packed.data_ptr(), (const unsigned*)watch.data_ptr<int>(), y.data_ptr(), sizes.data(),
                               result.strides.data(), stream) == 0,
                al_last_error());
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &seen = saved[0], &packed = saved[1], &dy = grads[0];
    const c10::cuda::CUDAGuard guard(dy.device());
    const int64_t oc = packed.size(0);
    Tensor g = std::get<1>(at::convolution_backward(dy, seen, packed, at::OptionalIntArrayRef(), {1, 1}, {0, 0}, {1, 1}, false, {0, 0}, 1, {false, true, false}));
    if (at::GradMode::is_enabled()) {   // a graph of the backward is wanted: channel = (row of the pair, column, image channel), zeros behind
      g = g.squeeze(3).slice(1, 0, 48).reshape({oc, 2, 8, 3, 4}).permute({0, 3, 4, 1, 2}).reshape({oc, 3, 8, 8});
      out[1] = g.slice(2, 0, 7).slice(3, 0, 7).to(at::kFloat);
      return out;
    }
    g = restored(g, {oc, 64, 4, 1}, seen.scalar_type(), dy, at::MemoryFormat::ChannelsLast);
    Tensor grad = at::empty_strided({oc, 3, 7, 7}, ctx->saved_data["strides"].toIntVector(), g.options().dtype(at::kFloat));
    const Shape s({seen.size(0), 3, 2 * (seen.size(2) - 3), 2 * seen.size(3)}, {0, 0, 0, 0}, grad);
    TORCH_CHECK(al_stem_scatter(type_code(g), g.data_ptr(), grad.data_ptr<float>(), s.sizes.data(), s.strides.data(),
                                c10::cuda::getCurrentCUDAStream().stream()) == 0,
                al_last_error());
    out[1] = grad;
    return out;
  }
};

/**
 * The weights of a block in a 16-bit type, and their gradients back in fp32, with one launch each way.  The gradients of a block come
 * together then, when the last of them is there.  For the 25 MB buckets that several ranks average meanwhile, ResNet-50 at batch 256, ms
 * after backward began: 0.58, 1.31, 1.94, 4.58, 12.69; with a cast per weight 0.59, 1.37, 1.77, 4.70, 12.90.
 */
struct CastAll : public torch::autograd::Function<CastAll> {
  /** Every tensor in `to`, dense and in the order of its memory. */
  static std::vector<Tensor> cast(at::TensorList tensors, at::ScalarType from, at::ScalarType to) {
    auto code = [](at::ScalarType t) { return (int)(t == at::kFloat ? Al::DType::f32 : t == at::kBFloat16 ? Al::DType::bf16 : Al::DType::f16); };
    std::vector<Tensor> made;
    std::vector<const void*> in;
    std::vector<void*> out;
    std::vector<size_t> n;
    for (const Tensor& t : tensors) {
      Tensor dense = t.is_non_overlapping_and_dense() && (uintptr_t)t.data_ptr() % 16 == 0 ? t : t.clone(at::MemoryFormat::Contiguous);
      made.push_back(at::empty_strided(dense.sizes(), dense.strides(), dense.options().dtype(to)));
      in.push_back(dense.data_ptr());
      out.push_back(made.back().data_ptr());
      n.push_back((size_t)dense.numel());
    }
    TORCH_CHECK(al_cast_all(out.data(), code(to), in.data(), code(from), n.data(), (int)n.size(), c10::cuda::getCurrentCUDAStream().stream()) == 0,
                al_last_error());
    return made;
  }

  static variable_list forward(AutogradContext* ctx, at::TensorList weights, at::ScalarType type) {
    const c10::cuda::CUDAGuard guard(weights[0].device());
    ctx->set_materialize_grads(false);
    return cast(weights, at::kFloat, type);
  }

  static variable_list backward(AutogradContext*, variable_list grads) {
    variable_list out(grads.size() + 1);
    std::vector<Tensor> given;
    for (const Tensor& g : grads)
      if (g.defined()) given.push_back(g);
    if (given.empty()) return out;
    const c10::cuda::CUDAGuard guard(given[0].device());
    const at::ScalarType type = given[0].scalar_type();
    bool plain = !at::GradMode::is_enabled() && (type == at::kBFloat16 || type == at::kHalf);   // (no graph of the backward is wanted)
    for (const Tensor& g : given) plain = plain && g.scalar_type() == type && g.layout() == at::kStrided && g.device() == given[0].device();
    const std::vector<Tensor> made = plain ? cast(given, type, at::kFloat) : std::vector<Tensor>();
    size_t next = 0;
    for (size_t i = 0; i < grads.size(); ++i)
      if (grads[i].defined()) out[i] = plain ? made[next++] : grads[i].to(at::kFloat);
    return out;
  }
};

std::vector<Tensor> cast_all(at::TensorList weights, at::ScalarType type) { return CastAll::apply(weights, type); }

Tensor stem_conv(const Tensor& x, const Tensor& weight, at::ScalarType type) { return StemConv::apply(x, weight, type); }

}  // namespace

TORCH_LIBRARY(aluminum_b200, m) {
  m.def("batch_norm_act(Tensor x, Tensor weight, Tensor bias, Tensor? residual, Tensor(a!) running_mean, Tensor(b!) running_var, "
        "Tensor(c!)? batches, float momentum, float eps, bool relu) -> Tensor",
        batch_norm_act);
  m.def("batch_norm_act_twice(Tensor x, Tensor weight, Tensor bias, Tensor? residual, Tensor(a!) running_mean, Tensor(b!) running_var, "
        "Tensor(c!)? batches, float momentum, float eps, bool relu) -> (Tensor, Tensor)",
        batch_norm_act_twice);
  m.def("cast_all(Tensor[] weights, ScalarType type) -> Tensor[]", cast_all);
  m.def("stem_conv(Tensor x, Tensor weight, ScalarType type) -> Tensor", stem_conv);
  m.def("max_pool(Tensor x, int k, int stride, int pad) -> Tensor", max_pool);
}
