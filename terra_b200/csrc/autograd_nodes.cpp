// The layers as autograd nodes in C++: the same launches as the Python nodes (which the multi-rank layouts, tracing and function
// transforms use), without the interpreter in the backward pass. A small layer is bound by the host: a Python node costs about
// 50 us of interpreter, argument lists and hand-over of the interpreter lock for its two directions, around 40 us of launches.
//
// A node keeps the operands that belong to the layer (bf16 weights, packed weights) beside the tensors saved for the backward pass, which go
// through whatever saved-tensor hooks are set. Parameter gradients are accumulated in place: the halves and linear layers into the
// accumulators that the forward call was given, the others into the parameter's `.grad` at the time of the backward pass, or returned to
// autograd where it has none by then. A parameter among the inputs (`anchor`) makes autograd call the node also when the activation needs no
// gradient.
// Us per pass, Python node / this: attention half of 512 rows of width 96 199 / 167, residual convolution and GroupNorm of 96 x 180 pixels
// 229 / 178, a training step of 19 such layers 2408 / 1994.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "check.h"
#include "host_api.h"
#include "launch_count.h"
#include "torch_ops.h"

namespace {

using torch::Tensor;
using OptTensor = c10::optional<torch::Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

template <class T>
using Held = c10::intrusive_ptr<T>;

template <class T>
void hold(AutogradContext* ctx, const Held<T>& layer) {
  ctx->saved_data["layer"] = c10::IValue::make_capsule(layer);
}
template <class T>
Held<T> held(AutogradContext* ctx) {
  return c10::static_intrusive_pointer_cast<T>(ctx->saved_data["layer"].toCapsule());
}

// fp32 zeros, cleared by a memory operation (half of the host time of a fill kernel)
Tensor zeroed(const Tensor& like, at::IntArrayRef sizes, const char* what) {
  Tensor t = torch::empty(sizes, like.options().dtype(torch::kFloat32));
  need(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), c10::cuda::getCurrentCUDAStream().stream()) == cudaSuccess, what);
  return t;
}

// Where a parameter's gradient goes: into its fp32 accumulator, or, where there is none to add into (dropped since the forward pass),
// into zeros that the node returns.
struct ParamGrad {
  Tensor into, returned;
  ParamGrad(const Tensor& param, const char* what) {
    const Tensor& g = param.grad();
    if (g.defined() && g.is_cuda() && g.scalar_type() == torch::kFloat32 && g.is_contiguous()) into = g;
    else into = returned = zeroed(param, param.sizes(), what);
  }
};

// ------------------------------------------------------------------------------------------------ attention half
struct AttnLayer : torch::CustomClassHolder {
  Tensor ln_w, ln_b, qkv_w, qkv_b, proj_w, proj_b, ln_wg, ln_bg, qkv_wg, qkv_bg, proj_wg, proj_bg, status;
  OptTensor table, table_g;
  std::vector<int64_t> geo;
  double scale, eps;
  bool fuse_bias;
};

struct AttnHalf : Function<AttnHalf> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& anchor, const Held<AttnLayer>& l) {
    auto r = terra_ops::attn_half_fwd(x, l->ln_w, l->ln_b, l->qkv_w, l->qkv_b, l->proj_w, l->proj_b, l->table, l->geo, l->scale, l->eps,
                                      l->status);
    ctx->save_for_backward({x, r[1], r[2], r[3], r[4], r[5]});
    hold(ctx, l);
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list dy) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<AttnLayer>(ctx);
    return {terra_ops::attn_half_bwd(dy[0].contiguous(), s[0], s[1], s[2], s[3], s[4], s[5], l->ln_w, l->qkv_w, l->proj_w, l->table, l->ln_wg,
                                     l->ln_bg, l->qkv_wg, l->qkv_bg, l->proj_wg, l->proj_bg, l->table_g, l->geo, l->scale, l->fuse_bias,
                                     l->status),
            Tensor(), Tensor()};
  }
};

Tensor attn_half(const Tensor& x, const Tensor& anchor, const std::vector<Tensor>& w, const std::vector<Tensor>& g, const OptTensor& table,
                 const OptTensor& table_g, std::vector<int64_t> geo, double scale, double eps, bool fuse_bias, const Tensor& status) {
  need(w.size() == 6 && g.size() == 6, "attention half: six weights and their gradients");
  auto l = c10::make_intrusive<AttnLayer>();
  l->ln_w = w[0], l->ln_b = w[1], l->qkv_w = w[2], l->qkv_b = w[3], l->proj_w = w[4], l->proj_b = w[5];
  l->ln_wg = g[0], l->ln_bg = g[1], l->qkv_wg = g[2], l->qkv_bg = g[3], l->proj_wg = g[4], l->proj_bg = g[5];
  l->table = table, l->table_g = table_g, l->geo = std::move(geo), l->scale = scale, l->eps = eps, l->fuse_bias = fuse_bias;
  l->status = status;
  return AttnHalf::apply(x, anchor, l);
}

// ------------------------------------------------------------------------------------------------ MLP half
struct MlpLayer : torch::CustomClassHolder {
  Tensor ln_w, ln_b, fc1_w, fc1_b, fc2_w, fc2_b, ln_wg, ln_bg, fc1_wg, fc1_bg, fc2_wg, fc2_bg, status;
  double eps;
  bool fuse_bias;
};

struct MlpHalf : Function<MlpHalf> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& anchor, const Held<MlpLayer>& l) {
    auto r = terra_ops::mlp_half_fwd(x, l->ln_w, l->ln_b, l->fc1_w, l->fc1_b, l->fc2_w, l->fc2_b, l->eps, l->status);
    ctx->save_for_backward({x, r[1], r[2], r[3], r[4], r[5]});
    hold(ctx, l);
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list dy) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<MlpLayer>(ctx);
    return {terra_ops::mlp_half_bwd(dy[0].contiguous(), s[0], s[1], s[2], s[3], s[4], s[5], l->ln_w, l->fc1_w, l->fc2_w, l->ln_wg, l->ln_bg,
                                    l->fc1_wg, l->fc1_bg, l->fc2_wg, l->fc2_bg, l->fuse_bias, l->status),
            Tensor(), Tensor()};
  }
};

Tensor mlp_half(const Tensor& x, const Tensor& anchor, const std::vector<Tensor>& w, const std::vector<Tensor>& g, double eps, bool fuse_bias,
                const Tensor& status) {
  need(w.size() == 6 && g.size() == 6, "MLP half: six weights and their gradients");
  if (!c10::GradMode::is_enabled() && !x._fw_grad(0).defined())
    return terra_ops::mlp_half_infer(x, w[0], w[1], w[2], w[3], w[4], w[5], eps, status);
  auto l = c10::make_intrusive<MlpLayer>();
  l->ln_w = w[0], l->ln_b = w[1], l->fc1_w = w[2], l->fc1_b = w[3], l->fc2_w = w[4], l->fc2_b = w[5];
  l->ln_wg = g[0], l->ln_bg = g[1], l->fc1_wg = g[2], l->fc1_bg = g[3], l->fc2_wg = g[4], l->fc2_bg = g[5];
  l->eps = eps, l->fuse_bias = fuse_bias, l->status = status;
  return MlpHalf::apply(x, anchor, l);
}

// ------------------------------------------------------------------------------------------------ linear
struct LinearLayer : torch::CustomClassHolder {
  Tensor w, wg, status;
  OptTensor b, bg;
  bool need_dx, fuse_bias, has_res;
};

struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& anchor, const OptTensor& residual, const Held<LinearLayer>& l) {
    Tensor y = terra_ops::linear_product(x, l->w, false, l->b, residual, l->status);
    ctx->save_for_backward({x});
    hold(ctx, l);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<LinearLayer>(ctx);
    const Tensor dy = grads[0].contiguous();
    terra_ops::wgrad(dy, s[0], l->wg, l->bg, l->fuse_bias, l->status);
    Tensor dx;
    if (l->need_dx) dx = terra_ops::linear_product(dy, l->w, true, c10::nullopt, c10::nullopt, l->status);
    return {dx, Tensor(), l->has_res ? dy : Tensor(), Tensor()};
  }
};

Tensor linear(const Tensor& x, const Tensor& anchor, const Tensor& w, const OptTensor& b, const Tensor& wg, const OptTensor& bg,
              const OptTensor& residual, bool need_dx, bool fuse_bias, const Tensor& status) {
  auto l = c10::make_intrusive<LinearLayer>();
  l->w = w, l->b = b, l->wg = wg, l->bg = bg, l->need_dx = need_dx, l->fuse_bias = fuse_bias, l->has_res = residual.has_value();
  l->status = status;
  return Linear::apply(x, anchor, residual, l);
}

// ------------------------------------------------------------------------------------------------ 3x3 convolution
struct ConvLayer : torch::CustomClassHolder {
  Tensor w_fwd, b, weight, bias, status;
  OptTensor w_dgrad;      // given where the input needs a gradient
  int64_t stride, split;
  bool fuse_bias;
};

struct Conv3x3 : Function<Conv3x3> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, const Held<ConvLayer>& l) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t st = l->stride;
    Tensor y = torch::empty({x.size(0), st == 1 ? x.size(1) : (x.size(1) + 1) / 2, x.size(2) / st, l->w_fwd.size(0)},
                            x.options().dtype(torch::kBFloat16));
    terra_ops::conv3x3_fwd(x, l->w_fwd, y, st, 1 /* with bias */, l->b, c10::nullopt, l->status, c10::nullopt, c10::nullopt);
    ctx->save_for_backward({x});
    hold(ctx, l);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<ConvLayer>(ctx);
    const Tensor& x = s[0];
    const Tensor dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(dy.device());
    ParamGrad gw(l->weight, "conv3x3: clearing the weight gradient"), gb(l->bias, "conv3x3: clearing the bias gradient");
    Tensor dw9 = terra_ops::scratch_take(x, {9, x.size(3), dy.size(3)});
    terra_ops::conv3x3_wgrad_taps(x, dy, dw9, l->stride, l->status, gb.into, l->fuse_bias, l->split);
    terra_ops::fold_taps(dw9, gw.into);
    terra_ops::scratch_give(dw9);
    Tensor dx;
    if (l->w_dgrad.has_value()) {
      dx = torch::empty_like(x);
      if (l->stride == 1)
        terra_ops::conv3x3_fwd(dy, *l->w_dgrad, dx, 1, 0, c10::nullopt, c10::nullopt, l->status, c10::nullopt, c10::nullopt);
      else
        terra_ops::conv3x3_s2_dgrad(dy, *l->w_dgrad, dx, l->status);
    }
    return {dx, gw.returned, gb.returned, Tensor()};
  }
};

Tensor conv3x3(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& w_fwd, const OptTensor& w_dgrad, const Tensor& b,
               int64_t stride, int64_t split, bool fuse_bias, const Tensor& status) {
  auto l = c10::make_intrusive<ConvLayer>();
  l->w_fwd = w_fwd, l->w_dgrad = w_dgrad, l->b = b, l->weight = weight, l->bias = bias, l->stride = stride, l->split = split, l->fuse_bias = fuse_bias;
  l->status = status;
  return Conv3x3::apply(x, weight, bias, l);
}

// ------------------------------------------------------------------------------------------------ transposed 2x2 convolution
struct ConvTLayer : torch::CustomClassHolder {
  Tensor w_fwd, b4, weight, bias, status;
  OptTensor w_dgrad;
  int64_t split;
  bool fuse_bias;
};

struct ConvT2x2 : Function<ConvT2x2> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, const Held<ConvTLayer>& l) {
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor y = torch::empty({x.size(0), 2 * x.size(1), 2 * x.size(2), l->weight.size(1)}, x.options().dtype(torch::kBFloat16));
    terra_ops::convt2x2(0, x.contiguous(), l->w_fwd, l->b4, y, l->status);
    ctx->save_for_backward({x});
    hold(ctx, l);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<ConvTLayer>(ctx);
    const Tensor x = s[0].contiguous(), dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(dy.device());
    const int64_t cout = dy.size(3);
    ParamGrad gw(l->weight, "conv_transpose2x2: clearing the weight gradient"), gb(l->bias, "conv_transpose2x2: clearing the bias gradient");
    Tensor dw4 = terra_ops::scratch_take(x, {4, cout, x.size(3)});
    terra_ops::convt2x2_wgrad_taps(x, dy, dw4, l->status, gb.into, l->fuse_bias, l->split);
    terra_ops::fold_taps(dw4, gw.into);
    terra_ops::scratch_give(dw4);
    Tensor dx;
    if (l->w_dgrad.has_value()) {
      dx = torch::empty(x.sizes(), x.options());
      terra_ops::convt2x2(1, dy, *l->w_dgrad, c10::nullopt, dx, l->status);
    }
    return {dx, gw.returned, gb.returned, Tensor()};
  }
};

Tensor conv_transpose2x2(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& w_fwd, const OptTensor& w_dgrad,
                         const Tensor& b4, int64_t split, bool fuse_bias, const Tensor& status) {
  auto l = c10::make_intrusive<ConvTLayer>();
  l->w_fwd = w_fwd, l->w_dgrad = w_dgrad, l->b4 = b4, l->weight = weight, l->bias = bias, l->split = split;
  l->fuse_bias = fuse_bias, l->status = status;
  return ConvT2x2::apply(x, weight, bias, l);
}

// ------------------------------------------------------------------------------------------------ GroupNorm + SiLU
struct NormLayer : torch::CustomClassHolder {
  Tensor g, b, gamma, beta;
  int64_t groups;
  double eps;
  bool has_res;
};

// (The launches on the tensors' own pointers: views of them as [B, pixels, C] were a third of the node's host time.)
struct GroupNormSilu : Function<GroupNormSilu> {
  struct Image {
    int B, C;
    long long HW;
    float inv_count;
    Image(const Tensor& x, int64_t groups) {
      need(x.is_cuda() && x.dim() == 4 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16, "groupnorm_silu: contiguous NHWC bf16");
      B = static_cast<int>(x.size(0)), C = static_cast<int>(x.size(3)), HW = x.size(1) * x.size(2);
      inv_count = static_cast<float>(1.0 / (static_cast<double>(HW) * (C / std::max<int64_t>(groups, 1))));
    }
  };
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gamma, const Tensor& beta, const OptTensor& residual,
                        const Held<NormLayer>& l) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Image im(x, l->groups);
    need(l->g.numel() == im.C && l->b.numel() == im.C && l->g.is_contiguous() && l->b.is_contiguous() && l->g.scalar_type() == torch::kBFloat16 &&
             l->b.scalar_type() == torch::kBFloat16,
         "groupnorm_silu: affine parameters bf16, one per channel");
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    Tensor stats = torch::empty({im.B, l->groups, 2}, x.options().dtype(torch::kFloat32));
    Tensor sums = terra_ops::scratch_take(x, {im.B * l->groups * 2 + 1});      // (and the ticket behind them)
    tb::note_launch(2);
    rc_check(tb::groupnorm_mean_rstd(x.data_ptr(), sums.data_ptr<float>(), stats.data_ptr<float>(), im.B, im.HW, im.C, static_cast<int>(l->groups),
                                     im.inv_count, static_cast<float>(l->eps), stream),
             "groupnorm_mean_rstd");
    terra_ops::scratch_give(sums);
    Tensor y = torch::empty_like(x), res;
    if (residual.has_value()) {
      need(residual->numel() == x.numel() && residual->is_cuda() && residual->scalar_type() == torch::kBFloat16,
           "groupnorm_silu: shortcut like the input");
      res = residual->contiguous();
    }
    rc_check(tb::groupnorm_silu_apply(x.data_ptr(), stats.data_ptr<float>(), l->g.data_ptr(), l->b.data_ptr(), res.defined() ? res.data_ptr() : nullptr,
                                      y.data_ptr(), im.B, im.HW, im.C, static_cast<int>(l->groups), stream),
             "groupnorm_silu_apply");
    ctx->save_for_backward({x, stats, l->g, l->b});
    hold(ctx, l);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto l = held<NormLayer>(ctx);
    const Tensor &x = s[0], &stats = s[1], &g = s[2], &b = s[3];
    const Tensor dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(dy.device());
    // (the saved tensors come back through whatever hooks the caller has set, so their form is checked like any input's)
    const Image im(x, l->groups);
    need(dy.sizes() == x.sizes() && dy.scalar_type() == torch::kBFloat16 && stats.is_cuda() && stats.is_contiguous() &&
             stats.scalar_type() == torch::kFloat32 && stats.numel() == 2 * im.B * l->groups && g.is_cuda() && g.is_contiguous() && b.is_cuda() &&
             b.is_contiguous() && g.numel() == im.C && b.numel() == im.C && g.scalar_type() == torch::kBFloat16 &&
             b.scalar_type() == torch::kBFloat16,
         "groupnorm_silu: saved tensors and the gradient like the forward pass's");
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    ParamGrad gg(l->gamma, "groupnorm: clearing the gradient"), gb(l->beta, "groupnorm: clearing the gradient");
    need(gg.into.numel() == im.C && gb.into.numel() == im.C, "groupnorm_silu: gradients of the affine parameters, one per channel");
    Tensor red = zeroed(x, {im.B, im.C, 2}, "groupnorm: clearing the gradient's sums"), dx = torch::empty_like(x);
    tb::note_launch(2);
    rc_check(tb::groupnorm_silu_bwd_reduce(dy.data_ptr(), x.data_ptr(), stats.data_ptr<float>(), g.data_ptr(), b.data_ptr(), red.data_ptr<float>(),
                                           gg.into.data_ptr<float>(), gb.into.data_ptr<float>(), im.B, im.HW, im.C, static_cast<int>(l->groups),
                                           stream),
             "groupnorm_silu_bwd_reduce");
    rc_check(tb::groupnorm_silu_bwd_apply(dy.data_ptr(), x.data_ptr(), stats.data_ptr<float>(), red.data_ptr<float>(), g.data_ptr(), b.data_ptr(),
                                          dx.data_ptr(), im.B, im.HW, im.C, static_cast<int>(l->groups), im.inv_count, stream),
             "groupnorm_silu_bwd_apply");
    return {dx, gg.returned, gb.returned, l->has_res ? dy : Tensor(), Tensor()};
  }
};

Tensor groupnorm_silu(const Tensor& x, const Tensor& gamma, const Tensor& beta, const OptTensor& residual, const Tensor& g, const Tensor& b,
                      int64_t groups, double eps) {
  auto l = c10::make_intrusive<NormLayer>();
  l->g = g, l->b = b, l->gamma = gamma, l->beta = beta, l->groups = groups, l->eps = eps, l->has_res = residual.has_value();
  return GroupNormSilu::apply(x, gamma, beta, residual, l);
}

// ------------------------------------------------------------------------------------------------ windows of an image and back
// x, seen as [outer, a, b, inner], with a and b exchanged, in the shape `sizes`
struct SwapMiddle : Function<SwapMiddle> {
  static Tensor copy(const Tensor& x, int64_t outer, int64_t a, int64_t b, at::IntArrayRef sizes) {
    const int64_t bytes = outer * a * b > 0 ? static_cast<int64_t>(x.nbytes()) / (outer * a * b) : 0;
    need(x.is_cuda() && x.is_contiguous() && bytes > 0 && bytes % 16 == 0 && bytes * outer * a * b == static_cast<int64_t>(x.nbytes()) &&
             reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0,
         "swap_middle: contiguous [outer, a, b, inner], inner whole 16-byte vectors");
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor y = torch::empty(sizes, x.options());
    need(y.numel() == x.numel(), "swap_middle: sizes");
    tb::note_launch();
    rc_check(tb::swap_middle_vectors(x.data_ptr(), y.data_ptr(), outer, a, b, bytes / 16, c10::cuda::getCurrentCUDAStream().stream()), "swap_middle");
    return y;
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t outer, int64_t a, int64_t b, std::vector<int64_t> sizes) {
    ctx->saved_data["dims"] = std::vector<int64_t>{outer, a, b};
    ctx->saved_data["sizes"] = x.sizes().vec();
    return copy(x, outer, a, b, sizes);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto d = ctx->saved_data["dims"].toIntVector(), sizes = ctx->saved_data["sizes"].toIntVector();
    Tensor dy = grads[0].contiguous();
    if (reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16 != 0) dy = dy.clone();
    return {SwapMiddle::apply(dy, d[0], d[2], d[1], sizes), Tensor(), Tensor(), Tensor(), Tensor()};   // itself differentiable, as the operators' is
  }
};

Tensor swap_middle(const Tensor& x, int64_t outer, int64_t a, int64_t b, std::vector<int64_t> sizes) {
  return SwapMiddle::apply(x, outer, a, b, std::move(sizes));
}

}  // namespace

void bind_nodes(pybind11::module_& m) {
  auto n = m.def_submodule("nodes", "layers as autograd nodes");
  n.def("attn_half", &attn_half);
  n.def("mlp_half", &mlp_half);
  n.def("linear", &linear);
  n.def("conv3x3", &conv3x3);
  n.def("conv_transpose2x2", &conv_transpose2x2);
  n.def("groupnorm_silu", &groupnorm_silu);
  n.def("swap_middle", &swap_middle, "x as [outer, a, b, inner] with a and b exchanged, in the shape given");
}
