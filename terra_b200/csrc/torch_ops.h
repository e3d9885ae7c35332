// The launches on torch tensors that the autograd nodes put together; each is defined beside its Python binding.
#pragma once
#include <torch/extension.h>
#include <vector>

namespace terra_ops {

using torch::Tensor;
using OptTensor = c10::optional<torch::Tensor>;

void conv3x3_fwd(const Tensor& x, const Tensor& w, Tensor& y, int64_t stride, int64_t flags, const OptTensor& bias, const OptTensor& residual,
                 const OptTensor& status, const OptTensor& halo_lo, const OptTensor& halo_hi);
void conv3x3_s2_dgrad(const Tensor& dy, const Tensor& w, Tensor& dx, const OptTensor& status);
void convt2x2(int64_t op, const Tensor& in, const Tensor& w, const OptTensor& bias4, Tensor& out, const OptTensor& status);
// The weight gradients of one rank, all taps in one product: dw [9, Cin, Cout] or [4, Cout, Cin], accumulated, for fold_taps; bias_grad
// [Cout] accumulated, by launches of its own unless `fuse_bias`. The contraction is cut into `least_split` parts at least. `plan`
// ({columns, CTAs, row blocks, split}) takes the place of the rule's.
using TapPlanRequest = c10::optional<std::vector<int64_t>>;
void conv3x3_wgrad_taps(const Tensor& x, const Tensor& dy, Tensor& dw, int64_t stride, const OptTensor& status, const OptTensor& bias_grad,
                        bool fuse_bias, int64_t least_split, const TapPlanRequest& plan = c10::nullopt);
void convt2x2_wgrad_taps(const Tensor& x, const Tensor& dy, Tensor& dw, const OptTensor& status, const OptTensor& bias_grad, bool fuse_bias,
                         int64_t least_split, const TapPlanRequest& plan = c10::nullopt);
void fold_taps(Tensor& src, Tensor& dst);

// fp32 scratch that a call takes zeroed, for itself, and gives back zeroed once everything it launches with it is queued (zero_scratch.cpp)
Tensor scratch_take(const Tensor& like, at::IntArrayRef sizes);
void scratch_give(const Tensor& scratch);

void colsum(const Tensor& x, Tensor& out);

void wgrad(const Tensor& dy, const Tensor& x, const Tensor& grad_w, const OptTensor& grad_b, bool fuse_bias, const Tensor& status);
Tensor linear_product(const Tensor& x, const Tensor& w, bool transposed, const OptTensor& bias, const OptTensor& residual, const Tensor& status);
std::vector<Tensor> attn_half_fwd(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& qkv_w, const Tensor& qkv_b,
                                  const Tensor& proj_w, const Tensor& proj_b, const OptTensor& table, const std::vector<int64_t>& geo,
                                  double scale, double eps, const Tensor& status);
Tensor attn_half_bwd(const Tensor& dy, const Tensor& x, const Tensor& mean, const Tensor& rstd, const Tensor& xn, const Tensor& qkv,
                     const Tensor& o, const Tensor& ln_w, const Tensor& qkv_w, const Tensor& proj_w, const OptTensor& table,
                     const Tensor& ln_wg, const Tensor& ln_bg, const Tensor& qkv_wg, const Tensor& qkv_bg, const Tensor& proj_wg,
                     const Tensor& proj_bg, const OptTensor& table_g, const std::vector<int64_t>& geo, double scale, bool fuse_bias,
                     const Tensor& status);
std::vector<Tensor> mlp_half_fwd(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& fc1_w, const Tensor& fc1_b,
                                 const Tensor& fc2_w, const Tensor& fc2_b, double eps, const Tensor& status);
Tensor mlp_half_infer(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& fc1_w, const Tensor& fc1_b, const Tensor& fc2_w,
                      const Tensor& fc2_b, double eps, const Tensor& status);
Tensor mlp_half_bwd(const Tensor& dy, const Tensor& x, const Tensor& mean, const Tensor& rstd, const Tensor& xn, const Tensor& pre,
                    const Tensor& act, const Tensor& ln_w, const Tensor& fc1_w, const Tensor& fc2_w, const Tensor& ln_wg,
                    const Tensor& ln_bg, const Tensor& fc1_wg, const Tensor& fc1_bg, const Tensor& fc2_wg, const Tensor& fc2_bg,
                    bool fuse_bias, const Tensor& status);

}  // namespace terra_ops
