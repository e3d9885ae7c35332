// Python bindings (torch tensors -> raw-pointer host API). Only this file sees torch headers.
#include <cstring>
#include <utility>
#include <vector>
#include <torch/extension.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAGuard.h>

#include "check.h"
#include "host_api.h"
#include "torch_ops.h"
#include "launch_count.h"

namespace {

cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int sm_count() {
  static const int n = [] {      // (once, whichever thread comes first)
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

const void* opt_ptr(const c10::optional<torch::Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }

void check_bf16_2d(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.scalar_type() == torch::kBFloat16, name, " must be bf16");
  TORCH_CHECK(t.dim() == 2 && t.stride(1) == 1, name, " must be 2-D with unit inner stride");
}

// C = epilogue(A_op * B_op^T). a: [M,K] (or [K,M] when a_mn), b: [N,K] (or [K,N] when b_mn).
void gemm(const torch::Tensor& a, bool a_mn, const torch::Tensor& b, bool b_mn, torch::Tensor& c, int64_t flags,
          const c10::optional<torch::Tensor>& bias, const c10::optional<torch::Tensor>& residual,
          const c10::optional<torch::Tensor>& aux, const c10::optional<torch::Tensor>& c2, double alpha,
          int64_t split_k, int64_t bn, const c10::optional<torch::Tensor>& status, int64_t sms,
          const std::vector<int64_t>& a_peer_ptrs, int64_t rank,
          const std::vector<int64_t>& c_peer_ptrs, int64_t a_flags_ptr, int64_t a_epoch, int64_t a_budget_ns,
          int64_t a_interleave, int64_t a_chunks, const c10::optional<torch::Tensor>& colsum) {
  check_bf16_2d(a, "a");
  check_bf16_2d(b, "b");
  const c10::cuda::CUDAGuard guard(a.device());
  // a_peer_ptrs: `a` is this GPU's shard and the operand is the concatenation of all GPUs' shards (all-gather fused
  // into the loads). c_peer_ptrs: fp32 accumulation buffers of the row blocks' owners (reduce-scatter fused into the
  // stores); `c` is then this GPU's own buffer and only gives the leading dimension.
  const int64_t gather = a_peer_ptrs.size() > 1 ? static_cast<int64_t>(a_peer_ptrs.size()) : 1;
  TORCH_CHECK(gather == 1 || !a_mn, "gemm: gathered A must be K-major");
  const int64_t M = (a_mn ? a.size(1) : a.size(0)) * gather;
  const int64_t K = a_mn ? a.size(0) : a.size(1);
  const int64_t N = b_mn ? b.size(1) : b.size(0);
  const int64_t Kb = b_mn ? b.size(0) : b.size(1);
  if (K != Kb) need(false, ("gemm: contraction mismatch " + std::to_string(K) + " vs " + std::to_string(Kb)).c_str());
  tb::GemmOperand A{a.data_ptr(), a.stride(0), a_mn ? 1 : 0};
  tb::GemmOperand B{b.data_ptr(), b.stride(0), b_mn ? 1 : 0};
  tb::GemmEpilogue e{};
  e.flags = static_cast<int>(flags);
  e.C = c.data_ptr();
  e.ldc = c.dim() >= 2 ? c.stride(c.dim() - 2) : c.size(-1);
  e.C2 = c2.has_value() ? c2->data_ptr() : nullptr;
  e.ldc2 = c2.has_value() ? c2->stride(0) : 0;
  e.bias = opt_ptr(bias);
  e.residual = opt_ptr(residual);
  e.ldr = residual.has_value() ? residual->stride(residual->dim() - 2) : 0;
  e.aux = opt_ptr(aux);
  e.ldaux = aux.has_value() ? aux->stride(0) : 0;
  e.alpha = static_cast<float>(alpha);
  e.status = status.has_value() ? status->data_ptr() : nullptr;
  if (colsum.has_value()) {
    TORCH_CHECK(colsum->scalar_type() == torch::kFloat32 && colsum->is_contiguous() && colsum->numel() == M,
                "gemm: colsum must be contiguous fp32 with one entry per output row");
    e.colsum = colsum->data_ptr<float>();
  }
  tb::note_launch();
  tb::GemmPeers peers;
  std::memset(&peers, 0, sizeof(peers));
  TORCH_CHECK(a_peer_ptrs.size() <= 8 && c_peer_ptrs.size() <= 8, "gemm: at most 8 peers");
  if (gather > 1) {
    peers.a_peers = static_cast<int>(gather);
    peers.a_rows = a.size(0);
    for (size_t i = 0; i < a_peer_ptrs.size(); ++i) peers.a_ptr[i] = reinterpret_cast<const void*>(a_peer_ptrs[i]);
  }
  peers.rank = static_cast<int>(rank);
  peers.a_flags = reinterpret_cast<const void*>(a_flags_ptr);
  peers.a_epoch = static_cast<unsigned int>(a_epoch);
  peers.a_budget_ns = static_cast<unsigned long long>(a_budget_ns);
  peers.a_interleave = static_cast<int>(a_interleave);
  peers.a_chunks = static_cast<int>(a_chunks);
  if (c_peer_ptrs.size() > 1) {
    peers.c_peers = static_cast<int>(c_peer_ptrs.size());
    TORCH_CHECK(M % peers.c_peers == 0, "gemm: rows not divisible by the number of owners");
    peers.c_rows = M / peers.c_peers;
    for (size_t i = 0; i < c_peer_ptrs.size(); ++i) peers.c_ptr[i] = reinterpret_cast<void*>(c_peer_ptrs[i]);
  }
  const int rc = tb::gemm_bf16_peers(A, B, M, N, K, e, peers, static_cast<int>(split_k), static_cast<int>(bn),
                                     sms > 0 ? static_cast<int>(sms) : sm_count(), cur_stream());
  if (rc != 0)
    rc_check(rc, ("gemm (M=" + std::to_string(M) + " N=" + std::to_string(N) + " K=" + std::to_string(K) + ") launch").c_str());
}

}  // namespace

namespace terra_ops {

// x: [B,H,W,Cin] bf16 NHWC, w: [Cout, 9*Cin_pad] bf16, y: [B,Ho,Wo,Cout]
void conv3x3_fwd(const torch::Tensor& x, const torch::Tensor& w, torch::Tensor& y, int64_t stride, int64_t flags,
                 const c10::optional<torch::Tensor>& bias, const c10::optional<torch::Tensor>& residual,
                 const c10::optional<torch::Tensor>& status, const c10::optional<torch::Tensor>& halo_lo,
                 const c10::optional<torch::Tensor>& halo_hi) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.is_contiguous() && x.dim() == 4, "x: NHWC bf16");
  TORCH_CHECK(w.scalar_type() == torch::kBFloat16 && w.is_contiguous() && w.dim() == 2, "w: [Cout, 9*Cin_pad] bf16");
  for (const auto* h : {&halo_lo, &halo_hi})
    TORCH_CHECK(!h->has_value() || ((*h)->is_contiguous() && (*h)->scalar_type() == torch::kBFloat16 &&
                                    (*h)->numel() == x.size(0) * x.size(2) * x.size(3)),
                "halo rows must be contiguous bf16 [B, 1, W, Cin]");
  TORCH_CHECK(y.is_contiguous(), "y must be contiguous");
  const c10::cuda::CUDAGuard guard(x.device());
  tb::GemmEpilogue e{};
  e.flags = static_cast<int>(flags);
  e.C = y.data_ptr();
  e.ldc = y.size(3);
  e.bias = opt_ptr(bias);
  e.residual = opt_ptr(residual);
  e.ldr = y.size(3);
  e.alpha = 1.0f;
  e.status = status.has_value() ? status->data_ptr() : nullptr;
  tb::note_launch();
  const int rc = tb::conv3x3_fwd_bf16(x.data_ptr(), w.data_ptr(), x.size(0), x.size(1), x.size(2), x.size(3), w.size(0),
                                      static_cast<int>(stride), e, sm_count(), cur_stream(), opt_ptr(halo_lo),
                                      opt_ptr(halo_hi));
  rc_check(rc, "conv3x3_fwd");
}

// dw: [9, Cout, Cin] fp32 (zeroed by the caller)
void conv3x3_wgrad(const torch::Tensor& x, const torch::Tensor& dy, torch::Tensor& dw, int64_t stride, int64_t split_k,
                   const c10::optional<torch::Tensor>& status, const c10::optional<torch::Tensor>& halo_lo,
                   const c10::optional<torch::Tensor>& halo_hi, const c10::optional<torch::Tensor>& bias_grad, int64_t stack) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.is_contiguous() && x.dim() == 4, "x: NHWC bf16");
  TORCH_CHECK(dy.scalar_type() == torch::kBFloat16 && dy.is_contiguous() && dy.dim() == 4, "dy: NHWC bf16");
  TORCH_CHECK(!bias_grad.has_value() || (bias_grad->scalar_type() == torch::kFloat32 && bias_grad->is_contiguous() &&
                                         bias_grad->numel() == dy.size(3)),
              "bias_grad: contiguous fp32 [Cout]");
  TORCH_CHECK(dw.scalar_type() == torch::kFloat32 && dw.is_contiguous(), "dw: fp32 [9,Cout,Cin]");
  const c10::cuda::CUDAGuard guard(x.device());
  tb::note_launch();
  const int rc = tb::conv3x3_wgrad_bf16(x.data_ptr(), dy.data_ptr(), dw.data_ptr<float>(), x.size(0), x.size(1),
                                        x.size(2), x.size(3), dy.size(3), static_cast<int>(stride),
                                        static_cast<int>(split_k), status.has_value() ? status->data_ptr() : nullptr,
                                        sm_count(), cur_stream(), opt_ptr(halo_lo), opt_ptr(halo_hi),
                                        bias_grad.has_value() ? bias_grad->data_ptr<float>() : nullptr,
                                        static_cast<int>(stack));
  rc_check(rc, "conv3x3_wgrad");
}

static void check_image(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.is_contiguous() && t.dim() == 4, name, ": NHWC bf16 contiguous");
}
static void check_packed(const torch::Tensor& w, int64_t rows, int64_t taps, int64_t channels) {
  TORCH_CHECK(w.scalar_type() == torch::kBFloat16 && w.is_contiguous() && w.dim() == 2 && w.size(0) == rows &&
                  w.size(1) == taps * ((channels + 63) / 64 * 64),
              "packed weights: bf16 [rows, taps * channels padded to 64]");
}
static void* status_ptr(const c10::optional<torch::Tensor>& s) { return s.has_value() ? s->data_ptr() : nullptr; }

// dy: [B, Ho, Wo, Cout], dx: [B, H, W, Cin] with Ho = (H + 1) / 2, Wo = W / 2; w: [Cin, 9 * Cout_pad]
void conv3x3_s2_dgrad(const torch::Tensor& dy, const torch::Tensor& w, torch::Tensor& dx,
                      const c10::optional<torch::Tensor>& status) {
  check_image(dy, "dy");
  check_image(dx, "dx");
  TORCH_CHECK(dy.size(0) == dx.size(0) && dy.size(1) == (dx.size(1) + 1) / 2 && 2 * dy.size(2) == dx.size(2),
              "conv3x3_s2_dgrad: dy must be the stride-2 output grid of dx");
  check_packed(w, dx.size(3), 9, dy.size(3));
  const c10::cuda::CUDAGuard guard(dy.device());
  tb::note_launch();
  const int rc = tb::conv3x3_s2_dgrad_bf16(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), dx.size(0), dx.size(1), dx.size(2), dx.size(3),
                                           dy.size(3), status_ptr(status), sm_count(), cur_stream());
  rc_check(rc, "conv3x3_s2_dgrad");
}

// The three products of the 2x2 / stride-2 transposed convolution, x [B, H, W, Cin] and y / dy [B, 2H, 2W, Cout]:
// op 0: y from x (w: [4 * Cout_pad, Cin_pad], bias [4 * Cout_pad]); op 1: dx from dy (w: [Cin, 4 * Cout_pad])
void convt2x2(int64_t op, const torch::Tensor& in, const torch::Tensor& w, const c10::optional<torch::Tensor>& bias4,
              torch::Tensor& out, const c10::optional<torch::Tensor>& status) {
  check_image(in, "in");
  check_image(out, "out");
  const torch::Tensor &x = op == 0 ? in : out, &y = op == 0 ? out : in;
  TORCH_CHECK(x.size(0) == y.size(0) && 2 * x.size(1) == y.size(1) && 2 * x.size(2) == y.size(2), "convt2x2: grids");
  const int64_t Cin = x.size(3), Cout = y.size(3);
  const int64_t phase = (Cout + 63) / 64 * 64;
  check_packed(w, op == 0 ? 4 * phase : Cin, op == 0 ? 1 : 4, op == 0 ? Cin : Cout);
  TORCH_CHECK(op != 0 || (bias4.has_value() && bias4->scalar_type() == torch::kBFloat16 && bias4->is_contiguous() &&
                          bias4->numel() == 4 * phase),
              "convt2x2: bias bf16 [4 * Cout_pad]");
  const c10::cuda::CUDAGuard guard(x.device());
  tb::note_launch();
  const int rc = op == 0 ? tb::convt2x2_fwd_bf16(x.data_ptr(), w.data_ptr(), opt_ptr(bias4), out.data_ptr(), x.size(0), x.size(1),
                                                 x.size(2), Cin, Cout, status_ptr(status), sm_count(), cur_stream())
                         : tb::convt2x2_dgrad_bf16(y.data_ptr(), w.data_ptr(), out.data_ptr(), x.size(0), x.size(1), x.size(2), Cin,
                                                   Cout, status_ptr(status), sm_count(), cur_stream());
  rc_check(rc, "convt2x2");
}

// dw: [4, Cout, Cin] fp32 and bias_grad: [Cout] fp32, accumulated
void convt2x2_wgrad(const torch::Tensor& x, const torch::Tensor& dy, torch::Tensor& dw, int64_t split_k,
                    const c10::optional<torch::Tensor>& status, int64_t stack,
                    const c10::optional<torch::Tensor>& bias_grad) {
  check_image(x, "x");
  check_image(dy, "dy");
  TORCH_CHECK(x.size(0) == dy.size(0) && 2 * x.size(1) == dy.size(1) && 2 * x.size(2) == dy.size(2), "convt2x2_wgrad: grids");
  TORCH_CHECK(dw.scalar_type() == torch::kFloat32 && dw.is_contiguous() && dw.numel() == 4 * x.size(3) * dy.size(3),
              "dw: fp32 [4, Cout, Cin]");
  TORCH_CHECK(!bias_grad.has_value() || (bias_grad->scalar_type() == torch::kFloat32 && bias_grad->is_contiguous() &&
                                         bias_grad->numel() == dy.size(3)),
              "bias_grad: contiguous fp32 [Cout]");
  const c10::cuda::CUDAGuard guard(x.device());
  tb::note_launch();
  const int rc = tb::convt2x2_wgrad_bf16(x.data_ptr(), dy.data_ptr(), dw.data_ptr<float>(), x.size(0), x.size(1), x.size(2),
                                         x.size(3), dy.size(3), static_cast<int>(split_k), status_ptr(status), sm_count(),
                                         cur_stream(), static_cast<int>(stack),
                                         bias_grad.has_value() ? bias_grad->data_ptr<float>() : nullptr);
  rc_check(rc, "convt2x2_wgrad");
}

static void check_patches(const Tensor& image, const Tensor& grid, const Tensor& w, const Tensor& bias, int64_t p, int64_t top, int64_t left) {
  check_image(image, "image");
  check_image(grid, "patches");
  TORCH_CHECK(grid.device() == image.device() && w.device() == image.device() && bias.device() == image.device(), "patches: operands on one GPU");
  TORCH_CHECK(image.numel() > 0 && image.size(0) == grid.size(0) && p >= 1 && p <= 4 && image.size(1) % p == 0 && image.size(2) % p == 0 && top >= 0 &&
                  left >= 0 && top + image.size(1) / p <= grid.size(1) && left + image.size(2) / p <= grid.size(2) && p * image.size(3) % 8 == 0 &&
                  grid.size(3) % 8 == 0 && p * ((p * image.size(3) + 63) / 64) <= 128 && (grid.size(3) + 63) / 64 <= 128,
              "patches: an image of whole patches inside the grid");
}

// image [B, H, W, C] -> y [B, rows, cols, N]; w [N, p * (p * C padded to 64)], bias [N]; top and left in patches
void embed_image(const Tensor& image, const Tensor& w, const Tensor& bias, Tensor& y, int64_t p, int64_t top, int64_t left, const OptTensor& status) {
  check_patches(image, y, w, bias, p, top, left);
  check_packed(w, y.size(3), p, p * image.size(3));
  TORCH_CHECK(bias.scalar_type() == torch::kBFloat16 && bias.is_contiguous() && bias.numel() == y.size(3), "embed_image: bias bf16 [N]");
  const c10::cuda::CUDAGuard guard(image.device());
  tb::note_launch();
  rc_check(tb::embed_image_bf16(image.data_ptr(), w.data_ptr(), bias.data_ptr(), y.data_ptr(), image.size(0), image.size(1), image.size(2),
                                image.size(3), p, top, left, y.size(1), y.size(2), y.size(3), status_ptr(status), sm_count(), cur_stream()),
           "embed_image");
}

// out = image + the patches of t [B, rows, cols, D] inside it; w [p * (p * C padded to 64), D padded to 64], bias alike
void recover_image(const Tensor& t, const Tensor& w, const Tensor& bias, const Tensor& image, Tensor& out, int64_t p, int64_t top, int64_t left,
                   const OptTensor& status) {
  check_patches(image, t, w, bias, p, top, left);
  check_image(out, "out");
  TORCH_CHECK(out.device() == image.device(), "recover_image: out on the image's GPU");
  const int64_t run = (p * image.size(3) + 63) / 64 * 64;
  check_packed(w, p * run, 1, t.size(3));
  TORCH_CHECK(out.sizes() == image.sizes() && bias.scalar_type() == torch::kBFloat16 && bias.is_contiguous() && bias.numel() == p * run,
              "recover_image: out like the image, bias bf16, a run padded to 64 per image row");
  const c10::cuda::CUDAGuard guard(image.device());
  tb::note_launch();
  rc_check(tb::recover_image_bf16(t.data_ptr(), w.data_ptr(), bias.data_ptr(), image.data_ptr(), out.data_ptr(), image.size(0), image.size(1),
                                  image.size(2), image.size(3), p, top, left, t.size(1), t.size(2), t.size(3), status_ptr(status), sm_count(),
                                  cur_stream()),
           "recover_image");
}

static tb::TapPlan tap_plan(const TapPlanRequest& request, int taps, int64_t channels, int64_t N, int64_t k_blocks, bool row_sums, bool column_sums,
                            int64_t least_split) {
  if (!request.has_value())
    return tb::plan_tap_wgrad(taps, static_cast<int>(channels), static_cast<int>(N), k_blocks, row_sums, column_sums, static_cast<int>(least_split),
                              sm_count());
  const auto& r = *request;
  TORCH_CHECK(r.size() == 4 && r[3] >= 1 && (r[1] == 1 ? (r[0] == 128 || r[0] == 192) && (r[2] == 1 || r[2] == 2)
                                                        : r[1] == 2 && r[2] == 1 && (r[0] == 384 || (r[0] == 256 && !column_sums))),
              "tap plan: {columns, CTAs, row blocks, split}");
  return {static_cast<int>(r[0]), static_cast<int>(r[1]), static_cast<int>(r[2]), static_cast<int>(r[3])};
}
static float* grad_ptr(const OptTensor& g, int64_t n) {
  TORCH_CHECK(!g.has_value() || (g->is_cuda() && g->scalar_type() == torch::kFloat32 && g->is_contiguous() && g->numel() == n),
              "bias_grad: contiguous fp32 [Cout]");
  return g.has_value() ? g->data_ptr<float>() : nullptr;
}

void conv3x3_wgrad_taps(const Tensor& x, const Tensor& dy, Tensor& dw, int64_t stride, const OptTensor& status, const OptTensor& bias_grad,
                        bool fuse_bias, int64_t least_split, const TapPlanRequest& request) {
  check_image(x, "x");
  check_image(dy, "dy");
  const int64_t Cin = x.size(3), Cout = dy.size(3), pixels = dy.numel() / std::max<int64_t>(Cout, 1);
  TORCH_CHECK((stride == 1 || (stride == 2 && x.size(2) % 2 == 0)) && x.size(0) == dy.size(0) && dy.size(1) == (x.size(1) + stride - 1) / stride &&
                  dy.size(2) == x.size(2) / stride && pixels > 0,
              "conv3x3_wgrad_taps: grids");
  TORCH_CHECK(dw.is_cuda() && dw.scalar_type() == torch::kFloat32 && dw.is_contiguous() && dw.numel() == 9 * Cin * Cout, "dw: fp32 [9, Cin, Cout]");
  float* const sums = grad_ptr(bias_grad, Cout);
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t k_blocks = (dy.size(2) + 63) / 64 * dy.size(1) * dy.size(0);
  const bool fused = fuse_bias && sums != nullptr;
  const tb::TapPlan plan = tap_plan(request, 9, Cin, Cout, k_blocks, fused, false, least_split);
  tb::note_launch();
  const int rc = tb::conv3x3_wgrad_taps_bf16(x.data_ptr(), dy.data_ptr(), dw.data_ptr<float>(), x.size(0), x.size(1), x.size(2), Cin, Cout,
                                             static_cast<int>(stride), plan, status_ptr(status), sm_count(), cur_stream(), fused ? sums : nullptr);
  rc_check(rc, "conv3x3_wgrad_taps");
  if (sums != nullptr && !fused) {
    Tensor out = *bias_grad;
    colsum(dy.view({-1, Cout}), out);
  }
}

void convt2x2_wgrad_taps(const Tensor& x, const Tensor& dy, Tensor& dw, const OptTensor& status, const OptTensor& bias_grad, bool fuse_bias,
                         int64_t least_split, const TapPlanRequest& request) {
  check_image(x, "x");
  check_image(dy, "dy");
  const int64_t Cin = x.size(3), Cout = dy.size(3), pixels = x.numel() / std::max<int64_t>(Cin, 1);
  TORCH_CHECK(x.size(0) == dy.size(0) && 2 * x.size(1) == dy.size(1) && 2 * x.size(2) == dy.size(2) && pixels > 0, "convt2x2_wgrad_taps: grids");
  TORCH_CHECK(dw.is_cuda() && dw.scalar_type() == torch::kFloat32 && dw.is_contiguous() && dw.numel() == 4 * Cin * Cout, "dw: fp32 [4, Cout, Cin]");
  float* const sums = grad_ptr(bias_grad, Cout);
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t k_blocks = (x.size(2) + 63) / 64 * x.size(1) * x.size(0);
  const bool fused = fuse_bias && sums != nullptr;
  const tb::TapPlan plan = tap_plan(request, 4, Cout, Cin, k_blocks, false, fused, least_split);
  tb::note_launch();
  const int rc = tb::convt2x2_wgrad_taps_bf16(x.data_ptr(), dy.data_ptr(), dw.data_ptr<float>(), x.size(0), x.size(1), x.size(2), Cin, Cout,
                                              plan, status_ptr(status), sm_count(), cur_stream(), fused ? sums : nullptr);
  rc_check(rc, "convt2x2_wgrad_taps");
  if (sums != nullptr && !fused) {
    Tensor out = *bias_grad;
    colsum(dy.view({-1, Cout}), out);
  }
}

}  // namespace terra_ops

using namespace terra_ops;

void bind_elementwise(pybind11::module_& m);
void bind_attention(pybind11::module_& m);
void bind_halves(pybind11::module_& m);
void bind_nodes(pybind11::module_& m);
void bind_copy_engine(pybind11::module_& m);
void bind_comm(pybind11::module_& m);

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("launch_count", []() { return static_cast<int64_t>(tb::g_kernel_launches.load()); });
  m.def("gemm_stall_counters", [](bool reset) {
    unsigned long long v[8];
    TORCH_CHECK(tb::gemm_stall_counters(v, reset ? 1 : 0) == 0, "gemm_stall_counters failed");
    std::vector<int64_t> out(v, v + 8);
    return out;
  });
  namespace py = pybind11;
  m.def("gemm", &gemm, "tcgen05 bf16 GEMM with fused epilogues", py::arg("a"), py::arg("a_mn"), py::arg("b"),
        py::arg("b_mn"), py::arg("c"), py::arg("flags"), py::arg("bias"), py::arg("residual"), py::arg("aux"),
        py::arg("c2"), py::arg("alpha"), py::arg("split_k"), py::arg("bn"), py::arg("status"), py::arg("sms"),
        py::arg("a_peer_ptrs"), py::arg("rank"),
        py::arg("c_peer_ptrs"), py::arg("a_flags_ptr"), py::arg("a_epoch"), py::arg("a_budget_ns"),
        py::arg("a_interleave"), py::arg("a_chunks"), py::arg("colsum") = py::none());
  m.def(
      "gemm_tile",
      [](int64_t M, int64_t N, int64_t K, bool b_mn, int64_t flags, int64_t sms, bool gathered) {
        int bn = 0, ctas = 0;
        tb::gemm_tile(M, N, K, b_mn, static_cast<int>(flags), gathered, static_cast<int>(sms), &bn, &ctas);
        return std::make_pair(bn, ctas);
      },
      "tile width and CTAs per tile that gemm takes when no width is asked for", py::arg("m"), py::arg("n"), py::arg("k"),
      py::arg("b_mn") = false, py::arg("flags") = 0, py::arg("sms") = 148, py::arg("gathered") = false);
  m.def("gemm_tma_epilogue", &tb::gemm_tma_epilogue, "whether the epilogue may go through TMA (TERRA_GEMM_TMA_EPILOGUE)");
  m.def("conv3x3_fwd", &conv3x3_fwd, "implicit-GEMM 3x3 convolution (NHWC bf16)");
  m.def("conv3x3_wgrad", &conv3x3_wgrad, "3x3 convolution weight gradient (fp32 atomics)", py::arg("x"), py::arg("dy"),
        py::arg("dw"), py::arg("stride"), py::arg("split_k"), py::arg("status"), py::arg("halo_lo"), py::arg("halo_hi"),
        py::arg("bias_grad") = py::none(), py::arg("stack") = 1);
  m.def("conv3x3_s2_dgrad", &conv3x3_s2_dgrad, "input gradient of the stride-2 3x3 convolution (NHWC bf16)");
  m.def("convt2x2", &convt2x2, "2x2 / stride-2 transposed convolution: forward (op 0), input gradient (op 1)", py::arg("op"),
        py::arg("input"), py::arg("w"), py::arg("bias4"), py::arg("out"), py::arg("status"));
  m.def("convt2x2_wgrad", &convt2x2_wgrad, "2x2 / stride-2 transposed convolution: weight gradient (fp32 atomics)",
        py::arg("x"), py::arg("dy"), py::arg("dw"), py::arg("split_k"), py::arg("status"), py::arg("stack") = 1, py::arg("bias_grad") = py::none());
  m.def("embed_image", &embed_image, "patch embedding that reads the image itself");
  m.def("recover_image", &recover_image, "patch recovery that adds to the image itself");
  m.def("conv3x3_wgrad_taps", &conv3x3_wgrad_taps, "3x3 convolution: weight gradients of all taps as one product", py::arg("x"), py::arg("dy"),
        py::arg("dw"), py::arg("stride"), py::arg("status"), py::arg("bias_grad") = py::none(), py::arg("fuse_bias") = true,
        py::arg("least_split") = 1, py::arg("plan") = py::none());
  m.def("convt2x2_wgrad_taps", &convt2x2_wgrad_taps, "2x2 / stride-2 transposed convolution: weight gradients of all taps as one product",
        py::arg("x"), py::arg("dy"), py::arg("dw"), py::arg("status"), py::arg("bias_grad") = py::none(), py::arg("fuse_bias") = true,
        py::arg("least_split") = 1, py::arg("plan") = py::none());
  m.def(
      "tap_wgrad_plan",
      [](int64_t taps, int64_t channels, int64_t N, int64_t k_blocks, bool row_sums, bool column_sums, int64_t least_split) {
        const tb::TapPlan p = tb::plan_tap_wgrad(static_cast<int>(taps), static_cast<int>(channels), static_cast<int>(N), k_blocks, row_sums,
                                                 column_sums, static_cast<int>(least_split), 148);
        return std::vector<int64_t>{p.bn, p.ctas, p.stack, p.split};
      },
      "the rule's plan on 148 SMs: columns, CTAs, row blocks, split", py::arg("taps"), py::arg("channels"), py::arg("n"), py::arg("k_blocks"),
      py::arg("row_sums"), py::arg("column_sums"), py::arg("least_split") = 1);
  bind_elementwise(m);
  bind_attention(m);
  bind_halves(m);
  bind_nodes(m);
  bind_copy_engine(m);
  bind_comm(m);
}
