// The transformer block halves as one native call per direction: the same launches in the same order as the Python form
// (which the multi-rank layouts use), without the interpreter between them. A small layer is bound by its launches: on 512
// rows of width 96 the Python form spent about 20 us per launch on the host against 1 to 10 us of kernel time.
#include <algorithm>
#include <tuple>
#include <vector>
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "check.h"
#include "host_api.h"
#include "launch_count.h"
#include "torch_ops.h"

namespace {

using torch::Tensor;
using OptTensor = c10::optional<torch::Tensor>;

cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
int sm_count() {
  static const int n = [] {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}
bool rows_bf16(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.is_contiguous();
}
// rows of any pitch (a product's operand)
bool rows_pitched(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.stride(1) == 1;
}
bool vec(const Tensor& t, at::ScalarType ty, int64_t n) { return t.is_cuda() && t.scalar_type() == ty && t.is_contiguous() && t.numel() == n; }

struct Epi {
  int flags = 0;
  const Tensor* bias = nullptr;
  const Tensor* residual = nullptr;
  const Tensor* aux = nullptr;
  const Tensor* pre = nullptr;
};

// an operand of the epilogue: rows like the output's
bool like_out(const Tensor* t, const Tensor& out) {
  return t == nullptr || (rows_pitched(*t) && t->sizes() == out.sizes() && t->device() == out.device());
}

// out [M, N] = epilogue(a [M, K] * w), w [N, K] or, with b_mn, [K, N]; the bias bf16 or fp32
void product(const Tensor& a, const Tensor& w, bool b_mn, const Tensor& out, const Epi& e, const Tensor& status) {
  need(rows_pitched(a) && rows_pitched(w) && rows_pitched(out) && a.device() == w.device() && a.device() == out.device(),
       "block half: operands must be 2-D bf16 rows on one GPU");
  need(a.size(1) == w.size(b_mn ? 0 : 1) && out.size(0) == a.size(0) && out.size(1) == w.size(b_mn ? 1 : 0), "block half: operand shapes");
  need(like_out(e.residual, out) && like_out(e.aux, out) && like_out(e.pre, out), "block half: operands of the epilogue");
  tb::GemmOperand A{a.data_ptr(), a.stride(0), 0}, B{w.data_ptr(), w.stride(0), b_mn ? 1 : 0};
  tb::GemmEpilogue g{};
  g.flags = e.flags;
  g.C = out.data_ptr();
  g.ldc = out.stride(0);
  if (e.bias != nullptr) {
    const bool f32 = e.bias->scalar_type() == torch::kFloat32;
    need(vec(*e.bias, f32 ? torch::kFloat32 : torch::kBFloat16, out.size(1)) && e.bias->device() == out.device(),
         "block half: bias bf16 or fp32, one entry per column");
    g.flags |= tb::EPI_BIAS | (f32 ? tb::EPI_BIAS_F32 : 0);
    g.bias = e.bias->data_ptr();
  }
  if (e.residual != nullptr) {
    g.flags |= tb::EPI_RESIDUAL;
    g.residual = e.residual->data_ptr();
    g.ldr = e.residual->stride(0);
  }
  if (e.aux != nullptr) {
    g.flags |= tb::EPI_MUL_DGELU;
    g.aux = e.aux->data_ptr();
    g.ldaux = e.aux->stride(0);
  }
  if (e.pre != nullptr) {
    g.flags |= tb::EPI_SAVE_PRE;
    g.C2 = e.pre->data_ptr();
    g.ldc2 = e.pre->stride(0);
  }
  g.alpha = 1.0f;
  g.status = status.data_ptr();
  tb::note_launch();
  rc_check(tb::gemm_bf16(A, B, a.size(0), out.size(1), a.size(1), g, 1, 0, sm_count(), cur_stream()), "gemm");
}

void column_sums(const Tensor& dy, const Tensor& out) {
  const int64_t parts = (dy.size(0) + tb::colsum_rows_per_block() - 1) / tb::colsum_rows_per_block();
  auto partials = torch::empty({parts, dy.size(1)}, dy.options().dtype(torch::kFloat32));
  tb::note_launch();
  rc_check(tb::colsum_bf16(dy.data_ptr(), out.data_ptr<float>(), partials.data_ptr<float>(), dy.size(0), dy.size(1), dy.stride(0),
                           cur_stream()),
           "colsum");
}

// Tile width, row blocks per tile and split of the contraction for N x K outputs over M rows. A k-block costs a CTA its
// operand fill plus the tensor core's reads through the shared-memory port, in KB; the column sums add 40 KB per row block,
// shared out over the column tiles. Every split pays its start and its pass of atomics (1100 KB a row block, and 1.3 KB per
// output block of the whole launch). Widths of 256 leave no room for the sums' accumulators: the column sums are then two
// launches of their own, which read dy once more (10 us and 5.6 TB/s against 3.7 us per 1000 KB).
// A pair of CTAs (request 1000 + width: 256 x 256 or 256 x 384 outputs) halves B's share and is bound by the tensor core instead: 512 or
// 768 cycles per k-block, 74 and 140 KB of that measure as timed. Only the 384-wide tile has room for the sums (16 KB, shared out alike).
// The constants of single CTAs were fitted to 11000 times: 64 to 557056 rows, 45 pairs of N and K between 96 and 4096, all widths, stacked
// or not, one to four rounds (passes back to back in a CUDA graph); the choice among them is 2 % slower than the best plan on average. Those of
// pairs are not part of that fit: the figures at the end are what they were set by. Without the 10 us the separate sums were taken for few rows
// too (us, that / this rule): 512 rows of 384 x 1536 22 / 9, 2048 of 256 x 1024 19 / 9, 17280 of
// 192 x 2208 39 / 23, 156672 of 3072 x 1024 839 / 799. Pairs (us, best single / pair): 557056 rows of 2976 x 384 with sums 1184 / 1032,
// without 1047 / 935, 139264 of 1536 x 384 231 / 202, 156672 of 3072 x 1024 without sums 704 / 647.
struct WgradPlan {
  int bn, stack, split;
  bool swapped;      // the transpose: rows are x's columns
};
WgradPlan plan_wgrad(int64_t N, int64_t K, int64_t M, bool sums) {
  const int64_t m_blocks = (N + 127) / 128, k_blocks = (M + 63) / 64, sms = sm_count();
  WgradPlan best{128, 1, 1, false};
  double least = -1.0;
  // `width` columns, `blocks` 128-row blocks a tile, `kb` KB a k-block, on `units` CTAs or pairs; `pair`: two CTAs share the blocks
  auto consider = [&](int request, int width, int stack, bool pair, double kb, double extra, bool swapped = false) {
    const int64_t blocks = pair ? 2 : stack, units = pair ? sms / 2 : sms;
    const int64_t rows = swapped ? (K + 127) / 128 : m_blocks;
    const int64_t n = ((swapped ? N : K) + width - 1) / width, tiles = (rows + blocks - 1) / blocks * n;
    if (sums && extra == 0.0 && !swapped) kb += (pair ? 16.0 : 40.0 * stack) / n;
    // whole rounds of CTAs: the largest split of one round, two rounds, ...
    for (int64_t rounds = 1; rounds <= 3; ++rounds) {
      const int64_t split = std::max<int64_t>(1, std::min(rounds * units / tiles, k_blocks));
      const int64_t per = (k_blocks + split - 1) / split;
      const double cost = static_cast<double>((tiles * split + units - 1) / units) * (per * kb + 1100.0 * (pair ? width / 128.0 : stack)) +
                          1.3 * tiles * split * blocks * width / 192 + (pair ? 600.0 : 0.0) + extra;   // (a pair starts 2 us later)
      if (least < 0.0 || cost < least * 0.995) {
        least = cost;
        best = {request, stack, static_cast<int>(split), swapped};
      }
    }
  };
  const double separate = sums ? (10.0 + 2.0 * M * N / 5.6e6) / 0.0037 : 0.0;
  for (int stack : {1, 2}) {
    if (stack > m_blocks) continue;
    for (int bn : {192, 128, 256})
      consider(bn, bn, stack, false, 16.0 * stack + bn / 8 + stack * (16.0 + bn / 8), bn == 256 ? separate : 0.0);
  }
  if (tb::gemm_pairs() && sms >= 2 && m_blocks >= 2) {
    if (K > 256) consider(1384, 384, 1, true, 140.0, 0.0);
    if (K > 128) consider(1256, 256, 1, true, 74.0, separate);
  }
  // few outputs of a wide layer (patch embedding: 384 x 2976): 384 rows fill one and a half pairs, 384 columns one tile
  if (tb::gemm_pairs() && sms >= 2 && N > 256 && K > 2 * N) consider(1384, 384, 1, true, 140.0, separate, true);
  return best;
}

}  // namespace

namespace terra_ops {

// grad_w [N, K] (fp32) += dy [M, N]^T x [M, K]; grad_b [N] += column sums of dy, from the same kernel (`fuse_bias`: a
// MMA of the dy tiles against ones) where its accumulators fit beside the tile's (single CTAs up to 192 columns, pairs of 384).
void wgrad(const Tensor& dy, const Tensor& x, const Tensor& grad_w, const OptTensor& grad_b, bool fuse_bias, const Tensor& status) {
  need(rows_pitched(dy) && rows_pitched(x) && dy.size(0) == x.size(0) && grad_w.scalar_type() == torch::kFloat32 && grad_w.dim() == 2 &&
           grad_w.is_cuda() && grad_w.stride(1) == 1 && grad_w.size(0) == dy.size(1) && grad_w.size(1) == x.size(1),
       "wgrad: dy [M, N], x [M, K] bf16, grad_w [N, K] fp32 rows");
  need(!grad_b.has_value() || vec(*grad_b, torch::kFloat32, dy.size(1)), "wgrad: grad_b fp32 [N]");
  need(dy.size(0) > 0 && dy.size(1) > 0 && x.size(1) > 0, "wgrad: empty operand");
  const c10::cuda::CUDAGuard guard(dy.device());
  const int64_t M = dy.size(0), N = dy.size(1), K = x.size(1);
  bool sums = grad_b.has_value();
  if (sums && !fuse_bias) {
    column_sums(dy, *grad_b);
    sums = false;
  }
  const WgradPlan plan = plan_wgrad(N, K, M, sums);
  if (sums && (plan.bn % 1000 == 256 || plan.swapped)) {
    column_sums(dy, *grad_b);
    sums = false;
  }
  tb::GemmOperand A{dy.data_ptr(), dy.stride(0), 1}, B{x.data_ptr(), x.stride(0), 1};
  if (plan.swapped) std::swap(A, B);
  tb::GemmEpilogue g{};
  g.flags = tb::EPI_OUT_F32 | tb::EPI_ATOMIC | (plan.swapped ? tb::EPI_TRANSPOSE : 0);
  g.C = grad_w.data_ptr();
  g.ldc = grad_w.stride(0);
  g.alpha = 1.0f;
  g.status = status.data_ptr();
  g.colsum = sums ? grad_b->data_ptr<float>() : nullptr;
  g.stack = plan.stack;
  tb::note_launch();
  rc_check(tb::gemm_bf16(A, B, plan.swapped ? K : N, plan.swapped ? N : K, M, g, plan.split, plan.bn, sm_count(), cur_stream()),
           "gemm (weight gradient)");
}

}  // namespace terra_ops

using namespace terra_ops;

namespace {

struct Norm {
  Tensor xn, mean, rstd;
};
Norm norm_fwd(const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
  need(rows_bf16(x) && vec(w, torch::kBFloat16, x.size(1)) && vec(b, torch::kBFloat16, x.size(1)), "block half: x [rows, C], norm weights bf16");
  Norm n;
  n.xn = torch::empty_like(x);
  n.mean = torch::empty({x.size(0)}, x.options().dtype(torch::kFloat32));
  n.rstd = torch::empty_like(n.mean);
  tb::note_launch();
  rc_check(tb::layernorm_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), n.xn.data_ptr(), n.mean.data_ptr<float>(),
                             n.rstd.data_ptr<float>(), x.size(0), static_cast<int>(x.size(1)), static_cast<float>(eps), cur_stream()),
           "layernorm_fwd");
  return n;
}
Tensor norm_bwd(const Tensor& dxn, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd, const Tensor& gw,
                const Tensor& gb, const Tensor& dres, const OptTensor& dres_sum) {
  need(rows_bf16(x) && rows_bf16(dxn) && rows_bf16(dres) && dxn.sizes() == x.sizes() && dres.sizes() == x.sizes(),
       "block half: x and its gradients must be contiguous [rows, C]");
  need(vec(w, torch::kBFloat16, x.size(1)) && vec(mean, torch::kFloat32, x.size(0)) && vec(rstd, torch::kFloat32, x.size(0)),
       "block half: norm weight bf16, row statistics fp32");
  need(vec(gw, torch::kFloat32, x.size(1)) && vec(gb, torch::kFloat32, x.size(1)), "block half: norm gradients fp32");
  need(!dres_sum.has_value() || vec(*dres_sum, torch::kFloat32, x.size(1)), "block half: bias gradient fp32, one entry per column");
  Tensor dx = torch::empty_like(x);
  tb::note_launch();
  rc_check(tb::layernorm_bwd(dxn.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(), dx.data_ptr(),
                             gw.data_ptr<float>(), gb.data_ptr<float>(), dres.data_ptr(), x.size(0), static_cast<int>(x.size(1)),
                             cur_stream(), dres_sum.has_value() ? dres_sum->data_ptr<float>() : nullptr),
           "layernorm_bwd");
  return dx;
}

// The bias gradient of a half's last product is the column sums of dy, which the LayerNorm's backward pass reads for the shortcut. For
// wide rows they are taken there: the weight gradient may then use tiles 256 wide, which have no room for them, without two launches that
// read dy once more (attention half of 156672 x 1024 4845 -> 4794 us). Narrower rows gain nothing (MLP half of 139264 x 384 1388 / 1401: the
// kernel spills), few rows would pay for half as many atomics again at the end of the kernel, and above 1024 columns it spills more.
bool sums_beside_norm(const Tensor& dy, bool fuse_bias) {
  return fuse_bias && dy.size(0) >= 32768 && dy.size(1) > 512 && dy.size(1) <= 1024;
}

// Window geometry of a rank that owns every window and token: {B, nWh, nWw, wh, ww, heads, sh, sw, use_mask}
tb::WindowAttnArgs window_args(const std::vector<int64_t>& g, int64_t C, const OptTensor& table, double scale, int64_t rows) {
  need(g.size() == 9 && g[5] > 0, "block half: window geometry");
  tb::WindowAttnArgs a{};
  a.B = static_cast<int>(g[0]);
  a.nWh = static_cast<int>(g[1]);
  a.nWw = static_cast<int>(g[2]);
  a.wh = static_cast<int>(g[3]);
  a.ww = static_cast<int>(g[4]);
  a.num_heads = static_cast<int>(g[5]);
  a.sh = static_cast<int>(g[6]);
  a.sw = static_cast<int>(g[7]);
  a.use_mask = g[8] != 0 ? 1 : 0;
  a.tp = a.n_wg = a.sp = 1;
  a.win_start[1] = a.nWh * a.nWw;
  a.shardN = a.wh * a.ww;
  a.C = static_cast<int>(C);
  a.scale = static_cast<float>(scale);
  need(static_cast<int64_t>(a.B) * a.win_start[1] * a.shardN == rows, "block half: rows = B * windows * tokens");
  if (table.has_value()) {
    need(vec(*table, torch::kFloat32, static_cast<int64_t>(2 * a.wh - 1) * (2 * a.ww - 1) * a.num_heads), "block half: bias table fp32");
    a.bias_table = table->data_ptr<float>();
  }
  return a;
}

}  // namespace

namespace terra_ops {

// y [M, N] = x [M, K] W^T (+ bias) (+ residual), or with `transposed` dx = dy W
Tensor linear_product(const Tensor& x, const Tensor& w, bool transposed, const OptTensor& bias, const OptTensor& residual, const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = torch::empty({x.size(0), w.size(transposed ? 1 : 0)}, x.options());
  Epi e;
  if (bias.has_value()) e.bias = &*bias;
  if (residual.has_value()) e.residual = &*residual;
  product(x, w, transposed, y, e, status);
  return y;
}

// -> y, mean, rstd, xn, qkv, o
std::vector<Tensor> attn_half_fwd(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& qkv_w, const Tensor& qkv_b,
                                  const Tensor& proj_w, const Tensor& proj_b, const OptTensor& table,
                                  const std::vector<int64_t>& geo, double scale, double eps, const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  Norm n = norm_fwd(x, ln_w, ln_b, eps);
  const int64_t rows = x.size(0), C = x.size(1);
  tb::WindowAttnArgs a = window_args(geo, C, table, scale, rows);
  Tensor qkv = torch::empty({rows, 3 * C}, x.options()), o = torch::empty_like(x), y = torch::empty_like(x);
  Epi e;
  e.bias = &qkv_b;
  product(n.xn, qkv_w, false, qkv, e, status);
  a.qkv[0] = qkv.data_ptr();
  a.out[0] = o.data_ptr();
  tb::note_launch();
  rc_check(tb::window_attn_fwd(a, cur_stream()), "window_attn_fwd");
  e.bias = &proj_b;
  e.residual = &x;
  product(o, proj_w, false, y, e, status);
  return {y, n.mean, n.rstd, n.xn, qkv, o};
}

// -> dx; the parameter gradients (fp32) are accumulated in place
Tensor attn_half_bwd(const Tensor& dy, const Tensor& x, const Tensor& mean, const Tensor& rstd, const Tensor& xn, const Tensor& qkv,
                     const Tensor& o, const Tensor& ln_w, const Tensor& qkv_w, const Tensor& proj_w, const OptTensor& table,
                     const Tensor& ln_wg, const Tensor& ln_bg, const Tensor& qkv_wg, const Tensor& qkv_bg, const Tensor& proj_wg,
                     const Tensor& proj_bg, const OptTensor& table_g, const std::vector<int64_t>& geo, double scale, bool fuse_bias,
                     const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  // (the saved tensors come back through whatever hooks the caller has set, so their form is checked like any input's)
  need(rows_bf16(x) && rows_bf16(dy) && dy.sizes() == x.sizes(), "block half: x and dy contiguous [rows, C]");
  need(rows_bf16(qkv) && qkv.size(0) == x.size(0) && qkv.size(1) == 3 * x.size(1), "block half: qkv contiguous [rows, 3 C]");
  tb::WindowAttnArgs a = window_args(geo, x.size(1), table, scale, x.size(0));
  const bool beside = sums_beside_norm(dy, fuse_bias);
  wgrad(dy, o, proj_wg, beside ? OptTensor() : OptTensor(proj_bg), fuse_bias, status);
  Tensor dout = torch::empty_like(x), dqkv = torch::empty_like(qkv), dxn = torch::empty_like(x);
  product(dy, proj_w, true, dout, Epi(), status);
  a.qkv[0] = qkv.data_ptr();
  a.dout[0] = dout.data_ptr();
  a.dqkv[0] = dqkv.data_ptr();
  if (table_g.has_value()) {
    need(table.has_value() && vec(*table_g, torch::kFloat32, table->numel()), "block half: bias table gradient fp32");
    a.dbias_table = table_g->data_ptr<float>();
  }
  tb::note_launch();
  rc_check(tb::window_attn_bwd(a, cur_stream()), "window_attn_bwd");
  wgrad(dqkv, xn, qkv_wg, qkv_bg, fuse_bias, status);
  product(dqkv, qkv_w, true, dxn, Epi(), status);
  return norm_bwd(dxn, x, ln_w, mean, rstd, ln_wg, ln_bg, dy, beside ? OptTensor(proj_bg) : OptTensor());
}

// y alone, where no backward pass follows: the pre-activation is not written
Tensor mlp_half_infer(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& fc1_w, const Tensor& fc1_b, const Tensor& fc2_w,
                      const Tensor& fc2_b, double eps, const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  Norm n = norm_fwd(x, ln_w, ln_b, eps);
  Tensor act = torch::empty({x.size(0), fc1_w.size(0)}, x.options()), y = torch::empty_like(x);
  Epi e;
  e.flags = tb::EPI_GELU;
  e.bias = &fc1_b;
  product(n.xn, fc1_w, false, act, e, status);
  Epi r;
  r.bias = &fc2_b;
  r.residual = &x;
  product(act, fc2_w, false, y, r, status);
  return y;
}

// -> y, mean, rstd, xn, pre, act
std::vector<Tensor> mlp_half_fwd(const Tensor& x, const Tensor& ln_w, const Tensor& ln_b, const Tensor& fc1_w, const Tensor& fc1_b,
                                 const Tensor& fc2_w, const Tensor& fc2_b, double eps, const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  Norm n = norm_fwd(x, ln_w, ln_b, eps);
  Tensor pre = torch::empty({x.size(0), fc1_w.size(0)}, x.options()), act = torch::empty_like(pre), y = torch::empty_like(x);
  Epi e;
  e.flags = tb::EPI_GELU;
  e.bias = &fc1_b;
  e.pre = &pre;
  product(n.xn, fc1_w, false, act, e, status);
  Epi r;
  r.bias = &fc2_b;
  r.residual = &x;
  product(act, fc2_w, false, y, r, status);
  return {y, n.mean, n.rstd, n.xn, pre, act};
}

Tensor mlp_half_bwd(const Tensor& dy, const Tensor& x, const Tensor& mean, const Tensor& rstd, const Tensor& xn, const Tensor& pre,
                    const Tensor& act, const Tensor& ln_w, const Tensor& fc1_w, const Tensor& fc2_w, const Tensor& ln_wg,
                    const Tensor& ln_bg, const Tensor& fc1_wg, const Tensor& fc1_bg, const Tensor& fc2_wg, const Tensor& fc2_bg,
                    bool fuse_bias, const Tensor& status) {
  const c10::cuda::CUDAGuard guard(x.device());
  need(rows_bf16(x) && rows_bf16(dy) && dy.sizes() == x.sizes(), "block half: x and dy contiguous [rows, C]");
  const bool beside = sums_beside_norm(dy, fuse_bias);
  wgrad(dy, act, fc2_wg, beside ? OptTensor() : OptTensor(fc2_bg), fuse_bias, status);
  Tensor dpre = torch::empty({x.size(0), fc2_w.size(1)}, x.options()), dxn = torch::empty_like(x);
  Epi e;
  e.aux = &pre;
  product(dy, fc2_w, true, dpre, e, status);
  wgrad(dpre, xn, fc1_wg, fc1_bg, fuse_bias, status);
  product(dpre, fc1_w, true, dxn, Epi(), status);
  return norm_bwd(dxn, x, ln_w, mean, rstd, ln_wg, ln_bg, dy, beside ? OptTensor(fc2_bg) : OptTensor());
}

}  // namespace terra_ops

void bind_halves(pybind11::module_& m) {
  m.def(
      "wgrad_plan",
      [](int64_t N, int64_t K, int64_t M, bool sums) {
        need(N > 0 && K > 0 && M > 0, "wgrad_plan: empty operand");
        const WgradPlan p = plan_wgrad(N, K, M, sums);
        return std::make_tuple(p.bn, p.stack, p.split);
      },
      "tile width, row blocks per tile and split of the contraction that wgrad takes");
  m.def(
      "wgrad_swapped",
      [](int64_t N, int64_t K, int64_t M, bool sums) {
        need(N > 0 && K > 0 && M > 0, "wgrad_swapped: empty operand");
        return plan_wgrad(N, K, M, sums).swapped;
      },
      "whether wgrad computes x^T dy and stores its transpose (the plan is then that of K x N outputs)");
  m.def("wgrad", &wgrad, "weight (and bias) gradient of a linear layer, accumulated in fp32");
  m.def("attn_half_fwd", &attn_half_fwd);
  m.def("attn_half_bwd", &attn_half_bwd);
  m.def("mlp_half_fwd", &mlp_half_fwd);
  m.def("mlp_half_bwd", &mlp_half_bwd);
}
