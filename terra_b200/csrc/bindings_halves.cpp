// The transformer block halves as one native call per direction: the same launches in the same order as the Python form
// (which the multi-rank layouts use), without the interpreter between them. A small layer is bound by its launches: on 512
// rows of width 96 the Python form spent about 20 us per launch on the host against 1 to 10 us of kernel time.
#include <algorithm>
#include <cstdint>
#include <tuple>
#include <vector>
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "check.h"
#include "host_api.h"
#include "launch_count.h"
#include "size_memo.h"
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

// Tile width, row blocks per tile and split of the contraction for N x K outputs over M rows: the plan of least time by a model, in us. Rounds of
// tiles over the CTAs (or pairs: request 1000 + width), each its k-blocks and a hand-over with the epilogue. A k-block costs less where fewer
// CTAs than there are SMs share L2's bandwidth; the column sums (the bias gradient) are more MMAs, shared out over the column tiles. Widths of
// 256 and transposed plans have no room for the sums' accumulators, or the wrong operand: there the sums are two launches that read dy once
// more, or rows of ones behind x's columns where the last pair has room for it (557056 rows of 384 x 2976 1003 / 890 us).
// Transposed: few outputs of a wide layer (patch embedding: 384 x 2976), 384 rows filling one and a half pairs, 384 columns one tile.
//
// Fitted to 9000 passes in CUDA graphs: 200 to 557056 rows, 22 pairs of N and K between 96 and 4096, with and without sums, all tiles, half
// a round to three; the choice is 0.9 % slower than the best plan on average, 9 % at most. The plans of the fit before, which was made with
// epilogues through the lanes, were 3.7 % slower than the best on average. Us, those plans / this: 17280 rows of 1024 x 1024 44 / 32, 40000
// of 3072 x 1024 with sums 220 / 186, 139264 of 1536 x 384 134 / 120, of 768 x 768 with sums 169 / 125, 156672 of 3072 x 1024 with sums 820
// / 730.
//
// The error of the tensor core's fp32 sums grows with their length (1.0e-6 of the norm at 15 k-blocks, 8.6e-6 at 128, 13e-6 at 192). So among
// plans within 3 % the one with most parts is taken; a part is longer than 32 k-blocks only where 128 x 256 tiles in one round would have it
// so; and it is no longer than 15 k-blocks or what the tiles that cover the outputs with least padding have in one round, where that costs
// no more than 15 %. Without the last of these one size in fifty had parts twice as long as with the 256-row tiles it took before. Error
// and us, without / with: 557056 rows of 192 x 192 8.4e-6 / 4.0e-6 and 67.5 / 67.7, 156672 of 768 x 192 7.2e-6 / 3.4e-6 and 52.7 / 53.3,
// 17280 of 1024 x 1024 4.7e-6 / 2.0e-6 and 30.3 / 30.3; at worst 36228 of 256 x 256 1.1e-6 / 0.6e-6 and 10.8 / 12.5. Shorter parts
// for all that would take them within 15 % cost 139264 rows of 1152 x 384 7 % for what no size had before.
struct WgradPlan {
  int bn, stack, split;
  bool swapped;      // the transpose: rows are x's columns
};
// How many of the tiles of 128 or 256 rows and 128, 192 or 256 columns it takes that cover N x K outputs with least padding: of several, the
// largest, but with sums 192 columns before 256, which have no room for them.
int64_t covering_tiles(int64_t N, int64_t K, bool sums) {
  std::tuple<int64_t, int, int64_t> least{INT64_MAX, 0, 0};
  for (int64_t h : {128, 256})
    for (int64_t w : {128, 192, 256}) {
      const int64_t count = (N + h - 1) / h * ((K + w - 1) / w);
      least = std::min(least, {count * h * w, !sums ? 0 : w == 192 ? 0 : w == 256 ? 1 : 2, count});
    }
  return std::get<2>(least);
}
WgradPlan model_wgrad(int64_t N, int64_t K, int64_t M, bool sums) {
  struct Tile {
    int request, stack;
    double kblock, tile;
  };
  static const Tile tiles[] = {{128, 1, 0.224, 1.91}, {192, 1, 0.307, 2.43}, {256, 1, 0.468, 2.42}, {128, 2, 0.523, 3.59}, {192, 2, 0.608, 4.73},
                               {256, 2, 0.682, 13.4}, {1256, 1, 0.342, 3.52}, {1384, 1, 0.512, 4.93}};
  const int64_t k_blocks = (M + 63) / 64, sms = sm_count();
  const int64_t blocks_256 = ((N + 127) / 128) * ((K + 255) / 256);
  const int64_t least_split = std::max<int64_t>(1, std::min((k_blocks + 31) / 32, sms / blocks_256));
  const double separate = sums ? 8.5 + 2e-6 * M * N / 4.71 : 0.0;
  const bool ones_row = tb::gemm_row_sums_fit(K, 2);      // (of a transposed plan: the sums are rows of ones behind x's columns)
  const bool pairs = tb::gemm_pairs() && sms >= 2;
  struct Choice {
    WgradPlan plan;
    int64_t length;
    double time;
  };
  std::vector<Choice> choices;
  for (const Tile& t : tiles) {
    const bool pair = t.request >= 1000;
    const int width = t.request % 1000;
    for (bool swapped : {false, true}) {
      if (swapped && !(t.request == 1384 && N > 256 && K > 2 * N)) continue;
      const int64_t rows = swapped ? K : N, cols = swapped ? N : K;
      if ((pair && (!pairs || rows <= 128 || width >= 2 * cols || (width == 384 && cols <= 256))) || (t.stack == 2 && rows <= 128) ||
          (width > 128 && !pair && cols <= width - 64))
        continue;
      const int64_t high = pair ? 2 : t.stack, units = pair ? sms / 2 : sms, n = (cols + width - 1) / width;
      const int64_t count = ((rows + 127) / 128 + high - 1) / high * n;
      const bool fused = sums && width != 256 && !swapped;
      const double sum_cost = fused ? (pair ? 0.128 : 0.158 * t.stack) / n : 0.0;
      for (int halves : {1, 2, 4, 6}) {
        const int64_t want = std::min(std::max(least_split, halves * units / 2 / count), k_blocks), per = (k_blocks + want - 1) / want;
        const int64_t split = (k_blocks + per - 1) / per, rounds = (count * split + units - 1) / units;
        const double full = std::min(1.0, static_cast<double>(count * split) / units);
        const double time = rounds * (per * (t.kblock * (0.77 + 0.23 * full) + sum_cost) + t.tile) + (pair ? 1.3 : 0.0) +
                            0.008 * 4e-6 * count * split * high * 128 * std::min<int64_t>(width, cols) + 3.4 +
                            (fused || (swapped && ones_row) ? 0.0 : separate);
        choices.push_back({{t.request, t.stack, static_cast<int>(split), swapped}, per, time});
      }
    }
  }
  double least = choices.front().time;
  for (const Choice& c : choices) least = std::min(least, c.time);
  const Choice* best = nullptr;
  for (const Choice& c : choices)
    if (c.time <= 1.03 * least && (best == nullptr || c.plan.split > best->plan.split || (c.plan.split == best->plan.split && c.time < best->time)))
      best = &c;
  const int64_t parts = std::max<int64_t>(1, sms / covering_tiles(N, K, sums)), longest = std::max<int64_t>(15, (k_blocks + parts - 1) / parts);
  if (best->length > longest) {      // the cheapest of those that keep to it, else the shortest parts
    for (const Choice& c : choices) {
      if (c.time > 1.15 * least) continue;
      const int64_t a = std::max(c.length, longest), b = std::max(best->length, longest);
      if (a < b || (a == b && c.time < best->time)) best = &c;
    }
  }
  return best->plan;
}
WgradPlan plan_wgrad(int64_t N, int64_t K, int64_t M, bool sums) {
  static thread_local tb::SizeMemo<WgradPlan, 4> known;
  return known.get({N, K, M, sums}, [&] { return model_wgrad(N, K, M, sums); });
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
  const bool ones_row = sums && plan.swapped && tb::gemm_row_sums_fit(K, 2) && tb::gemm_tma_epilogue() && grad_w.stride(0) % 4 == 0 &&
                        reinterpret_cast<uintptr_t>(grad_w.data_ptr()) % 16 == 0;
  if (sums && !ones_row && (plan.bn % 1000 == 256 || plan.swapped)) {
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
  g.colsum = sums && !ones_row ? grad_b->data_ptr<float>() : nullptr;
  g.row_sums = ones_row ? grad_b->data_ptr<float>() : nullptr;
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
