// Host-side construction of TMA tensor maps and GemmParams for the tcgen05 GEMM family.
// No allocation happens here: callers pass every buffer.
#include "gemm_sm100.cuh"
#include "host_api.h"
#include "size_memo.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace tb {

cudaError_t launch_gemm(const GemmParams& p, int bn, int ctas, int num_sms, cudaStream_t stream);
cudaError_t gemm_read_stalls(unsigned long long* out8, bool reset);
cudaError_t gemm_ones_rows(void** ptr);

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
  });
  return fn;
}

// rank <= 5, 128-byte swizzle, zero fill outside the tensor.
// dims/box are innermost first; strides (bytes) are for dims 1..rank-1.
static int make_tensor_map(CUtensorMap* out, CUtensorMapDataType type, const void* base, int rank, const unsigned long long* dims,
                           const unsigned long long* strides_bytes, const unsigned int* box) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return -1;
  // cuTensorMapEncodeTiled is a driver call: it needs the primary context bound to THIS thread. A thread that
  // has only queried the device so far (e.g. an autograd worker before its first runtime call) has none, so
  // bind it once per thread through the runtime.
  static thread_local bool context_bound = false;
  if (!context_bound) {
    cudaFree(nullptr);
    context_bound = true;
  }
  cuuint64_t gdim[5];
  cuuint64_t gstr[4];
  cuuint32_t bdim[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    estr[i] = 1;
  }
  for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides_bytes[i];
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return -2;
  for (int i = 0; i + 1 < rank; ++i)
    if (gstr[i] % 16 != 0) return -3;
  CUresult r = fn(out, type, static_cast<cuuint32_t>(rank), const_cast<void*>(base),
                  gdim, gstr, bdim, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -100 - static_cast<int>(r);
}

int make_tensor_map_bf16(CUtensorMap* out, const void* base, int rank, const unsigned long long* dims,
                         const unsigned long long* strides_bytes, const unsigned int* box) {
  return make_tensor_map(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, rank, dims, strides_bytes, box);
}

static int map_2d(CUtensorMap* out, const void* base, long long inner, long long outer, long long ld_elems,
                  int box_inner, int box_outer) {
  unsigned long long dims[2] = {static_cast<unsigned long long>(inner), static_cast<unsigned long long>(outer)};
  unsigned long long str[1] = {static_cast<unsigned long long>(ld_elems) * 2ull};
  unsigned int box[2] = {static_cast<unsigned int>(box_inner), static_cast<unsigned int>(box_outer)};
  return make_tensor_map_bf16(out, base, 2, dims, str, box);
}

// 32 x 64 unit of a row-major bf16 matrix in the 128-byte-swizzled layout (the epilogue's staging format)
static int map_chunk(CUtensorMap* out, const void* base, long long cols, long long rows, long long ld_elems) {
  unsigned long long dims[2] = {static_cast<unsigned long long>(cols), static_cast<unsigned long long>(rows)};
  unsigned long long str[1] = {static_cast<unsigned long long>(ld_elems) * 2ull};
  unsigned int box[2] = {64u, 32u};
  return make_tensor_map_bf16(out, base, 2, dims, str, box);
}

// TERRA_GEMM_TMA_EPILOGUE=0: outputs are stored and epilogue operands read by the lanes themselves.
bool gemm_tma_epilogue() {
  static const bool enabled = [] {
    const char* e = std::getenv("TERRA_GEMM_TMA_EPILOGUE");
    return e == nullptr || std::atoi(e) != 0;
  }();
  return enabled;
}

// Plain row-major bf16 outputs leave through TMA stores (and the residual / GELU-input operand arrives through TMA
// loads) when every matrix qualifies for a tensor map; otherwise the epilogue keeps its per-lane global accesses.
static void try_tma_epilogue(GemmParams& p, long long M, long long N) {
  p.epi_tma = 0;
  const int f = p.epi;
  if (!gemm_tma_epilogue() || (f & (EPI_OUT_F32 | EPI_ATOMIC | EPI_ROW_CONV))) return;
  if (((f & EPI_RESIDUAL) != 0) + ((f & EPI_MUL_DGELU) != 0) + ((f & EPI_SAVE_PRE) != 0) > 1) return;   // one second buffer
  if (p.a_peers > 1 || p.c_peers > 1 || p.groups != 1 || p.C == nullptr) return;
  if (map_chunk(&p.map_c, p.C, N, M, p.ldc) != 0) return;
  if ((f & EPI_SAVE_PRE) && map_chunk(&p.map_c2, p.C2, N, M, p.ldc2) != 0) return;
  if ((f & EPI_RESIDUAL) && map_chunk(&p.map_in, p.residual, N, M, p.ldr) != 0) return;
  if ((f & EPI_MUL_DGELU) && map_chunk(&p.map_in, p.aux, N, M, p.ldaux) != 0) return;
  p.epi_tma = 1;
}

// Accumulated fp32 outputs leave as TMA reductions of 32 x 32 units where they qualify: `groups` (taps) of `rows` x N, or the transpose of one.
static void try_tma_reduce(GemmParams& p, long long rows, long long N, long long groups, long long group_stride) {
  if (!gemm_tma_epilogue() || (p.epi & ~EPI_TRANSPOSE) != (EPI_OUT_F32 | EPI_ATOMIC) || p.a_peers > 1 || p.c_peers > 1 || p.C == nullptr) return;
  const bool turned = (p.epi & EPI_TRANSPOSE) != 0;
  unsigned long long dims[3] = {static_cast<unsigned long long>(turned ? rows : N), static_cast<unsigned long long>(turned ? N : rows),
                                static_cast<unsigned long long>(groups)};
  if (p.ldc < 0 || static_cast<unsigned long long>(p.ldc) < dims[0]) return;
  unsigned long long str[2] = {static_cast<unsigned long long>(p.ldc) * 4ull, static_cast<unsigned long long>(groups > 1 ? group_stride : p.ldc) * 4ull};
  unsigned int box[3] = {32u, 32u, 1u};
  if (make_tensor_map(&p.map_c, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.C, 3, dims, str, box) == 0) p.epi_tma = 3;
}

static int pick_bn(long long N, int requested) {
  if (requested == 64 || requested == 128 || requested == 192 || requested == 256) return requested;
  if (N <= 64) return 64;
  if (N % 256 == 0 && N >= 1024) return 256;
  if (N % 192 == 0) return 192;   // 384, 768, 1152: no partial tile, less operand traffic per flop than 128
  return 128;
}

// CTA pairs (256-row tiles, one MMA over two SMs). What bounds the main loop is the shared-memory port (128 B per clock
// and SM): a k-block of a 128 x BN tile costs (16 + BN / 8) KB of operand fill and as much again for the tensor core's
// reads. In a pair each CTA stages 128 rows of A and only half of B's BN rows, (16 + BN / 16) KB. A pair starts later (two
// cluster barriers) and its larger tiles leave more of the last round empty.
bool gemm_pairs() {
  static const bool on = [] {
    const char* e = std::getenv("TERRA_GEMM_2CTA");
    return e == nullptr || std::atoi(e) != 0;
  }();
  return on;
}

// Tile of a plain product or gathered convolution (no peers, no split, no column sums): the width and CTA count with the least time by a
// model, in us. Persistent CTAs (pairs) take rounds of tiles; a tile takes the longer of its main loop and its epilogue (rounds of
// 64-column units over the three warps of a lane quadrant, or of 32-column chunks where the lanes store themselves or fp32 sums are
// accumulated) and a fixed hand-over, and the shorter of the two shows once, before the first or after the last tile. Tiles of 384 columns
// (pairs) have one accumulator: main loop and most of the epilogue follow one another, for 40 KB of operands per k-block where two tiles of
// 192 read 56 (128 wide, the only even width of a pair with an MN-major B and N = 384: 72).
//
// The constants were fitted to measurements, passes in a CUDA graph at 1.9 GHz, falling to about 1.4 GHz under the
// power cap in the largest. Products: 512 to 139264 rows, 25 pairs of N and K between 96 and 3072, five epilogues, all seven
// tiles (3100 times). Convolutions: the five forms, 96 to 384 channels, 16 x 32 to 512 x 1088 pixels (1300 times). The choice was
// 0.5 % (0.4 %) slower than the best tile on average, more than 10 % in one case of 200. Since then epilogues with an input or GELU ask for the
// next unit's operands ahead and take up to a quarter less, which their terms do not know: 34816 x 384 x 384 with residual takes 20.1 us
// where pairs of 192 columns take 17.1, 34816 x 1536 x 384 with GELU 49.0 / 46.1. Before the fit and the 384-wide tiles (us, before /
// this, on one GPU): input gradients 139264 x 384 x 1152 118 / 104, 139264 x 384 x 1536 153 / 132, 557056 x 384 x 2976 1113 / 1054;
// patch embedding 557056 x 384 x 2976 1041 / 931, recovery 557056 x 2976 x 384 1662 / 1576.
struct TileCosts {
  double start[2], tile, tail, plain_unit, bias_unit, drain;   // start: single CTAs, pairs
  double kblock[2][4];                                         // main loop per 64-wide k-block, widths 128, 192, 256, 384
};
static void model_tile(long long m_blocks, long long N, int k_blocks, bool b_mn, int flags, bool gathered, int num_sms, int* bn_out,
                       int* ctas_out) {
  *bn_out = pick_bn(N, 0);
  *ctas_out = 1;
  if (N <= 64 || m_blocks < 1) return;
  static const TileCosts rows = {{4.04, 5.57}, 0.575, 0.93, 0.378, 0.806, 0.894, {{0.221, 0.320, 0.439}, {0.200, 0.274, 0.340, 0.535}}};
  static const TileCosts image = {{4.24, 6.3}, 0.754, 0.404, 0.925, 0.925, 0.830, {{0.267, 0.306, 0.372}, {0.255, 0.278, 0.320, 0.490}}};
  const TileCosts& cost = gathered ? image : rows;
  const bool input = (flags & (EPI_RESIDUAL | EPI_MUL_DGELU)) != 0;
  const double unit = (flags & EPI_MUL_DGELU) ? 2.14 : (flags & EPI_RESIDUAL) ? 1.77 : (flags & (EPI_GELU | EPI_SAVE_PRE)) ? 2.19
                      : (flags & EPI_BIAS) ? cost.bias_unit : cost.plain_unit;
  const bool chunks = !gemm_tma_epilogue() || (flags & (EPI_OUT_F32 | EPI_ATOMIC));
  double least = 0.0;
  for (int ctas : {1, 2}) {
    if (ctas == 2 && (!gemm_pairs() || num_sms < 2)) continue;
    for (int w = 0; w < 2 + ctas; ++w) {
      const int bn = w == 3 ? 384 : 128 + 64 * w;
      if (bn >= 2 * N || (bn == 384 && N <= 256)) continue;
      if (ctas == 2 && b_mn && bn == 192) continue;      // half of an MN-major B must be whole 64-row boxes
      const long long tiles = (m_blocks + ctas - 1) / ctas * ((N + bn - 1) / bn), units = num_sms / ctas;
      const long long cols = std::min<long long>(bn, N), rounds = (tiles + units - 1) / units;
      // (single tiles of 256 columns leave no room for the pre-activation's staging buffer beside the operand ring)
      const bool by_chunk = chunks || ((flags & EPI_SAVE_PRE) && !input && bn == 256 && ctas == 1);
      const double loop = k_blocks * cost.kblock[ctas - 1][w];
      const double epilogue = unit * (by_chunk ? ((cols + 31) / 32 + 2) / 3 : ((cols + 63) / 64 + 2) / 3);
      double time = cost.start[ctas - 1];
      if (bn == 384) time += rounds * (std::max(loop + epilogue * cost.drain, epilogue) + cost.tile) + (1.0 - cost.drain) * epilogue;
      else time += rounds * (std::max(loop, epilogue) + cost.tile) + cost.tail * std::min(loop, epilogue);
      if (ctas == 2) time *= 0.99;      // (a tie goes to the pair, which loads less)
      if (least == 0.0 || time < least) {
        least = time;
        *bn_out = bn;
        *ctas_out = ctas;
      }
    }
  }
}

static void pick_tile(long long m_blocks, long long N, int k_blocks, bool b_mn, int flags, bool gathered, int num_sms, int* bn_out,
                      int* ctas_out) {
  struct Choice {
    int bn, ctas;
  };
  static thread_local SizeMemo<Choice, 7> known;
  const Choice& c = known.get({m_blocks, N, k_blocks, b_mn, flags, gathered, num_sms}, [&] {
    Choice made;
    model_tile(m_blocks, N, k_blocks, b_mn, flags, gathered, num_sms, &made.bn, &made.ctas);
    return made;
  });
  *bn_out = c.bn;
  *ctas_out = c.ctas;
}

void gemm_tile(long long M, long long N, long long K, bool b_mn, int flags, bool gathered, int num_sms, int* bn, int* ctas) {
  pick_tile((M + GEMM_BM - 1) / GEMM_BM, N, static_cast<int>((K + GEMM_BK - 1) / GEMM_BK), b_mn, flags, gathered, num_sms, bn, ctas);
}

bool gemm_row_sums_fit(long long rows, int blocks) { return (rows + 63) / 64 % (2 * blocks) != 0; }

static void fill_epilogue(GemmParams& p, const GemmEpilogue& e) {
  p.epi = e.flags;
  p.C = e.C;
  p.C2 = e.C2;
  p.bias = e.bias;
  p.residual = static_cast<const __nv_bfloat16*>(e.residual);
  p.aux = static_cast<const __nv_bfloat16*>(e.aux);
  p.ldc = e.ldc;
  p.ldc2 = e.ldc2;
  p.ldr = e.ldr;
  p.ldaux = e.ldaux;
  p.alpha = e.alpha;
  p.status = static_cast<KernelStatus*>(e.status);
  p.colsum = e.colsum;
}

int gemm_bf16(const GemmOperand& A, const GemmOperand& B, long long M, long long N, long long K,
              const GemmEpilogue& epi, int split_k, int bn_request, int num_sms, cudaStream_t stream) {
  GemmPeers none;
  std::memset(&none, 0, sizeof(none));
  return gemm_bf16_peers(A, B, M, N, K, epi, none, split_k, bn_request, num_sms, stream);
}

int gemm_bf16_peers(const GemmOperand& A, const GemmOperand& B, long long M, long long N, long long K,
                    const GemmEpilogue& epi, const GemmPeers& peers, int split_k, int bn_request, int num_sms,
                    cudaStream_t stream) {
  GemmParams p;
  std::memset(&p, 0, sizeof(p));
  const bool gather_a = peers.a_peers > 1;
  const bool scatter_c = peers.c_peers > 1;
  if (gather_a && (A.mn_major || peers.a_peers > 8 || peers.a_rows <= 0 || M != peers.a_rows * peers.a_peers)) return -12;
  if (scatter_c && (peers.c_peers > 8 || peers.c_rows <= 0 || M != peers.c_rows * peers.c_peers)) return -13;
  // scattered output is either the fp32 atomic form or the plain bf16 form (one staging slot per source GPU)
  if (scatter_c && (epi.flags & EPI_OUT_F32) && !(epi.flags & EPI_ATOMIC)) return -13;
  if ((gather_a || scatter_c) && bn_request >= 1000) return -14;   // single-CTA tiles only
  // CTA pairs: explicit request 1000 + BN, or the rule of pick_tile where no tile width is asked for.
  int ctas = 1;
  if (bn_request >= 1000) {
    ctas = 2;
    bn_request -= 1000;
    if (bn_request != 128 && bn_request != 256 && !(bn_request == 192 && !B.mn_major) && bn_request != 384) return -11;
  } else if (bn_request == 0 && !A.mn_major && !gather_a && !scatter_c && split_k <= 1 && epi.colsum == nullptr) {
    gemm_tile(M, N, K, B.mn_major != 0, epi.flags, false, num_sms, &bn_request, &ctas);
  }
  if (epi.colsum != nullptr) {
    // column sums ride on the weight-gradient form only, and need room for their accumulators behind the tile's
    if (!A.mn_major || (epi.flags & EPI_BIAS) || !(epi.flags & EPI_ATOMIC) || (ctas != 1 && bn_request != 384) || gather_a || scatter_c) return -15;
    if (bn_request == 256 || (bn_request == 0 && pick_bn(N, 0) == 256)) bn_request = (N % 192 == 0) ? 192 : 128;
  }
  const int bn = ctas == 2 && bn_request == 384 ? 384 : pick_bn(N, bn_request);      // (single CTAs have no such tile: as any other width)
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(K);
  p.m_blocks = static_cast<int>((M + GEMM_BM - 1) / GEMM_BM);
  p.num_m_tiles = (p.m_blocks + ctas - 1) / ctas;
  if (epi.stack == 2) {
    if (!A.mn_major || ctas != 1 || gather_a || scatter_c || !(epi.flags & EPI_ATOMIC) || bn < 128 ||
        (bn == 256 && epi.colsum != nullptr))
      return -17;
    p.stack = 2;
    p.num_m_tiles = (p.m_blocks + 1) / 2;
  }
  if (gather_a || scatter_c) ctas = 1;
  if (gather_a) {
    p.a_peers = peers.a_peers;
    p.a_rows = static_cast<int>(peers.a_rows);
    p.a_tiles = static_cast<int>((peers.a_rows + GEMM_BM - 1) / GEMM_BM);
    p.a_first = peers.rank % peers.a_peers;
    p.a_flags = static_cast<const unsigned int*>(peers.a_flags);
    p.a_epoch = peers.a_epoch;
    p.a_budget_ns = peers.a_budget_ns > 0 ? peers.a_budget_ns : 2000000000ull;
    p.a_interleave = peers.a_interleave;
    p.a_chunks = peers.a_chunks < 1 ? 1 : (peers.a_chunks > 4 ? 4 : peers.a_chunks);
    p.a_chunk_tiles = (p.a_tiles + p.a_chunks - 1) / p.a_chunks;
    p.num_m_tiles = p.a_tiles * p.a_peers;
    for (int i = 0; i < peers.a_peers; ++i) {
      const int rc_i = map_2d(&p.map_a_peer[i], peers.a_ptr[i], K, peers.a_rows, A.ld, GEMM_BK, GEMM_BM);
      if (rc_i != 0) return rc_i - 3000;
    }
  }
  if (scatter_c) {
    p.c_peers = peers.c_peers;
    p.c_rows = static_cast<int>(peers.c_rows);
    p.c_slot = peers.rank % peers.c_peers;
    for (int i = 0; i < peers.c_peers; ++i) p.c_peer[i] = peers.c_ptr[i];
  }
  p.num_n_tiles = static_cast<int>((N + bn - 1) / bn);
  p.k_blocks = static_cast<int>((K + GEMM_BK - 1) / GEMM_BK);
  p.groups = 1;
  if (split_k < 1) split_k = 1;
  if (split_k > p.k_blocks) split_k = p.k_blocks;
  {
    const int per = (p.k_blocks + split_k - 1) / split_k;
    split_k = (p.k_blocks + per - 1) / per;   // no empty split
  }
  p.split_k = split_k;
  if (split_k > 1 && !((epi.flags & EPI_ATOMIC) && (epi.flags & EPI_OUT_F32))) return -10;
  if ((epi.flags & EPI_TRANSPOSE) && (!(epi.flags & EPI_ATOMIC) || !(epi.flags & EPI_OUT_F32) || !A.mn_major || scatter_c)) return -18;
  p.a_mode = A.mn_major ? OP_MNMAJOR_2D : OP_KMAJOR_2D;
  p.b_mode = B.mn_major ? OP_MNMAJOR_2D : OP_KMAJOR_2D;
  int rc;
  if (A.mn_major) rc = map_2d(&p.map_a, A.ptr, M, K, A.ld, 64, GEMM_BK);
  else rc = map_2d(&p.map_a, gather_a ? peers.a_ptr[p.a_first] : A.ptr, K, gather_a ? peers.a_rows : M, A.ld, GEMM_BK, GEMM_BM);
  if (rc != 0) return rc;
  if (B.mn_major) rc = map_2d(&p.map_b, B.ptr, N, K, B.ld, 64, GEMM_BK);
  else rc = map_2d(&p.map_b, B.ptr, K, N, B.ld, GEMM_BK, bn == 384 ? 64 : bn / ctas);   // a CTA of a pair stages half of B's rows
  if (rc != 0) return rc - 1000;
  fill_epilogue(p, epi);
  p.tile_n0 = 1;
  p.tile_n1 = 1;
  try_tma_epilogue(p, M, N);
  try_tma_reduce(p, M, N, 1, 0);
  if (epi.row_sums != nullptr) {
    if (!gemm_row_sums_fit(M, ctas * (p.stack == 2 ? 2 : 1)) || p.epi_tma != 3 || !A.mn_major) return -21;
    void* ones = nullptr;
    if (gemm_ones_rows(&ones) != cudaSuccess) return -20;
    rc = map_2d(&p.map_in, ones, 128, 256, 128, 64, 64);
    if (rc != 0) return rc - 2000;
    p.row_sums = epi.row_sums;
    p.ones_row = static_cast<int>((M + 63) / 64 * 64);
  }
  cudaError_t e = launch_gemm(p, bn, ctas, num_sms, stream);
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// 3x3 convolution, padding 1, stride 1 or 2, NHWC bf16, as implicit GEMM.
//   x: [B, H, W, Cin]   w: [Cout, 9 * Cin_pad] (tap-major, Cin padded to a multiple of 64 with zeros)
//   y: [B, Ho, Wo, Cout]
static int image_map(CUtensorMap* out, const void* base, int Cin, int par, int W, int rows, int B, int box_w, int box_h = 1) {
  unsigned long long dims[5] = {static_cast<unsigned long long>(Cin), static_cast<unsigned long long>(par),
                                static_cast<unsigned long long>(W / par), static_cast<unsigned long long>(rows),
                                static_cast<unsigned long long>(B)};
  unsigned long long str[4] = {static_cast<unsigned long long>(Cin) * 2ull,
                               static_cast<unsigned long long>(Cin) * 2ull * par,
                               static_cast<unsigned long long>(Cin) * 2ull * W,
                               static_cast<unsigned long long>(Cin) * 2ull * W * rows};
  unsigned int box[5] = {64, 1, static_cast<unsigned int>(box_w), static_cast<unsigned int>(box_h), 1};
  return make_tensor_map_bf16(out, base, 5, dims, str, box);
}

static int attach_halos(GemmParams& p, const void* halo_lo, const void* halo_hi, int Cin, int par, int W, int H, int B,
                        int box_w) {
  p.img_h = H;
  p.halo_flags = 0;
  if (halo_lo != nullptr) {
    const int rc = image_map(&p.map_halo_lo, halo_lo, Cin, par, W, 1, B, box_w);
    if (rc != 0) return rc - 3000;
    p.halo_flags |= 1;
  }
  if (halo_hi != nullptr) {
    const int rc = image_map(&p.map_halo_hi, halo_hi, Cin, par, W, 1, B, box_w);
    if (rc != 0) return rc - 4000;
    p.halo_flags |= 2;
  }
  return 0;
}

//
// The general form, shared by the transposed convolutions and the strided input gradients: output pixel (i, j) of the tile
// grid [tiles_h, tiles_w] sums, over the taps of its phase, input pixel (i * hmul + dh, columns split by parity `par`:
// j + dw of parity `parity`) times the tap's [N, Cin] weights; it is stored at (i * out_mul + oy, parity ox of column j).
// Measured (us, before -> now): transposed convolution 139264 x 384 -> 557056 x 384, forward 423 (per-lane pixel-shuffle
// stores) -> 259, input gradient with the un-shuffling copy 147 + 562 -> 182, weight gradient 145 -> 192; input gradient of
// the stride-2 convolution at 557056 pixels 397 (GEMM to per-tap columns) + 334 (gather) -> 394.
struct Tap {
  short parity, dw, dh;
};
struct GatherConv {
  const void* x;
  int B, H, W, Cin, par;            // input image
  int tiles_h, tiles_w, hmul;
  const Tap* taps;
  int ntaps;
  int groups;                       // phases with taps of their own (grp_taps[0 .. groups] = their ranges), or 1
  int grp_taps[5];
  const void* w;                    // [N, ntaps * Cin_pad], Cin padded to a multiple of 64 with zeros
  int N;
  void* y;
  int out_h, out_w, out_c, out_mul; // output image; out_w = columns of one parity
  int phase_cols;                   // > 0: phases side by side in N
  short out_off[4][2];
  // other layouts of the input and of the output (and the residual, which lies like the output): dimensions {channels, parity or row of a
  // patch, columns, rows, samples} with their strides in elements
  const struct ImageLayout* in_layout;
  const struct ImageLayout* out_layout;
};
struct ImageLayout {
  unsigned long long dims[5], strides[4];
};
static int layout_map(CUtensorMap* out, const void* base, const ImageLayout& l, int box_w, int box_h) {
  unsigned long long str[4];
  for (int i = 0; i < 4; ++i) str[i] = 2 * l.strides[i];
  unsigned int box[5] = {64, 1, static_cast<unsigned int>(box_w), static_cast<unsigned int>(box_h), 1};
  return make_tensor_map_bf16(out, base, 5, l.dims, str, box);
}

static int gather_conv(const GatherConv& c, const GemmEpilogue& epi, int num_sms, cudaStream_t stream, const void* halo_lo,
                       const void* halo_hi) {
  if (c.Cin % 8 != 0 || c.out_c % 8 != 0 || c.W % c.par != 0) return -13;
  const int cchunks = (c.Cin + 63) / 64;
  if (c.ntaps * cchunks > GEMM_MAX_KTABLE) return -14;
  GemmParams p;
  std::memset(&p, 0, sizeof(p));
  // (outputs that go to every second pixel, or into another layout, have no per-lane form)
  const bool strided = c.out_mul != 1 || c.phase_cols != 0;
  const bool tma_out = c.out_layout != nullptr || (!(epi.flags & ~(EPI_BIAS | EPI_BIAS_F32)) && (strided || gemm_tma_epilogue()));
  // Pixels of a tile: 128 of a row, or 64 of two rows or 32 of four where fewer tiles cover the image so (96 x 180: 144 instead of 192) and
  // rounds of CTAs can be saved by it. Not where rows come from a neighbour or every second row is read. Us, 128 x 1 / this: 3x3
  // convolutions of 96 x 180 pixels, 192 channels 21.8 / 14.5, of 2 x 76 x 131, 128 20.1 / 15.7, of 180 x 129, 192 30.6 / 23.2, of 200 x
  // 400, 192 54.8 / 46.9; in one round anyway 50 x 100 pixels of 384 to every second 12.9 / 14.1.
  int tile_w = GEMM_BM;
  long long m_blocks = 0;
  for (int w = GEMM_BM; w >= 32; w /= 2) {
    if (w < GEMM_BM && (!tma_out || c.hmul != 1 || halo_lo != nullptr || halo_hi != nullptr)) break;
    const int high = GEMM_BM / w;
    const long long count = static_cast<long long>((c.tiles_w + w - 1) / w) * ((c.tiles_h + high - 1) / high) * c.B;
    if (m_blocks == 0 || (count < m_blocks && m_blocks > num_sms)) {
      m_blocks = count;
      tile_w = w;
    }
  }
  const int tile_h = GEMM_BM / tile_w;
  int bn = 0, ctas = 1;
  pick_tile(m_blocks * c.groups, c.N, c.ntaps * cchunks / c.groups, false, epi.flags, true, num_sms, &bn, &ctas);
  p.M = c.B * c.tiles_h * c.tiles_w;
  p.N = c.N;
  p.K = c.ntaps * cchunks * 64;
  p.tile_shift = tile_w == 128 ? 7 : (tile_w == 64 ? 6 : 5);
  p.tile_n0 = (c.tiles_w + tile_w - 1) / tile_w;
  p.tile_n1 = (c.tiles_h + tile_h - 1) / tile_h;
  p.m_blocks = static_cast<int>(m_blocks);
  p.num_m_tiles = (p.m_blocks + ctas - 1) / ctas;
  p.num_n_tiles = (c.N + bn - 1) / bn;
  p.k_blocks = c.ntaps * cchunks;
  p.split_k = 1;
  p.groups = c.groups;
  if (c.groups > 1) {
    p.grp_ranges = 1;
    for (int g = 0; g <= c.groups; ++g) p.grp_kb[g] = c.grp_taps[g] * cchunks;
  }
  p.a_mode = OP_TABLE_5D;
  p.b_mode = OP_KMAJOR_2D;
  int rc = c.in_layout != nullptr ? layout_map(&p.map_a, c.x, *c.in_layout, tile_w, tile_h)
                                  : image_map(&p.map_a, c.x, c.Cin, c.par, c.W, c.H, c.B, tile_w, tile_h);
  if (rc != 0) return rc;
  rc = map_2d(&p.map_b, c.w, p.K, c.N, p.K, GEMM_BK, bn == 384 ? 64 : bn / ctas);
  if (rc != 0) return rc - 1000;
  rc = attach_halos(p, halo_lo, halo_hi, c.Cin, c.par, c.W, c.H, c.B, GEMM_BM);
  if (rc != 0) return rc;
  // tile (t0, t1, t2) = (w chunk, row, b): base coordinates
  p.a_mul0[2] = tile_w;
  p.a_mul1[3] = c.hmul * tile_h;
  p.a_mul2[4] = 1;
  for (int t = 0; t < c.ntaps; ++t)
    for (int k = 0; k < cchunks; ++k) {
      short* e = p.ktable[t * cchunks + k];
      e[0] = static_cast<short>(k * 64);
      e[1] = c.taps[t].parity;
      e[2] = c.taps[t].dw;
      e[3] = c.taps[t].dh;
    }
  fill_epilogue(p, epi);
  p.C = c.y;
  p.epi |= EPI_ROW_CONV;
  p.out_w = c.out_w;
  p.out_h = c.out_h;
  p.out_mul = c.out_mul;
  p.phase_cols = c.phase_cols;
  std::memcpy(p.out_off, c.out_off, sizeof(p.out_off));
  p.ldc = c.out_c;
  if (c.out_layout != nullptr) {
    rc = layout_map(&p.map_c, c.y, *c.out_layout, 32, 1);
    if (rc == 0 && (p.epi & EPI_RESIDUAL)) rc = layout_map(&p.map_in, p.residual, *c.out_layout, 32, 1);
    if (rc != 0) return rc - 5000;
    p.epi_tma = 2;
  } else if (tma_out) {
    // 32 pixels x 64 channels per store; rows and channels outside the image are clipped
    const unsigned long long C = static_cast<unsigned long long>(c.out_c), mul = static_cast<unsigned long long>(c.out_mul);
    const unsigned long long row = C * 2ull * mul * c.out_w;
    unsigned long long dims[5] = {C, mul, static_cast<unsigned long long>(c.out_w), static_cast<unsigned long long>(c.out_h),
                                  static_cast<unsigned long long>(c.B)};
    unsigned long long str[4] = {C * 2ull, C * 2ull * mul, row, row * c.out_h};
    unsigned int box[5] = {64, 1, 32, 1, 1};
    rc = make_tensor_map_bf16(&p.map_c, c.y, 5, dims, str, box);
    if (rc != 0) return rc - 5000;
    p.epi_tma = 2;
  } else if (strided) {
    return -16;
  }
  const cudaError_t e = launch_gemm(p, bn, ctas, num_sms, stream);
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

static void conv3x3_taps(Tap (&taps)[9], int stride) {
  for (int tap = 0; tap < 9; ++tap) {
    const int dyy = tap / 3, dxx = tap % 3;
    // stride 2: w_in = 2 wo + dxx - 1, so dxx = 0 -> parity 1 of column wo - 1; 1 -> parity 0 of wo; 2 -> parity 1 of wo
    taps[tap].parity = static_cast<short>(stride == 1 || dxx == 1 ? 0 : 1);
    taps[tap].dw = static_cast<short>(stride == 1 ? dxx - 1 : (dxx == 0 ? -1 : 0));
    taps[tap].dh = static_cast<short>(dyy - 1);
  }
}

int conv3x3_fwd_bf16(const void* x, const void* w, int B, int H, int W, int Cin, int Cout, int stride,
                     const GemmEpilogue& epi, int num_sms, cudaStream_t stream, const void* halo_lo,
                     const void* halo_hi) {
  if (stride != 1 && stride != 2) return -11;
  if (stride == 2 && (W % 2 != 0)) return -12;
  Tap taps[9];
  conv3x3_taps(taps, stride);
  const int Ho = (stride == 1) ? H : (H + 1) / 2, Wo = (stride == 1) ? W : W / 2;
  GatherConv c = {x, B, H, W, Cin, stride, Ho, Wo, stride, taps, 9, 1, {0, 9}, w, Cout, epi.C, Ho, Wo, Cout, 1, 0, {}};
  return gather_conv(c, epi, num_sms, stream, halo_lo, halo_hi);
}

// Input gradient of the stride-2 convolution: dy [B, Ho, Wo, Cout] -> dx [B, H, W, Cin] (W even). A row of dx of even index
// takes part in one tap row (ky = 1), one of odd index in two (ky = 0 of the next dy row, ky = 2), columns alike: four
// phases of 1, 2, 2 and 4 taps. w: [Cin, 9 * Cout_pad], taps in the order of `order` below.
int conv3x3_s2_dgrad_bf16(const void* dy, const void* w, void* dx, int B, int H, int W, int Cin, int Cout, void* status,
                          int num_sms, cudaStream_t stream) {
  if (W % 2 != 0) return -12;
  // {ky, kx} per tap, the phase with most taps first: its tiles are the longest
  static const short order[9][2] = {{0, 0}, {0, 2}, {2, 0}, {2, 2}, {1, 0}, {1, 2}, {0, 1}, {2, 1}, {1, 1}};
  Tap taps[9];
  for (int t = 0; t < 9; ++t) taps[t] = {0, static_cast<short>(order[t][1] == 0 ? 1 : 0), static_cast<short>(order[t][0] == 0 ? 1 : 0)};
  const int Ho = (H + 1) / 2, Wo = W / 2;
  GatherConv c = {dy, B, Ho, Wo, Cout, 1, Ho, Wo, 1, taps, 9, 4, {0, 4, 6, 8, 9}, w, Cin, dx, H, Wo, Cin, 2, 0,
                  {{1, 1}, {0, 1}, {1, 0}, {0, 0}}};
  GemmEpilogue epi = {};
  epi.alpha = 1.0f;
  epi.status = status;
  return gather_conv(c, epi, num_sms, stream, nullptr, nullptr);
}

// 2x2 / stride-2 transposed convolution: x [B, H, W, Cin] -> y [B, 2H, 2W, Cout]; w: [4 * Cout_pad, Cin_pad], rows (dy, dx, co);
// bias: [4 * Cout_pad] (padded to multiples of 64; the padding columns are clipped by the store). One tap, the four output phases side by
// side in N.
int convt2x2_fwd_bf16(const void* x, const void* w, const void* bias4, void* y, int B, int H, int W, int Cin, int Cout,
                      void* status, int num_sms, cudaStream_t stream) {
  const int pad = (Cout + 63) / 64 * 64;      // a 64-column unit of the epilogue lies inside one phase
  const Tap tap = {0, 0, 0};
  GatherConv c = {x, B, H, W, Cin, 1, H, W, 1, &tap, 1, 1, {0, 1}, w, 4 * pad, y, 2 * H, W, Cout, 2, pad,
                  {{0, 0}, {0, 1}, {1, 0}, {1, 1}}};
  GemmEpilogue epi = {};
  epi.flags = EPI_BIAS;
  epi.bias = bias4;
  epi.alpha = 1.0f;
  epi.status = status;
  return gather_conv(c, epi, num_sms, stream, nullptr, nullptr);
}

// Its input gradient: a 2x2 convolution of stride 2 over dy [B, 2H, 2W, Cout]; w: [Cin, 4 * Cout_pad], taps (dy, dx).
int convt2x2_dgrad_bf16(const void* dy, const void* w, void* dx, int B, int H, int W, int Cin, int Cout, void* status,
                        int num_sms, cudaStream_t stream) {
  const Tap taps[4] = {{0, 0, 0}, {1, 0, 0}, {0, 0, 1}, {1, 0, 1}};
  GatherConv c = {dy, B, 2 * H, 2 * W, Cout, 2, H, W, 2, taps, 4, 1, {0, 4}, w, Cin, dx, H, W, Cin, 1, 0, {}};
  GemmEpilogue epi = {};
  epi.alpha = 1.0f;
  epi.status = status;
  return gather_conv(c, epi, num_sms, stream, nullptr, nullptr);
}

// Patches of an image [B, H, W, C] (top and left patches of zeros before it, rows x cols of them in all) times w: y [B, rows, cols, N]. A patch's
// features are p runs of p * C neighbouring elements, one per image row, so that the products read the image itself: k-block
// padding (48 bytes a run of 138 or 186 channels) instead of a copy of the field in patch order. w: [N, p * (p * C padded to 64)].
// Us, 64800 patches of 16 x 138 features to 192 channels: copy and product 104 + 69, this 66.
int embed_image_bf16(const void* x, const void* w, const void* bias, void* y, int B, int H, int W, int C, int p, int top, int left, int rows,
                     int cols, int N, void* status, int num_sms, cudaStream_t stream) {
  if (p < 1 || p > 4 || H % p != 0 || W % p != 0 || (p * C) % 8 != 0 || N % 8 != 0) return -13;
  Tap taps[4];
  for (int r = 0; r < p; ++r) taps[r] = {static_cast<short>(r), static_cast<short>(-left), static_cast<short>(-top)};
  const unsigned long long run = static_cast<unsigned long long>(p) * C, line = static_cast<unsigned long long>(W) * C;
  const ImageLayout in = {{run, static_cast<unsigned long long>(p), static_cast<unsigned long long>(W / p), static_cast<unsigned long long>(H / p),
                           static_cast<unsigned long long>(B)},
                          {line, run, line * p, line * H}};
  GatherConv c = {x, B, H / p, W / p, static_cast<int>(run), 1, rows, cols, 1, taps, p, 1, {0, p}, w, N, y, rows, cols, N, 1, 0, {}, &in, nullptr};
  GemmEpilogue epi = {};
  epi.flags = EPI_BIAS;
  epi.bias = bias;
  epi.alpha = 1.0f;
  epi.status = status;
  return gather_conv(c, epi, num_sms, stream, nullptr, nullptr);
}

// The way back: t [B, rows, cols, D] times w, the patches inside the image [B, H, W, C] (top and left of them outside) plus the image x: out. The
// p runs of a patch are phases side by side in N. w: [p * (p * C padded to 64), D padded to 64], bias alike.
// Us, 64800 patches of 192 channels: product and copy with the sum 72 + 166, this 136 (floor of the fields 88).
int recover_image_bf16(const void* t, const void* w, const void* bias, const void* x, void* out, int B, int H, int W, int C, int p, int top,
                       int left, int rows, int cols, int D, void* status, int num_sms, cudaStream_t stream) {
  if (p < 1 || p > 4 || H % p != 0 || W % p != 0 || (p * C) % 8 != 0 || D % 8 != 0) return -13;
  const Tap tap = {0, static_cast<short>(left), static_cast<short>(top)};
  const unsigned long long run = static_cast<unsigned long long>(p) * C, line = static_cast<unsigned long long>(W) * C;
  const int pad = (p * C + 63) / 64 * 64;
  const ImageLayout image = {{run, static_cast<unsigned long long>(p), static_cast<unsigned long long>(W / p), static_cast<unsigned long long>(H / p),
                              static_cast<unsigned long long>(B)},
                             {line, run, line * p, line * H}};
  GatherConv c = {t, B, rows, cols, D, 1, H / p, W / p, 1, &tap, 1, 1, {0, 1}, w, p * pad, out, H / p, W / p, p * C, 1, pad,
                  {{0, 0}, {0, 1}, {0, 2}, {0, 3}}, nullptr, &image};
  GemmEpilogue epi = {};
  epi.flags = EPI_BIAS | EPI_RESIDUAL;
  epi.bias = bias;
  epi.residual = x;
  epi.alpha = 1.0f;
  epi.status = status;
  return gather_conv(c, epi, num_sms, stream, nullptr, nullptr);
}

// Weight gradients: dw[tap][M][N] (fp32, atomically accumulated) = sum over the pixels of `a` [B, Ho, Wo, M] of a[pix]^T
// times `b` [B, H, W, N] at the pixel's tap (hmul = par = stride of the grid of `a` in `b`). With disp_a the pixels are those of
// `b` [B, Ho, Wo, N], and `a` [B, H, W, M] is taken at the tap: its column sums then ride on the product.
static int gather_wgrad(const void* a, const void* b, float* dw, int B, int Ho, int Wo, int M, int H, int W, int N, int stride,
                        const Tap* taps, int ntaps, int split_k, void* status, int num_sms, cudaStream_t stream,
                        const void* halo_lo, const void* halo_hi, float* colsum, int stack, bool disp_a = false) {
  GemmParams p;
  std::memset(&p, 0, sizeof(p));
  const int bn = pick_bn(N, N % 192 == 0 ? 192 : 128);   // 384 columns: two tiles of 192, a fifth less operand traffic per flop
  p.M = M;
  p.N = N;
  p.pix_n0 = (Wo + GEMM_BK - 1) / GEMM_BK;
  p.pix_n1 = Ho;
  p.pix_hmul = stride;
  p.k_blocks = p.pix_n0 * Ho * B;
  p.K = p.k_blocks * GEMM_BK;
  p.m_blocks = (M + GEMM_BM - 1) / GEMM_BM;
  p.stack = stack == 2 && bn >= 128 ? 2 : 1;
  p.num_m_tiles = (p.m_blocks + p.stack - 1) / p.stack;
  p.num_n_tiles = (N + bn - 1) / bn;
  p.groups = ntaps;
  if (split_k < 1) split_k = 1;
  if (split_k > p.k_blocks) split_k = p.k_blocks;
  {
    const int per = (p.k_blocks + split_k - 1) / split_k;
    split_k = (p.k_blocks + per - 1) / per;
  }
  p.split_k = split_k;
  p.a_mode = OP_PIXELS_5D;
  p.b_mode = OP_PIXELS_5D;
  p.disp_a = disp_a ? 1 : 0;
  int rc = disp_a ? image_map(&p.map_a, a, M, stride, W, H, B, GEMM_BK) : image_map(&p.map_a, a, M, 1, Wo, Ho, B, GEMM_BK);
  if (rc != 0) return rc;
  rc = disp_a ? image_map(&p.map_b, b, N, 1, Wo, Ho, B, GEMM_BK) : image_map(&p.map_b, b, N, stride, W, H, B, GEMM_BK);
  if (rc != 0) return rc - 1000;
  rc = attach_halos(p, halo_lo, halo_hi, N, stride, W, H, B, GEMM_BK);
  if (rc != 0) return rc;
  for (int t = 0; t < ntaps; ++t) {
    p.grp_off[t][0] = taps[t].parity;
    p.grp_off[t][1] = taps[t].dw;
    p.grp_off[t][2] = taps[t].dh;
  }
  p.grp_c_stride = static_cast<long long>(M) * N;
  p.epi = EPI_OUT_F32 | EPI_ATOMIC;
  p.colsum = colsum;
  p.C = dw;
  p.ldc = N;
  p.alpha = 1.0f;
  p.status = static_cast<KernelStatus*>(status);
  p.tile_n0 = 1;
  p.tile_n1 = 1;
  try_tma_reduce(p, M, N, ntaps, p.grp_c_stride);
  const cudaError_t e = launch_gemm(p, bn, 1, num_sms, stream);
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// 3x3 convolution: dw[tap][Cout][Cin] (pre-zeroed), bias_grad[Cout] += the sums of dy from the same kernel.
int conv3x3_wgrad_bf16(const void* x, const void* dy, float* dw, int B, int H, int W, int Cin, int Cout, int stride,
                       int split_k, void* status, int num_sms, cudaStream_t stream, const void* halo_lo,
                       const void* halo_hi, float* bias_grad, int stack) {
  if (stride != 1 && stride != 2) return -11;
  if (stride == 2 && (W % 2 != 0)) return -12;
  if (Cin % 8 != 0 || Cout % 8 != 0) return -13;
  Tap taps[9];
  conv3x3_taps(taps, stride);
  const int Ho = (stride == 1) ? H : (H + 1) / 2, Wo = (stride == 1) ? W : W / 2;
  return gather_wgrad(dy, x, dw, B, Ho, Wo, Cout, H, W, Cin, stride, taps, 9, split_k, status, num_sms, stream, halo_lo,
                      halo_hi, bias_grad, stack);
}

// 2x2 / stride-2 transposed convolution: dw[tap][Cout][Cin] (pre-zeroed) from x [B, H, W, Cin] and dy [B, 2H, 2W, Cout], and
// bias_grad[Cout] += the sums of dy from the same kernel: dy is operand A, displaced by the tap. (As operand B its sums were two launches
// of their own, 90 of 290 us for 139264 pixels of 384 channels.)
int convt2x2_wgrad_bf16(const void* x, const void* dy, float* dw, int B, int H, int W, int Cin, int Cout, int split_k,
                        void* status, int num_sms, cudaStream_t stream, int stack, float* bias_grad) {
  if (Cin % 8 != 0 || Cout % 8 != 0) return -13;
  const Tap taps[4] = {{0, 0, 0}, {1, 0, 0}, {0, 0, 1}, {1, 0, 1}};
  return gather_wgrad(dy, x, dw, B, H, W, Cout, 2 * H, 2 * W, Cin, 2, taps, 4, split_k, status, num_sms, stream, nullptr,
                      nullptr, bias_grad, stack, true);
}

// All taps' weight gradients as one product (one rank): the channels of the displaced image, box after box of 64 and tap after tap, are the
// rows, and the other image's channels the columns, so that tiles of 256 rows need no whole number of them in a tap (9 x 384 rows are 13.5
// of a pair's, 9 x 192 seven stacked ones where two per tap made nine). With the undisplaced image as operand B its column sums, the bias
// gradient of a convolution, are one more box of rows, whose rows of ones share them out (g_ones_rows).
//
// The plan is the one with the least time by a model, in us: rounds of tiles over the CTAs (pairs), each its k-blocks and a hand-over with
// the epilogue. Fitted to 900 passes in CUDA graphs: the two layers at 512 to 557056 pixels, 96 to 384 channels, all tiles, half a round to
// three and more; the choice is 0.1 % slower than the best plan on average, at most 3 %.
// Us, a product per tap (two row blocks stacked where that was ahead) / this: 557056 pixels of 384 channels 1251 / 951, of 192 383 / 275,
// 80000 of 256 104 / 85, 17280 of 192 25 / 21; transposed, 139264 of 384 186 / 161, of 192 69 / 57, of 96 45 / 35. (Of 96 and 128 channels
// the row of ones costs a tile in ten: 17280 pixels 12.6 / 13.5 and 16.4 / 17.2; folding the gradients takes 2 to 10 us less than it did.)
// `least_split`: the contraction is cut into so many parts at least (the error of the tensor core's fp32 sums grows with their length:
// 139264 pixels of 384 channels, 18 parts 8.6e-6, 12 parts 13.0e-6), unless they are down to 15 k-blocks (1.0e-6; down to 24, 1.6e-6, is no
// faster: 2656 pixels of 384 channels 15.9 / 15.1 us, 600 to every second 14.5 / 14.2).
static TapPlan model_tap_wgrad(int taps, int channels, int N, long long k_blocks, bool row_sums, bool column_sums, int least_split, int num_sms) {
  struct Tile {
    int width, ctas, stack;
    double kblock, tile;
  };
  static const Tile tiles[] = {{128, 1, 1, 0.269, 1.56}, {192, 1, 1, 0.321, 1.92}, {128, 1, 2, 0.495, 3.34}, {192, 1, 2, 0.502, 4.65},
                               {256, 2, 1, 0.334, 2.84}, {384, 2, 1, 0.461, 5.38}};
  least_split = static_cast<int>(std::min<long long>(least_split, (k_blocks + 14) / 15));
  const long long boxes = static_cast<long long>(taps) * ((channels + 63) / 64) + (row_sums ? 1 : 0);
  TapPlan best = {128, 1, 1, 1};
  double least = -1.0;
  for (const Tile& t : tiles) {
    if (t.ctas == 2 && (!gemm_pairs() || num_sms < 2 || t.width >= 2 * N || (t.width == 384 && N <= 256) || (t.width == 256 && column_sums))) continue;
    if (t.width == 192 && N <= 128) continue;
    const long long units = num_sms / t.ctas, n = (N + t.width - 1) / t.width;
    const long long blocks = (boxes + 1) / 2, count = (blocks + t.stack * t.ctas - 1) / (t.stack * t.ctas) * n;
    const long long least_halves = 2 * ((std::min<long long>(least_split, k_blocks) * count + units - 1) / units);      // whole rounds
    for (long long halves : {1LL, 2LL, 4LL, 6LL, least_halves}) {      // half a round of CTAs, one, two, three, as many as it takes
      const long long want = std::max<long long>({1, least_split, halves * units / 2 / count});
      const long long per = (k_blocks + std::min(want, k_blocks) - 1) / std::min(want, k_blocks);
      const long long split = (k_blocks + per - 1) / per;
      const double full = std::min(1.0, static_cast<double>(count * split) / units);      // (fewer CTAs share L2's bandwidth)
      const double kblock = (t.kblock * (0.57 + 0.43 * full)) + (column_sums ? 0.151 * t.stack / n : 0.0);
      const double time = static_cast<double>((count * split + units - 1) / units) * (per * kblock + t.tile) + (t.ctas == 2 ? 1.0 : 0.0);
      if (least < 0.0 || time < least) {
        least = time;
        best = {t.width, t.ctas, t.stack, static_cast<int>(split)};
      }
    }
  }
  return best;
}

TapPlan plan_tap_wgrad(int taps, int channels, int N, long long k_blocks, bool row_sums, bool column_sums, int least_split, int num_sms) {
  static thread_local SizeMemo<TapPlan, 8> known;
  return known.get({taps, channels, N, k_blocks, row_sums, column_sums, least_split, num_sms},
                   [&] { return model_tap_wgrad(taps, channels, N, k_blocks, row_sums, column_sums, least_split, num_sms); });
}

// dw[tap][channels][N] (fp32, accumulated) = sum over the pixels of b [B, Ho, Wo, N] of a [B, H, W, channels] at the pixel's tap, times b.
// row_sums [N] += the sums of b, colsum [channels] += those of a over all taps.
static int tap_wgrad(const void* a, const void* b, float* dw, int B, int Ho, int Wo, int channels, int H, int W, int N, int stride,
                     const Tap* taps, int ntaps, const TapPlan& plan, void* status, int num_sms, cudaStream_t stream, float* row_sums,
                     float* colsum) {
  GemmParams p;
  std::memset(&p, 0, sizeof(p));
  p.M = channels;
  p.N = N;
  p.pix_n0 = (Wo + GEMM_BK - 1) / GEMM_BK;
  p.pix_n1 = Ho;
  p.pix_hmul = stride;
  p.k_blocks = p.pix_n0 * Ho * B;
  p.K = p.k_blocks * GEMM_BK;
  p.taps = ntaps;
  p.tap_boxes = (channels + 63) / 64;
  p.tap_channels = channels;
  p.row_sums = row_sums;
  p.ones_row = ntaps * p.tap_boxes * 64;
  p.m_blocks = (ntaps * p.tap_boxes + (row_sums != nullptr ? 1 : 0) + 1) / 2;
  p.stack = plan.stack;
  p.num_m_tiles = (p.m_blocks + plan.stack * plan.ctas - 1) / (plan.stack * plan.ctas);
  p.num_n_tiles = (N + plan.bn - 1) / plan.bn;
  p.groups = 1;
  int split = std::max(1, std::min(plan.split, p.k_blocks));
  {
    const int per = (p.k_blocks + split - 1) / split;
    split = (p.k_blocks + per - 1) / per;      // no empty split
  }
  p.split_k = split;
  p.a_mode = OP_PIXELS_5D;
  p.b_mode = OP_PIXELS_5D;
  p.disp_a = 1;
  int rc = image_map(&p.map_a, a, channels, stride, W, H, B, GEMM_BK);
  if (rc != 0) return rc;
  rc = image_map(&p.map_b, b, N, 1, Wo, Ho, B, GEMM_BK);
  if (rc != 0) return rc - 1000;
  void* ones = nullptr;      // (boxes behind the last tap are read in any case)
  if (gemm_ones_rows(&ones) != cudaSuccess) return -20;
  rc = map_2d(&p.map_in, ones, 128, 256, 128, 64, 64);
  if (rc != 0) return rc - 2000;
  for (int t = 0; t < ntaps; ++t) {
    p.grp_off[t][0] = taps[t].parity;
    p.grp_off[t][1] = taps[t].dw;
    p.grp_off[t][2] = taps[t].dh;
  }
  p.epi = EPI_OUT_F32 | EPI_ATOMIC;
  p.colsum = colsum;
  p.C = dw;
  p.ldc = N;
  p.alpha = 1.0f;
  p.status = static_cast<KernelStatus*>(status);
  p.tile_n0 = 1;
  p.tile_n1 = 1;
  try_tma_reduce(p, channels, N, ntaps, static_cast<long long>(channels) * N);
  const cudaError_t e = launch_gemm(p, plan.bn, plan.ctas, num_sms, stream);
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// 3x3 convolution on one rank: dw[tap][Cin][Cout] += ..., and bias_grad[Cout] += the sums of dy.
int conv3x3_wgrad_taps_bf16(const void* x, const void* dy, float* dw, int B, int H, int W, int Cin, int Cout, int stride, const TapPlan& plan,
                            void* status, int num_sms, cudaStream_t stream, float* bias_grad) {
  if (stride != 1 && stride != 2) return -11;
  if (stride == 2 && (W % 2 != 0)) return -12;
  if (Cin % 8 != 0 || Cout % 8 != 0) return -13;
  Tap taps[9];
  conv3x3_taps(taps, stride);
  const int Ho = (stride == 1) ? H : (H + 1) / 2, Wo = (stride == 1) ? W : W / 2;
  return tap_wgrad(x, dy, dw, B, Ho, Wo, Cin, H, W, Cout, stride, taps, 9, plan, status, num_sms, stream, bias_grad, nullptr);
}

// 2x2 / stride-2 transposed convolution: dw[tap][Cout][Cin] += ..., bias_grad[Cout] += the sums of dy
int convt2x2_wgrad_taps_bf16(const void* x, const void* dy, float* dw, int B, int H, int W, int Cin, int Cout, const TapPlan& plan,
                             void* status, int num_sms, cudaStream_t stream, float* bias_grad) {
  if (Cin % 8 != 0 || Cout % 8 != 0) return -13;
  const Tap taps[4] = {{0, 0, 0}, {1, 0, 0}, {0, 0, 1}, {1, 0, 1}};
  return tap_wgrad(dy, x, dw, B, H, W, Cout, 2 * H, 2 * W, Cin, 2, taps, 4, plan, status, num_sms, stream, nullptr, bias_grad);
}

int gemm_stall_counters(unsigned long long* out8, int reset) {
  return gemm_read_stalls(out8, reset != 0) == cudaSuccess ? 0 : -1;
}

}  // namespace tb
