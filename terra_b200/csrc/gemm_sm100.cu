// Persistent, warp-specialised bf16 GEMM / implicit-GEMM for sm_100a.
//
//   D[M,N] (+)= A[M,K] * B[N,K]^T, fp32 accumulation in tensor memory.
//
// Roles inside a 480-thread CTA (one CTA per SM, tiles assigned round-robin):
//   warp 0, warp 14  one elected lane each issues the TMA loads of A and of B (per-CTA, no cluster fan-out) into a ring of
//            128-byte-swizzled shared-memory stages, signalling `full[s]` (of a pair: the leader's) by transaction bytes;
//   warp 1   owns the TMEM allocation; one elected lane issues tcgen05.mma (M=128, N=BN, K=16)
//            and commits to `empty[s]` (stage reusable) and `tfull[a]` (accumulator a complete);
//   warps 2-13 epilogue (three per 32-lane TMEM quadrant, interleaved over the columns): tcgen05.ld, fused bias / GELU /
//            residual / GELU-gradient; bf16 outputs leave as units of 32 rows (or pixels) x 64 columns through TMA stores,
//            accumulated fp32 outputs as TMA reductions of 32 x 32 units, what does not fit a tensor map as 32-column chunks through an
//            exchange buffer.
// Two accumulators (2*BN TMEM columns) let the epilogue of tile i overlap the main loop of tile i+1 (tiles 384 wide have one).
//
// Operand addressing is data driven (see gemm_sm100.cuh) so that the same kernel serves
//   * linear layers forward (K-major x K-major),
//   * their input gradients (B read MN-major: the weight is used untransposed),
//   * their weight gradients (both operands MN-major, contraction over tokens, split-K atomics),
//   * 3x3 convolutions (stride 1 and 2) as implicit GEMM: A rows gathered by 5-D TMA boxes with
//     zero fill outside the image, k-blocks enumerate (tap, channel chunk),
//   * 2x2 / stride-2 transposed convolutions, their input gradient, and the input gradient of the stride-2 3x3
//     convolution: the same gather with other tap tables, outputs stored to every second pixel through 5-D TMA boxes,
//   * convolution weight gradients (contraction over pixels; the rows of all taps one after the other, or a tile group per tap).
// Two further instantiations: CTA pairs (a cluster of two drives one cta_group::2 MMA over a 256-row tile, see GemmCfg)
// and the tensor-parallel forms (A gathered from the peers' buffers, output scattered to the owners' buffers, see
// gemm_sm100.cuh).
//
// Every wait is bounded; on expiry the CTA sets its abort flag, records the site in the
// KernelStatus word, drains, releases TMEM and returns.
#include <atomic>
#include <type_traits>
#include "chained_launch.cuh"
#include "gemm_sm100.cuh"
#include "shared_limit.h"

namespace tb {

// warp 0: TMA of A, warp 1: MMA, warps 2..13: epilogue (three per TMEM lane quadrant, interleaved over the columns), warp 14:
// TMA of B. 15 warps keep every scheduler at four warps or fewer, which allows 128 registers per thread: with 18 warps
// the cap is 96 and the epilogue spills, and its reloads miss the small L1 left beside 227 KB of shared memory.
constexpr int GEMM_EPI_WARPS = 12;
// The last warp issues the loads of B: one thread's chain of wait, expect and load instructions for both operands took about
// as long per k-block as the loads themselves, and the MMA thread waited for it two thirds of its time (K = 384).
constexpr int GEMM_B_WARP = 2 + GEMM_EPI_WARPS;
constexpr int GEMM_THREADS = 32 * (GEMM_B_WARP + 1);

// CTAS = 2: a cluster of two CTAs (two SMs of one TPC) computes a 256 x BN tile with one pair-wide MMA. Each CTA stages
// its own 128 rows of A and its own half of B, so a k-block costs each SM (16 + BN / 16) KB of shared-memory fill instead
// of (16 + BN / 8) KB: the operand traffic per flop through shared memory, which bounds the single-CTA main loop, drops
// by a third at BN = 256.
//
// STACK = 2 (weight gradients, one CTA): two 128-row blocks of A share a tile of B, 256 x BN outputs in both accumulators.
// The operand stream through L2 bounds those products (12 TB/s measured with 128 x 192 tiles: 40 KB per k-block); stacked, a
// k-block costs 56 KB for twice the outputs. There is no second accumulator set to overlap the epilogue with the next
// tile, which a contraction over thousands of k-blocks does not need.
//
// BN = 384 (pairs): one tile of A meets 384 columns of B, as two MMAs of 256 and 128 columns (their halves are whole 64-column boxes in
// either orientation of B).
template <int BN, int CTAS, int STACK = 1>
struct GemmCfg {
  static constexpr bool WIDE = BN == 384;
  static_assert(!WIDE || (CTAS == 2 && STACK == 1), "wide tiles: pairs");
  static constexpr int BLOCK_BYTES = GEMM_BM * GEMM_BK * 2;   // one 128-row block of A
  static constexpr int A_BYTES = STACK * BLOCK_BYTES;
  static constexpr int ACCS = STACK == 1 && !WIDE ? 2 : 1;          // accumulator sets
  static constexpr int B_ROWS = BN / CTAS;                 // rows of B staged by one CTA
  static constexpr int B_BYTES = B_ROWS * GEMM_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // After the operand ring: 1 KB of barriers, the per-warp bias slots (together 4 KB), then `bufs` buffers of
  // 2 KB per epilogue warp: one (the exchange buffer of the per-lane epilogue), or two (a 32 x 64 unit of the output on its
  // way to a TMA store), or four (another such unit: the saved pre-activation, or the operand the epilogue reads). The
  // ring takes what is left: the launcher passes the stage count to the kernel.
  static constexpr int BAR_BYTES = 1024;
  static constexpr int FIXED_BASE = 4096;
  static constexpr int EPI_BUF = 2048;
  static constexpr int MAX_SMEM = 232448;   // 227 KB, the per-block limit of sm_100
  static constexpr int MAX_STAGES = 8;
  static constexpr int fixed_bytes(int bufs) { return FIXED_BASE + GEMM_EPI_WARPS * bufs * EPI_BUF; }
  static constexpr int stages_for(int bufs) {
    return (MAX_SMEM - 1024 - fixed_bytes(bufs)) / STAGE_BYTES > MAX_STAGES ? MAX_STAGES
                                                                            : (MAX_SMEM - 1024 - fixed_bytes(bufs)) / STAGE_BYTES;
  }
  static constexpr int smem_bytes(int bufs) { return stages_for(bufs) * STAGE_BYTES + fixed_bytes(bufs) + 1024; }   // + alignment slack
  // two accumulators (of alternating tiles, or of a tile's two row blocks); the allocation must be a power of two
  // behind them two 32-column accumulators of the column sums (weight-gradient form with a bias gradient; single
  // CTAs up to 192 columns, and pairs of 384 behind their one accumulator)
  static constexpr int SUM_COL0 = WIDE ? BN : 2 * BN;
  static constexpr int TMEM_COLS = (SUM_COL0 + 64 <= 256) ? 256 : 512;
  static constexpr bool CAN_COLSUM = (CTAS == 1 || WIDE) && SUM_COL0 + 64 <= 512;
  static_assert((STACK == 2 ? stages_for(1) : stages_for(2)) >= 3 && smem_bytes(1) <= MAX_SMEM && smem_bytes(2) <= MAX_SMEM, "shared memory budget");
  static_assert(GEMM_EPI_WARPS * 64 * 4 + BAR_BYTES <= FIXED_BASE && GEMM_EPI_WARPS * 64 * 4 >= 4 * 512, "bias slots");
  // a CTA's half of an MN-major B must be whole 64-row boxes; K-major rows only need whole 8-row swizzle atoms
  static constexpr bool CAN_B_MN = B_ROWS % 64 == 0;
  static_assert(B_ROWS % 8 == 0 && B_BYTES % 1024 == 0, "B tile: whole swizzle atoms");
};

// Cycle counters of the three roles, summed over CTAs and launches since the last reset (read by gemm_read_stalls):
// [0] MMA thread busy span, [1] of it waiting for a free accumulator, [2] waiting for operand stages,
// [3] TMA thread span, [4] of it waiting for free stages, [5] first epilogue warp span, [6] of it waiting for tiles.
__device__ unsigned long long g_gemm_stalls[8];

// Operand rows whose product with B is B's column sums (GemmParams::row_sums): 4 x 64 rows of 128 bf16, of which rows 64 j to 64 j + 63
// have a one in column 56 + j. A box of 64 x 64 of them from column 56 - 8 i and row 64 j on is a box of A whose row 8 i + j is ones. The
// others are 2^-126, not zeros, which would turn an infinity of B into a NaN.
#define TB_8(...) __VA_ARGS__, __VA_ARGS__, __VA_ARGS__, __VA_ARGS__, __VA_ARGS__, __VA_ARGS__, __VA_ARGS__, __VA_ARGS__
#define TB_LOW 0x00800080u
#define TB_LOW_4 TB_LOW, TB_LOW, TB_LOW, TB_LOW
#define TB_ROW(a, b) TB_8(TB_LOW), TB_8(TB_LOW), TB_8(TB_LOW), TB_LOW_4, a, b, TB_LOW, TB_LOW, TB_8(TB_LOW_4)
#define TB_64_ROWS(a, b) TB_8(TB_8(TB_ROW(a, b)))
__device__ __align__(1024) uint32_t g_ones_rows[4 * 64 * 64] = {TB_64_ROWS(0x00803F80u, TB_LOW), TB_64_ROWS(0x3F800080u, TB_LOW),
                                                                TB_64_ROWS(TB_LOW, 0x00803F80u), TB_64_ROWS(TB_LOW, 0x3F800080u)};
#undef TB_8
#undef TB_LOW
#undef TB_LOW_4
#undef TB_ROW
#undef TB_64_ROWS

// A k-block's box of g_ones_rows: each of 32 rows of A takes every 32nd k-block, since the tensor core's fp32 sums lose with their length.
// Error of the bias gradient of 557056 pixels (parts of 871 k-blocks), a row for all k-blocks 2.6e-6, 32 rows 1.1e-7; of 139264 (231)
// 4.2e-7 and 1.0e-7; of a patch embedding of 557056 patches (484) 1.1e-6 and 1.3e-7. The time is the same.
__device__ __forceinline__ int ones_col(int kb) { return 56 - (kb & 7) * 8; }
__device__ __forceinline__ int ones_line(int kb) { return (kb >> 3 & 3) * 64; }

struct TileCoord {
  int grp, m_blk, n_blk, split;
  int kb_begin, kb_end;
};

// Column sums of A (weight-gradient form): every tile of a row block streams the same A tiles, so the sums are shared out by k-block, kb %
// ways == the tile's place among its row block's `ways` tiles (with a displaced A those of its group). (A 16-column MMA costs as much of
// the tensor pipe and of the shared-memory port as 40 KB of operand stream: left to the first column tile it made that tile half as slow
// again, and the launch waits for the slowest.) Returns this tile's first such k-block.
__device__ __forceinline__ int first_sum_kb(const GemmParams& p, const TileCoord& t, int ways) {
  const int place = p.disp_a ? t.n_blk : t.grp * p.num_n_tiles + t.n_blk;
  return t.kb_begin + (place + ways - t.kb_begin % ways) % ways;
}

// Walks over the tiles of a CTA (pair): tile t is a mixed-radix number, and a step adds the digits of the tile step. (Decoded by
// divisions a tile cost every role about 600 cycles, once per tile for the loads and the MMAs and three times for the epilogue: as long as
// two k-blocks.) The digits are, from the fastest, (n, m, group, split): the tiles of one part of the contraction run side by side and share
// its operands in L2, where a launch has more of them than CTAs.
// p.num_m_tiles counts tiles of ctas * 128 rows; m_blk is in units of 128 rows for CTA `rank` of the pair.
// Stacked tiles (p.stack = 2 blocks of rows) go by (split, n, group, m): the row tile varies slowest, so that the last one, which may hold a
// single block, is handed out last.
template <int CTAS, int STACK>
struct TileWalk {
  int tile, split, n, lo, hi;          // (lo, hi) = (m, group), stacked tiles (group, m)
  int step, d_split, d_n, d_lo, d_hi;
  __device__ __forceinline__ TileWalk(const GemmParams& p, int first, int by) : tile(first), step(by) {
    digits(p, first, split, n, lo, hi);
    digits(p, by, d_split, d_n, d_lo, d_hi);
  }
  static __device__ __forceinline__ void digits(const GemmParams& p, int t, int& split, int& n, int& lo, int& hi) {
    split = 0;
    if (STACK > 1 && p.split_k > 1) {
      split = t % p.split_k;
      t /= p.split_k;
    }
    n = t % p.num_n_tiles;
    t /= p.num_n_tiles;
    const int radix = STACK > 1 ? p.groups : p.num_m_tiles;
    lo = t % radix;
    hi = t / radix;
    if (STACK == 1 && p.split_k > 1) {
      split = hi / p.groups;
      hi -= split * p.groups;
    }
  }
  __device__ __forceinline__ void next(const GemmParams& p) {
    tile += step;
    int carry = 0;
    if (STACK > 1) {
      split += d_split;
      carry = split >= p.split_k;
      split -= carry ? p.split_k : 0;
    }
    n += d_n + carry;
    carry = n >= p.num_n_tiles;
    n -= carry ? p.num_n_tiles : 0;
    lo += d_lo + carry;
    const int radix = STACK > 1 ? p.groups : p.num_m_tiles;
    carry = lo >= radix;
    lo -= carry ? radix : 0;
    hi += d_hi + carry;
    if (STACK == 1 && p.split_k > 1) {
      carry = hi >= p.groups;
      hi -= carry ? p.groups : 0;
      split += d_split + carry;
    }
  }
  __device__ __forceinline__ int m_blk(int rank) const { return STACK > 1 ? hi * STACK : lo * CTAS + rank; }
  __device__ __forceinline__ TileCoord coord(const GemmParams& p, int rank, int per_split) const {
    TileCoord t;
    t.split = split;
    t.n_blk = n;
    t.m_blk = m_blk(rank);
    t.grp = STACK > 1 ? lo : hi;
    if (p.grp_ranges) {
      t.kb_begin = p.grp_kb[t.grp];
      t.kb_end = p.grp_kb[t.grp + 1];
    } else {
      t.kb_begin = split * per_split;
      t.kb_end = min(p.k_blocks, t.kb_begin + per_split);
    }
    return t;
  }
};

// Image position of a k-block of 64 pixels (OP_PIXELS_5D). Stepped: its four divisions per k-block kept the producers at 800 to 1030 cycles
// a k-block, above the 384 to 768 that the tensor core needs.
struct PixelWalk {
  int w, h, b;
  __device__ __forceinline__ void start(const GemmParams& p, int kb) {
    w = kb % p.pix_n0;
    kb /= p.pix_n0;
    h = kb % p.pix_n1;
    b = kb / p.pix_n1;
  }
  __device__ __forceinline__ void next(const GemmParams& p) {
    if (++w < p.pix_n0) return;
    w = 0;
    if (++h < p.pix_n1) return;
    h = 0;
    ++b;
  }
};

// A unit of 32 consecutive pixels of an image row (EPI_ROW_CONV): coordinates in the output image, and in an operand that lies like it.
struct PixelUnit {
  int c, par, w, h, b;
};
__device__ __forceinline__ PixelUnit pixel_unit(const GemmParams& p, int m_blk, int q, int col, int grp) {
  const int phase = p.phase_cols > 0 ? col / p.phase_cols : grp;
  const int line = m_blk / p.tile_n0, b = line / p.tile_n1, row = q * 32 >> p.tile_shift;
  return {p.phase_cols > 0 ? col - phase * p.phase_cols : col, p.out_off[phase][1], ((m_blk - line * p.tile_n0 - row) << p.tile_shift) + q * 32,
          (((line - b * p.tile_n1) << 7 >> p.tile_shift) + row) * p.out_mul + p.out_off[phase][0], b};
}

// mbar_wait that adds the time spent to `waited`; a barrier that is complete costs one test and reads no clock.
template <bool PAIR>
__device__ __forceinline__ bool wait_counted(uint64_t* bar, uint32_t parity, volatile int* abort_flag, KernelStatus* st,
                                             unsigned int where, uint32_t budget, long long& waited) {
  if (mbar_test(bar, parity)) return true;
  const long long begin = clock64();
  const bool ok = mbar_wait<PAIR>(bar, parity, abort_flag, st, where, budget);
  waited += clock64() - begin;
  return ok;
}

// PEERS: the tensor-parallel variants (A gathered from peer buffers, output scattered to peer buffers). A separate
// instantiation, so that the plain kernel carries none of their registers and branches.
template <int BN, int CTAS, bool PEERS, int STACK = 1>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_tcgen05_kernel(const __grid_constant__ GemmParams p) {
  static_assert(STACK == 1 || (CTAS == 1 && !PEERS), "stacked tiles: one CTA, no peers");
  using Cfg = GemmCfg<BN, CTAS, STACK>;
  constexpr bool PAIR = CTAS == 2, WIDE = Cfg::WIDE;
  auto start = []() {
    if constexpr (PEERS) chain_wait();
    else chain_begin();
  };
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stages = p.stages;
  uint8_t* fixed = smem + stages * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(fixed);
  uint64_t* empty = full + Cfg::MAX_STAGES;
  uint64_t* tfull = empty + Cfg::MAX_STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* in_bar = tempty + 2;   // two per epilogue warp: "the epilogue operand's unit has landed"
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(in_bar + 2 * GEMM_EPI_WARPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * Cfg::MAX_STAGES + 4 + 2 * GEMM_EPI_WARPS) * 8 + 8 <= Cfg::BAR_BYTES, "barrier block");
  float* bias_slots = reinterpret_cast<float*>(fixed + Cfg::BAR_BYTES);
  uint8_t* xchg = fixed + Cfg::FIXED_BASE;
  // The ring needs a 1024-byte aligned base (128-byte swizzle atoms). The dynamic window normally starts aligned; if
  // the alignment shift does not fit into the slack the launch is refused as a whole, before any barrier exists.
  if (stages < 1 || stages > Cfg::MAX_STAGES ||
      xchg + GEMM_EPI_WARPS * p.epi_bufs * Cfg::EPI_BUF > smem_raw + p.smem_bytes) {
    start();
    if (threadIdx.x == 0) report_error(p.status, TB_ERR_BAD_ARG, 0x700u, blockIdx.x, 0u);
    return;
  }

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = PAIR ? static_cast<int>(cluster_ctarank()) : 0;     // 0 = leader (issues the MMAs)
  const int unit = PAIR ? blockIdx.x >> 1 : blockIdx.x;                 // CTA or CTA pair
  const int units = PAIR ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::MAX_STAGES; ++s) {
      mbar_init(&full[s], 2);         // both producers (a pair: the leader's, for the loads of both CTAs)
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2 * GEMM_EPI_WARPS; ++i) mbar_init(&in_bar[i], 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], GEMM_EPI_WARPS * CTAS);   // pair mode: both CTAs' epilogue warps release the leader's
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.map_a);
    tma_prefetch_desc(&p.map_b);
    if (p.epi_tma) {
      tma_prefetch_desc(&p.map_c);
      if (p.epi & EPI_SAVE_PRE) tma_prefetch_desc(&p.map_c2);
      if (p.epi & (EPI_RESIDUAL | EPI_MUL_DGELU)) tma_prefetch_desc(&p.map_in);
    }
    if (PEERS)
      for (int i = 0; i < p.a_peers && p.a_peers > 1; ++i) tma_prefetch_desc(&p.map_a_peer[i]);
  }
  if (warp == 1) {
    tmem_alloc<Cfg::TMEM_COLS, CTAS>(tmem_slot);
    tmem_relinquish<CTAS>();
  }
  if (Cfg::CAN_COLSUM && p.colsum != nullptr && threadIdx.x >= 64 && threadIdx.x < 64 + 128) {
    // In the bias slots, which this form does not use: a 16 x 16 tile (four core matrices of eight rows of 16 bytes) for each of the four
    // MMAs of a k-block, with ones in rows i and i + 8 of tile i. So each of them sums in a column of its own, over a fourth of the additions:
    // error of the sums of 156672 x 3072 in one column 2.4e-7, in four 1.1e-7, of 557056 x 2976 1.2e-6 and 2.2e-7. The other rows are 2^-126
    // (see g_ones_rows).
#pragma unroll
    for (int i = 0; i < 4; ++i)
      reinterpret_cast<uint32_t*>(bias_slots)[i * 128 + threadIdx.x - 64] = (threadIdx.x - 64) % 32 / 4 == i ? 0x3F803F80u : 0x00800080u;
    fence_proxy_async_smem();
  }
  tc_fence_before();
  if (PAIR) cluster_sync_all(); else __syncthreads();   // barriers and allocations of both CTAs exist from here on
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  start();        // global memory is touched from here on
  if (PAIR) {
    // the pair-wide MMA names one tensor-memory address for both CTAs: the two allocations must coincide
    if (threadIdx.x == 0 && ld_shared_cluster_u32(map_to_cta(tmem_slot, rank ^ 1)) != tmem_base) {
      *abort_flag = 1;
      report_error(p.status, TB_ERR_BAD_ARG, 0x701u, tmem_base, 0u);
    }
    cluster_sync_all();
    if (*abort_flag == 0 && ld_shared_cluster_u32(map_to_cta(const_cast<int*>(abort_flag), rank ^ 1)) != 0) *abort_flag = 1;
    cluster_sync_all();
  }

  const int total_tiles = p.groups * p.num_m_tiles * p.num_n_tiles * p.split_k;
  const int per_split = p.split_k > 1 ? (p.k_blocks + p.split_k - 1) / p.split_k : p.k_blocks;
  using Walk = TileWalk<CTAS, STACK>;
  // Bound of the CTA-internal waits, in units of about a second of polling. The producer of the tensor-parallel form
  // may wait a_budget_ns (global timer) for a peer's shard; the roles that consume its stages must outlast that wait,
  // or ordinary rank skew would abort a tile whose data arrives in time. Measured polling rates put one unit between
  // 0.3 and 2 s, so 4 units per second of peer budget (+ 1) stay above it.
  const uint32_t mbar_budget = PEERS ? 1u + 4u * static_cast<uint32_t>((p.a_budget_ns + 999999999ull) / 1000000000ull) : 1u;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer of A
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      const long long t_begin = clock64();
      long long t_wait = 0;
      unsigned int peers_ready = 0u;   // bit per (peer, chunk) whose flag has been seen
      for (Walk walk(p, unit, units); walk.tile < total_tiles && !*abort_flag; walk.next(p)) {
        const TileCoord tc = walk.coord(p, rank, per_split);
        const int m0 = tc.m_blk * GEMM_BM;
        const int blocks = STACK > 1 ? min(STACK, p.m_blocks - tc.m_blk) : 1;   // 128-row blocks of this tile
        int abase[5] = {0, 0, 0, 0, 0};
        if (p.a_mode == OP_TABLE_5D) {
          const int t0 = tc.m_blk % p.tile_n0;
          const int t1 = (tc.m_blk / p.tile_n0) % p.tile_n1;
          const int t2 = tc.m_blk / (p.tile_n0 * p.tile_n1);
#pragma unroll
          for (int d = 0; d < 5; ++d) abase[d] = t0 * p.a_mul0[d] + t1 * p.a_mul1[d] + t2 * p.a_mul2[d];
        }
        // rows over all taps: channel and displacement of this tile's boxes of 64 rows (channel < 0: ones or nothing)
        constexpr int BOXES = PEERS ? 1 : STACK * GEMM_BM / 64;
        short box_c[BOXES], box_p[BOXES], box_w[BOXES], box_h[BOXES];
        if (!PEERS && p.tap_boxes > 0) {
#pragma unroll
          for (int j = 0; j < BOXES; ++j) {
            const int box = tc.m_blk * (GEMM_BM / 64) + j, tap = box / p.tap_boxes;
            const short* g = p.grp_off[min(tap, p.taps - 1)];
            box_c[j] = tap < p.taps ? static_cast<short>((box - tap * p.tap_boxes) * 64) : -1;
            box_p[j] = g[0];
            box_w[j] = g[1];
            box_h[j] = g[2];
          }
        }
        PixelWalk pix = {};
        if (p.a_mode == OP_PIXELS_5D) pix.start(p, tc.kb_begin);
        for (int kb = tc.kb_begin; kb < tc.kb_end; ++kb, ph ^= (s + 1 == stages), s = (s + 1 == stages) ? 0 : s + 1) {
          if (!wait_counted<PAIR>(&empty[s], ph ^ 1u, abort_flag, p.status, 0x100u + s, mbar_budget, t_wait)) break;
          uint8_t* sA = smem + s * Cfg::STAGE_BYTES;
          if (rank == 0) mbar_expect_tx(&full[s], STACK > 1 ? blocks * Cfg::BLOCK_BYTES : CTAS * Cfg::BLOCK_BYTES);
          const uint32_t bar = PAIR ? map_to_cta(&full[s], 0) : smem_u32(&full[s]);
          // ---- operand A
          if (p.a_mode == OP_KMAJOR_2D) {
            if (PEERS && p.a_peers > 1) {
              const int slot = p.a_interleave ? tc.m_blk % p.a_peers : tc.m_blk / p.a_tiles;
              const int lm = p.a_interleave ? tc.m_blk / p.a_peers : tc.m_blk % p.a_tiles;
              const int peer = (slot + p.a_first) % p.a_peers;
              const int fidx = peer * p.a_chunks + min(lm / p.a_chunk_tiles, p.a_chunks - 1);
              if (p.a_flags != nullptr && peer != p.a_first && !((peers_ready >> fidx) & 1u)) {
                // first tile from this peer: its shard must have been published (bounded wait on its flag)
                const unsigned long long w_begin = global_timer_ns();
                unsigned int seen, polls = 0;
                while (true) {
                  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.a_flags + fidx) : "memory");
                  if (static_cast<int>(seen - p.a_epoch) >= 0) break;
                  if ((++polls & 31u) == 0u && global_timer_ns() - w_begin > p.a_budget_ns) {
                    *abort_flag = 1;
                    report_error(p.status, TB_ERR_PEER_TIMEOUT, 0x500u + peer, seen, p.a_epoch);
                    break;
                  }
                  __nanosleep(50);
                }
                if (*abort_flag) break;
                fence_proxy_async_all();   // order the acquire before the asynchronous-proxy reads of the shard
                peers_ready |= 1u << fidx;
              }
              tma_load_2d<PAIR>(sA, &p.map_a_peer[peer], bar, kb * GEMM_BK, lm * GEMM_BM);
            } else {
              tma_load_2d<PAIR>(sA, &p.map_a, bar, kb * GEMM_BK, m0);
            }
          } else if (p.a_mode == OP_MNMAJOR_2D) {
#pragma unroll
            for (int j = 0; j < STACK * GEMM_BM / 64; ++j)
              if (STACK == 1 || j < blocks * (GEMM_BM / 64)) {
                if (!PEERS && p.row_sums != nullptr && m0 + j * 64 == p.ones_row)
                  tma_load_2d<PAIR>(sA + j * (GEMM_BK * 128), &p.map_in, bar, ones_col(kb), ones_line(kb));
                else tma_load_2d<PAIR>(sA + j * (GEMM_BK * 128), &p.map_a, bar, m0 + j * 64, kb * GEMM_BK);
              }
          } else if (p.a_mode == OP_TABLE_5D) {
            const short* e = p.ktable[kb];
            int h = abase[3] + e[3];
            const CUtensorMap* m = &p.map_a;
            if (h < 0 && (p.halo_flags & 1)) {
              m = &p.map_halo_lo;
              h += 1;
            } else if (h >= p.img_h && (p.halo_flags & 2)) {
              m = &p.map_halo_hi;
              h -= p.img_h;
            }
            tma_load_5d<PAIR>(sA, m, bar, abase[0] + e[0], abase[1] + e[1], abase[2] + e[2], h, abase[4]);
          } else if (!PEERS && p.tap_boxes > 0) {   // OP_PIXELS_5D, a tap per box
#pragma unroll
            for (int j = 0; j < BOXES; ++j) {
              if (STACK > 1 && j >= blocks * (GEMM_BM / 64)) break;
              if (box_c[j] >= 0)
                tma_load_5d<PAIR>(sA + j * (GEMM_BK * 128), &p.map_a, bar, box_c[j], box_p[j], pix.w * GEMM_BK + box_w[j],
                                  pix.h * p.pix_hmul + box_h[j], pix.b);
              else
                tma_load_2d<PAIR>(sA + j * (GEMM_BK * 128), &p.map_in, bar, ones_col(kb), ones_line(kb));
            }
            pix.next(p);
          } else {  // OP_PIXELS_5D: {channels, parity, w, h, b}
            const short* g = p.grp_off[tc.grp];
            const int par = p.disp_a ? g[0] : 0, w = pix.w * GEMM_BK + (p.disp_a ? g[1] : 0);
            const int h = p.disp_a ? pix.h * p.pix_hmul + g[2] : pix.h;
#pragma unroll
            for (int j = 0; j < STACK * GEMM_BM / 64; ++j)
              if (STACK == 1 || j < blocks * (GEMM_BM / 64))
                tma_load_5d<PAIR>(sA + j * (GEMM_BK * 128), &p.map_a, bar, m0 + j * 64, par, w, h, pix.b);
            pix.next(p);
          }
        }
      }
      atomicAdd(&g_gemm_stalls[3], static_cast<unsigned long long>(clock64() - t_begin));
      atomicAdd(&g_gemm_stalls[4], static_cast<unsigned long long>(t_wait));
    }
  } else if (warp == GEMM_B_WARP) {
    // ------------------------------------------------------------------ TMA producer of B
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      long long t_wait = 0;
      for (Walk walk(p, unit, units); walk.tile < total_tiles && !*abort_flag; walk.next(p)) {
        const TileCoord tc = walk.coord(p, rank, per_split);
        // this CTA's rows of B, in boxes of 64 where they are not one (wide tiles: its halves of 256 and of 128)
        const int n0 = tc.n_blk * BN + rank * (WIDE ? 128 : Cfg::B_ROWS);
        auto box_at = [&](int j) { return WIDE && j == 2 ? tc.n_blk * BN + 256 + rank * 64 : n0 + j * 64; };
        PixelWalk pix = {};
        if (p.b_mode == OP_PIXELS_5D) pix.start(p, tc.kb_begin);
        for (int kb = tc.kb_begin; kb < tc.kb_end; ++kb, ph ^= (s + 1 == stages), s = (s + 1 == stages) ? 0 : s + 1) {
          if (!wait_counted<PAIR>(&empty[s], ph ^ 1u, abort_flag, p.status, 0x140u + s, mbar_budget, t_wait)) break;
          uint8_t* sB = smem + s * Cfg::STAGE_BYTES + Cfg::A_BYTES;
          if (rank == 0) mbar_expect_tx(&full[s], CTAS * Cfg::B_BYTES);
          const uint32_t bar = PAIR ? map_to_cta(&full[s], 0) : smem_u32(&full[s]);
          if (p.b_mode == OP_KMAJOR_2D) {
            if (WIDE) {
#pragma unroll
              for (int j = 0; j < 3; ++j) tma_load_2d<PAIR>(sB + j * (64 * 128), &p.map_b, bar, kb * GEMM_BK, box_at(j));
            } else {
              tma_load_2d<PAIR>(sB, &p.map_b, bar, kb * GEMM_BK, n0);
            }
          } else if (p.b_mode == OP_MNMAJOR_2D) {
#pragma unroll
            for (int j = 0; Cfg::CAN_B_MN && j < Cfg::B_ROWS / 64; ++j)
              tma_load_2d<PAIR>(sB + j * (GEMM_BK * 128), &p.map_b, bar, box_at(j), kb * GEMM_BK);
          } else {  // OP_PIXELS_5D with per-group (tap) displacement
            const short* g = p.grp_off[tc.grp];
            const int par = p.disp_a ? 0 : g[0], w = pix.w * GEMM_BK + (p.disp_a ? 0 : g[1]);
            int h = p.disp_a ? pix.h : pix.h * p.pix_hmul + g[2];
            const CUtensorMap* m = &p.map_b;
            if (h < 0 && (p.halo_flags & 1)) {
              m = &p.map_halo_lo;
              h += 1;
            } else if (h >= p.img_h && (p.halo_flags & 2)) {
              m = &p.map_halo_hi;
              h -= p.img_h;
            }
#pragma unroll
            for (int j = 0; j < Cfg::B_ROWS / 64; ++j)
              tma_load_5d<PAIR>(sB + j * (GEMM_BK * 128), m, bar, box_at(j), par, w, h, pix.b);
            pix.next(p);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA in pair mode)
    if (rank == 0 && elect_one()) {
      const bool a_mn = (p.a_mode == OP_MNMAJOR_2D || p.a_mode == OP_PIXELS_5D);
      const bool b_mn = (p.b_mode == OP_MNMAJOR_2D || p.b_mode == OP_PIXELS_5D);
      const uint32_t idesc = make_idesc_bf16(GEMM_BM * CTAS, WIDE ? 256 : BN, a_mn, b_mn);
      const uint32_t idesc_rest = make_idesc_bf16(GEMM_BM * CTAS, 128, a_mn, b_mn);      // wide tiles: columns 256 to 383
      const uint32_t a_lbo = a_mn ? GEMM_BK * 128 : 16, b_lbo = b_mn ? GEMM_BK * 128 : 16;
      const uint32_t a_kstep = a_mn ? (16 * 128) >> 4 : 32 >> 4;   // descriptor units of 16 bytes
      const uint32_t b_kstep = b_mn ? (16 * 128) >> 4 : 32 >> 4;
      const uint32_t idesc_sums = make_idesc_bf16(GEMM_BM * CTAS, PAIR ? 32 : 16, a_mn, 0);   // (16 rows of ones per CTA)
      const uint64_t d_ones = make_smem_desc_plain(smem_u32(bias_slots), 128, 256);
      int s = 0;
      bool landed = false;                   // the next stage has been seen full
      uint32_t ph = 0, tcount = 0;
      const long long t_begin = clock64();
      long long t_acc = 0, t_ops = 0;
      for (Walk walk(p, unit, units); walk.tile < total_tiles && !*abort_flag; walk.next(p), ++tcount) {
        const TileCoord tc = walk.coord(p, rank, per_split);
        const int acc = tcount % Cfg::ACCS;
        const uint32_t aph = (tcount / Cfg::ACCS) & 1u;
        const int blocks = STACK > 1 ? min(STACK, p.m_blocks - tc.m_blk) : 1;
        const long long w0 = clock64();
        if (!mbar_wait<PAIR>(&tempty[acc], aph ^ 1u, abort_flag, p.status, 0x200u + acc, mbar_budget)) break;
        t_acc += clock64() - w0;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        bool ok = true;
        // (Column sums have a loop of their own: with their test inside, the four MMAs of a k-block took 200 to 280 cycles to issue
        // instead of 60.)
        auto k_loop = [&](auto with_sums) {
          constexpr bool SUMS = decltype(with_sums)::value;
          const int ways = p.disp_a ? p.num_n_tiles : p.groups * p.num_n_tiles;
          const int sum_first = SUMS ? first_sum_kb(p, tc, ways) : 0;
          int sum_kb = sum_first;
          const uint32_t d_sums = tmem_base + Cfg::SUM_COL0 + acc * 32;
          for (int kb = tc.kb_begin; kb < tc.kb_end; ++kb) {
            if (!landed && !wait_counted<PAIR>(&full[s], ph, abort_flag, p.status, 0x300u + s, mbar_budget, t_ops)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sA = smem_u32(smem + s * Cfg::STAGE_BYTES);
            const uint32_t sB = sA + Cfg::A_BYTES;
            uint64_t* const freed = &empty[s];
            ph ^= (s + 1 == stages);
            s = (s + 1 == stages) ? 0 : s + 1;
            landed = mbar_test(&full[s], ph);       // (a look at the next stage, whose latency the MMAs cover)
            const uint64_t da = make_smem_desc(sA, a_lbo, 1024);
            const uint64_t db = make_smem_desc(sB, b_lbo, 1024);
#pragma unroll
            for (int mb = 0; mb < STACK; ++mb) {
              if (STACK > 1 && mb >= blocks) break;
              const uint64_t dm = da + mb * (Cfg::BLOCK_BYTES >> 4);
#pragma unroll
              for (int kk = 0; kk < GEMM_BK / 16; ++kk) {
                umma_bf16<CTAS>(d_tmem + mb * BN, dm + kk * a_kstep, db + kk * b_kstep, idesc, (kb > tc.kb_begin || kk > 0) ? 1u : 0u);
                if (WIDE)
                  umma_bf16<CTAS>(d_tmem + 256, dm + kk * a_kstep, db + (128 * 128 >> 4) + kk * b_kstep, idesc_rest,
                                  (kb > tc.kb_begin || kk > 0) ? 1u : 0u);
              }
              if (SUMS && kb == sum_kb) {   // column sums of A: the same A tiles against columns of ones
#pragma unroll
                for (int kk = 0; kk < GEMM_BK / 16; ++kk)
                  umma_bf16<CTAS>(d_sums + mb * 32, dm + kk * a_kstep, d_ones + kk * (512 >> 4), idesc_sums, (kb > sum_first || kk > 0) ? 1u : 0u);
              }
            }
            if (SUMS && kb == sum_kb) sum_kb += ways;
            umma_commit<CTAS>(freed);     // frees the stage (in both CTAs of a pair)
          }
        };
        if constexpr (Cfg::CAN_COLSUM) {
          if (p.colsum != nullptr) k_loop(std::true_type{});
          else k_loop(std::false_type{});
        } else {
          k_loop(std::false_type{});
        }
        if (!ok) break;
        umma_commit<CTAS>(&tfull[acc]);     // accumulator complete (in both CTAs of a pair)
      }
      atomicAdd(&g_gemm_stalls[0], static_cast<unsigned long long>(clock64() - t_begin));
      atomicAdd(&g_gemm_stalls[1], static_cast<unsigned long long>(t_acc));
      atomicAdd(&g_gemm_stalls[2], static_cast<unsigned long long>(t_ops));
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..13)
    // tcgen05.ld hands lane l the 32 columns of accumulator row l. Global memory wants the opposite: neighbouring
    // lanes on neighbouring addresses. The TMA forms (first two branches below) stage units for bulk stores and reductions. In the other form
    // (fp32 output that is not accumulated, peers, matrices or operand mixes without a tensor map, TERRA_GEMM_TMA_EPILOGUE=0) every
    // transfer of a 32 x 32 chunk goes through the warp's 2 KB exchange buffer: row-per-lane on one side, four lanes per
    // row (eight rows, 64 contiguous bytes each, per instruction) on the global side. 16-byte vectors are XOR
    // swizzled by (row >> 1); the profiler still counts about two wavefronts per ideal one on the row-gathering
    // side (a padded 80-byte pitch measured worse), which costs a few percent of the short-K GEMMs.
    const int q = warp & 3;               // TMEM lane quadrant this warp may read
    const int part = (warp - 2) >> 2;     // chunks (units) part, part + 3, ... of the tile's columns
    constexpr int CHUNKS = BN / 32;
    float* my_bias = bias_slots + (warp - 2) * 64;
    uint8_t* my_x = xchg + (warp - 2) * 2048;
    const bool has_bias = (p.epi & EPI_BIAS) != 0;
    const int grow = lane >> 2, gvec = lane & 3;      // global side: rows grow + 8 i, vector gvec
    uint32_t tcount = 0;
    const long long e_begin = clock64();
    long long e_wait = 0;
    auto xaddr = [&](int rr, int vec) -> uint4* {
      return reinterpret_cast<uint4*>(my_x + rr * 64 + (((vec ^ (rr >> 1)) & 3) << 4));
    };
    constexpr int CPW = (CHUNKS + GEMM_EPI_WARPS / 4 - 1) / (GEMM_EPI_WARPS / 4);   // chunks per warp
    // the bias gradient that rides on a weight gradient: columns 0 to 3 of the sums accumulator, lane l holding the sums of A's column (row of
    // D) q * 32 + l
    auto add_column_sums = [&](const TileCoord& tc, int dcol) {
      if (!Cfg::CAN_COLSUM || p.colsum == nullptr || part != 0 ||
          first_sum_kb(p, tc, p.disp_a ? p.num_n_tiles : p.groups * p.num_n_tiles) >= tc.kb_end)
        return;
      uint32_t v[32];
      tmem_ld_32x32(tmem_base + Cfg::SUM_COL0 + dcol * 32 + (static_cast<uint32_t>(q * 32) << 16), v);
      tmem_ld_wait();
      int g = tc.m_blk * GEMM_BM + q * 32 + lane;
      if (p.tap_boxes > 0) {      // (the taps' sums add up)
        const int tap = (g >> 6) / p.tap_boxes;
        g = tap < p.taps ? g - tap * p.tap_boxes * 64 : p.M;
      }
      const float sum = (__uint_as_float(v[0]) + __uint_as_float(v[1])) + (__uint_as_float(v[2]) + __uint_as_float(v[3]));
      if (g < p.M) atomicAdd(p.colsum + g, sum * p.alpha);
    };
    if (!PEERS && STACK == 1 && p.epi_tma && p.epi_tma != 3) {
      // ---- bf16 outputs through TMA, and the operand the epilogue reads. A warp works on units of 32 rows x 64 columns (128
      // bytes per row in the 128-byte-swizzled layout, conflict-free for the row-per-lane 16-byte accesses). Tiles of 192
      // columns are one unit per warp and tile.
      //
      // What bounds a unit is latency, three warps per scheduler being all there is to hide it. So the form of the epilogue is a
      // compile-time constant (with the flags tested inside, every pair of elements became a basic block of its own), a unit's two
      // tensor-memory loads are issued together, the bias of a unit is spread through shared memory once, and the input unit arrives in the
      // buffer its output is staged in: a lane reads and writes the same 16 bytes. With two such buffers the next unit's load has this
      // unit's processing time to arrive; with one (long contractions, which want the ring and hide the epilogue) it is on its way from HBM
      // to L2 meanwhile and issued when the store has read the buffer. The first buffer (4 KB) stages the output; the second takes the
      // saved pre-activation, or alternates with the first. Cycles per unit with the flags tested inside: bias 2400 (now under 1300), bias
      // and residual 3400 + 800 waiting for the input, GELU with the pre-activation 4500, times GELU' 6100 + 800. Launches, before / now:
      // 139264 x 1536 x 384 times GELU' 334 -> 261 us, the same with GELU 260 -> 243, 139264 x 384 x 384 63 -> 54, 156672 x 1024 x 1024
      // with residual 316 -> 279, 17280 x 576 x 192 12.4 -> 10.0. Where the epilogue bounds the launch no wait for a tile hides a latency,
      // so the next unit's bias is loaded and its input asked for before this one is worked on, at coordinates that the walk over the tiles
      // has anyway (two walks of units of their own took about 500 cycles a unit, a bias loaded with its tile 600): times GELU' 254 -> 217
      // us and 139264 x 2976 x 384 503 -> 440, with residual 388 -> 375 and x 2208 x 192 366 -> 277.
      constexpr int UNITS = BN / 64, WARPS_PER_Q = GEMM_EPI_WARPS / 4;
      uint8_t* my_out = xchg + (warp - 2) * p.epi_bufs * Cfg::EPI_BUF;
      uint64_t* my_in = in_bar + 2 * (warp - 2);
      const uint32_t out_base = smem_u32(my_out) + static_cast<uint32_t>(lane) * 128u;
      const uint32_t swz = (static_cast<uint32_t>(lane) & 7u) << 4;
      const uint32_t bias_base = smem_u32(my_bias);
      // column of this warp's first unit in the tile that a walk stands at, or -1
      auto first_col = [&](const Walk& w) -> int {
        const int col = w.n * BN + part * 64;
        return part < UNITS && w.tile < total_tiles && col < p.N ? col : -1;
      };

      auto run = [&](auto form_const) __attribute__((always_inline)) {
        constexpr int FORM = decltype(form_const)::value;      // EPI_* flags of the form, or -1: tested at run time
        const int flags = FORM >= 0 ? FORM : p.epi;
        const bool with_bias = (flags & EPI_BIAS) != 0, gelu = (flags & EPI_GELU) != 0, save_pre = (flags & EPI_SAVE_PRE) != 0;
        const bool has_in = (flags & (EPI_RESIDUAL | EPI_MUL_DGELU)) != 0, dgelu = (flags & EPI_MUL_DGELU) != 0;
        const f32x2 alpha2 = f2_both(p.alpha);
        // (GELU's chains are long enough to alternate between two runs of columns; the other forms lose by it: 139264 x 2976 x 384 with
        // GELU 381 / 344 us, times GELU' 455 / 470)
        constexpr int RUN = FORM >= 0 && (FORM & EPI_GELU) ? 2 : 1;
        const int in_bufs = p.epi_bufs / 2;
        auto bias_pair = [&](int col) -> float2 {     // columns col, col + 1 (col even)
          float2 b = make_float2(0.f, 0.f);
          if (p.epi & EPI_BIAS_F32) {
            if (col < p.N) b.x = __ldg(static_cast<const float*>(p.bias) + col);
            if (col + 1 < p.N) b.y = __ldg(static_cast<const float*>(p.bias) + col + 1);
          } else {
            if (col < p.N) b.x = __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]);
            if (col + 1 < p.N) b.y = __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col + 1]);
          }
          return b;
        };
        // the input unit at column `col` of row block `m_blk` on its way into buffer `buf`, or (buf < 0) into L2; one lane
        auto fetch_in = [&](int col, int m_blk, int buf) {
          if (lane != 0) return;
          uint8_t* const to = my_out + max(buf, 0) * 2 * Cfg::EPI_BUF;
          if (buf >= 0) mbar_expect_tx(my_in + buf, 2 * Cfg::EPI_BUF);
          if (p.epi_tma == 2) {
            const PixelUnit u = pixel_unit(p, m_blk, q, col, 0);
            if (buf >= 0) tma_load_5d(to, &p.map_in, smem_u32(my_in + buf), u.c, u.par, u.w, u.h, u.b);
            else tma_prefetch_l2_5d(&p.map_in, u.c, u.par, u.w, u.h, u.b);
          } else {
            if (buf >= 0) tma_load_2d(to, &p.map_in, my_in + buf, col, m_blk * GEMM_BM + q * 32);
            else tma_prefetch_l2_2d(&p.map_in, col, m_blk * GEMM_BM + q * 32);
          }
        };
        Walk walk(p, unit, units);
        float2 bias_here = make_float2(0.f, 0.f);      // of the unit to come
        {
          const int col = first_col(walk);
          if (with_bias && col >= 0) bias_here = bias_pair(col + 2 * lane);
          if (has_in && col >= 0) fetch_in(col, walk.m_blk(rank), 0);
        }
        uint32_t count = 0;                  // units of this warp so far
        bool failed = false;
        for (; walk.tile < total_tiles && !failed; ++tcount) {
          const TileCoord tc = walk.coord(p, rank, per_split);
          Walk after = walk;
          after.next(p);
          const int acc = tcount % Cfg::ACCS;
          const uint32_t aph = (tcount / Cfg::ACCS) & 1u;
          const int n0 = tc.n_blk * BN;
          const long long ew0 = clock64();
          const bool tile_ready = mbar_wait<PAIR>(&tfull[acc], aph, abort_flag, p.status, 0x400u + acc, mbar_budget);
          if (!__all_sync(0xffffffffu, tile_ready)) break;
          e_wait += clock64() - ew0;
          tc_fence_after();
          bool released = false;
          auto release = [&]() {   // the accumulator has been read: the MMA thread may start the tile after next
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if (PAIR && rank == 1) mbar_arrive_remote(map_to_cta(&tempty[acc], 0));   // the leader's MMA thread waits
              else mbar_arrive(&tempty[acc]);
            }
            released = true;
          };
#pragma unroll 1
          for (int u = part; u < UNITS && n0 + u * 64 < p.N; u += WARPS_PER_Q) {   // warp-uniform
            const int nb0 = n0 + u * 64;
            const bool last = u + WARPS_PER_Q >= UNITS || nb0 + 64 * WARPS_PER_Q >= p.N;
            const int buf = has_in && in_bufs == 2 ? static_cast<int>(count & 1u) : 0;
            uint32_t v[2][32];
            const uint32_t tcol = tmem_base + acc * BN + u * 64 + (static_cast<uint32_t>(q * 32) << 16);
            tmem_ld_32x32(tcol, v[0]);
            tmem_ld_32x32(tcol + 32, v[1]);
            // the next unit's bias and input are asked for now: where the epilogue is what bounds the launch, nothing else hides their latency
            const int next_col = last ? first_col(after) : nb0 + 64 * WARPS_PER_Q;
            const int next_blk = last ? after.m_blk(rank) : tc.m_blk;
            if (with_bias) {
              __syncwarp();
              asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(bias_base + lane * 8), "f"(bias_here.x), "f"(bias_here.y) : "memory");
              if (next_col >= 0) bias_here = bias_pair(next_col + 2 * lane);
            }
            if (has_in) {
              const bool in_ready = mbar_wait<false>(my_in + buf, (in_bufs == 2 ? count >> 1 : count) & 1u, abort_flag, p.status, 0x600u,
                                                     mbar_budget);
              if (!__all_sync(0xffffffffu, in_ready)) {
                tmem_ld_wait();
                failed = true;
                break;
              }
            }
            ++count;
            tmem_ld_wait();
            if (last) release();
            if (lane == 0) bulk_wait_group_read<0>();     // the unit before has left its buffer
            __syncwarp();
            if (has_in && next_col >= 0) fetch_in(next_col, next_blk, in_bufs == 2 ? buf ^ 1 : -1);
            const uint32_t row_out = out_base + buf * 2 * Cfg::EPI_BUF;
            const int row0 = tc.m_blk * GEMM_BM + q * 32;
#pragma unroll
            for (int g2 = 0; g2 < 8; g2 += RUN) {      // 8 columns (16 bytes of the output row) at a time, or twice 8
              f32x2 f[RUN][4];
              float bias[RUN][8];
              uint32_t in[RUN][4];
#pragma unroll
              for (int e = 0; e < RUN; ++e) {
                const int g = g2 + e;
                if (with_bias) {
#pragma unroll
                  for (int k = 0; k < 8; k += 4)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(bias[e][k]), "=f"(bias[e][k + 1]), "=f"(bias[e][k + 2]), "=f"(bias[e][k + 3])
                                 : "r"(bias_base + g * 32 + k * 4));
                }
                if (has_in)
                  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                               : "=r"(in[e][0]), "=r"(in[e][1]), "=r"(in[e][2]), "=r"(in[e][3])
                               : "r"(row_out + ((static_cast<uint32_t>(g) << 4) ^ swz))
                               : "memory");
              }
#pragma unroll
              for (int e = 0; e < RUN; ++e)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const int at = ((g2 + e) & 3) * 8 + 2 * k;
                  f32x2 x = f2_pack(__uint_as_float(v[g2 >> 2][at]), __uint_as_float(v[g2 >> 2][at + 1]));
                  if (with_bias) {
                    const f32x2 add = f2_pack(bias[e][2 * k], bias[e][2 * k + 1]);
                    x = FORM >= 0 ? f2_add(x, add) : f2_fma(x, alpha2, add);
                  } else if (FORM < 0) {
                    x = f2_mul(x, alpha2);
                  }
                  f[e][k] = x;
                }
              if (save_pre) {
#pragma unroll
                for (int e = 0; e < RUN; ++e)
                  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_out + 2 * Cfg::EPI_BUF + ((static_cast<uint32_t>(g2 + e) << 4) ^ swz)),
                               "r"(f2_to_bf16x2(f[e][0])), "r"(f2_to_bf16x2(f[e][1])), "r"(f2_to_bf16x2(f[e][2])), "r"(f2_to_bf16x2(f[e][3]))
                               : "memory");
              }
#pragma unroll
              for (int e = 0; e < RUN; ++e)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  if (gelu) f[e][k] = gelu_erf2(f[e][k]);
                  if (has_in) {
                    if (dgelu) {
                      f[e][k] = f2_mul(f[e][k], gelu_erf_grad2_bf16(in[e][k]));
                    } else {
                      const float2 r = unpack_bf16x2(in[e][k]);
                      f[e][k] = f2_add(f[e][k], f2_pack(r.x, r.y));
                    }
                  }
                }
#pragma unroll
              for (int e = 0; e < RUN; ++e)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_out + ((static_cast<uint32_t>(g2 + e) << 4) ^ swz)),
                             "r"(f2_to_bf16x2(f[e][0])), "r"(f2_to_bf16x2(f[e][1])), "r"(f2_to_bf16x2(f[e][2])), "r"(f2_to_bf16x2(f[e][3]))
                             : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const uint32_t src = smem_u32(my_out) + buf * 2 * Cfg::EPI_BUF;
              if (p.epi_tma == 2) {
                // (decoded by this one lane)
                const PixelUnit o = pixel_unit(p, tc.m_blk, q, nb0, tc.grp);
                if (tc.m_blk < p.m_blocks && o.w < p.out_w && o.h < p.out_h) tma_store_5d(&p.map_c, src, o.c, o.par, o.w, o.h, o.b);
              } else {
                if (row0 < p.M) {
                  if (save_pre) tma_store_2d(&p.map_c2, src + 2 * Cfg::EPI_BUF, nb0, row0);
                  tma_store_2d(&p.map_c, src, nb0, row0);
                }
              }
              bulk_commit_group();
            }
            if (has_in && in_bufs == 1 && next_col >= 0) {
              if (lane == 0) bulk_wait_group_read<0>();
              __syncwarp();
              fetch_in(next_col, next_blk, 0);
            }
          }
          if (!released && !failed) {   // a warp without a unit in this tile
            release();
            const int col = first_col(after);
            if (with_bias && col >= 0) bias_here = bias_pair(col + 2 * lane);
            if (has_in && col >= 0) {
              if (lane == 0) bulk_wait_group_read<0>();
              fetch_in(col, after.m_blk(rank), in_bufs == 2 ? static_cast<int>(count & 1u) : 0);
            }
          }
          walk = after;
        }
        if (lane == 0) bulk_wait_group_read<0>();
      };
      const int form = p.epi & (EPI_BIAS | EPI_GELU | EPI_RESIDUAL | EPI_MUL_DGELU | EPI_SAVE_PRE);
      if (p.alpha != 1.0f) run(std::integral_constant<int, -1>{});
      else if (form == 0) run(std::integral_constant<int, 0>{});
      else if (form == EPI_BIAS) run(std::integral_constant<int, EPI_BIAS>{});
      else if (form == (EPI_BIAS | EPI_GELU | EPI_SAVE_PRE)) run(std::integral_constant<int, EPI_BIAS | EPI_GELU | EPI_SAVE_PRE>{});
      else if (form == (EPI_BIAS | EPI_GELU)) run(std::integral_constant<int, EPI_BIAS | EPI_GELU>{});
      else if (form == (EPI_BIAS | EPI_RESIDUAL)) run(std::integral_constant<int, EPI_BIAS | EPI_RESIDUAL>{});
      else if (form == EPI_MUL_DGELU) run(std::integral_constant<int, EPI_MUL_DGELU>{});
      else run(std::integral_constant<int, -1>{});
    } else if (!PEERS && p.epi_tma == 3) {
      // ---- accumulated fp32 outputs as TMA reductions of 32 x 32 units, 128 bytes a row in the 128-byte-swizzled layout. (By the lanes, as
      // vector reductions behind the exchange buffer, an SM got 16 bytes per clock to L2: 14500 cycles for a tile of 256 x 192, which
      // nothing hides where a tile is the CTA's only one.) Weight gradients, us, lanes / this, the same plans: 2048 rows of 384 x 384 10.4 / 6.9,
      // 17280 of 192 x 192 11.4 / 8.8, 139264 of 384 x 384 49.6 / 46.3; convolution of 17280 pixels, 192 channels 20.8 / 18.
      uint8_t* my_out = xchg + (warp - 2) * p.epi_bufs * Cfg::EPI_BUF;
      const uint32_t out_base = smem_u32(my_out);
      for (Walk walk(p, unit, units); walk.tile < total_tiles; walk.next(p), ++tcount) {
        const TileCoord first = walk.coord(p, rank, per_split);
        const int acc = tcount % Cfg::ACCS, n0 = first.n_blk * BN;
        const long long ew0 = clock64();
        const bool tile_ready = mbar_wait<PAIR>(&tfull[acc], (tcount / Cfg::ACCS) & 1u, abort_flag, p.status, 0x400u + acc, mbar_budget);
        if (!__all_sync(0xffffffffu, tile_ready)) break;
        e_wait += clock64() - ew0;
        tc_fence_after();
#pragma unroll 1
        for (int mb = 0; mb < STACK; ++mb) {
          TileCoord tc = first;
          tc.m_blk += mb;
          if (STACK > 1 && tc.m_blk >= p.m_blocks) break;
          const int dcol = STACK > 1 ? mb : acc;
          int row = tc.m_blk * GEMM_BM + q * 32, group = tc.grp, rows = p.M;      // this warp's rows of the group (tap)
          const bool ones = p.row_sums != nullptr && (row & ~63) == p.ones_row;
          if (p.tap_boxes > 0) {
            group = (row >> 6) / p.tap_boxes;
            row -= group * p.tap_boxes * 64;
            if (group >= p.taps) rows = 0;
          }
          if (row < rows || ones) {
#pragma unroll 1
            for (int c = part; c < CHUNKS && n0 + c * 32 < p.N; c += GEMM_EPI_WARPS / 4) {      // warp-uniform
              const int cb = n0 + c * 32;
              uint32_t v[32];
              tmem_ld_32x32(tmem_base + dcol * BN + c * 32 + (static_cast<uint32_t>(q * 32) << 16), v);
              if (lane == 0) bulk_wait_group_read<0>();      // the unit before has left the buffer
              tmem_ld_wait();
              if (p.alpha != 1.0f) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * p.alpha);
              }
              __syncwarp();
              if (p.epi & EPI_TRANSPOSE) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  asm volatile("st.shared.b32 [%0], %1;" ::"r"(out_base + j * 128 + (((lane >> 2) ^ (j & 7)) << 4) + ((lane & 3) << 2)), "r"(v[j])
                               : "memory");
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(out_base + lane * 128 + ((j ^ (lane & 7)) << 4)), "r"(v[4 * j]),
                               "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                               : "memory");
              }
              if (ones) {      // the rows of a column add up to its share of the column sums of B; a lane per column
                __syncwarp();
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int r = 0; r < 32; ++r) {
                  const int at = (p.epi & EPI_TRANSPOSE) ? lane * 128 + (((r >> 2) ^ (lane & 7)) << 4) + ((r & 3) << 2)
                                                         : r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + ((lane & 3) << 2);
                  sum[r & 3] += *reinterpret_cast<const float*>(my_out + at);
                }
                if (cb + lane < p.N) atomicAdd(p.row_sums + cb + lane, (sum[0] + sum[1]) + (sum[2] + sum[3]));
                continue;
              }
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (p.epi & EPI_TRANSPOSE) tma_reduce_add_3d(&p.map_c, out_base, row, cb, 0);
                else tma_reduce_add_3d(&p.map_c, out_base, cb, row, group);
                bulk_commit_group();
              }
            }
          }
          add_column_sums(tc, dcol);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR && rank == 1) mbar_arrive_remote(map_to_cta(&tempty[acc], 0));   // the leader's MMA thread waits
          else mbar_arrive(&tempty[acc]);
        }
      }
      if (lane == 0) bulk_wait_group_read<0>();
    } else
    for (Walk walk(p, unit, units); walk.tile < total_tiles; walk.next(p), ++tcount) {
      const TileCoord first = walk.coord(p, rank, per_split);
      const int acc = tcount % Cfg::ACCS;
      const uint32_t aph = (tcount / Cfg::ACCS) & 1u;
      const int n0 = first.n_blk * BN;
      bool failed = false;
#pragma unroll 1
      for (int mb = 0; mb < STACK; ++mb) {       // the tile's row blocks
        TileCoord tc = first;
        tc.m_blk += mb;
        if (STACK > 1 && tc.m_blk >= p.m_blocks) break;
        const int dcol = (STACK > 1 ? mb : acc);    // which of the two accumulators
        // ---- tile row -> output row index (-1: outside the output)
        auto out_row = [&](int r) -> long long {
          if (p.epi & EPI_ROW_CONV) {
            const int t0 = tc.m_blk % p.tile_n0;
            const int t1 = (tc.m_blk / p.tile_n0) % p.tile_n1;
            const int t2 = tc.m_blk / (p.tile_n0 * p.tile_n1);
            const int w = t0 * GEMM_BM + r;
            return (w < p.out_w && tc.m_blk < p.m_blocks) ? (static_cast<long long>(t2) * p.tile_n1 + t1) * p.out_w + w : -1;
          } else if (PEERS && p.a_peers > 1) {
            const int slot = p.a_interleave ? tc.m_blk % p.a_peers : tc.m_blk / p.a_tiles;
            const int peer = (slot + p.a_first) % p.a_peers;
            const int lr = (p.a_interleave ? tc.m_blk / p.a_peers : tc.m_blk % p.a_tiles) * GEMM_BM + r;
            return (lr < p.a_rows) ? static_cast<long long>(peer) * p.a_rows + lr : -1;
          } else if (!PEERS && p.tap_boxes > 0) {
            const int g = tc.m_blk * GEMM_BM + r, tap = (g >> 6) / p.tap_boxes, c = g - tap * p.tap_boxes * 64;
            if (tap >= p.taps) return (g & ~63) == p.ones_row ? -2 : -1;      // -2: a share of the column sums of B
            return c < p.tap_channels ? static_cast<long long>(tap) * p.tap_channels + c : -1;
          } else {
            const long long g = static_cast<long long>(tc.m_blk) * GEMM_BM + r;
            return (g < p.M) ? g : -1;
          }
        };
        int grows[4];   // row indices fit 32 bits (element offsets may not)
  #pragma unroll
        for (int i = 0; i < 4; ++i) grows[i] = static_cast<int>(out_row(q * 32 + grow + 8 * i));
        const long long gofs = static_cast<long long>(tc.grp) * p.grp_c_stride;
        const int ncols_out = p.N;

        // bf16 chunk from global memory, global-side layout (zeros outside the output)
        auto fetch_chunk = [&](const __nv_bfloat16* base, long long ld, int cb, uint4 (&t)[4]) {
  #pragma unroll
          for (int i = 0; i < 4; ++i) {
            t[i] = make_uint4(0, 0, 0, 0);
            if (grows[i] >= 0 && cb + gvec * 8 < ncols_out)
              t[i] = *reinterpret_cast<const uint4*>(base + static_cast<long long>(grows[i]) * ld + cb + gvec * 8);
          }
        };
        // global-side registers -> row-per-lane registers
        auto turn_chunk = [&](const uint4 (&t)[4], uint4 (&u)[4]) {
          __syncwarp();
  #pragma unroll
          for (int i = 0; i < 4; ++i) *xaddr(grow + 8 * i, gvec) = t[i];
          __syncwarp();
  #pragma unroll
          for (int j = 0; j < 4; ++j) u[j] = *xaddr(lane, j);
        };
        // 32 floats of the row-per-lane layout to bf16 global memory
        auto store_chunk = [&](__nv_bfloat16* base, long long ld, int cb, const float (&f)[32]) {
          __syncwarp();
  #pragma unroll
          for (int j = 0; j < 4; ++j)
            *xaddr(lane, j) = make_uint4(pack_bf16x2(f[8 * j], f[8 * j + 1]), pack_bf16x2(f[8 * j + 2], f[8 * j + 3]),
                                         pack_bf16x2(f[8 * j + 4], f[8 * j + 5]), pack_bf16x2(f[8 * j + 6], f[8 * j + 7]));
          __syncwarp();
  #pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 t = *xaddr(grow + 8 * i, gvec);
            if (grows[i] >= 0 && cb + gvec * 8 < ncols_out) {
              __nv_bfloat16* o = base + static_cast<long long>(grows[i]) * ld + cb + gvec * 8;
              if (PEERS && p.c_peers > 1 && base == static_cast<__nv_bfloat16*>(p.C) + gofs)   // the row's owner stages it
                o = static_cast<__nv_bfloat16*>(p.c_peer[grows[i] / p.c_rows]) + gofs +
                    (static_cast<long long>(p.c_slot) * p.c_rows + grows[i] % p.c_rows) * ld + cb + gvec * 8;
              *reinterpret_cast<uint4*>(o) = t;
            }
          }
        };

        // The operand the epilogue reads (GELU input of the backward pass, or the residual) does not depend on the
        // accumulator: pull it into L2 before waiting for the tile, so the DRAM latency hides behind the main loop;
        // the chunk loop then fetches it (an L2 hit) under the latency of its tcgen05.ld.
        const bool pre_aux = (p.epi & EPI_MUL_DGELU) != 0;
        const bool pre_res = !pre_aux && (p.epi & EPI_RESIDUAL) != 0;
        const __nv_bfloat16* pre_ptr = pre_aux ? p.aux : p.residual;
        const long long pre_ld = pre_aux ? p.ldaux : p.ldr;
        if (pre_aux || pre_res) {
  #pragma unroll
          for (int ci = 0; ci < CPW; ++ci) {
            const int c = part + ci * (GEMM_EPI_WARPS / 4);
            if (c < CHUNKS && n0 + c * 32 < p.N) {
  #pragma unroll
              for (int i = 0; i < 4; ++i)
                if (grows[i] >= 0 && n0 + c * 32 + gvec * 8 < ncols_out)
                  asm volatile("prefetch.global.L2 [%0];" ::"l"(pre_ptr + static_cast<long long>(grows[i]) * pre_ld + n0 + c * 32 + gvec * 8));
            }
          }
        }
        if (mb == 0) {
          const long long ew0 = clock64();
          // Every lane polls for itself and may leave the wait in a different iteration; the vote reconverges the warp
          // before the warp-collective tcgen05.ld below (and makes a failed wait leave the loop as one warp).
          const bool tile_ready = mbar_wait<PAIR>(&tfull[acc], aph, abort_flag, p.status, 0x400u + acc, mbar_budget);
          if (!__all_sync(0xffffffffu, tile_ready)) {
            failed = true;
            break;
          }
          e_wait += clock64() - ew0;
          tc_fence_after();
        }

  #pragma unroll
        for (int ci = 0; ci < CPW; ++ci) {
          const int c = part + ci * (GEMM_EPI_WARPS / 4);
          if (c >= CHUNKS || n0 + c * 32 >= p.N) break;   // warp-uniform
          const int cb = n0 + c * 32;          // first output column of this chunk
          uint4 pre[4];
          if (pre_aux || pre_res) fetch_chunk(pre_ptr, pre_ld, cb, pre);
          if (has_bias) {
            // one coalesced load per warp and chunk; the 32 values are then read back as broadcast float4
            float b = 0.f;
            if (cb + lane < p.N)
              b = (p.epi & EPI_BIAS_F32) ? __ldg(static_cast<const float*>(p.bias) + cb + lane)
                                         : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[cb + lane]);
            __syncwarp();
            my_bias[lane] = b;
            __syncwarp();
          }
          uint32_t v[32];
          tmem_ld_32x32(tmem_base + dcol * BN + c * 32 + (static_cast<uint32_t>(q * 32) << 16), v);
          tmem_ld_wait();
          float f[32];
          if (has_bias) {
  #pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 b4 = *reinterpret_cast<const float4*>(my_bias + j);
              f[j] = fmaf(__uint_as_float(v[j]), p.alpha, b4.x);
              f[j + 1] = fmaf(__uint_as_float(v[j + 1]), p.alpha, b4.y);
              f[j + 2] = fmaf(__uint_as_float(v[j + 2]), p.alpha, b4.z);
              f[j + 3] = fmaf(__uint_as_float(v[j + 3]), p.alpha, b4.w);
            }
          } else if (p.alpha != 1.0f) {
  #pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]) * p.alpha;
          } else {
  #pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
          }
          if (p.epi & EPI_SAVE_PRE) store_chunk(static_cast<__nv_bfloat16*>(p.C2), p.ldc2, cb, f);
          if (p.epi & EPI_GELU) {
  #pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = gelu_erf(f[j]);
          }
          if (p.epi & EPI_MUL_DGELU) {
            uint4 u[4];
            turn_chunk(pre, u);
  #pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t w4[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
  #pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 x = unpack_bf16x2(w4[k]);
                f[8 * j + 2 * k] *= gelu_erf_grad(x.x);
                f[8 * j + 2 * k + 1] *= gelu_erf_grad(x.y);
              }
            }
          }
          if (p.epi & EPI_RESIDUAL) {
            uint4 u[4];
            if (pre_res) {
              turn_chunk(pre, u);
            } else {
              uint4 t[4];
              fetch_chunk(p.residual, p.ldr, cb, t);
              turn_chunk(t, u);
            }
  #pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t w4[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
  #pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 x = unpack_bf16x2(w4[k]);
                f[8 * j + 2 * k] += x.x;
                f[8 * j + 2 * k + 1] += x.y;
              }
            }
          }
          if (p.epi & EPI_TRANSPOSE) {
            // a column of the chunk is 32 consecutive rows, one per lane: 128 bytes of the transposed output
            const int g = static_cast<int>(out_row(q * 32 + lane));
            float* o = static_cast<float*>(p.C) + g;
            if (g >= 0) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (cb + j < ncols_out) atomicAdd(o + static_cast<long long>(cb + j) * p.ldc, f[j]);
            }
          } else if (p.epi & EPI_OUT_F32) {
            // fp32 output: two passes of 16 columns through the exchange buffer (4 floats per 16-byte vector)
            float* obase = static_cast<float*>(p.C) + gofs;
            const bool vec_ok = ((reinterpret_cast<uintptr_t>(obase) & 15) == 0) && ((p.ldc & 3) == 0);
  #pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              __syncwarp();
  #pragma unroll
              for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(xaddr(lane, j)) =
                    make_float4(f[16 * hf + 4 * j], f[16 * hf + 4 * j + 1], f[16 * hf + 4 * j + 2], f[16 * hf + 4 * j + 3]);
              __syncwarp();
  #pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float4 t = *reinterpret_cast<const float4*>(xaddr(grow + 8 * i, gvec));
                const int col = cb + 16 * hf + gvec * 4;
                if (!PEERS && grows[i] == -2 && p.row_sums != nullptr) {
                  const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e)
                    if (col + e < ncols_out) atomicAdd(p.row_sums + col + e, tv[e]);
                  continue;
                }
                if (grows[i] < 0 || col >= ncols_out) continue;
                float* o = obase + static_cast<long long>(grows[i]) * p.ldc + col;
                if (PEERS && p.c_peers > 1)   // the row's owner accumulates it
                  o = static_cast<float*>(p.c_peer[grows[i] / p.c_rows]) + gofs +
                      static_cast<long long>(grows[i] % p.c_rows) * p.ldc + col;
                const bool full4 = vec_ok && col + 4 <= ncols_out;
                if (p.epi & EPI_ATOMIC) {
                  if (full4) {
                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o), "f"(t.x), "f"(t.y), "f"(t.z),
                                 "f"(t.w)
                                 : "memory");
                  } else {
                    const float tv[4] = {t.x, t.y, t.z, t.w};
  #pragma unroll
                    for (int e = 0; e < 4; ++e)
                      if (col + e < ncols_out) atomicAdd(o + e, tv[e]);
                  }
                } else {
                  if (full4) {
                    *reinterpret_cast<float4*>(o) = t;
                  } else {
                    const float tv[4] = {t.x, t.y, t.z, t.w};
  #pragma unroll
                    for (int e = 0; e < 4; ++e)
                      if (col + e < ncols_out) o[e] = tv[e];
                  }
                }
              }
            }
          } else {
            store_chunk(static_cast<__nv_bfloat16*>(p.C) + gofs, p.ldc, cb, f);
          }
        }
        add_column_sums(tc, dcol);
      }
      if (failed) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && rank == 1) mbar_arrive_remote(map_to_cta(&tempty[acc], 0));   // the leader's MMA thread waits
        else mbar_arrive(&tempty[acc]);
      }
    }
    if (warp == 2 && lane == 0) {
      atomicAdd(&g_gemm_stalls[5], static_cast<unsigned long long>(clock64() - e_begin));
      atomicAdd(&g_gemm_stalls[6], static_cast<unsigned long long>(e_wait));
    }
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_flag) {
    // Give copies that are still in flight time to land before shared memory is released.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  // pair mode: neither CTA may leave while the other can still signal its barriers or read its operands
  if (PAIR) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc<Cfg::TMEM_COLS, CTAS>(tmem_base);
  }
}

// ------------------------------------------------------------------------------ host side
template <int BN, int CTAS, bool PEERS = false, int STACK = 1>
static cudaError_t launch_bn(const GemmParams& p_in, int num_sms, cudaStream_t stream) {
  using Cfg = GemmCfg<BN, CTAS, STACK>;
  static SharedLimit limit;      // (the backward pass launches without the interpreter's lock)
  const cudaError_t raised = limit.raise(reinterpret_cast<const void*>(gemm_tcgen05_kernel<BN, CTAS, PEERS, STACK>), Cfg::MAX_SMEM);
  if (raised != cudaSuccess) return raised;
  GemmParams p = p_in;
  if (PEERS || (STACK > 1 && p.epi_tma != 3) || (p.epi_tma == 3 && Cfg::stages_for(2) < 3)) p.epi_tma = 0;
  // (a long contraction hides the epilogue behind its main loop and wants the deeper ring: one buffer for input and output)
  const bool has_in = (p.epi & (EPI_RESIDUAL | EPI_MUL_DGELU)) != 0;
  p.epi_bufs = p.epi_tma == 0 ? 1 : ((p.epi & EPI_SAVE_PRE) || (has_in && p.k_blocks <= 12) ? 4 : 2);
  if (p.epi_bufs == 4 && has_in && Cfg::stages_for(4) < 3) p.epi_bufs = 2;
  if (p.epi_tma == 1 && Cfg::stages_for(p.epi_bufs) < 3) {   // single-CTA tiles 256 wide: the ring needs the room
    p.epi_tma = 0;
    p.epi_bufs = 1;
  }
  p.stages = Cfg::stages_for(p.epi_bufs);
  p.smem_bytes = Cfg::smem_bytes(p.epi_bufs);
  const int total = p.groups * p.num_m_tiles * p.num_n_tiles * p.split_k;
  const int max_units = num_sms / CTAS;
  if (total <= 0) return cudaSuccess;
  if (max_units < 1) return cudaErrorInvalidValue;   // a pair on one SM
  const int units = total < max_units ? total : max_units;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(units * CTAS);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = p.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int attrs = 0;
  if (!PEERS) {      // (kernels that wait for another GPU are not chained)
    attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (CTAS > 1) {
    attr[attrs].id = cudaLaunchAttributeClusterDimension;
    attr[attrs].val.clusterDim.x = CTAS;
    attr[attrs].val.clusterDim.y = 1;
    attr[attrs++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = attrs;
  return cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<BN, CTAS, PEERS, STACK>, p);
}

cudaError_t gemm_ones_rows(void** ptr) {
  static std::atomic<void*> known[64];      // per device: the look-up takes a microsecond
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  *ptr = dev < 64 ? known[dev].load(std::memory_order_relaxed) : nullptr;
  if (*ptr != nullptr) return cudaSuccess;
  e = cudaGetSymbolAddress(ptr, g_ones_rows);
  if (e == cudaSuccess && dev < 64) known[dev].store(*ptr, std::memory_order_relaxed);
  return e;
}

cudaError_t gemm_read_stalls(unsigned long long* out8, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out8, g_gemm_stalls, 8 * sizeof(unsigned long long));
  if (e != cudaSuccess) return e;
  if (reset) {
    unsigned long long zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    e = cudaMemcpyToSymbol(g_gemm_stalls, zero, sizeof(zero));
  }
  return e;
}

cudaError_t launch_gemm(const GemmParams& p, int bn, int ctas, int num_sms, cudaStream_t stream) {
  if (ctas == 2) {
    switch (bn) {
      case 384: return launch_bn<384, 2>(p, num_sms, stream);
      case 128: return launch_bn<128, 2>(p, num_sms, stream);
      case 192: return p.b_mode == OP_KMAJOR_2D ? launch_bn<192, 2>(p, num_sms, stream) : cudaErrorInvalidValue;
      case 256: return launch_bn<256, 2>(p, num_sms, stream);
      default: return cudaErrorInvalidValue;
    }
  }
  if (p.stack == 2) {
    switch (bn) {
      case 128: return launch_bn<128, 1, false, 2>(p, num_sms, stream);
      case 192: return launch_bn<192, 1, false, 2>(p, num_sms, stream);
      case 256: return p.colsum == nullptr ? launch_bn<256, 1, false, 2>(p, num_sms, stream) : cudaErrorInvalidValue;
      default: return cudaErrorInvalidValue;
    }
  }
  if (p.a_peers > 1 || p.c_peers > 1) {
    switch (bn) {
      case 64: return launch_bn<64, 1, true>(p, num_sms, stream);
      case 128: return launch_bn<128, 1, true>(p, num_sms, stream);
      case 192: return launch_bn<192, 1, true>(p, num_sms, stream);
      case 256: return launch_bn<256, 1, true>(p, num_sms, stream);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (bn) {
    case 64: return launch_bn<64, 1>(p, num_sms, stream);
    case 128: return launch_bn<128, 1>(p, num_sms, stream);
    case 192: return launch_bn<192, 1>(p, num_sms, stream);
    case 256: return launch_bn<256, 1>(p, num_sms, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace tb
