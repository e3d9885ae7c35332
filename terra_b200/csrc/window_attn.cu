// Swin window attention (forward and backward) over a window-major activation layout, with the
// shifted-window roll / partition / reverse, the window-parallel halo and the sequence-parallel K/V
// gather all expressed as index math on the loads and stores:
//
//   * activations are stored unshifted, window-major: rank p of the window dimension holds
//     [B, nW_p, shardN, *] rows for its flat window range [win_start[p], win_start[p+1]);
//   * a CTA walks over windows of the *shifted* frame for a fixed group of heads; every token of a window is
//     located (owner rank, row) in closed form and its Q/K/V row is read from the owner's buffer
//     (a peer pointer over NVLink when the owner is another GPU); outputs are stored to the token's
//     home row, again possibly on a peer;
//   * relative-position bias comes from a shared-memory copy of the table, the shifted-window mask
//     from the token's region id in the rolled frame; nothing of size [nW, N, N] is materialised.
//
// Windows here are small (N = wh*ww <= 128 keys), far below the tile sizes at which tcgen05 pays off, so the products
// run on warp-level mma.sync. The kernels are bound by instruction issue: every score element costs a scale + bias, a
// max, an exponential and a sum besides its share of the products, so what the design buys is few other instructions
// per element and enough independent warps:
//   * one warp owns one 16-row block of the window for the whole kernel (block = NPAD / 16 warps), so everything that
//     depends on (row, column) only is computed once: bias addresses become a register plus an immediate for windows 8
//     or 12 wide, and the bias gradient of a thread's score elements is summed over all windows in registers (windows
//     of 64 tokens) or in a private shared-memory slot (larger ones) and folded into the table once at the end;
//   * the rows of the next window are fetched by cp.async while the current one is computed (two stages where the
//     shared memory allows it); the token tables are computed two windows ahead;
//   * a window's results are staged over its own dead operand rows and leave as 16-byte vectors, warp by warp.
//   * elementwise work on neighbouring columns goes through the two-wide fp32 instructions.
//   * where a block holds two heads (forward, 16 and 32 channels) a warp takes 32 rows of one head, not 16 of both: two independent
//     chains to issue from, and half the reads of K and V through the shared-memory port;
//   * accumulator tiles go to shared memory four 8 x 8 tiles an instruction;
//   * windows of at most 32 tokens have blocks of their own size, and padding columns cost a comparison, not the masked form.
// Us, before these three / now (shifted, with bias): 2176 windows of 8 x 8, 12 heads of 32 channels, forward 105 / 87 (66 of HBM
// traffic), backward 236 / 227 (115); 2448 of 8 x 8, 8 heads of 128 channels 237 / 236 and 626 / 599; 180 of 8 x 12, 12 heads of 16
// channels 26 / 16 and 50 / 44; 1020 of 7 x 7, 12 heads of 32 channels 93 / 52 and 140 / 122; 1800 of 4 x 8, 8 heads of 32 channels
// 89 / 23 and 120 / 57. What is left is issue and latency: the shared-memory port is busy 50 (forward) and 70 % (backward) of the time.
#include <atomic>
#include "chained_launch.cuh"
#include "common.cuh"
#include "host_api.h"
#include "shared_limit.h"
#include "window_geo.cuh"

namespace tb {
namespace {

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}

// four 8 x 8 tiles of the accumulator layout (bf16 pairs) to rows of shared memory, lane l giving the address of row l & 7 of tile l >> 3
__device__ __forceinline__ void stsm_x4(void* p, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(smem_u32(p)), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}

// 16-byte asynchronous copy global -> shared
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr float WA_LOG2E = 1.4426950408889634f;

// Shared-memory layout of one instantiation. G = channels of a row handled by the CTA (HPC heads), rows padded by 16
// bytes so that the eight rows of an ldmatrix fall into different banks for every G (16, 32, 64, 128).
template <int HD, int NPAD, int HPC, bool BWD>
struct WaCfg {
  static constexpr int G = HD * HPC;
  static constexpr int PITCH = G + 8;
  static constexpr int PP = NPAD + 8;                            // pitch of the P / dS stash (backward)
  static constexpr int THREADS = NPAD * 2;                       // a warp per 16 rows
  static constexpr int MT = !BWD && HPC == 2 ? 2 : 1;            // 16-row tiles of a warp (two: half of the warps per head)
  static constexpr int MATS = BWD ? 4 : 3;                       // q, k, v [, dO]
  static constexpr int MAT = NPAD * PITCH;                       // elements
  static constexpr int STAGE = MATS * MAT;
  static constexpr int STASH = BWD ? 2 * NPAD * PP : 0;          // P and dS, bf16
  // dQ is staged in the warp's own stash rows before P and dS go there; a 128-channel head does not fit into them
  static constexpr bool DQ_IN_STASH = HD <= NPAD;
  static constexpr int DQ = (BWD && !DQ_IN_STASH) ? MAT : 0;
  static constexpr bool ACC_REGS = NPAD <= 64;                   // bias-gradient sums: registers or shared memory
  static constexpr int ACC = (BWD && !ACC_REGS) ? NPAD * NPAD : 0;   // floats
  static constexpr int FIXED = (STASH + DQ) * 2 + ACC * 4 + 3 * NPAD * 8 + NPAD * 4;
  // Resident CTAs that shared memory allows, with the kilobyte that every CTA reserves and a small bias table (that of an 8 x 8
  // window makes three of four where 64 channels are staged). Two stages where three (two for windows above 64 tokens) fit.
  static constexpr int fits(int stages) { return 228 * 1024 / (FIXED + stages * STAGE * 2 + 1024); }
  static constexpr int STAGES = fits(2) >= (NPAD <= 64 ? 3 : 2) ? 2 : 1;
  static constexpr size_t bytes(int nrel) { return static_cast<size_t>(FIXED) + STAGES * STAGE * 2 + HPC * nrel * 4; }
  // Resident CTAs asked of the compiler, which bounds the registers per thread: no more than shared memory allows. (Asked for
  // five where two stages of 64 channels let four or three fit, the compiler spilled for nothing: 2176 windows of 8 x 8, 12 heads
  // of 32 channels, forward without / with shift 116 / 125 us, for four 96 / 105. For three it would be 94 / 103, but then
  // 4 x 4 windows lose the fourth: 6 heads of 64 channels 67 / 71 us, for four 65 / 70, for three 75 / 80. One stage and five
  // CTAs: 100 / 109.)
  // (Two tiles a warp: three blocks of 160 registers instead of four of 128, 96 / 102 us for the 2176 windows above.)
  static constexpr int WANTED = MT == 2 && NPAD <= 64 ? (NPAD == 64 ? 3 : 8) : NPAD == 32 ? (BWD ? (HD > 64 ? 4 : 6) : 8) : NPAD > 96 ? 1 : (BWD ? (NPAD > 64 ? (HD > 64 ? 1 : 2) : (HD > 64 ? 2 : 3))
                                                     : (NPAD > 64 ? 2 : (HD > 64 ? 4 : 5)));
  // (128-token windows of 128-channel heads do not fit backward at all: their launch is refused)
  static constexpr int MIN_CTAS = fits(STAGES) < 1 ? 1 : (WANTED < fits(STAGES) ? WANTED : fits(STAGES));
};

struct WaItem {
  int b, ii, jj;
};

__device__ __forceinline__ WaItem wa_item(const WindowAttnArgs& a, int item, int my_nw) {
  WaItem w;
  w.b = 0;
  if (a.B > 1) {
    w.b = item / my_nw;
    item -= w.b * my_nw;
  }
  const int flat = a.win_start[a.my_wg] + item;
  w.ii = flat / a.nWw;
  w.jj = flat - w.ii * a.nWw;
  return w;
}

// Row tables of one window: {row in the owner's buffer (-1: no such token), peer slot | region << 8} per token. Thread
// `tid` < NPAD writes its token's entry.
__device__ __forceinline__ void wa_table(const WindowAttnArgs& a, const Geo& geo, const WaItem& w, int ti, int tj, int2* entry) {
  if (a.n_wg * a.sp * a.tp == 1 && !TB_DEBUG_BOUNDS) {
    // one rank owns every token: a shifted token lies in its own window or the next one per axis
    int ri = ti + a.sh, wi = w.ii, rj = tj + a.sw, wj = w.jj;
    if (ri >= a.wh) {
      ri -= a.wh;
      wi = wi + 1 == a.nWh ? 0 : wi + 1;
    }
    if (rj >= a.ww) {
      rj -= a.ww;
      wj = wj + 1 == a.nWw ? 0 : wj + 1;
    }
    const int rh = (a.sh > 0 && w.ii == a.nWh - 1) ? (ti < a.wh - a.sh ? 1 : 2) : 0;
    const int rw = (a.sw > 0 && w.jj == a.nWw - 1) ? (tj < a.ww - a.sw ? 1 : 2) : 0;
    *entry = make_int2(((w.b * a.nWh + wi) * a.nWw + wj) * geo.N + ri * a.ww + rj, (rh * 3 + rw) << 8);
  } else {
    const Home h = locate_ij(a, geo, w.b, w.ii, w.jj, ti, tj);
    *entry = make_int2(static_cast<int>(h.row), h.slot | (h.region << 8));
  }
}

// Row-wise copies of one window into a stage: VPR lanes per row move its 16-byte vectors of q, k, v [and dO].
template <class Cfg, bool BWD>
__device__ __forceinline__ void wa_gather(const WindowAttnArgs& a, const int2* tab, uint32_t stage, int ch0, int tid, int q0, int q1) {
  constexpr int VPR = Cfg::G / 8, RPP = Cfg::THREADS / VPR, NPAD = Cfg::MAT / Cfg::PITCH;
  static_assert(Cfg::THREADS % VPR == 0, "lanes per row");
  const int v = tid % VPR;
#pragma unroll
  for (int i = 0; i < (NPAD + RPP - 1) / RPP; ++i) {
    const int r = tid / VPR + i * RPP;
    if (NPAD % RPP != 0 && r >= NPAD) break;
    const int2 e = tab[r];
    if (e.x < 0) continue;                   // a padding row: zero since the start
    const int slot = e.y & 255;
    const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.qkv[slot]) + static_cast<long long>(e.x) * (3 * a.C) + ch0 + v * 8;
    const uint32_t dst = stage + (r * Cfg::PITCH + v * 8) * 2;
    if (BWD || (r >= q0 && r < q1)) cp_async16(dst, src);
    cp_async16(dst + Cfg::MAT * 2, src + a.C);
    cp_async16(dst + Cfg::MAT * 4, src + 2 * a.C);
    if (BWD)
      cp_async16(dst + Cfg::MAT * 6,
                 static_cast<const __nv_bfloat16*>(a.dout[slot]) + static_cast<long long>(e.x) * a.C + ch0 + v * 8);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// 16 rows x CH channels staged in shared memory (pitch in elements) to the rows' home buffers.
template <int CH>
__device__ __forceinline__ void wa_store(void* const* bases, long long ld, int col, const __nv_bfloat16* src, int pitch,
                                         const int2* tab, int row0, int lane, int q0, int q1) {
  constexpr int VPR = CH / 8;
#pragma unroll
  for (int i = 0; i < (16 * VPR + 31) / 32; ++i) {
    const int idx = lane + 32 * i;
    const int r = idx / VPR, v = idx % VPR;
    if (row0 + r >= q0 && row0 + r < q1) {
      const int2 e = tab[row0 + r];
      __nv_bfloat16* o = static_cast<__nv_bfloat16*>(bases[e.y & 255]) + static_cast<long long>(e.x) * ld + col + v * 8;
      *reinterpret_cast<uint4*>(o) = *reinterpret_cast<const uint4*>(src + r * pitch + v * 8);
    }
  }
}

// Pairs of neighbouring columns go through the two-wide fp32 instructions (one issue slot for both, same rounding).
__device__ __forceinline__ f32x2 wa_pair(const float (&v)[4], int i) { return f2_pack(v[i], v[i + 1]); }
__device__ __forceinline__ void wa_set(float (&v)[4], int i, f32x2 x) { f2_unpack(x, v[i], v[i + 1]); }

// Scores of a 16-row block: s <- s * scale + bias, base-2 domain, and the row maxima of this thread's columns.
// `tb` is the head's table in shared memory, pre-multiplied by log2(e). The table index of (query r, key c) is
// cofs(r) - cofs(c) + rel0 with cofs(t) = (t / ww) (2 ww - 1) + t % ww. For windows 8 (12) wide the columns of a thread
// repeat every 1 (3) blocks of 8, so an index is one of 1 (3) per-thread bases plus a compile-time constant; other
// widths read cofs from shared memory.
// A warp's block is MT tiles of 16 rows (rows r0 + 16 t and r0 + 16 t + 8 of this thread).
//
// MASK: of a window that the shifted frame's last row or column cuts; the mask is added where query and key lie in different regions (`tab`).
// Without the pairs and the constant offsets that took three times as long per element, and the blocks that met such a window finished last.
// Us, forward and backward, so / this: 180 windows of 8 x 12, 12 heads of 16 channels 24.4 / 15.7 and 51 / 44; 2176 of 8 x 8, 12 heads
// of 32 93.5 / 87 and 235 / 228. (The mask over the scale as what the products are added to, 16.3 and 44.5, 88.8 and 227, sums a
// masked product at the mask's magnitude, which rounds HD / 16 times where this rounds once: gradient of the bias table where such
// products decide 5.2e-6 off instead of 2.0e-6. 32 channels in windows of 8 x 12 spill more here: forward 11.5 / 12.1.)
template <int NPAD, int WW, int MT, bool MASK>
__device__ __forceinline__ void wa_scores(float (&s)[MT][NPAD / 8][4], float scale2, const float* tb, int rel0, const int* cofs, const int2* tab,
                                          int r0, int tq, int N, float (&mx)[MT][2]) {
  auto mask = [&](float (&v)[4], int t, int nb) {
    if constexpr (MASK) {
      const int e0 = tab[nb * 8 + tq * 2].y, e1 = tab[nb * 8 + tq * 2 + 1].y;      // regions in bits 8 and up
      const int f0 = tab[r0 + 16 * t].y, f1 = tab[r0 + 16 * t + 8].y;
      if ((e0 ^ f0) >> 8) v[0] += -100.f * WA_LOG2E;
      if ((e1 ^ f0) >> 8) v[1] += -100.f * WA_LOG2E;
      if ((e0 ^ f1) >> 8) v[2] += -100.f * WA_LOG2E;
      if ((e1 ^ f1) >> 8) v[3] += -100.f * WA_LOG2E;
    }
  };
  if constexpr (WW == 8) {
    // row r0 + 8 is the next window row, same column: its bias at key block nb is row r0's at block nb - 1, and so on for the rows below
    const float* p = tb + ((r0 >> 3) * 15 + (r0 & 7) - 2 * tq + rel0);
    float b[2 * MT][2];      // this key block's bias of rows r0, r0 + 8, ...
#pragma unroll
    for (int i = 1; i < 2 * MT; ++i) b[i][0] = p[15 * i], b[i][1] = p[15 * i - 1];
#pragma unroll
    for (int nb = 0; nb < NPAD / 8; ++nb) {
      b[0][0] = p[-15 * nb];
      b[0][1] = p[-15 * nb - 1];
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          wa_set(s[t][nb], 2 * h, f2_fma(wa_pair(s[t][nb], 2 * h), f2_both(scale2), f2_pack(b[2 * t + h][0], b[2 * t + h][1])));
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        mask(s[t][nb], t, nb);
#pragma unroll
        for (int h = 0; h < 2; ++h) mx[t][h] = fmaxf(mx[t][h], fmaxf(s[t][nb][2 * h], s[t][nb][2 * h + 1]));
      }
#pragma unroll
      for (int i = 2 * MT - 1; i > 0; --i) b[i][0] = b[i - 1][0], b[i][1] = b[i - 1][1];
    }
  } else if constexpr (WW == 12) {
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const int ra = r0 + 16 * t;
      const int ro0 = cofs[ra] + rel0, dr = cofs[ra + 8] - cofs[ra];
      // columns 8 m + 2 tq of the first three blocks, m = 0, 1, 2; later blocks are whole window rows (2 per 3 blocks) on
      const float* p[3];
      p[0] = tb + ro0 - 2 * tq;
      p[1] = tb + ro0 - (tq < 2 ? 8 + 2 * tq : 23 + 2 * tq - 4);
      p[2] = tb + ro0 - (23 + 4 + 2 * tq);
#pragma unroll
      for (int nb = 0; nb < NPAD / 8; ++nb) {
        const float* c = p[nb % 3] - (nb / 3) * 46;
        wa_set(s[t][nb], 0, f2_fma(wa_pair(s[t][nb], 0), f2_both(scale2), f2_pack(c[0], c[-1])));
        wa_set(s[t][nb], 2, f2_fma(wa_pair(s[t][nb], 2), f2_both(scale2), f2_pack(c[dr], c[dr - 1])));
        mask(s[t][nb], t, nb);
        mx[t][0] = fmaxf(mx[t][0], fmaxf(s[t][nb][0], s[t][nb][1]));
        mx[t][1] = fmaxf(mx[t][1], fmaxf(s[t][nb][2], s[t][nb][3]));
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const float *t0 = tb + cofs[r0 + 16 * t] + rel0, *t1 = tb + cofs[r0 + 16 * t + 8] + rel0;
#pragma unroll
      for (int nb = 0; nb < NPAD / 8; ++nb) {
        const int2 co = *reinterpret_cast<const int2*>(cofs + nb * 8 + tq * 2);
        s[t][nb][0] = fmaf(s[t][nb][0], scale2, t0[-co.x]);
        s[t][nb][1] = fmaf(s[t][nb][1], scale2, t0[-co.y]);
        s[t][nb][2] = fmaf(s[t][nb][2], scale2, t1[-co.x]);
        s[t][nb][3] = fmaf(s[t][nb][3], scale2, t1[-co.y]);
        mask(s[t][nb], t, nb);
        if (nb * 8 + 8 > N) {      // padding columns: their scores are lowest, their probabilities zero
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (nb * 8 + tq * 2 + (k & 1) >= N) s[t][nb][k] = -1e30f;
        }
        mx[t][0] = fmaxf(mx[t][0], fmaxf(s[t][nb][0], s[t][nb][1]));
        mx[t][1] = fmaxf(mx[t][1], fmaxf(s[t][nb][2], s[t][nb][3]));
      }
    }
  }
}

template <int NPAD, int MT>
__device__ __forceinline__ void wa_zero(float (&d)[MT][NPAD / 8][4]) {
#pragma unroll
  for (int t = 0; t < MT; ++t)
#pragma unroll
    for (int nb = 0; nb < NPAD / 8; ++nb)
#pragma unroll
      for (int k = 0; k < 4; ++k) d[t][nb][k] = 0.f;
}

// d[t] += A(16 rows at `arow` + 16 t, HD channels) * B(NPAD rows at `bmat`)^T, both row-major bf16 in shared memory
template <int HD, int NPAD, int PITCH, int MT>
__device__ __forceinline__ void wa_mma_nt(float (&d)[MT][NPAD / 8][4], const __nv_bfloat16* arow, const __nv_bfloat16* bmat, int lane) {
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    uint32_t af[MT][4];
#pragma unroll
    for (int t = 0; t < MT; ++t) ldsm_x4(af[t], arow + (16 * t + (lane & 15)) * PITCH + kk * 16 + (lane >> 4) * 8);
#pragma unroll
    for (int nb = 0; nb < NPAD / 8; nb += 2) {
      uint32_t bf[4];
      ldsm_x4(bf, bmat + (nb * 8 + (lane & 7) + (lane >> 4) * 8) * PITCH + kk * 16 + ((lane >> 3) & 1) * 8);
      const uint32_t b0[2] = {bf[0], bf[1]}, b1[2] = {bf[2], bf[3]};
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        mma_bf16_16816(d[t][nb], af[t], b0);
        mma_bf16_16816(d[t][nb + 1], af[t], b1);
      }
    }
  }
}

// o[t] = P[t] (16 x NPAD, fp32 accumulator layout, rounded to bf16) * B (NPAD rows, HD channels, row-major in shared memory)
template <int HD, int NPAD, int PITCH, int MT>
__device__ __forceinline__ void wa_mma_pn(float (&o)[MT][HD / 8][4], const float (&p)[MT][NPAD / 8][4], const __nv_bfloat16* bmat, int lane) {
#pragma unroll
  for (int t = 0; t < MT; ++t)
#pragma unroll
    for (int nb = 0; nb < HD / 8; ++nb)
#pragma unroll
      for (int k = 0; k < 4; ++k) o[t][nb][k] = 0.f;
#pragma unroll
  for (int j = 0; j < NPAD / 16; ++j) {
    uint32_t pf[MT][4];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      pf[t][0] = pack_bf16x2(p[t][2 * j][0], p[t][2 * j][1]);
      pf[t][1] = pack_bf16x2(p[t][2 * j][2], p[t][2 * j][3]);
      pf[t][2] = pack_bf16x2(p[t][2 * j + 1][0], p[t][2 * j + 1][1]);
      pf[t][3] = pack_bf16x2(p[t][2 * j + 1][2], p[t][2 * j + 1][3]);
    }
#pragma unroll
    for (int nb = 0; nb < HD / 8; nb += 2) {
      uint32_t bf[4];
      ldsm_x4_t(bf, bmat + (j * 16 + (lane & 15)) * PITCH + nb * 8 + (lane >> 4) * 8);
      const uint32_t b0[2] = {bf[0], bf[1]}, b1[2] = {bf[2], bf[3]};
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        mma_bf16_16816(o[t][nb], pf[t], b0);
        mma_bf16_16816(o[t][nb + 1], pf[t], b1);
      }
    }
  }
}

// Softmax numerators of the block (in place) and the reciprocal row sums.
template <int NPAD>
__device__ __forceinline__ void wa_softmax(float (&s)[NPAD / 8][4], float mx0, float mx1, float& inv0, float& inv1) {
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
  f32x2 t0 = f2_both(0.f), t1 = f2_both(0.f);
#pragma unroll
  for (int nb = 0; nb < NPAD / 8; ++nb) {
    wa_set(s[nb], 0, f2_add(wa_pair(s[nb], 0), f2_both(-mx0)));
    wa_set(s[nb], 2, f2_add(wa_pair(s[nb], 2), f2_both(-mx1)));
#pragma unroll
    for (int k = 0; k < 4; ++k) s[nb][k] = exp2f(s[nb][k]);
    t0 = f2_add(t0, wa_pair(s[nb], 0));
    t1 = f2_add(t1, wa_pair(s[nb], 2));
  }
  float sum0, sum1, odd0, odd1;
  f2_unpack(t0, sum0, odd0);
  f2_unpack(t1, sum1, odd1);
  sum0 += odd0;
  sum1 += odd1;
  sum0 += __shfl_xor_sync(0xffffffffu, sum0, 1);
  sum0 += __shfl_xor_sync(0xffffffffu, sum0, 2);
  sum1 += __shfl_xor_sync(0xffffffffu, sum1, 1);
  sum1 += __shfl_xor_sync(0xffffffffu, sum1, 2);
  inv0 = 1.f / sum0;
  inv1 = 1.f / sum1;
}

// A warp's 16 x W accumulator tile, scaled per row (r0 = gq and r0 + 8), to bf16 rows in shared memory.
template <int W>
__device__ __forceinline__ void wa_stage(__nv_bfloat16* dst, int pitch, const float (&o)[W / 8][4], float f0, float f1, int lane) {
  __nv_bfloat16* at = dst + (lane & 15) * pitch + (lane >> 4) * 8;
#pragma unroll
  for (int nb = 0; nb < W / 8; nb += 2)
    stsm_x4(at + nb * 8, pack_bf16x2(o[nb][0] * f0, o[nb][1] * f0), pack_bf16x2(o[nb][2] * f1, o[nb][3] * f1),
            pack_bf16x2(o[nb + 1][0] * f0, o[nb + 1][1] * f0), pack_bf16x2(o[nb + 1][2] * f1, o[nb + 1][3] * f1));
}
// The same where rows may be padding, which stays as it is (K and V rows of later windows must find zeros there).
template <int W>
__device__ __forceinline__ void wa_stage_rows(__nv_bfloat16* dst, int pitch, const float (&o)[W / 8][4], float f, int lane, bool ok0, bool ok1) {
  const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
  for (int nb = 0; nb < W / 8; ++nb) {
    if (ok0) *reinterpret_cast<uint32_t*>(dst + gq * pitch + nb * 8 + tq * 2) = pack_bf16x2(o[nb][0] * f, o[nb][1] * f);
    if (ok1) *reinterpret_cast<uint32_t*>(dst + (gq + 8) * pitch + nb * 8 + tq * 2) = pack_bf16x2(o[nb][2] * f, o[nb][3] * f);
  }
}

__host__ __device__ __forceinline__ bool one_rank(const WindowAttnArgs& a) { return a.n_wg * a.sp * a.tp == 1; }

template <int HD, int NPAD, int HPC, int WW, bool BWD>
__global__ void __launch_bounds__(WaCfg<HD, NPAD, HPC, BWD>::THREADS, (WaCfg<HD, NPAD, HPC, BWD>::MIN_CTAS))
    window_attn_kernel(const __grid_constant__ WindowAttnArgs a) {
  using Cfg = WaCfg<HD, NPAD, HPC, BWD>;
  static_assert(!BWD || HPC == 1, "the backward kernel keeps one head's bias-gradient sums");
  constexpr int G = Cfg::G, PITCH = Cfg::PITCH, PP = Cfg::PP, STAGES = Cfg::STAGES, NB = NPAD / 8, MT = Cfg::MT;
  extern __shared__ __align__(16) uint8_t smem[];
  __nv_bfloat16* stages = reinterpret_cast<__nv_bfloat16*>(smem);
  __nv_bfloat16* Ps = stages + STAGES * Cfg::STAGE;             // backward: [NPAD][PP] each
  __nv_bfloat16* dSs = Ps + Cfg::STASH / 2;
  __nv_bfloat16* dQs = dSs + Cfg::STASH / 2;                     // backward, 128-channel heads
  float* acc_s = reinterpret_cast<float*>(dQs + Cfg::DQ);        // backward: [NB / 1][THREADS][4] bias-gradient sums
  int2* tabs = reinterpret_cast<int2*>(acc_s + Cfg::ACC);        // [3][NPAD]
  int* cofs = reinterpret_cast<int*>(tabs + 3 * NPAD);           // [NPAD]
  float* bias_s = reinterpret_cast<float*>(cofs + NPAD);         // [HPC][nrel], times log2(e)

  Geo geo;
  geo.N = a.wh * a.ww;
  geo.nrel = (2 * a.wh - 1) * (2 * a.ww - 1);
  geo.Hg = a.nWh * a.wh;
  geo.Wg = a.nWw * a.ww;
  const int N = geo.N;
  const int rel0 = (a.wh - 1) * (2 * a.ww - 1) + (a.ww - 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int head0 = blockIdx.y * HPC, ch0 = blockIdx.y * G;
  const bool use_bias = a.bias_table != nullptr;
  const bool bias_grad = BWD && use_bias && a.dbias_table != nullptr;
  const int my_nw = a.win_start[a.my_wg + 1] - a.win_start[a.my_wg];
  const int items = a.B * my_nw;
  const int q0 = a.my_sp * a.shardN;
  const int q1 = min(N, q0 + a.shardN);
  const float scale2 = a.scale * WA_LOG2E;
  const int ti = tid / a.ww, tj = tid % a.ww;                    // token `tid` of a window

  if (tid < NPAD) {
    cofs[tid] = tid < N ? ti * (2 * a.ww - 1) + tj : 0;      // (a padding token's bias is read, from inside the table, and not used)
    if (tid >= N)
      for (int k = 0; k < 3; ++k) tabs[k * NPAD + tid] = make_int2(-1, 15 << 8);
  }
  if (N < NPAD)   // padding rows are never written again
    for (int i = tid; i < STAGES * Cfg::MATS * (NPAD - N) * (PITCH / 2); i += Cfg::THREADS) {
      const int m = i / ((NPAD - N) * (PITCH / 2)), o = i % ((NPAD - N) * (PITCH / 2));
      reinterpret_cast<uint32_t*>(stages + m * Cfg::MAT + N * PITCH)[o] = 0u;
    }
  for (int i = tid; i < Cfg::ACC; i += Cfg::THREADS) acc_s[i] = 0.f;

  float acc[(BWD && Cfg::ACC_REGS) ? NB : 1][4];
#pragma unroll
  for (int nb = 0; nb < (BWD && Cfg::ACC_REGS ? NB : 1); ++nb)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[nb][k] = 0.f;

  const int step = gridDim.x;
  const int my_head = MT == 1 ? 0 : warp / (NPAD / (16 * MT));
  const int row0 = (MT == 1 ? warp : warp % (NPAD / (16 * MT))) * 16 * MT, r0 = row0 + gq, r1 = r0 + 8;
  const float own0 = (r0 >= q0 && r0 < q1) ? 1.f : 0.f, own1 = (r1 >= q0 && r1 < q1) ? 1.f : 0.f;   // this rank's query rows

  WaItem next = wa_item(a, blockIdx.x, my_nw);      // the item whose table was written last
  WaItem cur = next;
  if (tid < N) wa_table(a, geo, next, ti, tj, tabs + tid);
  __syncthreads();
  if (one_rank(a)) chain_begin(); else chain_wait();        // global memory is touched from here on
  if (STAGES == 2) wa_gather<Cfg, BWD>(a, tabs, smem_u32(stages), ch0, tid, q0, q1);
  for (int i = tid; i < HPC * geo.nrel; i += Cfg::THREADS) {
    const int h = i / geo.nrel, r = i % geo.nrel;
    bias_s[i] = use_bias ? a.bias_table[r * a.num_heads + head0 + h] * WA_LOG2E : 0.f;
  }      // (seen after the barrier that opens the first window)
  if (static_cast<int>(blockIdx.x) + step < items) {
    next = wa_item(a, blockIdx.x + step, my_nw);
    if (tid < N) wa_table(a, geo, next, ti, tj, tabs + NPAD + tid);
  }

  int slot = 0, buf = 0;
  for (int item = blockIdx.x; item < items; item += step) {
    const int2* tab = tabs + slot * NPAD;
    const int slot1 = slot == 2 ? 0 : slot + 1, slot2 = slot1 == 2 ? 0 : slot1 + 1;
    __nv_bfloat16* Qs = stages + buf * Cfg::STAGE;
    __nv_bfloat16 *Ks = Qs + Cfg::MAT, *Vs = Ks + Cfg::MAT, *dOs = Vs + Cfg::MAT;
    if (STAGES == 1) {
      __syncthreads();          // the previous window has been consumed, this window's table is visible
      wa_gather<Cfg, BWD>(a, tab, smem_u32(Qs), ch0, tid, q0, q1);
    }
    cp_async_wait_all();
    __syncthreads();            // this window's rows are visible; with two stages the previous one has been consumed
    const WaItem mine = cur;
    cur = next;
    if (STAGES == 2 && item + step < items)
      wa_gather<Cfg, BWD>(a, tabs + slot1 * NPAD, smem_u32(stages + (buf ^ 1) * Cfg::STAGE), ch0, tid, q0, q1);
    if (item + 2 * step < items) {
      next = wa_item(a, item + 2 * step, my_nw);
      if (tid < N) wa_table(a, geo, next, ti, tj, tabs + slot2 * NPAD + tid);
    }
    const bool masked = a.use_mask && ((a.sh > 0 && mine.ii == a.nWh - 1) || (a.sw > 0 && mine.jj == a.nWw - 1));

    if constexpr (!BWD) {
      if (row0 < q1 && row0 + 16 * MT > q0) {
#pragma unroll 1
        for (int hh = MT == 1 ? 0 : my_head; hh < (MT == 1 ? HPC : my_head + 1); ++hh) {
          float s[MT][NB][4];
          wa_zero<NPAD, MT>(s);
          wa_mma_nt<HD, NPAD, PITCH, MT>(s, Qs + row0 * PITCH + hh * HD, Ks + hh * HD, lane);
          float mx[MT][2], inv[MT][2];
#pragma unroll
          for (int t = 0; t < MT; ++t) mx[t][0] = mx[t][1] = -1e30f;
          if (masked) wa_scores<NPAD, WW, MT, true>(s, scale2, bias_s + hh * geo.nrel, rel0, cofs, tab, r0, tq, N, mx);
          else wa_scores<NPAD, WW, MT, false>(s, scale2, bias_s + hh * geo.nrel, rel0, cofs, tab, r0, tq, N, mx);
#pragma unroll
          for (int t = 0; t < MT; ++t) wa_softmax<NPAD>(s[t], mx[t][0], mx[t][1], inv[t][0], inv[t][1]);
          // O = P V with the numerators as P, the row normalisation applied to the (smaller) output; staged over this
          // warp's own Q rows, which no other warp reads
          float o[MT][HD / 8][4];
          wa_mma_pn<HD, NPAD, PITCH, MT>(o, s, Vs + hh * HD, lane);
          __syncwarp();
#pragma unroll
          for (int t = 0; t < MT; ++t)
            wa_stage<HD>(Qs + (row0 + 16 * t) * PITCH + hh * HD, PITCH, o[t], inv[t][0], inv[t][1], lane);
        }
        __syncwarp();
        if constexpr (MT == 1) {
          wa_store<G>(a.out, a.C, ch0, Qs + row0 * PITCH, PITCH, tab, row0, lane, q0, q1);
        } else {
#pragma unroll
          for (int t = 0; t < MT; ++t)
            wa_store<HD>(a.out, a.C, ch0 + my_head * HD, Qs + (row0 + 16 * t) * PITCH + my_head * HD, PITCH, tab, row0 + 16 * t, lane, q0, q1);
        }
      }
    } else {
      // ---- phase 1, a warp per 16 query rows: P, dS, dQ
      if (row0 < N) {
        float s1[1][NB][4], dp1[1][NB][4], mx[1][2] = {{-1e30f, -1e30f}}, inv0, inv1;
        float(&s)[NB][4] = s1[0], (&dp)[NB][4] = dp1[0];
        wa_zero<NPAD, 1>(s1);
        wa_mma_nt<HD, NPAD, PITCH, 1>(s1, Qs + row0 * PITCH, Ks, lane);
        // (128 channels: with both forms of constant offsets the compiler spills, 655 / 710 us; WW = 0 reads them, and spares registers)
        if (masked) wa_scores<NPAD, HD < 128 ? WW : 0, 1, true>(s1, scale2, bias_s, rel0, cofs, tab, r0, tq, N, mx);
        else wa_scores<NPAD, WW, 1, false>(s1, scale2, bias_s, rel0, cofs, tab, r0, tq, N, mx);
        wa_softmax<NPAD>(s, mx[0][0], mx[0][1], inv0, inv1);
        wa_zero<NPAD, 1>(dp1);
        wa_mma_nt<HD, NPAD, PITCH, 1>(dp1, dOs + row0 * PITCH, Vs, lane);        // dP = dO V^T
        f32x2 e0 = f2_both(0.f), e1 = f2_both(0.f);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          wa_set(s[nb], 0, f2_mul(wa_pair(s[nb], 0), f2_both(inv0)));
          wa_set(s[nb], 2, f2_mul(wa_pair(s[nb], 2), f2_both(inv1)));
          e0 = f2_fma(wa_pair(s[nb], 0), wa_pair(dp[nb], 0), e0);
          e1 = f2_fma(wa_pair(s[nb], 2), wa_pair(dp[nb], 2), e1);
        }
        float d0, d1, odd0, odd1;
        f2_unpack(e0, d0, odd0);
        f2_unpack(e1, d1, odd1);
        d0 += odd0;
        d1 += odd1;
        d0 += __shfl_xor_sync(0xffffffffu, d0, 1);
        d0 += __shfl_xor_sync(0xffffffffu, d0, 2);
        d1 += __shfl_xor_sync(0xffffffffu, d1, 1);
        d1 += __shfl_xor_sync(0xffffffffu, d1, 2);
        // dS = P (dP - rowsum(P dP)); its sum over the windows is the gradient of the bias
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          wa_set(dp[nb], 0, f2_mul(wa_pair(s[nb], 0), f2_add(wa_pair(dp[nb], 0), f2_both(-d0))));
          wa_set(dp[nb], 2, f2_mul(wa_pair(s[nb], 2), f2_add(wa_pair(dp[nb], 2), f2_both(-d1))));
          if constexpr (Cfg::ACC_REGS) {
            wa_set(acc[nb], 0, f2_fma(wa_pair(dp[nb], 0), f2_both(own0), wa_pair(acc[nb], 0)));
            wa_set(acc[nb], 2, f2_fma(wa_pair(dp[nb], 2), f2_both(own1), wa_pair(acc[nb], 2)));
          } else if (bias_grad) {
            float4* t = reinterpret_cast<float4*>(acc_s) + nb * Cfg::THREADS + tid;
            float4 v = *t;
            v.x = fmaf(dp[nb][0], own0, v.x);
            v.y = fmaf(dp[nb][1], own0, v.y);
            v.z = fmaf(dp[nb][2], own1, v.z);
            v.w = fmaf(dp[nb][3], own1, v.w);
            *t = v;
          }
        }
        {
          float dq1[1][HD / 8][4];
          float(&dq)[HD / 8][4] = dq1[0];
          wa_mma_pn<HD, NPAD, PITCH, 1>(dq1, dp1, Ks, lane);
          // the stash rows of this block were last read before the barrier that opened this window
          __nv_bfloat16* st = Cfg::DQ_IN_STASH ? Ps + row0 * PP : dQs + row0 * PITCH;
          constexpr int stp = Cfg::DQ_IN_STASH ? PP : PITCH;
          wa_stage<HD>(st, stp, dq, a.scale, a.scale, lane);
          __syncwarp();
          wa_store<HD>(a.dqkv, 3LL * a.C, ch0, st, stp, tab, row0, lane, q0, q1);
          __syncwarp();
        }
        if constexpr (HD == 64 && NPAD == 64) {      // (the compiler spills here with the tile stores: 127 us instead of 114)
          wa_stage_rows<NPAD>(Ps + row0 * PP, PP, s, 1.f, lane, true, true);
          wa_stage_rows<NPAD>(dSs + row0 * PP, PP, dp, 1.f, lane, true, true);
        } else {
          wa_stage<NPAD>(Ps + row0 * PP, PP, s, 1.f, 1.f, lane);
          wa_stage<NPAD>(dSs + row0 * PP, PP, dp, 1.f, 1.f, lane);
        }
      }
      __syncthreads();
      // ---- phase 2, a warp per 16 keys: dV = P^T dO, dK = scale dS^T Q. (Half of the warps for dV and half for dK, 32 keys each, read
      // less of dO and Q but measured up to 6 % slower at 64 tokens.) K and V are dead: their rows stage the results. With sequence
      // parallelism every rank of the window recomputes the whole window (cheap) and keeps only the gradients of its own token shard, so no
      // cross-rank reduction of dK / dV is needed.
      const int qblocks = (N + 15) >> 4;
      if (row0 < N) {
        float dv[HD / 8][4], dk[HD / 8][4];
#pragma unroll
        for (int nb = 0; nb < HD / 8; ++nb)
#pragma unroll
          for (int k = 0; k < 4; ++k) dv[nb][k] = dk[nb][k] = 0.f;
#pragma unroll
        for (int j = 0; j < NPAD / 16; ++j) {   // query blocks (contraction); blocks without a token were not stashed
          if (j >= qblocks) break;
          uint32_t pa[4], sa[4];
          const int prow = j * 16 + (lane & 7) + (lane >> 4) * 8;
          const int pcol = row0 + ((lane >> 3) & 1) * 8;
          ldsm_x4_t(pa, Ps + prow * PP + pcol);
          ldsm_x4_t(sa, dSs + prow * PP + pcol);
#pragma unroll
          for (int nb = 0; nb < HD / 8; nb += 2) {
            uint32_t bf[4];
            ldsm_x4_t(bf, dOs + (j * 16 + (lane & 15)) * PITCH + nb * 8 + (lane >> 4) * 8);
            const uint32_t b0[2] = {bf[0], bf[1]}, b1[2] = {bf[2], bf[3]};
            mma_bf16_16816(dv[nb], pa, b0);
            mma_bf16_16816(dv[nb + 1], pa, b1);
            ldsm_x4_t(bf, Qs + (j * 16 + (lane & 15)) * PITCH + nb * 8 + (lane >> 4) * 8);
            const uint32_t c0[2] = {bf[0], bf[1]}, c1[2] = {bf[2], bf[3]};
            mma_bf16_16816(dk[nb], sa, c0);
            mma_bf16_16816(dk[nb + 1], sa, c1);
          }
        }
        if (WW != 0 || N == NPAD) {
          wa_stage<HD>(Ks + row0 * PITCH, PITCH, dk, a.scale, a.scale, lane);
          wa_stage<HD>(Vs + row0 * PITCH, PITCH, dv, 1.f, 1.f, lane);
        } else {
          wa_stage_rows<HD>(Ks + row0 * PITCH, PITCH, dk, a.scale, lane, r0 < N, r1 < N);
          wa_stage_rows<HD>(Vs + row0 * PITCH, PITCH, dv, 1.f, lane, r0 < N, r1 < N);
        }
        __syncwarp();
        wa_store<HD>(a.dqkv, 3LL * a.C, a.C + ch0, Ks + row0 * PITCH, PITCH, tab, row0, lane, q0, q1);
        wa_store<HD>(a.dqkv, 3LL * a.C, 2 * a.C + ch0, Vs + row0 * PITCH, PITCH, tab, row0, lane, q0, q1);
      }
    }
    slot = slot1;
    if (STAGES == 2) buf ^= 1;
  }

  if (bias_grad) {
    // Spread the sums out as an [N][NPAD + 1] matrix over the operand stages, then fold its diagonals into the table: entry
    // (di, dj) collects the pairs with query - key = (di, dj).
    float* D = reinterpret_cast<float*>(smem);
    static_assert(!BWD || static_cast<size_t>(NPAD) * (NPAD + 1) * 4 <= static_cast<size_t>(STAGES * Cfg::STAGE + Cfg::STASH) * 2,
                  "scratch of the bias-gradient fold");
    __syncthreads();
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float4 v;
      if constexpr (BWD && Cfg::ACC_REGS) v = make_float4(acc[nb][0], acc[nb][1], acc[nb][2], acc[nb][3]);
      else v = reinterpret_cast<const float4*>(acc_s)[nb * Cfg::THREADS + tid];
      const int col = nb * 8 + tq * 2;
      D[r0 * (NPAD + 1) + col] = v.x;
      D[r0 * (NPAD + 1) + col + 1] = v.y;
      D[r1 * (NPAD + 1) + col] = v.z;
      D[r1 * (NPAD + 1) + col + 1] = v.w;
    }
    __syncthreads();
    const int ndj = 2 * a.ww - 1;
    for (int i = tid; i < geo.nrel; i += Cfg::THREADS) {
      const int di = i / ndj - (a.wh - 1), dj = i % ndj - (a.ww - 1);
      float t = 0.f;
      for (int y = max(0, di); y < min(a.wh, a.wh + di); ++y)
        for (int x = max(0, dj); x < min(a.ww, a.ww + dj); ++x)
          t += D[(y * a.ww + x) * (NPAD + 1) + (y - di) * a.ww + x - dj];
      atomicAdd(&a.dbias_table[i * a.num_heads + head0], t);
    }
  }
}

template <int HD, int NPAD, int HPC, int WW, bool BWD>
int launch(WindowAttnArgs a, cudaStream_t stream) {
  using Cfg = WaCfg<HD, NPAD, HPC, BWD>;
  const int nrel = (2 * a.wh - 1) * (2 * a.ww - 1);
  const size_t sb = Cfg::bytes(nrel);
  if (sb > 227 * 1024) return -20;
  auto kernel = window_attn_kernel<HD, NPAD, HPC, WW, BWD>;
  static SharedLimit limit;
  if (limit.raise(reinterpret_cast<const void*>(kernel), 227 * 1024) != cudaSuccess) return -21;
  // resident CTAs per SM for the last shared-memory size seen (one word, so that threads read a matching pair)
  static std::atomic<unsigned long long> known{0};
  unsigned long long k = known.load(std::memory_order_relaxed);
  if ((k >> 8) != sb) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, Cfg::THREADS, sb) != cudaSuccess || occ < 1) occ = 1;
    k = (static_cast<unsigned long long>(sb) << 8) | static_cast<unsigned long long>(occ);
    known.store(k, std::memory_order_relaxed);
  }
  const int occupancy = static_cast<int>(k & 255);
  const int my_nw = a.win_start[a.my_wg + 1] - a.win_start[a.my_wg];
  const int items = a.B * my_nw;
  if (items <= 0) return 0;
  a.heads_per_cta = HPC;
  const int groups = a.num_heads / HPC;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int gx = sms * occupancy / groups;             // one resident wave: a CTA of a second wave would repeat the set-up
  if (gx < 1) gx = 1;
  if (gx > items) gx = items;
  // (with peers a neighbour's flags order the buffers: launched plainly)
  if (one_rank(a)) launch_chained(kernel, dim3(gx, groups), dim3(Cfg::THREADS), sb, stream, a);
  else kernel<<<dim3(gx, groups), Cfg::THREADS, sb, stream>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -22;
}

template <int HD, int NPAD, bool BWD>
int launch_hd(const WindowAttnArgs& a, cudaStream_t stream) {
  // Forward: 64 channels per CTA (128-byte row segments) where the head count allows it, so that a window's set-up is
  // shared by several heads. Backward: one head, whose bias-gradient sums stay in registers.
  constexpr int HPC = (BWD || HD >= 64) ? 1 : 2;
  const bool grouped = HPC > 1 && a.num_heads % HPC == 0;
#define TB_WA_WIDTH(WW_)                                                                       \
  return grouped ? launch<HD, NPAD, HPC, WW_, BWD>(a, stream) : launch<HD, NPAD, 1, WW_, BWD>(a, stream)
  // (the specialised widths serve windows without padding tokens; 96 = 8 x 12 or 12 x 8)
  const bool whole = a.wh * a.ww == NPAD;
  if constexpr (NPAD != 96) { if (whole && a.ww == 8) { TB_WA_WIDTH(8); } }
  if constexpr (NPAD == 96) { if (whole && a.ww == 12) { TB_WA_WIDTH(12); } }
  TB_WA_WIDTH(0);
#undef TB_WA_WIDTH
}

template <bool BWD>
int dispatch(const WindowAttnArgs& a, cudaStream_t stream) {
  const int N = a.wh * a.ww;
  if (a.num_heads <= 0 || a.C % a.num_heads != 0) return -10;
  const int hd = a.C / a.num_heads;
  if (N > 128) return -11;
  if (a.sp < 1 || a.shardN < 1 || a.n_wg < 1 || a.n_wg > 8 || a.n_wg * a.sp > WA_MAX_PEERS) return -12;
  const int npad = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 96 ? 96 : 128));
#define TB_WA_CASE(HD_, NP_) \
  if (hd == HD_ && npad == NP_) return launch_hd<HD_, NP_, BWD>(a, stream);
  TB_WA_CASE(16, 32) TB_WA_CASE(32, 32) TB_WA_CASE(64, 32) TB_WA_CASE(128, 32)
  TB_WA_CASE(16, 64) TB_WA_CASE(32, 64) TB_WA_CASE(64, 64) TB_WA_CASE(128, 64)
  TB_WA_CASE(16, 96) TB_WA_CASE(32, 96) TB_WA_CASE(64, 96) TB_WA_CASE(128, 96)
  TB_WA_CASE(16, 128) TB_WA_CASE(32, 128) TB_WA_CASE(64, 128) TB_WA_CASE(128, 128)
#undef TB_WA_CASE
  return -13;
}

}  // namespace

int window_attn_fwd(const WindowAttnArgs& a, cudaStream_t stream) { return dispatch<false>(a, stream); }
int window_attn_bwd(const WindowAttnArgs& a, cudaStream_t stream) { return dispatch<true>(a, stream); }

}  // namespace tb
