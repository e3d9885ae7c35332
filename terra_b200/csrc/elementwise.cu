// Memory-bound kernels: LayerNorm, GroupNorm(+SiLU), column sums, masked loss, fused AdamW.
// All are single-pass over HBM where the math allows it, with 16-byte vector accesses.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include "chained_launch.cuh"
#include "common.cuh"
#include "host_api.h"
#include "shared_limit.h"

namespace tb {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// += of four neighbouring values, as one vector reduction where they are a whole 16-byte vector
__device__ __forceinline__ void add4(float* to, const float4& v) {
  if ((reinterpret_cast<uintptr_t>(to) & 15u) == 0) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
  } else {
    atomicAdd(to, v.x);
    atomicAdd(to + 1, v.y);
    atomicAdd(to + 2, v.z);
    atomicAdd(to + 3, v.w);
  }
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 x = unpack_bf16x2(w[k]);
    f[2 * k] = x.x;
    f[2 * k + 1] = x.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

__device__ __forceinline__ f32x2 f2_of_bf16x2(uint32_t v) {
  const float2 f = unpack_bf16x2(v);
  return f2_pack(f.x, f.y);
}

// A thread's own 16-byte vectors on their way through shared memory: K tensors, S steps ahead, read two steps at a time (instructions of
// one issue between those of the other). What kernels over HBM lack beside bandwidth is loads in flight: held in registers, a round's loads
// are issued, waited for and used in turn, while cp.async fetches the next rounds meanwhile and costs no register. Every thread reads only
// what it fetched, so there is no barrier.
template <int K, int S>
struct LaneRing {
  static_assert(S % 2 == 0 && S >= 4, "rounds of two steps");
  uint32_t at, stride;      // this thread's slot; bytes between slots
  int s = 0;                // the step to be read next
  static constexpr int bytes(int threads) { return K * S * 16 * threads; }
  __device__ __forceinline__ LaneRing(void* smem, int thread, int threads) : at(smem_u32(smem) + thread * 16), stride(threads * 16) {}
  __device__ __forceinline__ void put(int slot, int k, const void* src) const {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + (slot * K + k) * stride), "l"(src) : "memory");
  }
  // the vectors of round `p`, two pixels `by` apart, into the slots read last (or, at the start, slots `slot` and `slot` + 1)
  template <class Src>
  __device__ __forceinline__ void fetch(int slot, long long p, long long by, long long end, long long pitch, const Src* const* src) const {
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (p + u * by < end) {
#pragma unroll
        for (int k = 0; k < K; ++k)
          put(slot + u, k, src[k] + (p + u * by) * pitch);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  template <class Src>
  __device__ __forceinline__ void start(long long p, long long by, long long end, long long pitch, const Src* const* src) const {
#pragma unroll
    for (int u = 0; u < S; u += 2) fetch(u, p + u * by, by, end, pitch, src);
  }
  __device__ __forceinline__ void wait() const { asm volatile("cp.async.wait_group %0;" ::"n"(S / 2 - 1) : "memory"); }
  __device__ __forceinline__ uint4 read(int u, int k) const {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(at + ((s + u) * K + k) * stride)
                 : "memory");
    return v;
  }
  __device__ __forceinline__ void next() { s = s + 2 == S ? 0 : s + 2; }
};

// ------------------------------------------------------------------------------------------ LayerNorm
// Both kernels are bound by HBM. A row is held in registers by LPR lanes of VPL 16-byte vectors each, so that a warp carries 32 / LPR rows:
// a row of 48 vectors (C = 384) takes 16 lanes x 3 vectors, with no idle lane, where a whole warp would leave half of its lanes idle in the
// second vector. LPR is the largest power of two that divides the row's vectors; rows of more than 3 odd vectors per lane fall back to 32
// lanes with a bounds test. The backward kernel has the next rows on their way through shared memory, reads a row there twice (three blocks
// of four warps then share an SM), works on two columns per instruction and ends in vector reductions without shared-memory atomics, which
// are compare-and-swap loops for floats.
// 139264 x 384, one row per warp -> this: forward 49 -> 37 us (33 us at 6.5 TB/s). Backward with shortcut, us, rows in registers and scalar
// atomics / the rest of this / those ends too: 139264 x 384 79 / 69 / 65 (65 at 6.5 TB/s), 156672 x 1024 262 / 204 / 202 (196), 17280 x 192
// 11.4 / 11.2 / 8.4, 2048 x 384 10.8 / 10.8 / 6.4, 20000 x 512 23.6 / 21.5 / 15.5; with the shortcut's sums 156672 x 1024 380 / 262 / -.
template <int LPR>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int LPR, int VPL, bool EXACT>
__global__ void __launch_bounds__(256, VPL == 1 ? 6 : (VPL == 2 ? 5 : (VPL <= 4 ? 4 : (VPL == 6 ? 3 : 2)))) layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ gamma,
                                                            const __nv_bfloat16* __restrict__ beta,
                                                            __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out,
                                                            float* __restrict__ rstd_out, long long rows, int C,
                                                            float eps) {
  chain_begin();
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  const int nvec = EXACT ? LPR * VPL : C >> 3;
  const long long step = static_cast<long long>(gridDim.x) * (blockDim.x >> 5) * RPW;
  // (the loop is warp-uniform: every lane takes part in the shuffles)
  for (long long base = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * RPW; base < rows;
       base += step) {
    const long long row = base + lane / LPR;
    const bool live = RPW == 1 || row < rows;
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * C);
    float v[VPL][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = sub + i * LPR;
      if (live && (EXACT || vi < nvec)) {
        unpack8(xr[vi], v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[i][j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
      }
    }
    const float mean = group_sum<LPR>(s) / C;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (EXACT || sub + i * LPR < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = v[i][j] - mean;
          q += d * d;
        }
      }
    }
    const float rstd = rsqrtf(group_sum<LPR>(q) / C + eps);
    if (live) {
      uint4* yr = reinterpret_cast<uint4*>(y + row * C);
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = sub + i * LPR;
        if (EXACT || vi < nvec) {
          float g[8], b[8], o[8];
          unpack8(reinterpret_cast<const uint4*>(gamma)[vi], g);
          unpack8(reinterpret_cast<const uint4*>(beta)[vi], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * g[j] + b[j];
          yr[vi] = pack8(o);
        }
      }
      if (sub == 0) {
        mean_out[row] = mean;
        rstd_out[row] = rstd;
      }
    }
  }
}

// Rows in flight per warp of the backward kernel beside the one in its registers, through shared memory by cp.async (see LaneRing; here the
// K = vectors of x, dy and the shortcut's gradient that a lane has of a row).
__host__ __device__ constexpr int ln_bwd_ahead(int vpl) { return vpl <= 4 ? 3 : 2; }

// RES: dres is added. SUMS: dsum += the column sums of dres as well, which passes through here anyway (the bias gradient of the layer before the
// shortcut).
template <int LPR, int VPL, bool EXACT, bool RES, bool SUMS>
__global__ void __launch_bounds__(128, VPL == 1 ? 5 : (VPL == 2 ? 4 : (VPL <= 4 ? 3 : 2))) layernorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                            const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ gamma,
                                                            const float* __restrict__ mean, const float* __restrict__ rstd,
                                                            __nv_bfloat16* __restrict__ dx, float* __restrict__ dgamma,
                                                            float* __restrict__ dbeta, const __nv_bfloat16* __restrict__ dres,
                                                            long long rows, int C, float* __restrict__ dsum) {
  static_assert(RES || !SUMS, "the sums are of dres");
  chain_begin();
  constexpr int RPW = 32 / LPR, K = (RES ? 3 : 2) * VPL, S = ln_bwd_ahead(VPL);
  extern __shared__ __align__(16) float sh[];   // the lanes' rows in flight, then [warp][2 or 3][C] sums
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  const int nvec = EXACT ? LPR * VPL : C >> 3;
  const long long step = static_cast<long long>(gridDim.x) * (blockDim.x >> 5) * RPW;
  // (two columns per instruction)
  f32x2 ag[VPL][4], ab[VPL][4], as[SUMS ? VPL : 1][4];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      ag[i][j] = ab[i][j] = f2_both(0.f);
      if (SUMS) as[i][j] = f2_both(0.f);
    }
  uint4 gq[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int vi = sub + i * LPR;
    if (EXACT || vi < nvec) gq[i] = reinterpret_cast<const uint4*>(gamma)[vi];
  }
  const uint32_t ring = smem_u32(sh) + threadIdx.x * 16;
  constexpr uint32_t SLOT = 128 * 16;
  auto fetch = [&](int slot, long long row) {
    if (row < rows) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = sub + i * LPR;
        if (!EXACT && vi >= nvec) break;
        const __nv_bfloat16* from[3] = {x, dy, dres};
#pragma unroll
        for (int t = 0; t < (RES ? 3 : 2); ++t)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + (slot * K + t * VPL + i) * SLOT), "l"(from[t] + row * C + vi * 8)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto read = [&](int slot, int k) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(ring + (slot * K + k) * SLOT) : "memory");
    return v;
  };
  const long long first = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * RPW;
  int slot = 0;
#pragma unroll
  for (int u = 0; u < S; ++u) fetch(u, first + u * step + lane / LPR);
  float mu_next = 0.f, rs_next = 0.f;
  if (first + lane / LPR < rows) {
    mu_next = mean[first + lane / LPR];
    rs_next = rstd[first + lane / LPR];
  }
#pragma unroll 1
  for (long long base = first; base < rows; base += step) {
    const long long row = base + lane / LPR;
    const bool live = RPW == 1 || row < rows;
    const float mu = mu_next, rs = rs_next;
    if (row + step < rows) {
      mu_next = mean[row + step];
      rs_next = rstd[row + step];
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
    const f32x2 nmu = f2_both(-mu), rs2 = f2_both(rs);
    f32x2 t1 = f2_both(0.f), t2 = f2_both(0.f);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (live && (EXACT || sub + i * LPR < nvec)) {
        const uint4 xq = read(slot, i), dq = read(slot, VPL + i);
        const uint32_t x4[4] = {xq.x, xq.y, xq.z, xq.w}, d4[4] = {dq.x, dq.y, dq.z, dq.w}, g4[4] = {gq[i].x, gq[i].y, gq[i].z, gq[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 xh = f2_mul(f2_add(f2_of_bf16x2(x4[j]), nmu), rs2), d = f2_of_bf16x2(d4[j]), dv = f2_mul(d, f2_of_bf16x2(g4[j]));
          ag[i][j] = f2_fma(d, xh, ag[i][j]);
          ab[i][j] = f2_add(ab[i][j], d);
          t1 = f2_add(t1, dv);
          t2 = f2_fma(dv, xh, t2);
        }
      }
    }
    float s1, s2, odd1, odd2;
    f2_unpack(t1, s1, odd1);
    f2_unpack(t2, s2, odd2);
    s1 = group_sum<LPR>(s1 + odd1) / C;
    s2 = group_sum<LPR>(s2 + odd2) / C;
    if (live) {
      uint4* or_ = reinterpret_cast<uint4*>(dx + row * C);
      const f32x2 n1 = f2_both(-s1), n2 = f2_both(-s2);
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = sub + i * LPR;
        if (EXACT || vi < nvec) {
          // (read again: held in registers the operands would spill, or take a block's place)
          const uint4 xq = read(slot, i), dq = read(slot, VPL + i);
          const uint32_t x4[4] = {xq.x, xq.y, xq.z, xq.w}, d4[4] = {dq.x, dq.y, dq.z, dq.w}, g4[4] = {gq[i].x, gq[i].y, gq[i].z, gq[i].w};
          uint32_t r4[4] = {}, o[4];
          if constexpr (RES) {
            const uint4 rq = read(slot, 2 * VPL + i);
            r4[0] = rq.x, r4[1] = rq.y, r4[2] = rq.z, r4[3] = rq.w;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const f32x2 xh = f2_mul(f2_add(f2_of_bf16x2(x4[j]), nmu), rs2), dv = f2_mul(f2_of_bf16x2(d4[j]), f2_of_bf16x2(g4[j]));
            f32x2 v = f2_mul(rs2, f2_fma(xh, n2, f2_add(dv, n1)));
            if constexpr (RES) {
              const f32x2 r = f2_of_bf16x2(r4[j]);
              v = f2_add(v, r);
              if constexpr (SUMS) as[i][j] = f2_add(as[i][j], r);
            }
            o[j] = f2_to_bf16x2(v);
          }
          or_[vi] = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
    fetch(slot, row + S * step);
    slot = slot + 1 == S ? 0 : slot + 1;
  }
  // the warp's row groups first (lanes sub, sub + LPR, ... hold the same columns), then the block's warps through shared memory where the rows
  // were, then one vector reduction per four columns: the blocks' ends meet on the same addresses, and take turns there
  constexpr int SETS = SUMS ? 3 : 2;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int vi = sub + i * LPR;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      auto fold = [&](f32x2 v, int set) {
        float e0, e1;
        f2_unpack(v, e0, e1);
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) {
          e0 += __shfl_xor_sync(0xffffffffu, e0, o);
          e1 += __shfl_xor_sync(0xffffffffu, e1, o);
        }
        if (lane < LPR && (EXACT || vi < nvec))
          *reinterpret_cast<float2*>(sh + ((threadIdx.x >> 5) * SETS + set) * C + vi * 8 + 2 * j) = make_float2(e0, e1);
      };
      fold(ag[i][j], 0);
      fold(ab[i][j], 1);
      if constexpr (SUMS) fold(as[i][j], 2);
    }
  }
  __syncthreads();
  float* const out[3] = {dgamma, dbeta, dsum};
#pragma unroll
  for (int set = 0; set < SETS; ++set)
    for (int c = threadIdx.x * 4; c < C; c += blockDim.x * 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float4 t = *reinterpret_cast<const float4*>(sh + (w * SETS + set) * C + c);
        v.x += t.x, v.y += t.y, v.z += t.z, v.w += t.w;
      }
      add4(out[set] + c, v);
    }
}

// ------------------------------------------------------------------------------------------ column sums
__global__ void __launch_bounds__(256) colsum_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ partials,
                                                     long long rows, int C, long long ld, int rows_per_block) {
  chain_begin();
  // thread -> one 8-wide column vector; blockDim.y rows in flight. blockDim.x spans the whole row when it has at most
  // 64 vectors (a row is then one contiguous read), otherwise 32 vectors per block column.
  const int nvec = C >> 3;
  const int vi = blockIdx.y * blockDim.x + threadIdx.x;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const long long r0 = static_cast<long long>(blockIdx.x) * rows_per_block;
  const long long r1 = min(rows, r0 + rows_per_block);
  if (vi < nvec) {
    // four independent 16-byte loads in flight per thread
    const long long step = blockDim.y;
    long long r = r0 + threadIdx.y;
    for (; r + 3 * step < r1; r += 4 * step) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = *reinterpret_cast<const uint4*>(x + (r + u * step) * ld + vi * 8);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float f[8];
        unpack8(q[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += f[j];
      }
    }
    for (; r < r1; r += step) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(x + r * ld + vi * 8), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
  }
  extern __shared__ float csh[];              // [blockDim.y][blockDim.x * 8 + 1]
  const int pitch = blockDim.x * 8 + 1;
#pragma unroll
  for (int j = 0; j < 8; ++j) csh[threadIdx.y * pitch + threadIdx.x * 8 + j] = acc[j];
  __syncthreads();
  if (threadIdx.y == 0 && vi < nvec) {
    // one partial row per row block: many blocks adding into the same few hundred addresses serialise in L2
    // (about 80 ns per atomic on one address), so the partials are written out and a second kernel adds them up
    float* prow = partials + static_cast<long long>(blockIdx.x) * C;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float s = 0.f;
      for (int y = 0; y < blockDim.y; ++y) s += csh[y * pitch + threadIdx.x * 8 + j];
      prow[vi * 8 + j] = s;
    }
  }
}

// out[c] += sum over r of partials[r][c]. Block = 32 columns x 32 row lanes.
__global__ void __launch_bounds__(1024) colsum_finish_kernel(const float* __restrict__ partials, float* __restrict__ out,
                                                             int nparts, int C) {
  chain_begin();
  __shared__ float sh[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (c < C)
    for (int r = threadIdx.y; r < nparts; r += 32) s += partials[static_cast<long long>(r) * C + c];
  sh[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += sh[y][threadIdx.x];
    out[c] += t;
  }
}

// ------------------------------------------------------------------------------------------ GroupNorm
// x: [B, HW, C] bf16. Every kernel is one pass over the image, bound by HBM: a block is (column vectors) x (pixels in flight), so a
// thread's column constants (statistics, affine parameters) are loaded once for all of its pixels, and it keeps several independent 16-byte
// loads in flight (LaneRing). blockIdx.y is the sample; the pixel range of a sample is split over blockIdx.x so that the grid is about one
// resident wave. (Before, the apply kernels divided to find every vector's channel and loaded its constants again, and one load per thread
// was in flight. 557056 pixels x 384, before -> now: statistics 98 -> 90 us, apply with shortcut 355 -> 225, backward sums 366 -> 258,
// backward apply 406 -> 264; one copy of the image each way at 6.65 TB/s is 129 us. Then, loads in registers -> in shared memory: apply 228
// -> 212 with the shortcut and 190 -> 143 without, backward sums 192 -> 160, backward apply 264 -> 199; 17280 x 192, with one wave of
// blocks for images that stay in L2: 6.4 -> 4.9, 6.0 -> 4.7, 8.6 -> 8.3, 7.3 -> 6.3, statistics 5.0 -> 4.2.)
//
// Adds a thread's 16 sums (s, q of its eight channels) over the block's threadIdx.y and leaves them in sh[c] and sh[C + c]. Every thread of
// the block takes part. Through a buffer of the block's own rather than by shared-memory atomics, which
// are compare-and-swap loops for floats and met `blockDim.y` at a time on one address: they were half of the time of images of some MB.
__device__ __forceinline__ void gn_block_sums(float* sh, float* buf, const float (&s)[8], const float (&q)[8], int C, int vi) {
  const int bx = blockDim.x, t = threadIdx.y * bx + threadIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    buf[(threadIdx.y * 16 + j) * bx + threadIdx.x] = s[j];
    buf[(threadIdx.y * 16 + 8 + j) * bx + threadIdx.x] = q[j];
  }
  __syncthreads();
  for (int i = t; i < 16 * bx; i += bx * blockDim.y) {
    float sum = 0.f;
    for (int y = 0; y < static_cast<int>(blockDim.y); ++y) sum += buf[y * 16 * bx + i];
    const int j = i / bx, c = (vi - static_cast<int>(threadIdx.x) + i % bx) * 8 + (j & 7);
    if (c < C) sh[(j >> 3) * C + c] = sum;
  }
  __syncthreads();
}

constexpr int GN_AHEAD = 4;      // pixels in flight per thread
using GnStatsRing = LaneRing<1, GN_AHEAD>;
using GnPairRing = LaneRing<2, GN_AHEAD>;

__device__ __forceinline__ void gn_finalize_cell(float* sums, float* stats, int i, float inv_count, float eps) {
  const float mean = __ldcg(sums + 2 * i) * inv_count;
  const float var = fmaxf(__ldcg(sums + 2 * i + 1) * inv_count - mean * mean, 0.f);
  stats[2 * i] = mean;
  stats[2 * i + 1] = rsqrtf(var + eps);
  sums[2 * i] = 0.f;
  sums[2 * i + 1] = 0.f;
}

// Statistics: per-channel sums of the block, folded to groups, two atomics per (block, group). With `stats` the last block to finish turns
// the sums into mean and reciprocal deviation and clears them and the ticket counter. They belong to this launch alone while it runs: shared
// by two launches at once, one would finalize what the other still adds to, and a ticket left at a remainder would spoil every launch after them.
__global__ void __launch_bounds__(512) groupnorm_stats_kernel(const __nv_bfloat16* __restrict__ x,
                                                              float* __restrict__ sums, long long HW, int C, int groups,
                                                              int pix_per_block, float* __restrict__ stats, unsigned int* __restrict__ ticket,
                                                              float inv_count, float eps) {
  chain_begin();
  extern __shared__ __align__(16) float sh[];  // [2][C], then the threads' sums
  const int nvec = C >> 3;
  const int b = blockIdx.y;
  const long long p0 = static_cast<long long>(blockIdx.x) * pix_per_block;
  const long long p1 = min(HW, p0 + pix_per_block);
  for (int v0 = 0; v0 < nvec; v0 += blockDim.x) {
    const int vi = v0 + threadIdx.x;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (vi < nvec) {
      const uint4* src = reinterpret_cast<const uint4*>(x) + static_cast<long long>(b) * HW * nvec + vi;
      const uint4* const from[1] = {src};
      GnStatsRing ring(sh + 2 * C, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
      const long long by = blockDim.y;
      ring.start(p0 + threadIdx.y, by, p1, nvec, from);
#pragma unroll 1
      for (long long p = p0 + threadIdx.y; p < p1; p += 2 * by) {
        ring.wait();
        const uint4 t[2] = {ring.read(0, 0), ring.read(1, 0)};
        ring.fetch(ring.s, p + GN_AHEAD * by, by, p1, nvec, from);
        ring.next();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (u == 1 && p + by >= p1) break;
          float f[8];
          unpack8(t[u], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            s[j] += f[j];
            q[j] += f[j] * f[j];
          }
        }
      }
    }
    __syncthreads();      // (the sums' buffer lies where the rings were)
    gn_block_sums(sh, sh + 2 * C, s, q, C, vi);
  }
  const int cpg = C / groups, tid = threadIdx.y * blockDim.x + threadIdx.x;
  for (int g = 2 * tid; g < groups; g += 2 * blockDim.x * blockDim.y) {      // two groups: their four sums lie side by side
    const bool two = g + 1 < groups;
    float s[2] = {0.f, 0.f}, q[2] = {0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (k == 0 || two)
        for (int c = (g + k) * cpg; c < (g + k + 1) * cpg; ++c) {
          s[k] += sh[c];
          q[k] += sh[C + c];
        }
    float* to = sums + (b * groups + g) * 2;
    if (two) {
      add4(to, make_float4(s[0], q[0], s[1], q[1]));
    } else {
      atomicAdd(to, s[0]);
      atomicAdd(to + 1, q[0]);
    }
  }
  if (stats == nullptr) return;
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(ticket, 1u) + 1u == gridDim.x * gridDim.y;
  __syncthreads();
  if (last) {
    __threadfence();
    for (int i = tid; i < static_cast<int>(gridDim.y) * groups; i += blockDim.x * blockDim.y) gn_finalize_cell(sums, stats, i, inv_count, eps);
    if (tid == 0) *ticket = 0u;
  }
}

// Two channels' constants, and SiLU's derivative part of them: xhat and dz = dy * silu'(z), z = xhat * gamma + beta.
struct GnPair {
  f32x2 nmu, rs, g, bt;      // minus the mean, reciprocal deviation, affine parameters
};
__device__ __forceinline__ GnPair gn_pair(const float* __restrict__ stats, uint32_t gamma2, uint32_t beta2, int b, int c, int cpg, int groups) {
  const float* s0 = stats + (b * groups + c / cpg) * 2;
  const float* s1 = stats + (b * groups + (c + 1) / cpg) * 2;
  const float2 g = unpack_bf16x2(gamma2), bt = unpack_bf16x2(beta2);
  return {f2_pack(-s0[0], -s1[0]), f2_pack(s0[1], s1[1]), f2_pack(g.x, g.y), f2_pack(bt.x, bt.y)};
}
// a thread's eight channels
__device__ __forceinline__ void gn_pairs(GnPair (&c)[4], const float* __restrict__ stats, const __nv_bfloat16* __restrict__ gamma,
                                         const __nv_bfloat16* __restrict__ beta, int b, int vi, int cpg, int groups) {
  const uint4 gq = reinterpret_cast<const uint4*>(gamma)[vi], bq = reinterpret_cast<const uint4*>(beta)[vi];
  const uint32_t g4[4] = {gq.x, gq.y, gq.z, gq.w}, b4[4] = {bq.x, bq.y, bq.z, bq.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) c[j] = gn_pair(stats, g4[j], b4[j], b, vi * 8 + 2 * j, cpg, groups);
}
// 1 / (1 + exp(-z)), two elements per instruction
__device__ __forceinline__ f32x2 f2_sigmoid(f32x2 z) {
  float a, b;
  f2_unpack(f2_mul(z, f2_both(-1.4426950408889634f)), a, b);
  f2_unpack(f2_add(f2_pack(exp2f(a), exp2f(b)), f2_both(1.f)), a, b);
  return f2_pack(__fdividef(1.f, a), __fdividef(1.f, b));
}
// RES: a shortcut is added (without it twice the pixels ahead make up for the second tensor's loads)
template <bool RES>
__global__ void __launch_bounds__(256, 2) groupnorm_silu_apply_kernel(const __nv_bfloat16* __restrict__ x,
                                                                      const float* __restrict__ stats,
                                                                      const __nv_bfloat16* __restrict__ gamma,
                                                                      const __nv_bfloat16* __restrict__ beta,
                                                                      const __nv_bfloat16* __restrict__ res,
                                                                      __nv_bfloat16* __restrict__ y, long long HW, int C,
                                                                      int groups, int pix_per_block) {
  chain_begin();
  extern __shared__ uint4 gn_ring[];
  const int nvec = C >> 3;
  const int b = blockIdx.y;
  const long long p0 = static_cast<long long>(blockIdx.x) * pix_per_block;
  const long long p1 = min(HW, p0 + pix_per_block);
  for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
    GnPair c[4];
    gn_pairs(c, stats, gamma, beta, b, vi, C / groups, groups);
    const long long first = static_cast<long long>(b) * HW * nvec + vi;
    const uint4* from[RES ? 2 : 1];
    from[0] = reinterpret_cast<const uint4*>(x) + first;
    if constexpr (RES) from[1] = reinterpret_cast<const uint4*>(res) + first;
    uint4* dst = reinterpret_cast<uint4*>(y) + first;
    constexpr int AHEAD = RES ? GN_AHEAD : 2 * GN_AHEAD;
    LaneRing<RES ? 2 : 1, AHEAD> ring(gn_ring, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
    const long long by = blockDim.y;
    ring.start(p0 + threadIdx.y, by, p1, nvec, from);
#pragma unroll 1
    for (long long p = p0 + threadIdx.y; p < p1; p += 2 * by) {
      ring.wait();
      const uint4 t[2] = {ring.read(0, 0), ring.read(1, 0)};
      uint4 r[2] = {};
      if constexpr (RES) r[0] = ring.read(0, 1), r[1] = ring.read(1, 1);
      ring.fetch(ring.s, p + AHEAD * by, by, p1, nvec, from);
      ring.next();
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (u == 1 && p + by >= p1) break;
        const uint32_t x4[4] = {t[u].x, t[u].y, t[u].z, t[u].w}, r4[4] = {r[u].x, r[u].y, r[u].z, r[u].w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 z = f2_fma(f2_mul(f2_add(f2_of_bf16x2(x4[j]), c[j].nmu), c[j].rs), c[j].g, c[j].bt);
          f32x2 v = f2_mul(z, f2_sigmoid(z));
          if constexpr (RES) v = f2_add(v, f2_of_bf16x2(r4[j]));
          o[j] = f2_to_bf16x2(v);
        }
        dst[(p + u * by) * nvec] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

__device__ __forceinline__ f32x2 gn_dz(const GnPair& c, f32x2 x, f32x2 dy, f32x2& xh) {
  xh = f2_mul(f2_add(x, c.nmu), c.rs);
  const f32x2 z = f2_fma(xh, c.g, c.bt), sg = f2_sigmoid(z);
  return f2_mul(f2_mul(dy, sg), f2_fma(z, f2_fma(sg, f2_both(-1.f), f2_both(1.f)), f2_both(1.f)));
}

// pass 1 of the backward: red[b][c] = {sum dz, sum dz * xhat}. Bound by issue and the special functions beside HBM: two channels per instruction,
// no shared-memory atomics, one block of 16 warps (us, 557056 pixels x 384: two blocks of 8 warps with eight loads in registers 192, three with
// the ring and one pixel at a time 168, this 160; HBM alone 131).
__global__ void __launch_bounds__(512, 1) groupnorm_silu_bwd_reduce_kernel(
    const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const float* __restrict__ stats,
    const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ beta, float* __restrict__ red,
    long long HW, int C, int groups, int pix_per_block, float* __restrict__ dgamma, float* __restrict__ dbeta) {
  chain_begin();
  extern __shared__ __align__(16) float sh[];  // [2][C], then the threads' sums
  const int nvec = C >> 3;
  const int b = blockIdx.y;
  const long long p0 = static_cast<long long>(blockIdx.x) * pix_per_block;
  const long long p1 = min(HW, p0 + pix_per_block);
  for (int v0 = 0; v0 < nvec; v0 += blockDim.x) {
    const int vi = v0 + threadIdx.x;
    f32x2 s2[4], q2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s2[j] = q2[j] = f2_both(0.f);
    if (vi < nvec) {
      GnPair c[4];
      gn_pairs(c, stats, gamma, beta, b, vi, C / groups, groups);
      const long long first = static_cast<long long>(b) * HW * nvec + vi;
      const uint4* xs = reinterpret_cast<const uint4*>(x) + first;
      const uint4* ds = reinterpret_cast<const uint4*>(dy) + first;
      const uint4* const from[2] = {xs, ds};
      GnPairRing ring(sh + 2 * C, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
      const long long by = blockDim.y;
      ring.start(p0 + threadIdx.y, by, p1, nvec, from);
#pragma unroll 1
      for (long long p = p0 + threadIdx.y; p < p1; p += 2 * by) {
        ring.wait();
        const uint4 t[2] = {ring.read(0, 0), ring.read(1, 0)}, d[2] = {ring.read(0, 1), ring.read(1, 1)};
        ring.fetch(ring.s, p + GN_AHEAD * by, by, p1, nvec, from);
        ring.next();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (u == 1 && p + by >= p1) break;
          const uint32_t x4[4] = {t[u].x, t[u].y, t[u].z, t[u].w}, d4[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f32x2 xh;
            const f32x2 dz = gn_dz(c[j], f2_of_bf16x2(x4[j]), f2_of_bf16x2(d4[j]), xh);
            s2[j] = f2_add(s2[j], dz);
            q2[j] = f2_fma(dz, xh, q2[j]);
          }
        }
      }
    }
    __syncthreads();      // (the sums' buffer lies where the rings were)
    float s[8], q[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f2_unpack(s2[j], s[2 * j], s[2 * j + 1]);
      f2_unpack(q2[j], q[2 * j], q[2 * j + 1]);
    }
    gn_block_sums(sh, sh + 2 * C, s, q, C, vi);
  }
  // (vector reductions: the blocks' ends meet on the same addresses)
  for (int c = 4 * (threadIdx.y * blockDim.x + threadIdx.x); c < C; c += 4 * blockDim.x * blockDim.y) {
    const float4 dz = *reinterpret_cast<const float4*>(sh + c), dzx = *reinterpret_cast<const float4*>(sh + C + c);
    float* r = red + (static_cast<long long>(b) * C + c) * 2;
    add4(r, make_float4(dz.x, dzx.x, dz.y, dzx.y));
    add4(r + 4, make_float4(dz.z, dzx.z, dz.w, dzx.w));
    // the affine parameters' gradients are the same sums taken over the batch as well
    if (dbeta != nullptr) add4(dbeta + c, dz);
    if (dgamma != nullptr) add4(dgamma + c, dzx);
  }
}

// {sum, sum of squares} per (sample, group) -> {mean, rstd}; the sums are cleared
__global__ void groupnorm_finalize_kernel(float* __restrict__ sums, float* __restrict__ stats, int cells, float inv_count,
                                          float eps) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cells) gn_finalize_cell(sums, stats, i, inv_count, eps);
}

// dst[a * sa + b * sb + c * sc] += src[(a * nb + b) * nc + c] (fp32); the source is zeroed behind the read. Used to fold tap-major convolution
// weight gradients into the (Cout, Cin, kh, kw) layout of the gradient arena.
__global__ void __launch_bounds__(256) strided_add_kernel(float* __restrict__ src, float* __restrict__ dst, int na, int nb,
                                                          int nc, long long sa, long long sb, long long sc) {
  chain_begin();
  const long long total = static_cast<long long>(na) * nb * nc;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % nc);
    const long long t = i / nc;
    const int b = static_cast<int>(t % nb), a2 = static_cast<int>(t / nb);
    dst[a2 * sa + b * sb + c * sc] += src[i];
    src[i] = 0.f;
  }
}

// dst[c][r][t] += src[t][r][c] (fp32), the source zeroed behind the read: weight gradients of all taps ([tap][displaced channel][column]) into
// the parameter's layout. Both sides move whole lines, through a tile of 32 columns x 16 rows x taps in shared memory.
constexpr int FOLD_COLS = 32, FOLD_ROWS = 16, FOLD_TAPS = 9;
__global__ void __launch_bounds__(256) fold_taps_kernel(float* __restrict__ src, float* __restrict__ dst, int taps, int rows, int cols) {
  chain_begin();
  __shared__ float tile[FOLD_COLS][FOLD_ROWS * FOLD_TAPS + 1];
  const int c0 = blockIdx.x * FOLD_COLS, r0 = blockIdx.y * FOLD_ROWS;
  const int nr = min(FOLD_ROWS, rows - r0), nc = min(FOLD_COLS, cols - c0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // all loads of a thread are issued before the first use: 2 rows of every tap, 4 columns of the destination
  constexpr int RUN = (FOLD_ROWS * FOLD_TAPS + 31) / 32;
  float v[FOLD_ROWS / 8][FOLD_TAPS], old[FOLD_COLS / 8][RUN];
  float* const s = src + static_cast<long long>(r0) * cols + c0 + lane;
#pragma unroll
  for (int k = 0; k < FOLD_ROWS / 8; ++k)
#pragma unroll
    for (int t = 0; t < FOLD_TAPS; ++t)
      if (t < taps && warp + 8 * k < nr && lane < nc) v[k][t] = s[(static_cast<long long>(t) * rows + warp + 8 * k) * cols];
#pragma unroll
  for (int k = 0; k < FOLD_COLS / 8; ++k)
#pragma unroll
    for (int i = 0; i < RUN; ++i)
      if (warp + 8 * k < nc && lane + 32 * i < nr * taps)
        old[k][i] = dst[(static_cast<long long>(c0 + warp + 8 * k) * rows + r0) * taps + lane + 32 * i];
#pragma unroll
  for (int k = 0; k < FOLD_ROWS / 8; ++k)
#pragma unroll
    for (int t = 0; t < FOLD_TAPS; ++t)
      if (t < taps && warp + 8 * k < nr && lane < nc) {
        tile[lane][(warp + 8 * k) * taps + t] = v[k][t];
        s[(static_cast<long long>(t) * rows + warp + 8 * k) * cols] = 0.f;
      }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < FOLD_COLS / 8; ++k)
#pragma unroll
    for (int i = 0; i < RUN; ++i)
      if (warp + 8 * k < nc && lane + 32 * i < nr * taps)
        dst[(static_cast<long long>(c0 + warp + 8 * k) * rows + r0) * taps + lane + 32 * i] = old[k][i] + tile[warp + 8 * k][lane + 32 * i];
}

// out[p][b][a][r] = in[p][a][b][r] (16-byte vectors): image rows of windows to windows of rows and back. Bound by HBM: four vectors a
// thread, all asked for before the first is stored. Against the tensor operators' copy, which moves two bytes per lane, cold: 23040 x 192
// 18.4 -> 10.2 us, 139264 x 384 141.2 -> 38.9 us (5.5 TB/s).
__global__ void __launch_bounds__(256) swap_middle_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, unsigned int A, unsigned int B,
                                                          unsigned int run, unsigned int total) {
  chain_begin();
  constexpr int EACH = 4;
  uint4 v[EACH];
  const unsigned int first = blockIdx.x * (256u * EACH) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < EACH; ++k) {
    const unsigned int i = first + 256u * k;
    if (i >= total) break;
    const unsigned int t = i / run, q = t / A, a = t - q * A, p = q / B, b = q - p * B;
    v[k] = in[static_cast<size_t>((p * A + a) * B + b) * run + (i - t * run)];
  }
#pragma unroll
  for (int k = 0; k < EACH; ++k)
    if (first + 256u * k < total) out[first + 256u * k] = v[k];
}

// pass 2: dx = rstd * (dz*gamma - s1/n - xhat * s2/n), s1 = sum_c gamma_c red[b][c][0], s2 likewise with [1]
__global__ void __launch_bounds__(256, 2) groupnorm_silu_bwd_apply_kernel(
    const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const float* __restrict__ stats,
    const float* __restrict__ red, const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ beta,
    __nv_bfloat16* __restrict__ dx, long long HW, int C, int groups, float inv_count, int pix_per_block) {
  chain_begin();
  extern __shared__ float gs[];  // [groups][2] of this block's sample
  const int cpg = C / groups, nvec = C >> 3;
  const int b = blockIdx.y;
  for (int g = threadIdx.y * blockDim.x + threadIdx.x; g < groups; g += blockDim.x * blockDim.y) {
    float s1 = 0.f, s2 = 0.f;
    for (int c = g * cpg; c < (g + 1) * cpg; ++c) {
      const float gm = __bfloat162float(gamma[c]);
      const float2 r = reinterpret_cast<const float2*>(red)[static_cast<long long>(b) * C + c];
      s1 += gm * r.x;
      s2 += gm * r.y;
    }
    gs[g * 2] = s1 * inv_count;
    gs[g * 2 + 1] = s2 * inv_count;
  }
  __syncthreads();
  const long long p0 = static_cast<long long>(blockIdx.x) * pix_per_block;
  const long long p1 = min(HW, p0 + pix_per_block);
  for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
    GnPair c[4];
    f32x2 nm1[4], nm2[4];
    {
      gn_pairs(c, stats, gamma, beta, b, vi, cpg, groups);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int ch = vi * 8 + 2 * j;
        nm1[j] = f2_pack(-gs[ch / cpg * 2], -gs[(ch + 1) / cpg * 2]);
        nm2[j] = f2_pack(-gs[ch / cpg * 2 + 1], -gs[(ch + 1) / cpg * 2 + 1]);
      }
    }
    const long long first = static_cast<long long>(b) * HW * nvec + vi;
    const uint4* xs = reinterpret_cast<const uint4*>(x) + first;
    const uint4* ds = reinterpret_cast<const uint4*>(dy) + first;
    uint4* dst = reinterpret_cast<uint4*>(dx) + first;
    const uint4* const from[2] = {xs, ds};
    GnPairRing ring(gs + (groups * 2 + 3) / 4 * 4, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
    const long long by = blockDim.y;
    ring.start(p0 + threadIdx.y, by, p1, nvec, from);
#pragma unroll 1
    for (long long p = p0 + threadIdx.y; p < p1; p += 2 * by) {
      ring.wait();
      const uint4 t[2] = {ring.read(0, 0), ring.read(1, 0)}, d[2] = {ring.read(0, 1), ring.read(1, 1)};
      ring.fetch(ring.s, p + GN_AHEAD * by, by, p1, nvec, from);
      ring.next();
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (u == 1 && p + by >= p1) break;
        const uint32_t x4[4] = {t[u].x, t[u].y, t[u].z, t[u].w}, d4[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f32x2 xh;
          const f32x2 dz = gn_dz(c[j], f2_of_bf16x2(x4[j]), f2_of_bf16x2(d4[j]), xh);
          o[j] = f2_to_bf16x2(f2_mul(c[j].rs, f2_fma(xh, nm2[j], f2_fma(dz, c[j].g, nm1[j]))));
        }
        dst[(p + u * by) * nvec] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ masked loss
__global__ void __launch_bounds__(256) masked_loss_kernel(const __nv_bfloat16* __restrict__ pred,
                                                          const __nv_bfloat16* __restrict__ label,
                                                          const __nv_bfloat16* __restrict__ mask, long long nvec,
                                                          long long mask_period_vec, int kind, float grad_scale,
                                                          float* __restrict__ loss_sum, __nv_bfloat16* __restrict__ grad) {
  chain_begin();
  float acc = 0.f;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float p[8], l[8], m[8], g[8];
    unpack8(reinterpret_cast<const uint4*>(pred)[i], p);
    unpack8(reinterpret_cast<const uint4*>(label)[i], l);
    if (mask != nullptr) {
      unpack8(reinterpret_cast<const uint4*>(mask)[i % mask_period_vec], m);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) m[j] = 1.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float d = p[j] * m[j] - l[j];
      if (kind == 0) {
        acc += fabsf(d);
        g[j] = (d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f)) * m[j] * grad_scale;
      } else {
        acc += d * d;
        g[j] = 2.f * d * m[j] * grad_scale;
      }
    }
    if (grad != nullptr) reinterpret_cast<uint4*>(grad)[i] = pack8(g);
  }
  acc = warp_sum(acc);
  __shared__ float sh[8];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < (blockDim.x >> 5); ++w) s += sh[w];
    atomicAdd(loss_sum, s);
  }
}

// ------------------------------------------------------------------------------------------ attention row dots
// drow[row, head] = sum over the head's channels of dO * O: the "D" term of the attention backward pass. A warp per row;
// lanes stride over the row's 16-byte vectors, then the lanes of one head are summed.
__global__ void __launch_bounds__(256) attn_rowdot_kernel(const uint4* __restrict__ o, const uint4* __restrict__ dout,
                                                          float* __restrict__ drow, long long rows, int vec_per_row,
                                                          int vec_per_head, int heads) {
  chain_begin();
  const int lane = threadIdx.x & 31;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long r = warp; r < rows; r += nwarps) {
    for (int v0 = 0; v0 < vec_per_row; v0 += 32) {
      const int v = v0 + lane;
      float acc = 0.f;
      if (v < vec_per_row) {
        float x[8], y[8];
        unpack8(o[r * vec_per_row + v], x);
        unpack8(dout[r * vec_per_row + v], y);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fmaf(x[j], y[j], acc);
      }
      // vec_per_head is 2, 4, 8 or 16 (head dims 16 .. 128): sum groups of that many neighbouring lanes
      for (int d = 1; d < vec_per_head && d < 32; d <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (v < vec_per_row && (v % vec_per_head) == 0) drow[r * heads + v / vec_per_head] = acc;
    }
  }
}

// ------------------------------------------------------------------------------------------ gradient inspection
// One pass over a flat fp32 gradient buffer for the loss-scaling path: out[0] += sum of squares (for the clipping
// norm), out[1] becomes non-zero when any element is inf or nan (the step is then skipped and the scale backed off).
__global__ void __launch_bounds__(256) grad_inspect_kernel(const float* __restrict__ g, long long n, float* __restrict__ out) {
  chain_begin();
  float acc = 0.f;
  bool bad = false;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float v = g[i];
    bad |= !(fabsf(v) <= 3.0e38f);     // false for inf and for nan
    acc = fmaf(v, v, acc);
  }
  acc = warp_sum(acc);
  const unsigned int any_bad = __ballot_sync(0xffffffffu, bad);
  __shared__ float sh[8];
  __shared__ unsigned int shb[8];
  if ((threadIdx.x & 31) == 0) {
    sh[threadIdx.x >> 5] = acc;
    shb[threadIdx.x >> 5] = any_bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    unsigned int b = 0u;
    for (int w = 0; w < (blockDim.x >> 5); ++w) {
      s += sh[w];
      b |= shb[w];
    }
    if (b == 0u) atomicAdd(out, s);           // a poisoned sum would only hide the flag's meaning
    else out[1] = 1.f;
  }
}

// ------------------------------------------------------------------------------------------ AdamW
template <bool GRAD_BF16>
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ master, float* __restrict__ m,
                                                    float* __restrict__ v, const void* __restrict__ grad,
                                                    __nv_bfloat16* __restrict__ param, long long n, float lr, float b1,
                                                    float b2, float eps, float wd, float bc1, float bc2s,
                                                    float gscale) {
  chain_begin();
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float g = GRAD_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(grad)[i])
                        : static_cast<const float*>(grad)[i];
    g *= gscale;
    float p = master[i];
    p *= 1.f - lr * wd;
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    const float denom = sqrtf(vi) / bc2s + eps;
    p -= (lr / bc1) * (mi / denom);
    m[i] = mi;
    v[i] = vi;
    master[i] = p;
    if (param != nullptr) param[i] = __float2bfloat16(p);
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ d, long long n) {
  chain_begin();
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    d[i] = __float2bfloat16(s[i]);
}

__global__ void add_bf16_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, uint4* __restrict__ o,
                                long long nvec) {
  chain_begin();
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8], y[8];
    unpack8(a[i], x);
    unpack8(b[i], y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    o[i] = pack8(x);
  }
}

// Packed operands of the implicit GEMMs: out[(n1 * N2 + n2)][t][c] = w[n1 * s1 + n2 * s2 + c * sc + off[t]], zero for c >= C and for n2 >=
// V2 (rows that only pad). One launch per operand and optimizer step (zero fill, permutation, flip and copy were three to five); the reads
// are strided by the taps, which the caches absorb (a weight is at most a few MB).
struct PackTaps {
  int N2, V2, T, C, Cpad;
  long long s1, s2, sc;
  int off[9];
};
__global__ void __launch_bounds__(256) pack_taps_kernel(const __nv_bfloat16* __restrict__ w, uint32_t* __restrict__ out,
                                                        PackTaps p, long long total) {
  chain_begin();
  const int half = p.Cpad >> 1;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % half) * 2;
    const long long r = i / half;
    const int t = static_cast<int>(r % p.T);
    const long long n = r / p.T;
    const __nv_bfloat16* src = w + n / p.N2 * p.s1 + n % p.N2 * p.s2 + p.off[t];
    __nv_bfloat162 v = __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0));
    const bool row = n % p.N2 < p.V2;
    if (row && c < p.C) v.x = src[c * p.sc];
    if (row && c + 1 < p.C) v.y = src[(c + 1) * p.sc];
    out[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
}

// Input gradient of the 3x3 stride-2 convolution from its per-tap columns: dcol[b, ho, wo, tap, c] (tap = ky * 3 + kx)
// is the contribution of output pixel (ho, wo) to padded input pixel (2 ho + ky, 2 wo + kx). Every padded input pixel
// gathers its (at most four) contributions; the result is written for padded rows [r0, r0 + rows) and padded columns
// [1, W + 1) as fp32 (F32: with the halo rows, for the multi-rank fold) or bf16.
template <bool F32>
__global__ void conv_s2_col2im_kernel(const uint4* __restrict__ dcol, void* __restrict__ out, int B, int Ho, int Wo, int W,
                                      int cvec, int r0, int rows) {
  chain_begin();
  const long long total = static_cast<long long>(B) * rows * W * cvec;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int cv = static_cast<int>(i % cvec);
    long long t = i / cvec;
    const int w = static_cast<int>(t % W);
    t /= W;
    const int r = static_cast<int>(t % rows);
    const int b = static_cast<int>(t / rows);
    const int ph = r0 + r, pw = w + 1;                     // padded coordinates
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    // ky in {ph & 1, (ph & 1) + 2 if even}: ph = 2 ho + ky
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int ky = (ph & 1) + 2 * a;
      if (ky > 2) continue;
      const int ho = (ph - ky) >> 1;
      if (ph - ky < 0 || ho >= Ho) continue;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int kx = (pw & 1) + 2 * c;
        if (kx > 2) continue;
        const int wo = (pw - kx) >> 1;
        if (pw - kx < 0 || wo >= Wo) continue;
        float f[8];
        unpack8(dcol[((static_cast<long long>(b) * Ho + ho) * Wo + wo) * 9 * cvec + (ky * 3 + kx) * cvec + cv], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += f[j];
      }
    }
    if (F32) {
      float4* o = reinterpret_cast<float4*>(static_cast<float*>(out) + i * 8);
      o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
      reinterpret_cast<uint4*>(out)[i] = pack8(acc);
    }
  }
}

// Image [B, H, W, C] <-> patches [B, Hp / p, Wp / p, (p1, p2, c)] of the image padded to Hp x Wp (`top` rows above, `left`
// columns left). A patch row (p2, c) is p * C contiguous elements on both sides, so the rearrangement is one pass of
// contiguous copies, bound by HBM; V (16, 8, 4 or 2 bytes) divides the byte length of a patch row, of an image row and of
// the left padding, so that no vector crosses the edge of the image. `row_units` = vectors of a padded row,
// `seg_units` = vectors of a patch row. Thread block: one padded row (blockIdx.y) and PATCH_UNROLL vectors per thread.
// 720 x 1440 x 138 padded to 768 rows, L2 flushed before: 94 us in (591 MB, 90 us at 6.54 TB/s), 132 us out with the addition
// (858 MB, 131 us; the padding is not read); the tensor operators took 1100 us for both.
constexpr int PATCH_UNROLL = 4;
template <class V>
__global__ void __launch_bounds__(256) pad_patchify_kernel(const V* __restrict__ x, V* __restrict__ patches, int H, int p, int hn,
                                                           int top, int left_units, int img_units, int row_units, int seg_units) {
  chain_begin();
  const int yy = blockIdx.y % (hn * p), b = blockIdx.y / (hn * p);
  const int y = yy - top;
  const V* src = x + (static_cast<long long>(b) * H + y) * img_units - left_units;
  V* dst = patches + (static_cast<long long>(b) * hn + yy / p) * p * row_units + static_cast<long long>(yy % p) * seg_units;
  V t[PATCH_UNROLL];
#pragma unroll
  for (int u = 0; u < PATCH_UNROLL; ++u) {
    const int e = (blockIdx.x * PATCH_UNROLL + u) * blockDim.x + threadIdx.x;
    t[u] = V{};
    if (e < row_units && y >= 0 && y < H && e >= left_units && e < left_units + img_units) t[u] = src[e];
  }
#pragma unroll
  for (int u = 0; u < PATCH_UNROLL; ++u) {
    const int e = (blockIdx.x * PATCH_UNROLL + u) * blockDim.x + threadIdx.x;
    if (e < row_units) dst[static_cast<long long>(e / seg_units) * p * seg_units + e % seg_units] = t[u];
  }
}

__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
  const float2 x = unpack_bf16x2(a), y = unpack_bf16x2(b);
  return pack_bf16x2(x.x + y.x, x.y + y.y);
}
__device__ __forceinline__ uint4 add_bf16v(uint4 a, uint4 b) {
  return make_uint4(add_bf16x2(a.x, b.x), add_bf16x2(a.y, b.y), add_bf16x2(a.z, b.z), add_bf16x2(a.w, b.w));
}
__device__ __forceinline__ uint2 add_bf16v(uint2 a, uint2 b) { return make_uint2(add_bf16x2(a.x, b.x), add_bf16x2(a.y, b.y)); }
__device__ __forceinline__ uint32_t add_bf16v(uint32_t a, uint32_t b) { return add_bf16x2(a, b); }
__device__ __forceinline__ unsigned short add_bf16v(unsigned short a, unsigned short b) {
  return static_cast<unsigned short>(add_bf16x2(a, b) & 0xffffu);
}

// The inverse, cropped to the image, with `add` (an image, or null) added in fp32 before the rounding.
template <class V>
__global__ void __launch_bounds__(256) unpatchify_crop_kernel(const V* __restrict__ patches, const V* __restrict__ add,
                                                              V* __restrict__ out, int H, int p, int hn, int top, int left_units,
                                                              int img_units, int row_units, int seg_units) {
  chain_begin();
  const int y = blockIdx.y % H, b = blockIdx.y / H;
  const int yy = y + top;
  const V* src = patches + (static_cast<long long>(b) * hn + yy / p) * p * row_units + static_cast<long long>(yy % p) * seg_units;
  const long long row = (static_cast<long long>(b) * H + y) * img_units;
  V t[PATCH_UNROLL], r[PATCH_UNROLL];
#pragma unroll
  for (int u = 0; u < PATCH_UNROLL; ++u) {
    const int e = (blockIdx.x * PATCH_UNROLL + u) * blockDim.x + threadIdx.x;
    if (e < img_units) {
      const int k = e + left_units;
      t[u] = src[static_cast<long long>(k / seg_units) * p * seg_units + k % seg_units];
      if (add != nullptr) r[u] = add[row + e];
    }
  }
#pragma unroll
  for (int u = 0; u < PATCH_UNROLL; ++u) {
    const int e = (blockIdx.x * PATCH_UNROLL + u) * blockDim.x + threadIdx.x;
    if (e < img_units) out[row + e] = add != nullptr ? add_bf16v(t[u], r[u]) : t[u];
  }
}

// out = sum over `slots` consecutive bf16 buffers of `nvec` 16-byte vectors each (fp32 accumulation), optionally
// + bias[col] (bf16, `cvec` vectors per row) + residual (bf16, same shape as out): the owner's side of the slot-staged
// reduce-scatter with the row-parallel layer's bias and the block's shortcut folded in.
__global__ void sum_slots_bf16_kernel(const uint4* __restrict__ src, uint4* __restrict__ o, int slots, long long nvec,
                                      const uint4* __restrict__ bias, const uint4* __restrict__ res, int cvec) {
  chain_begin();
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float acc[8];
    unpack8(src[i], acc);
    for (int s = 1; s < slots; ++s) {
      float y[8];
      unpack8(src[i + s * nvec], y);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += y[j];
    }
    if (bias != nullptr) {
      float y[8];
      unpack8(bias[i % cvec], y);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += y[j];
    }
    if (res != nullptr) {
      float y[8];
      unpack8(res[i], y);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += y[j];
    }
    o[i] = pack8(acc);
  }
}

int grid_for(long long work_items, int block, int max_blocks = 148 * 16) {
  long long g = (work_items + block - 1) / block;
  if (g > max_blocks) g = max_blocks;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

}  // namespace

// CALL sees LPR, VPL and EXACT (see the LayerNorm kernels) for rows of NVEC 16-byte vectors. MANY: rows enough for groups of 32 / LPR of
// them; below that a row per warp finishes sooner (shorter chains, more warps). The lines are LN_FWD_GROUPS and LN_BWD_GROUPS rows: beyond
// them a row per warp means several rows one after the other in every warp, each waiting for its loads and its shuffles, and backward as
// many more blocks that end in atomics on the same sums. Inputs in L2, us, a row per warp / groups. Forward: C = 192, 1024 rows 1.70 /
// 1.97, 2048 1.88 / 1.98, 4096 2.59 / 2.06, 17280 5.23 / 3.17; 384, 2048 2.33 / 2.13, 17280 7.29 / 5.39; 96, 2048 1.88 / 1.98, 17280 5.17 /
// 2.41. Backward: 96, 512 2.06 / 2.59, 2048 3.59 / 2.66; 192, 512 2.79 / 2.67, 1024 3.84 / 2.83, 2048 6.21 / 3.41, 8192 7.76 / 6.88; 384,
// 2048 6.31 / 4.68, 8192 9.09 / 7.95.
constexpr long long LN_FWD_GROUPS = 2048, LN_BWD_GROUPS = 1024;
#define TB_LN_CASE(L, V, E, ...) { constexpr int LPR = L; constexpr int VPL = V; constexpr bool EXACT = E; __VA_ARGS__; }
#define TB_LN_DISPATCH(NVEC, MANY, ...)                         \
  switch ((MANY) ? (NVEC) : 0) {                                               \
    case 4: TB_LN_CASE(4, 1, true, __VA_ARGS__) break;                 \
    case 8: TB_LN_CASE(8, 1, true, __VA_ARGS__) break;                 \
    case 12: TB_LN_CASE(4, 3, true, __VA_ARGS__) break;                \
    case 16: TB_LN_CASE(16, 1, true, __VA_ARGS__) break;               \
    case 24: TB_LN_CASE(8, 3, true, __VA_ARGS__) break;                \
    case 48: TB_LN_CASE(16, 3, true, __VA_ARGS__) break;               \
    default:                                                    \
      switch (((NVEC) + 31) / 32) {                             \
        case 1: TB_LN_CASE(32, 1, false, __VA_ARGS__) break;           \
        case 2: TB_LN_CASE(32, 2, false, __VA_ARGS__) break;           \
        case 3: TB_LN_CASE(32, 3, false, __VA_ARGS__) break;           \
        case 4: TB_LN_CASE(32, 4, false, __VA_ARGS__) break;           \
        case 5: case 6: TB_LN_CASE(32, 6, false, __VA_ARGS__) break;   \
        case 7: case 8: TB_LN_CASE(32, 8, false, __VA_ARGS__) break;   \
        default: return -1;                                     \
      }                                                         \
  }

// Blocks of the LayerNorm kernels. Forward: one resident wave where the rows of a warp are many vectors or few, more blocks than
// that for wide rows (278528 rows, us, 4 / 6 / 16 blocks per SM: C = 384 70 / 77 / 71, 768 142 / 160 / 142, 1024 195 / 198 / 177).
constexpr int ln_fwd_blocks(int vpl) { return 148 * (vpl == 1 ? 6 : (vpl == 2 ? 5 : (vpl == 3 ? 4 : (vpl == 8 ? 2 : 16)))); }
// Backward: every block ends in 2 C atomics on the same addresses, so few rows take three blocks per SM and many rows one
// resident wave (139264 rows with shortcut, us, 2 / 3 / resident: C = 72 70 / 55 / 42, 256 116 / 87 / 62, 512 158 / 124 / 108; 4096 rows
// of 256 7.5 / 9 / 15). Rows of five vectors per lane and more have room for two blocks; a third waits for both (2048 columns
// 1186 / 1452).
inline int ln_bwd_blocks(int vpl, long long rows) {
  if (vpl > 4) return 148 * 2;
  const bool many = rows >= 148LL * 3 * 4 * 32;       // 32 rows for every warp of three blocks per SM
  return 148 * (many && vpl == 1 ? 5 : (many && vpl == 2 ? 4 : 3));
}

int layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                  long long rows, int C, float eps, cudaStream_t stream) {
  if (C % 8 != 0 || C > 2048) return -1;
  TB_LN_DISPATCH(C / 8, rows >= LN_FWD_GROUPS,
                 launch_chained(layernorm_fwd_kernel<LPR, VPL, EXACT>, grid_for(rows, 8 * (32 / LPR), ln_fwd_blocks(VPL)), 256, 0, stream,
                                static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma),
                                static_cast<const __nv_bfloat16*>(beta), static_cast<__nv_bfloat16*>(y), mean, rstd, rows, C, eps));
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

template <int LPR, int VPL, bool EXACT, bool RES, bool SUMS>
static int ln_bwd_launch(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* gamma, const float* mean, const float* rstd,
                         __nv_bfloat16* dx, float* dgamma, float* dbeta, const __nv_bfloat16* dres, long long rows, int C, float* dsum,
                         cudaStream_t stream) {
  const size_t bytes = std::max<size_t>(4 * (SUMS ? 3 : 2) * C * sizeof(float), static_cast<size_t>(RES ? 3 : 2) * VPL * ln_bwd_ahead(VPL) * 128 * 16);
  auto kernel = layernorm_bwd_kernel<LPR, VPL, EXACT, RES, SUMS>;
  static SharedLimit limit;
  if (bytes > 48 * 1024 && limit.raise(reinterpret_cast<const void*>(kernel), 112 * 1024) != cudaSuccess) return -3;
  launch_chained(kernel, grid_for(rows, 4 * (32 / LPR), ln_bwd_blocks(VPL, rows)), 128, bytes, stream, dy, x, gamma, mean, rstd, dx, dgamma,
                 dbeta, dres, rows, C, dsum);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int layernorm_bwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, void* dx,
                  float* dgamma, float* dbeta, const void* dres, long long rows, int C, cudaStream_t stream, float* dres_sum) {
  if (C % 8 != 0 || C > 2048 || (dres_sum != nullptr && dres == nullptr)) return -1;
  auto go = [&](auto launch) {
    return launch(static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), mean, rstd,
                  static_cast<__nv_bfloat16*>(dx), dgamma, dbeta, static_cast<const __nv_bfloat16*>(dres), rows, C, dres_sum, stream);
  };
  if (dres_sum != nullptr) {
    // (of the widths that gain by it: bindings_halves.cpp, sums_beside_norm)
    if (C <= 512 || C > 1024) return -1;
    return C <= 768 ? go(ln_bwd_launch<32, 3, false, true, true>) : go(ln_bwd_launch<32, 4, false, true, true>);
  }
  if (dres != nullptr) {
    TB_LN_DISPATCH(C / 8, rows >= LN_BWD_GROUPS, return go(ln_bwd_launch<LPR, VPL, EXACT, true, false>));
  } else {
    TB_LN_DISPATCH(C / 8, rows >= LN_BWD_GROUPS, return go(ln_bwd_launch<LPR, VPL, EXACT, false, false>));
  }
  return -1;
}

int colsum_rows_per_block() { return 256; }

// out[c] += sum over rows of x[r][c]. `partials`: fp32 scratch of ceil(rows / colsum_rows_per_block()) x C elements.
int colsum_bf16(const void* x, float* out, float* partials, long long rows, int C, long long ld, cudaStream_t stream) {
  if (C % 8 != 0 || partials == nullptr) return -1;
  const int nvec = C / 8;
  const int bx = nvec <= 64 ? nvec : 32;
  const int by = 256 / bx > 0 ? 256 / bx : 1;
  dim3 block(bx, by);
  const int rows_per_block = colsum_rows_per_block();
  const int nparts = static_cast<int>((rows + rows_per_block - 1) / rows_per_block);
  dim3 grid(static_cast<unsigned>(nparts), (nvec + bx - 1) / bx);
  const size_t sh = static_cast<size_t>(by) * (bx * 8 + 1) * sizeof(float);
  launch_chained(colsum_kernel, grid, block, sh, stream, static_cast<const __nv_bfloat16*>(x), partials, rows, C, ld, rows_per_block);
  launch_chained(colsum_finish_kernel, (C + 31) / 32, dim3(32, 32), 0, stream, partials, out, nparts, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Launch shape of the GroupNorm kernels: `threads` per block as (column vectors) x (pixels), pixels split over at most `waves`
// blocks per SM in all (one block beyond a resident wave would double the time: eight samples of 17280 x 384 rounded up made 448
// blocks of 444, 106 us instead of 70 in the backward sums) and at least one loop round of `unroll` pixels per thread, so that
// tiny images do not pay for more blocks than they fill.
struct GnShape {
  dim3 block, grid;
  int pix;
  GnShape(int B, long long HW, int C, int threads, int waves, int unroll) {
    const int nvec = C / 8;
    const int bx = nvec < 64 ? nvec : 64;
    const int by = threads / bx > 0 ? threads / bx : 1;
    block = dim3(bx, by);
    const long long blocks = B < 148 * waves ? 148LL * waves / B : 1;
    const long long least = static_cast<long long>(by) * unroll;
    long long p = (HW + blocks - 1) / blocks;
    p = (p + least - 1) / least * least;
    pix = static_cast<int>(p);
    grid = dim3(static_cast<unsigned>((HW + p - 1) / p), B);
  }
};

// (GnShape divides by the sizes: an empty batch or image is refused here, as an empty grid would be by the launch)
static bool gn_sizes_ok(int B, long long HW, int C, int groups) {
  return B >= 1 && HW >= 1 && C >= 8 && C % 8 == 0 && groups >= 1 && C % groups == 0;
}

// Images that stay in L2 are through before a second wave's blocks have paid for their set-up.
static bool gn_small(int B, long long HW, int C) { return static_cast<long long>(B) * HW * C * 2 <= 72000000LL; }

// [2][C] sums of the block, and 16 per thread where the threads' rings were. Beyond the 48 KB that every launch may have the kernel is
// asked for more.
constexpr int GN_MAX_CHANNELS = 6144;
template <class Ring>
static size_t gn_smem(const GnShape& s, int C) {
  const int threads = s.block.x * s.block.y;
  return 2 * static_cast<size_t>(C) * sizeof(float) + std::max<size_t>(16 * sizeof(float) * threads, Ring::bytes(threads));
}
template <class Kernel>
static bool gn_limit(SharedLimit& limit, Kernel kernel, size_t bytes) {
  return bytes <= 47 * 1024 || limit.raise(reinterpret_cast<const void*>(kernel), 160 * 1024) == cudaSuccess;
}

static int groupnorm_stats_launch(const void* x, float* sums, int B, long long HW, int C, int groups, float* stats, unsigned int* ticket,
                                  float inv_count, float eps, cudaStream_t stream) {
  if (!gn_sizes_ok(B, HW, C, groups) || C > GN_MAX_CHANNELS) return -1;
  // Every block ends in two atomics per group on the same addresses, and its warps meet in shared memory before. While the image
  // is L2-sized the passes over it are shorter than that, and one block per SM is enough (us, 1 / 3 blocks per SM: 64800 x 192 13 / 21,
  // 139264 x 128 15 / 22, 139264 x 256 20 / 23, 139264 x 384 52 / 29).
  const GnShape s(B, HW, C, 512, gn_small(B, HW, C) ? 1 : 3, 2);
  const size_t bytes = gn_smem<GnStatsRing>(s, C);
  static SharedLimit limit;
  if (!gn_limit(limit, groupnorm_stats_kernel, bytes)) return -3;
  launch_chained(groupnorm_stats_kernel, s.grid, s.block, bytes, stream, static_cast<const __nv_bfloat16*>(x), sums, HW, C, groups, s.pix, stats,
                 ticket, inv_count, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
int groupnorm_stats(const void* x, float* sums, int B, long long HW, int C, int groups, cudaStream_t stream) {
  return groupnorm_stats_launch(x, sums, B, HW, C, groups, nullptr, nullptr, 0.f, 0.f, stream);
}
// Mean and reciprocal deviation in one launch; sums [B * groups * 2] and the ticket behind them zero before and after.
int groupnorm_mean_rstd(const void* x, float* sums, float* stats, int B, long long HW, int C, int groups, float inv_count, float eps,
                        cudaStream_t stream) {
  return groupnorm_stats_launch(x, sums, B, HW, C, groups, stats, reinterpret_cast<unsigned int*>(sums + 2LL * B * groups), inv_count, eps, stream);
}

int groupnorm_silu_apply(const void* x, const float* stats, const void* gamma, const void* beta, const void* res, void* y,
                         int B, long long HW, int C, int groups, cudaStream_t stream) {
  if (!gn_sizes_ok(B, HW, C, groups)) return -1;
  const GnShape s(B, HW, C, 256, gn_small(B, HW, C) ? 2 : 4, 2);
  launch_chained(res != nullptr ? groupnorm_silu_apply_kernel<true> : groupnorm_silu_apply_kernel<false>, s.grid, s.block,
                 GnPairRing::bytes(s.block.x * s.block.y), stream, static_cast<const __nv_bfloat16*>(x), stats,
                 static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta), static_cast<const __nv_bfloat16*>(res),
                 static_cast<__nv_bfloat16*>(y), HW, C, groups, s.pix);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int groupnorm_silu_bwd_reduce(const void* dy, const void* x, const float* stats, const void* gamma, const void* beta,
                              float* red, float* dgamma, float* dbeta, int B, long long HW, int C, int groups,
                              cudaStream_t stream) {
  if (!gn_sizes_ok(B, HW, C, groups) || C > GN_MAX_CHANNELS) return -1;
  const bool tiny = static_cast<long long>(B) * HW * C <= 1500000LL;      // (not enough pixels for larger blocks)
  const GnShape s(B, HW, C, tiny ? 256 : 512, tiny ? 2 : 1, 2);
  const size_t bytes = gn_smem<GnPairRing>(s, C);
  static SharedLimit limit;
  if (!gn_limit(limit, groupnorm_silu_bwd_reduce_kernel, bytes)) return -3;
  launch_chained(groupnorm_silu_bwd_reduce_kernel, s.grid, s.block, bytes, stream,
                 static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), stats, static_cast<const __nv_bfloat16*>(gamma),
                 static_cast<const __nv_bfloat16*>(beta), red, HW, C, groups, s.pix, dgamma, dbeta);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int groupnorm_finalize(float* sums, float* stats, int cells, float inv_count, float eps, cudaStream_t stream) {
  if (cells <= 0) return 0;
  launch_chained(groupnorm_finalize_kernel, (cells + 255) / 256, 256, 0, stream, sums, stats, cells, inv_count, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int strided_add_f32(float* src, float* dst, int na, int nb, int nc, long long sa, long long sb, long long sc, cudaStream_t stream) {
  const long long total = static_cast<long long>(na) * nb * nc;
  if (total <= 0) return 0;
  launch_chained(strided_add_kernel, grid_for(total, 256), 256, 0, stream, src, dst, na, nb, nc, sa, sb, sc);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int swap_middle_vectors(const void* in, void* out, long long P, long long A, long long B, long long run, cudaStream_t stream) {
  const long long total = P * A * B * run;
  if (P < 0 || A < 0 || B < 0 || run < 0 || total > 0x70000000LL) return -1;
  if (total == 0) return 0;
  launch_chained(swap_middle_kernel, static_cast<unsigned>((total + 1023) / 1024), 256, 0, stream, static_cast<const uint4*>(in),
                 static_cast<uint4*>(out), static_cast<unsigned>(A), static_cast<unsigned>(B), static_cast<unsigned>(run), static_cast<unsigned>(total));
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int fold_taps_f32(float* src, float* dst, int taps, int rows, int cols, cudaStream_t stream) {
  if (taps < 1 || taps > FOLD_TAPS) return -1;
  if (rows <= 0 || cols <= 0) return 0;
  const dim3 grid((cols + FOLD_COLS - 1) / FOLD_COLS, (rows + FOLD_ROWS - 1) / FOLD_ROWS);
  launch_chained(fold_taps_kernel, grid, dim3(256), 0, stream, src, dst, taps, rows, cols);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int groupnorm_silu_bwd_apply(const void* dy, const void* x, const float* stats, const float* red, const void* gamma,
                             const void* beta, void* dx, int B, long long HW, int C, int groups, float inv_count,
                             cudaStream_t stream) {
  if (!gn_sizes_ok(B, HW, C, groups)) return -1;
  const GnShape s(B, HW, C, 256, gn_small(B, HW, C) ? 2 : 4, 2);
  const size_t bytes = (groups * 2 + 3) / 4 * 4 * sizeof(float) + GnPairRing::bytes(s.block.x * s.block.y);
  static SharedLimit limit;
  if (!gn_limit(limit, groupnorm_silu_bwd_apply_kernel, bytes)) return -3;
  launch_chained(groupnorm_silu_bwd_apply_kernel, s.grid, s.block, bytes, stream,
                 static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), stats, red, static_cast<const __nv_bfloat16*>(gamma),
                 static_cast<const __nv_bfloat16*>(beta), static_cast<__nv_bfloat16*>(dx), HW, C, groups, inv_count, s.pix);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int masked_loss_fwd_bwd(const void* pred, const void* label, const void* mask, long long n, long long mask_period,
                        int kind, float grad_scale, float* loss_sum, void* grad, cudaStream_t stream) {
  if (n % 8 != 0 || (mask != nullptr && mask_period % 8 != 0)) return -1;
  const long long nvec = n / 8;
  launch_chained(masked_loss_kernel, grid_for(nvec, 256), 256, 0, stream, static_cast<const __nv_bfloat16*>(pred),
                 static_cast<const __nv_bfloat16*>(label), static_cast<const __nv_bfloat16*>(mask), nvec, mask != nullptr ? mask_period / 8 : 1, kind,
                 grad_scale, loss_sum, static_cast<__nv_bfloat16*>(grad));
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int adamw_step(float* master, float* exp_avg, float* exp_avg_sq, const void* grad, int grad_is_bf16, void* param_bf16,
               long long n, float lr, float beta1, float beta2, float eps, float weight_decay, float bias_corr1,
               float bias_corr2_sqrt, float grad_scale, cudaStream_t stream) {
  const int grid = grid_for(n, 256);
  if (grad_is_bf16)
    launch_chained(adamw_kernel<true>, grid, 256, 0, stream, master, exp_avg, exp_avg_sq, grad, static_cast<__nv_bfloat16*>(param_bf16), n,
                   lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2_sqrt, grad_scale);
  else
    launch_chained(adamw_kernel<false>, grid, 256, 0, stream, master, exp_avg, exp_avg_sq, grad, static_cast<__nv_bfloat16*>(param_bf16), n,
                   lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2_sqrt, grad_scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int cast_f32_to_bf16(const float* src, void* dst, long long n, cudaStream_t stream) {
  launch_chained(cast_f32_bf16_kernel, grid_for(n, 256), 256, 0, stream, src, static_cast<__nv_bfloat16*>(dst), n);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int add_bf16(const void* a, const void* b, void* out, long long n, cudaStream_t stream) {
  if (n % 8 != 0) return -1;
  launch_chained(add_bf16_kernel, grid_for(n / 8, 256), 256, 0, stream, static_cast<const uint4*>(a), static_cast<const uint4*>(b),
                 static_cast<uint4*>(out), n / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int conv_s2_col2im(const void* dcol, void* out, int B, int Ho, int Wo, int W, int C, int r0, int rows, int out_f32,
                   cudaStream_t stream) {
  if (C % 8 != 0 || rows <= 0) return -1;
  const long long total = static_cast<long long>(B) * rows * W * (C / 8);
  if (out_f32)
    launch_chained(conv_s2_col2im_kernel<true>, grid_for(total, 256), 256, 0, stream, static_cast<const uint4*>(dcol), out, B, Ho, Wo, W,
                   C / 8, r0, rows);
  else
    launch_chained(conv_s2_col2im_kernel<false>, grid_for(total, 256), 256, 0, stream, static_cast<const uint4*>(dcol), out, B, Ho, Wo, W,
                   C / 8, r0, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int patch_relayout(const void* image, const void* add, void* patches, void* image_out, int to_patches, int B, int H, int W, int C,
                   int p, int Hp, int Wp, int top, int left, cudaStream_t stream) {
  if (p < 1 || Hp % p != 0 || Wp % p != 0 || top < 0 || left < 0 || top + H > Hp || left + W > Wp || B < 1 || H < 1 || W < 1) return -1;
  const int hn = Hp / p;
  const long long rows = static_cast<long long>(B) * (to_patches ? Hp : H);
  if (rows > 65535 || static_cast<long long>(Wp) * C > (1LL << 30)) return -1;
  unsigned long long bytes = (static_cast<unsigned long long>(p) * C * 2) | (static_cast<unsigned long long>(W) * C * 2) |
                             (static_cast<unsigned long long>(left) * C * 2) | 16ull;
  for (const void* q : {image, add, static_cast<const void*>(patches), static_cast<const void*>(image_out)})
    bytes |= reinterpret_cast<unsigned long long>(q);
  const auto launch = [&](auto unit) {
    using V = decltype(unit);
    const int per = static_cast<int>(sizeof(V) / 2);
    const int row_units = Wp * C / per, img_units = W * C / per, seg = p * C / per, lu = left * C / per;
    const int span = to_patches ? row_units : img_units;
    const dim3 grid((span + 256 * PATCH_UNROLL - 1) / (256 * PATCH_UNROLL), static_cast<unsigned>(rows));
    if (to_patches)
      launch_chained(pad_patchify_kernel<V>, grid, 256, 0, stream, static_cast<const V*>(image), static_cast<V*>(patches), H, p, hn, top,
                     lu, img_units, row_units, seg);
    else
      launch_chained(unpatchify_crop_kernel<V>, grid, 256, 0, stream, static_cast<const V*>(patches), static_cast<const V*>(add),
                     static_cast<V*>(image_out), H, p, hn, top, lu, img_units, row_units, seg);
  };
  if (bytes % 16 == 0) launch(uint4{});
  else if (bytes % 8 == 0) launch(uint2{});
  else if (bytes % 4 == 0) launch(uint32_t{});
  else launch(static_cast<unsigned short>(0));
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int pack_taps_bf16(const void* w, void* out, int N1, int N2, int V2, int T, int C, int Cpad, long long s1, long long s2, long long sc,
                   const int* offsets, cudaStream_t stream) {
  if (T < 1 || T > 9 || Cpad % 2 != 0 || C > Cpad || N1 < 1 || N2 < 1) return -1;
  PackTaps p = {N2, V2, T, C, Cpad, s1, s2, sc, {}};
  for (int t = 0; t < T; ++t) p.off[t] = offsets[t];
  const long long total = static_cast<long long>(N1) * N2 * T * (Cpad / 2);
  launch_chained(pack_taps_kernel, grid_for(total, 256), 256, 0, stream, static_cast<const __nv_bfloat16*>(w), static_cast<uint32_t*>(out),
                 p, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int attn_rowdot(const void* o, const void* dout, float* drow, long long rows, int C, int heads, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (heads <= 0 || C % heads != 0) return -1;
  const int hd = C / heads;
  if (hd != 16 && hd != 32 && hd != 64 && hd != 128) return -1;
  launch_chained(attn_rowdot_kernel, grid_for(rows * 32, 256), 256, 0, stream, static_cast<const uint4*>(o),
                 static_cast<const uint4*>(dout), drow, rows, C / 8, hd / 8, heads);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int grad_inspect(const float* grad, long long n, float* out2, cudaStream_t stream) {
  if (n <= 0) return 0;
  launch_chained(grad_inspect_kernel, grid_for(n, 256 * 8, 148 * 8), 256, 0, stream, grad, n, out2);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sum_slots_bf16(const void* src, void* out, int slots, long long n, cudaStream_t stream, const void* bias,
                   const void* residual, int cols) {
  if (n % 8 != 0 || slots < 1) return -1;
  if (bias != nullptr && (cols <= 0 || cols % 8 != 0 || n % cols != 0)) return -1;
  launch_chained(sum_slots_bf16_kernel, grid_for(n / 8, 256), 256, 0, stream, static_cast<const uint4*>(src), static_cast<uint4*>(out),
                 slots, n / 8, static_cast<const uint4*>(bias), static_cast<const uint4*>(residual), cols > 0 ? cols / 8 : 1);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace tb
