// Prefill of the gated delta rule on bf16 inputs, 64 tokens at a time, in two kernels.  The equations of a chunk are those of
// gdn_chunk.cu: with the running sum G of the log decays, the incoming state S0 and T = (I + A)^-1,
//
//   U = T diag(beta) V - T diag(beta exp(G)) K S0,   O = exp(G) (Q S0) + (M * Q K^T) U,   S = exp(G_C) S0 + K^T (exp(G_C - G) U).
//
// One kernel that walks a request's chunks and does all of that per chunk spends its time on what does not depend on the state
// at all (31 us a chunk, of which the products with the state are under 2).  So:
//   * gdn_prepare_kernel takes every (chunk, head) by itself, all of them side by side: unit norms, decays, K K^T and Q K^T, the
//     inverse T (16 x 16 blocks by substitution, joined by products, in fp32), and from it -W = -T diag(beta exp(G)) K and
//     U0 = T diag(beta) V.
//   * gdn_scan_kernel walks the chunks with the state in registers.  A CTA owns a block of 64 value features, whose columns of the
//     state never mix.
// Products enter the tensor cores in 16 bits.  K, Q and V are bf16 and enter as they are; every fp32 operand (T, W, the state, U, the
// decayed scores) enters as two bf16 terms, its rounding and the remainder: 16 bits of it, against the 11 of a tf32 operand, for as many
// instructions.  Sums and the state are fp32.  The first kernel's products are warp-level MMAs, chained through element-wise steps; the
// scan's are tcgen05 with accumulators in tensor memory: what bounds the scan is the chain from one chunk's state to the next, and of a
// chunk's 2032 warp-level MMAs, their fragment loads and the addresses of its copies it made 12300 cycles.
//
// Measured (16 heads of 128 x 128, the longest length given; one kernel with tf32 operands, two kernels with warp-level MMAs in both, these):
// 4 x 2000 tokens 1274, 375, 212 us, 1 x 2048 582, 128, 113; 8 x 1000 374 -> 217, 8 x 2048 734 -> 412, 1 x 300 33.3 -> 31.5.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace mb200 {
namespace {

constexpr int kC = 64;                 // tokens of a chunk
constexpr int kD = 128;                // key features, zero-padded
constexpr int kThreads = 256;
constexpr int kLd = kC + 4;            // row stride (floats) of chunk x chunk matrices
constexpr int kXLd = 18;               // of 16 x 16 blocks
constexpr int kTileBytes = kC * kD * 2;  // 16 KB: a chunk of K, Q or V, two planes
constexpr int kScalars = 160;          // floats: exp(G) / |q|, exp(G_C - G) / |k|, exp(G_C)
constexpr int kBV = 64;                // value features of a scan CTA
constexpr int kPlane = kC * 128;       // 8 KB: 64 rows of 64 16-bit values, one swizzle span each

// What the first kernel leaves for a (chunk, head): the scan's operands as they lie in its shared memory (planes of 64 rows with the
// 128-byte swizzle, so that one bulk copy moves them all), the scalars behind them, and U0 in the order in which the scan's threads
// take it, [block of 64 value features][four features][token][4].
struct Slot {
  // for each half of the key features W (rounding), Q, W (remainder): rows 0 - 127 of the left operand are W and Q together
  static constexpr int kWhi = 0, kQ = kPlane, kWlo = 2 * kPlane, kHalf = 3 * kPlane;
  static constexpr int kK = 2 * kHalf, kP = kK + 2 * kPlane;       // K: two halves; decayed scores: rounding, remainder
  static constexpr int kScal = kP + 2 * kPlane, kBulk = kScal + kScalars * 4;
  static constexpr int64_t kU = kBulk;
};
static_assert(Slot::kBulk % 16 == 0, "bulk copies move multiples of 16 bytes");
__host__ __device__ inline int value_blocks(int dv) { return (dv + kBV - 1) / kBV; }
__host__ __device__ inline int64_t slot_bytes(int dv) { return Slot::kU + static_cast<int64_t>(value_blocks(dv)) * kBV * kC * 4; }

struct PrefillParams {
  GdnRuleParams r;
  uint8_t* ws;
  int* status;
  int chunk0, span;      // chunks chunk0 .. chunk0 + span of every request are in the workspace
  int wide;              // state and outputs may be moved 16 bytes at a time
};

// 16-byte piece of a row of 128 values in two planes: eight neighbouring rows lie in different banks
__device__ __forceinline__ uint32_t at128(int row, int chunk) { return (chunk >> 3) * kPlane + row * 128 + (((chunk & 7) ^ (row & 7)) << 4); }
// (a, b) as the pair of their roundings and the pair of the remainders
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(a, b);
  const float2 r = unpack_bf16x2(hi);
  lo = pack_bf16x2(a - r.x, b - r.y);
}
using BF = __nv_bfloat16;

// fragments of four 8 x 8 tiles to their rows, whose addresses the lanes give (8 lanes a tile)
__device__ __forceinline__ void stsm4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

__global__ void __launch_bounds__(kThreads, 2) gdn_prepare_kernel(const PrefillParams pp) {
  const GdnRuleParams& p = pp.r;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint8_t* sK = smem;
  uint8_t* sQ = sK + kTileBytes;
  uint8_t* sV = sQ + kTileBytes;
  float* sA = reinterpret_cast<float*>(sV + kTileBytes);
  float* sT = sA + kC * kLd;
  float* sX = sT + kC * kLd;             // [3][16][kXLd]
  float* sG = sX + 3 * 16 * kXLd;
  float* sB = sG + kC;
  float* sRk = sB + kC;
  float* sRq = sRk + kC;
  float* sE = sRq + kC;
  uint8_t* sP = reinterpret_cast<uint8_t*>(sE + kC);       // the decayed scores, two planes
  // -W, planes as they lie in the slot: where A was, and Q
  auto w_plane = [&](int half) { return half == 0 ? reinterpret_cast<uint8_t*>(sA) : sQ; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int h = blockIdx.y, b = blockIdx.z;
  pdl_wait_loads();
  pdl_launch_dependents();
  const int n = p.lens[b];
  const int c0 = (pp.chunk0 + static_cast<int>(blockIdx.x)) * kC;
  if (c0 >= n) return;
  const int nv = min(kC, n - c0);
  const int hk = h / (p.heads / p.k_heads);
  const int64_t row0 = static_cast<int64_t>(p.q_start[b]) + c0;
  uint8_t* slot = pp.ws + ((static_cast<int64_t>(b) * pp.span + blockIdx.x) * p.heads + h) * slot_bytes(p.dv);

  const BF* q = static_cast<const BF*>(p.q) + static_cast<int64_t>(hk) * p.dk;
  const BF* k = static_cast<const BF*>(p.k) + static_cast<int64_t>(hk) * p.dk;
  for (int i = tid; i < kC * 16; i += kThreads) {
    const int r = i >> 4, ch = i & 15;
    const bool ok = r < nv && ch * 8 < p.dk;
    const int64_t row = row0 + (ok ? r : 0);
    cp16_zfill(smem_u32(sK) + at128(r, ch), k + row * p.k_ld + (ok ? ch * 8 : 0), ok);
    cp16_zfill(smem_u32(sQ) + at128(r, ch), q + row * p.q_ld + (ok ? ch * 8 : 0), ok);
  }
  auto load_v = [&](int v0) {
    const BF* v = static_cast<const BF*>(p.v) + static_cast<int64_t>(h) * p.dv + v0;
    for (int i = tid; i < kC * 16; i += kThreads) {
      const int r = i >> 4, ch = i & 15;
      const bool ok = r < nv && v0 + ch * 8 < p.dv;
      cp16_zfill(smem_u32(sV) + at128(r, ch), v + (row0 + (ok ? r : 0)) * p.v_ld + (ok ? ch * 8 : 0), ok);
    }
    cp_commit();
  };
  load_v(0);
  if (tid < kC) {
    const int64_t at = (row0 + min(tid, nv - 1)) * p.heads + h;
    sG[tid] = tid < nv ? p.g[at] : 0.f;
    sB[tid] = tid < nv ? p.beta[at] : 0.f;
  }
  cp_wait<0>();
  fence_proxy_async_smem();
  __syncthreads();

  // ---- Q and K as the scan takes them ----
  if (tid == 0) {
    bulk_store(slot + Slot::kK, smem_u32(sK), 2 * kPlane);
    bulk_store(slot + Slot::kQ, smem_u32(sQ), kPlane);
    bulk_store(slot + Slot::kHalf + Slot::kQ, smem_u32(sQ) + kPlane, kPlane);
    bulk_commit();
  }
  // ---- norms of the rows, two threads to a row of K or of Q (in an order that keeps their pieces in different banks) ----
  const float qscale = 1.f / sqrtf(static_cast<float>(p.dk));
  {
    const int r = (tid >> 1) & (kC - 1), half = tid & 1;
    const uint8_t* from = tid < 2 * kC ? sK : sQ;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 v = *reinterpret_cast<const uint4*>(from + at128(r, half * 8 + (i ^ (half * 4))));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16x2(w[j]);
        ss = fmaf(a.x, a.x, fmaf(a.y, a.y, ss));
      }
    }
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    if (half == 0) {
      if (tid < 2 * kC) sRk[r] = 1.f / sqrtf(ss + 1e-6f);
      else sRq[r] = qscale / sqrtf(ss + 1e-6f);
    }
  }
  __syncthreads();
  if (warp == 0) {
    const float a = sG[2 * lane], ab = a + sG[2 * lane + 1];
    float incl = ab;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    const float before = incl - ab, total = __shfl_sync(0xffffffffu, incl, 31);
    float* scal = reinterpret_cast<float*>(slot + Slot::kScal);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * lane + i;
      const float G = i ? before + ab : before + a;
      sG[r] = G;
      sE[r] = expf(G);
      scal[r] = expf(G) * sRq[r];
      scal[kC + r] = expf(total - G) * sRk[r];
    }
    if (lane == 0) scal[2 * kC] = expf(total);
  }
  __syncthreads();

  // ---- K K^T (warps 0 - 3) and Q K^T (4 - 7), a row tile each, on and below the diagonal ----
  {
    const int ti = warp & 3;
    const bool is_q = warp >= 4;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
    const uint32_t left = smem_u32(is_q ? sQ : sK), right = smem_u32(sK);
#pragma unroll
    for (int kk = 0; kk < kD / 16; ++kk) {
      uint32_t a[4];
      ldsm4(a, left + at128(ti * 16 + (lane & 15), kk * 2 + (lane >> 4)));
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        if (np <= ti) {
          uint32_t w[4];
          ldsm4(w, right + at128(np * 16 + (lane & 7) + ((lane >> 4) << 3), kk * 2 + ((lane >> 3) & 1)));
          mma_16816<BF>(acc[2 * np], a[0], a[1], a[2], a[3], w[0], w[1]);
          mma_16816<BF>(acc[2 * np + 1], a[0], a[1], a[2], a[3], w[2], w[3]);
        }
      }
    }
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (np > ti && !is_q) continue;            // (the scores' tiles above the diagonal are written too: zero)
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int nt = 2 * np + (e >> 1), half = e & 1;
        const int i = ti * 16 + g + half * 8, j = nt * 8 + 2 * t;
        float v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const bool in = is_q ? j + c <= i : j + c < i;
          const float f = (is_q ? sRq[i] : sB[i] * sRk[i]) * sRk[j + c];
          v[c] = in ? __expf(sG[i] - sG[j + c]) * (f * acc[nt][half * 2 + c]) : 0.f;
        }
        if (is_q) split2(v[0], v[1], hi[e], lo[e]);
        else *reinterpret_cast<float2*>(sA + i * kLd + j) = make_float2(v[0], v[1]);
      }
      if (is_q) {
        const uint32_t at = smem_u32(sP) + at128(ti * 16 + (lane & 15), 2 * np + (lane >> 4));
        stsm4(at, hi[0], hi[1], hi[2], hi[3]);
        stsm4(at + kPlane, lo[0], lo[1], lo[2], lo[3]);
      }
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (tid == 0) {
    bulk_store(slot + Slot::kP, smem_u32(sP), 2 * kPlane);
    bulk_commit();
  }

  // ---- T = (I + A)^-1: the diagonal blocks by substitution, a thread per column ----
  if (tid < kC) {
    const int blk = (tid >> 4) * 16, col = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = i == col ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) s = fmaf(-sA[(blk + i) * kLd + blk + j], x[j], s);
      x[i] = s;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) sT[(blk + i) * kLd + blk + col] = x[i];
  }
  __syncthreads();
  // ---- the blocks below, diagonal by diagonal: T_ij = -T_ii sum_k A_ik T_kj.  Half the threads to a block, two neighbouring columns each,
  // so that a load serves two to four products (one value at a time the block products were bound by shared memory) ----
  {
    const int grp = tid >> 7, r = (tid >> 3) & 15, c = (tid & 7) * 2;
    for (int d = 1; d < 4; ++d) {
      for (int bi = d + grp; bi < 4; bi += 2) {
        const int bj = bi - d;
        float s0 = 0.f, s1 = 0.f;
        for (int m = bj * 16; m < bi * 16; m += 4) {
          const float4 a = *reinterpret_cast<const float4*>(sA + (bi * 16 + r) * kLd + m);
          const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = *reinterpret_cast<const float2*>(sT + (m + e) * kLd + bj * 16 + c);
            s0 = fmaf(av[e], x.x, s0);
            s1 = fmaf(av[e], x.y, s1);
          }
        }
        *reinterpret_cast<float2*>(sX + (bj * 16 + r) * kXLd + c) = make_float2(s0, s1);
      }
      __syncthreads();
      for (int bi = d + grp; bi < 4; bi += 2) {
        const int bj = bi - d;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int m = 0; m < 16; m += 4) {
          const float4 a = *reinterpret_cast<const float4*>(sT + (bi * 16 + r) * kLd + bi * 16 + m);
          const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = *reinterpret_cast<const float2*>(sX + (bj * 16 + m + e) * kXLd + c);
            s0 = fmaf(av[e], x.x, s0);
            s1 = fmaf(av[e], x.y, s1);
          }
        }
        *reinterpret_cast<float2*>(sT + (bi * 16 + r) * kLd + bj * 16 + c) = make_float2(-s0, -s1);
      }
      // the copies have read Q, whose place W takes
      if (d == 3 && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncthreads();
    }
  }

  // ---- -W = -T diag(beta exp(G) / |k|) K (warps 0 - 3) and U0 = T diag(beta) V (4 - 7) ----
  {
    const int ti = warp & 3;
    const bool is_u = warp >= 4;
    const int blocks = value_blocks(p.dv);
    for (int v0 = 0; v0 < p.dv; v0 += kD) {
      if (v0 > 0) {
        __syncthreads();
        load_v(v0);
        cp_wait<0>();
        __syncthreads();
        if (!is_u) continue;
      }
      float acc[16][4];
#pragma unroll
      for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
      const uint32_t right = smem_u32(is_u ? sV : sK);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks <= ti) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = ti * 16 + g + (i & 1) * 8, j = ks * 16 + 2 * t + (i >> 1) * 8;
            const float2 v = *reinterpret_cast<const float2*>(sT + row * kLd + j);
            const float f0 = is_u ? sB[j] : sB[j] * sE[j] * sRk[j], f1 = is_u ? sB[j + 1] : sB[j + 1] * sE[j + 1] * sRk[j + 1];
            split2(v.x * f0, v.y * f1, hi[i], lo[i]);
          }
#pragma unroll
          for (int np = 0; np < 8; ++np) {
            uint32_t w[4];
            ldsm4_t(w, right + at128(ks * 16 + (lane & 15), np * 2 + (lane >> 4)));
            mma_16816<BF>(acc[2 * np], hi[0], hi[1], hi[2], hi[3], w[0], w[1]);
            mma_16816<BF>(acc[2 * np + 1], hi[0], hi[1], hi[2], hi[3], w[2], w[3]);
            mma_16816<BF>(acc[2 * np], lo[0], lo[1], lo[2], lo[3], w[0], w[1]);
            mma_16816<BF>(acc[2 * np + 1], lo[0], lo[1], lo[2], lo[3], w[2], w[3]);
          }
        }
      }
      if (is_u) {
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int row = ti * 16 + g + half * 8, vc = v0 + nt * 8 + 2 * t, vb = vc / kBV;
            if (vb < blocks)
              *reinterpret_cast<float2*>(slot + Slot::kU + (static_cast<int64_t>(vb * (kBV / 4) + (vc % kBV) / 4) * kC + row) * 16 + (vc & 3) * 4) =
                  make_float2(acc[nt][half * 2], acc[nt][half * 2 + 1]);
          }
        }
      } else {
#pragma unroll
        for (int np = 0; np < 8; ++np) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int nt = 2 * np + (e >> 1), half = e & 1;
            split2(-acc[nt][half * 2], -acc[nt][half * 2 + 1], hi[e], lo[e]);
          }
          const uint32_t at = smem_u32(w_plane(np >> 2)) + at128(ti * 16 + (lane & 15), 2 * (np & 3) + (lane >> 4));
          stsm4(at, hi[0], hi[1], hi[2], hi[3]);
          stsm4(at + kPlane, lo[0], lo[1], lo[2], lo[3]);
        }
        fence_proxy_async_smem();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (tid == 0) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            bulk_store(slot + half * Slot::kHalf + Slot::kWhi, smem_u32(w_plane(half)), kPlane);
            bulk_store(slot + half * Slot::kHalf + Slot::kWlo, smem_u32(w_plane(half)) + kPlane, kPlane);
          }
          bulk_commit();
        }
      }
    }
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------------------------------
// The scan.  Warps 0 - 15 hold the state (a thread has 16 value features of one key feature) and form the operands; one thread of warp
// 16 moves the chunks and issues the products:
//   D1 = [W; Q] [S_hi | S_lo] and D2 = W_lo S_hi (rows 0 - 63 of D1 and D2 make W S, rows 64 - 127 of D1 are Q S),
//   dS = K^T [U'_hi | U'_lo],   D3 = P_hi [U_hi | U_lo] + P_lo U_hi  (rows 64 - 127; what stands in the other rows is not read).
// The two terms of a right operand are side by side, so that one instruction takes both.  What bounds it is the chain of a chunk: state ->
// operands -> D1, D2 (1000 cycles) -> U -> operands -> dS (300) -> state, with four handovers; D3, the outputs, the next chunk's copy
// and U0 lie beside it.  (Eight warps with 32 value features a thread: the element-wise parts of the chain took twice as long, and a
// chunk 7500 cycles.)
// Tensor memory: D1 0 - 127, D2 128 - 191, dS 256 - 383, D3 384 - 511.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kScanWarps = 16, kScanCols = kBV / (kScanWarps / 4), kScanThreads = 32 * (kScanWarps + 1);
constexpr int kOperand = kD * 128;                                   // 16 KB: one term of the state, [128][64]
constexpr int kScanSmem = 1024 + 2 * Slot::kScal + 2 * kOperand + 4 * kPlane + 2 * kScalars * 4 + 256;
static_assert(kScanSmem <= 232448, "shared memory");

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(smem_u32(bar))
               : "memory");
}

__global__ void __launch_bounds__(kScanThreads, 1) gdn_scan_kernel(const PrefillParams pp) {
  const GdnRuleParams& p = pp.r;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stages = smem;                                  // two chunks' operands
  uint8_t* sS = stages + 2 * Slot::kScal;                  // two terms of the state, [key feature][64]
  uint8_t* sU = sS + 2 * kOperand;                         // two terms of U, then of exp(G_C - G) / |k| U, [token][64]
  float* scalars = reinterpret_cast<float*>(sU + 4 * kPlane);
  uint64_t* loaded = reinterpret_cast<uint64_t*>(scalars + 2 * kScalars);      // [stage] bytes of the copies
  uint64_t* left = loaded + 2;               // [stage] commit: the chunk's products are complete (and its D3)
  uint64_t* state_ready = left + 2;          // all threads of the state
  uint64_t* u_ready = state_ready + 1;       // the same
  uint64_t* d_full = u_ready + 1;            // commit: D1, D2
  uint64_t* ds_full = d_full + 1;            // commit: dS
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(ds_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int vb = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  pdl_wait_loads();
  const int n = p.lens[b];
  const int chunks = (n + kC - 1) / kC;
  const int c_end = min(pp.chunk0 + pp.span, chunks);
  if (pp.chunk0 >= c_end) return;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&loaded[i], 1);
      mbar_init(&left[i], 1);
    }
    mbar_init(state_ready, 32 * kScanWarps);
    mbar_init(u_ready, 32 * kScanWarps);
    mbar_init(d_full, 1);
    mbar_init(ds_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kScanWarps) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  const uint32_t t_d1 = tmem, t_d2 = tmem + 128, t_ds = tmem + 256, t_d3 = tmem + 384;
  pdl_launch_dependents();

  auto slot_of = [&](int c) {
    return pp.ws + ((static_cast<int64_t>(b) * pp.span + (c - pp.chunk0)) * p.heads + h) * slot_bytes(p.dv);
  };
  if (warp == kScanWarps) {
    if (elect_one()) {
      auto load = [&](int c) {
        const int st = (c - pp.chunk0) & 1;
        const uint8_t* src = slot_of(c);
        mbar_arrive_expect_tx(&loaded[st], Slot::kBulk);
        bulk_load(smem_u32(stages) + st * Slot::kScal, src, Slot::kScal, &loaded[st]);
        bulk_load(smem_u32(scalars) + st * (kScalars * 4), src + Slot::kScal, kScalars * 4, &loaded[st]);
      };
      const uint32_t fmt = 1;                              // bf16 operands, fp32 sums
      const uint32_t id_128 = umma_idesc(128, 128, 1, fmt, fmt, 0, 1), id_64 = umma_idesc(128, 64, 1, fmt, fmt, 0, 1);
      const uint32_t id_kt = umma_idesc(128, 128, 1, fmt, fmt, 1, 1);
      const uint64_t st0 = umma_desc_k_sw128(smem_u32(stages));
      const uint64_t k0 = umma_desc_mn_sw128(smem_u32(stages + Slot::kK), kPlane, 1024);
      const uint64_t s_desc = umma_desc_mn_sw128(smem_u32(sS), kOperand, 1024);
      const uint64_t u_desc = umma_desc_mn_sw128(smem_u32(sU), kPlane, 1024);
      bool ok = true;
      auto wait_on = [&](uint64_t* bar, uint32_t parity) {
        if (ok && !mbar_wait(bar, parity, abort_flag)) ok = false;
        if (ok) tc_fence_after_sync();
      };
      load(pp.chunk0);
      if (pp.chunk0 + 1 < c_end) load(pp.chunk0 + 1);
      for (int c = pp.chunk0; c < c_end && ok; ++c) {
        const int i = c - pp.chunk0, st = i & 1;
        const uint32_t ph = i & 1, ph_stage = (i >> 1) & 1;
        const uint32_t off = st * (Slot::kScal >> 4);
        wait_on(&loaded[st], ph_stage);
        wait_on(state_ready, ph);
        if (!ok) break;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t a = st0 + off + (kk >> 2) * (Slot::kHalf >> 4) + (kk & 3) * 2;
          umma_f16(t_d1, a, s_desc + kk * (2048 >> 4), id_128, kk > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t a = st0 + off + ((Slot::kWlo + (kk >> 2) * Slot::kHalf) >> 4) + (kk & 3) * 2;
          umma_f16(t_d2, a, s_desc + kk * (2048 >> 4), id_64, kk > 0 ? 1u : 0u);
        }
        umma_commit(d_full);
        // every thread has left the chunk before, and its products were complete before these began: its stage is free
        if (i >= 1 && c + 1 < c_end) {
          wait_on(&left[st ^ 1], ((i - 1) >> 1) & 1);
          if (ok) load(c + 1);
        }
        wait_on(u_ready, ph);
        if (!ok) break;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16(t_ds, k0 + off + kk * (2048 >> 4), u_desc + ((2 * kPlane + kk * 2048) >> 4), id_kt, kk > 0 ? 1u : 0u);
        umma_commit(ds_full);
        // rows 64 - 127 of the left operand are the scores; the plane in front fills the others.  16 tokens at a time, into the rows of
        // these tokens and of those behind them: above the diagonal the scores are 0, and 0 times an infinity or a NaN is a NaN
        auto scores_by_u = [&](int plane, uint32_t idesc, bool first) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint32_t off_rows[4] = {~0u, ~0u, kk == 0 ? 0u : kk == 1 ? 0xFFFFu : ~0u, kk == 3 ? 0xFFFFu : 0u};
            umma_f16_rows(t_d3, st0 + off + ((plane - kPlane) >> 4) + kk * 2, u_desc + kk * (2048 >> 4), idesc, first && kk == 0 ? 0u : 1u, off_rows);
          }
        };
        scores_by_u(Slot::kP, id_128, true);
        scores_by_u(Slot::kP + kPlane, id_64, false);
        umma_commit(&left[st]);
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    constexpr int N = kScanCols;
    const int quad = warp & 3, col0 = (warp >> 2) * N;           // this warp's lanes of tensor memory, and its value features
    const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
    const int key = quad * 32 + lane, tok = (quad & 1) * 32 + lane;
    const bool is_o = quad >= 2;                                 // rows 64 - 127: outputs; rows 0 - 63: U
    const int cols = min(N, p.dv - vb * kBV - col0);             // may be negative
    float* S = p.state + ((static_cast<int64_t>(p.slots[b]) * p.heads + h) * p.dk + min(key, p.dk - 1)) * p.dv + vb * kBV + col0;
    const bool resume = p.has_state[b] != 0 || pp.chunk0 > 0;
    float s[N];
#pragma unroll
    for (int j = 0; j < N; j += 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (resume && key < p.dk && j < cols) v = pp.wide ? *reinterpret_cast<const float4*>(S + j) : make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
      s[j] = v.x;
      s[j + 1] = v.y;
      s[j + 2] = v.z;
      s[j + 3] = v.w;
    }
    float u0[N];
    auto load_u0 = [&](int c) {
      if (is_o) return;
      const float4* src = reinterpret_cast<const float4*>(slot_of(c) + Slot::kU) + static_cast<int64_t>(vb * (kBV / 4) + col0 / 4) * kC + tok;
#pragma unroll
      for (int j = 0; j < N / 4; ++j) {
        const float4 v = __ldcg(src + j * kC);
        u0[4 * j] = v.x;
        u0[4 * j + 1] = v.y;
        u0[4 * j + 2] = v.z;
        u0[4 * j + 3] = v.w;
      }
    };
    // values of a row as two terms into planes of 128-byte rows, `second` bytes apart
    auto put = [&](uint8_t* plane, int row, const float (&v)[N], float f, uint32_t second) {
#pragma unroll
      for (int q = 0; q < N / 8; ++q) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split2(v[q * 8 + 2 * j] * f, v[q * 8 + 2 * j + 1] * f, hi[j], lo[j]);
        uint8_t* to = plane + row * 128 + (((col0 / 8 + q) ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(to + second) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
    };
    // v += f * (the columns at `at` and, where there are two terms, those 64 on)
    auto add_columns = [&](uint32_t at, float (&v)[N], float f, bool two) {
      uint32_t r[N], r2[N];
      tmem_ld_32x16(at + lanes + col0, r);
      if (two) tmem_ld_32x16(at + 64 + lanes + col0, r2);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < N; ++j) {
        v[j] = fmaf(__uint_as_float(r[j]), f, v[j]);
        if (two) v[j] = fmaf(__uint_as_float(r2[j]), f, v[j]);
      }
    };
    static_assert(N == 16, "loads of tensor memory");
    bool ok = true;
    auto wait_on = [&](uint64_t* bar, uint32_t parity) {
      if (ok && !mbar_wait(bar, parity, abort_flag)) ok = false;
      tc_fence_after_sync();
    };
    float v[N];
    auto finish_outputs = [&](int c) {       // v: exp(G) Q S of the chunk
      const int i = c - pp.chunk0;
      wait_on(&left[i & 1], (i >> 1) & 1);
      add_columns(t_d3, v, 1.f, true);
      if (!ok || c * kC + tok >= n) return;
      BF* out = static_cast<BF*>(p.out) + ((static_cast<int64_t>(p.q_start[b]) + static_cast<int64_t>(c) * kC + tok) * p.heads + h) * p.dv + vb * kBV + col0;
      if (cols == N && pp.wide) {
#pragma unroll
        for (int q = 0; q < N / 8; ++q)
          reinterpret_cast<uint4*>(out)[q] = make_uint4(pack_bf16x2(v[q * 8], v[q * 8 + 1]), pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]),
                                                        pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]), pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]));
      } else {
#pragma unroll
        for (int j = 0; j < N; j += 2)
          if (j < cols) *reinterpret_cast<uint32_t*>(out + j) = pack_bf16x2(v[j], v[j + 1]);
      }
    };
    load_u0(pp.chunk0);
    for (int c = pp.chunk0; c < c_end && ok; ++c) {
      const int i = c - pp.chunk0, st = i & 1;
      const uint32_t ph = i & 1, ph_stage = (i >> 1) & 1;
      put(sS, key, s, 1.f, kOperand);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(state_ready);
      if (is_o && i > 0) finish_outputs(c - 1);
      wait_on(&loaded[st], ph_stage);
      const float* scal = scalars + st * kScalars;
      const float f = scal[is_o ? tok : kC + tok], carry = scal[2 * kC];
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = is_o ? 0.f : u0[j];
      wait_on(d_full, ph);
      if (is_o) {
        add_columns(t_d1, v, f, true);
      } else {
        add_columns(t_d1, v, 1.f, true);
        add_columns(t_d2, v, 1.f, false);
        put(sU + 2 * kPlane, tok, v, f, kPlane);
        put(sU, tok, v, 1.f, kPlane);
        fence_proxy_async_smem();
      }
      tc_fence_before_sync();
      mbar_arrive(u_ready);
      if (c + 1 < c_end) load_u0(c + 1);
#pragma unroll
      for (int j = 0; j < N; ++j) s[j] *= carry;
      wait_on(ds_full, ph);
      add_columns(t_ds, s, 1.f, true);
    }
    if (is_o && ok) finish_outputs(c_end - 1);
    if (!ok) *abort_flag = 1;
    if (key < p.dk && ok) {
#pragma unroll
      for (int j = 0; j < N; j += 4) {
        if (j >= cols) continue;
        if (pp.wide) {
          *reinterpret_cast<float4*>(S + j) = make_float4(s[j], s[j + 1], s[j + 2], s[j + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j + e] = s[j + e];
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0 && pp.status != nullptr) atomicExch(pp.status, kStatusPipelineTimeout);
    // copies may still be in flight: give them time to land before the CTA's memory is reused
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == kScanWarps) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

constexpr int kPrepareSmem = 3 * kTileBytes + (2 * kC * kLd + 3 * 16 * kXLd + 5 * kC) * 4 + 2 * kPlane + 128;
static_assert(2 * (kPrepareSmem + 1024) <= 228 * 1024, "two CTAs of the first kernel per SM");

}  // namespace

bool gdn_prefill_covers(const GdnRuleParams& p) { return p.dt == kBF16 && !p.split_tf32 && gdn_chunk_covers(p); }

// As many chunks of all requests as `most_bytes` have room for; where not even one fits, one chunk of equal groups of requests.  The
// least is a chunk of one request.  A (chunk, head) takes 115328 bytes at 128 value features, Q and K as the scan's operands among them:
// 512 MB are 72 chunks of four requests of 16 heads.  A span costs a start of both kernels and the state's way through memory: 32 x 1024
// tokens 854 us with 512 MB, 1186 with 128 MB, 788 with 4 GB; 4 x 2000 212, 230 and 212.  (Groups of requests that fill the GPU once, with
// longer spans, leave the scan's last CTAs of every group alone; with the scan by warp-level MMAs 1467 us instead of 1388.)
GdnPrefillPlan gdn_prefill_plan(const GdnRuleParams& p, int max_len, int64_t most_bytes) {
  const int64_t chunk = slot_bytes(p.dv) * p.heads, slots = std::max<int64_t>(1, most_bytes / chunk);
  const int64_t batch = std::max(1, p.batch), groups = (batch + slots - 1) / slots, group = (batch + groups - 1) / groups;
  const int64_t span = std::max<int64_t>(1, std::min<int64_t>((max_len + kC - 1) / kC, slots / group));
  return {static_cast<int>(group), static_cast<int>(span), group * span * chunk};
}

int launch_gdn_prefill(const GdnRuleParams& p, void* ws, const GdnPrefillPlan& plan, int max_len, int* status, cudaStream_t s) {
  if (p.batch <= 0 || max_len <= 0) return 0;
  if (!gdn_prefill_covers(p) || p.heads % p.k_heads != 0 || p.g == nullptr || (reinterpret_cast<uintptr_t>(p.out) & 3) != 0) return -1;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_prepare_kernel), kPrepareSmem) != cudaSuccess) return -3;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_scan_kernel), kScanSmem) != cudaSuccess) return -3;
  const int wide = ((reinterpret_cast<uintptr_t>(p.state) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0;
  const int chunks = (max_len + kC - 1) / kC;
  for (int b0 = 0; b0 < p.batch; b0 += plan.group) {
    GdnRuleParams r = p;
    r.batch = std::min(plan.group, p.batch - b0);
    r.slots += b0;
    r.lens += b0;
    r.has_state += b0;
    r.q_start += b0;
    for (int c0 = 0; c0 < chunks; c0 += plan.span) {
      PrefillParams pp{r, static_cast<uint8_t*>(ws), status, c0, plan.span, wide};
      cudaError_t err = launch_pdl(gdn_prepare_kernel, dim3(std::min(plan.span, chunks - c0), r.heads, r.batch), dim3(kThreads), kPrepareSmem, s, pp);
      note_launch();      // the pair counts as one: the rule over a span
      if (err != cudaSuccess) return -4;
      err = launch_pdl(gdn_scan_kernel, dim3(value_blocks(r.dv), r.heads, r.batch), dim3(kScanThreads), kScanSmem, s, pp);
      if (err != cudaSuccess) return -4;
    }
  }
  return 0;
}

}  // namespace mb200
