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
//   * gdn_scan_kernel walks the chunks with the state in its accumulators: U = U0 - W S0, then O and the next S; two barriers a
//     chunk, the next chunk's operands on their way meanwhile.  A CTA owns a block of the value features, whose columns of the
//     state never mix.
// Products are warp-level MMAs.  K, Q and V are bf16 and enter as they are; every fp32 operand (T, W, the state, U, the decayed
// scores) enters as two bf16 terms, its rounding and the remainder: 16 bits of it, against the 11 of a tf32 operand, for as many
// instructions.  Sums and the state are fp32.
//
// Measured (16 heads of 128 x 128; one kernel with tf32 operands, then these two): 4 x 2000 tokens
// 1274 -> 433 us, 1 x 2048 582 -> 126, 8 x 2048 1612 -> 732, 32 x 1024 2849 -> 1388; the state's error against 64 bits 2e-4 -> 4e-6.
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
constexpr int kRow = kD * 2;           // bytes of a K, Q, V or W row in shared memory
constexpr int kTileBytes = kC * kRow;  // 16 KB
constexpr int kPBytes = kC * kC * 2;   // 8 KB
constexpr int kScalars = 160;          // floats: exp(G) / |q|, exp(G_C - G) / |k|, exp(G_C)

// what the first kernel leaves for a (chunk, head)
struct Slot {
  static constexpr int64_t kW = 0, kP = 2 * kTileBytes, kScal = kP + 2 * kPBytes, kU = kScal + kScalars * 4;
};
__host__ __device__ inline int64_t slot_bytes(int dv) { return Slot::kU + static_cast<int64_t>(kC) * ((dv + 15) / 16 * 16) * 4; }

struct PrefillParams {
  GdnRuleParams r;
  uint8_t* ws;
  int chunk0, span;      // chunks chunk0 .. chunk0 + span of every request are in the workspace
};

__device__ __forceinline__ uint32_t at128(int row, int chunk) { return row * kRow + ((chunk ^ (row & 7)) << 4); }   // 256-byte rows
__device__ __forceinline__ uint32_t at64(int row, int chunk) { return row * (kC * 2) + ((chunk ^ (row & 7)) << 4); }  // 128-byte rows
// rows of BV 16-bit values: eight rows of a fragment load fall on different 16-byte groups of the banks
template <int BV>
__device__ __forceinline__ uint32_t at_v(int row, int chunk) {
  constexpr int kCh = BV / 8, kPer = 8 / kCh;
  return row * (BV * 2) + ((chunk ^ ((row / kPer) & (kCh - 1))) << 4);
}
// (a, b) as the pair of their roundings and the pair of the remainders
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(a, b);
  const float2 r = unpack_bf16x2(hi);
  lo = pack_bf16x2(a - r.x, b - r.y);
}
using BF = __nv_bfloat16;

__global__ void __launch_bounds__(kThreads, 2) gdn_prepare_kernel(const PrefillParams pp) {
  const GdnRuleParams& p = pp.r;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint8_t* sK = smem;
  uint8_t* sQ = sK + kTileBytes;
  uint8_t* sV = sQ + kTileBytes;
  float* sA = reinterpret_cast<float*>(sV + kTileBytes);
  float* sT = sA + kC * kLd;
  float* sX = sT + kC * kLd;             // [3][16][17]
  float* sG = sX + 3 * 16 * 17;
  float* sB = sG + kC;
  float* sRk = sB + kC;
  float* sRq = sRk + kC;
  float* sE = sRq + kC;
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
  __syncthreads();

  // ---- norms of the rows (a warp takes eight), running sum of the log decays ----
  const float qscale = 1.f / sqrtf(static_cast<float>(p.dk));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = warp * 8 + i;
    float s[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint2 v = *reinterpret_cast<const uint2*>((w ? sQ : sK) + at128(r, lane >> 1) + (lane & 1) * 8);
      const float2 a = unpack_bf16x2(v.x), c = unpack_bf16x2(v.y);
      s[w] = warp_sum(a.x * a.x + a.y * a.y + c.x * c.x + c.y * c.y);
    }
    if (lane == 0) {
      sRk[r] = 1.f / sqrtf(s[0] + 1e-6f);
      sRq[r] = qscale / sqrtf(s[1] + 1e-6f);
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
    for (int nt = 0; nt < 8; ++nt) {
      if (nt >= 2 * (ti + 1)) continue;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = ti * 16 + g + half * 8, j = nt * 8 + 2 * t;
        float v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const bool in = is_q ? j + c <= i : j + c < i;
          const float f = (is_q ? sRq[i] : sB[i] * sRk[i]) * sRk[j + c];
          v[c] = in ? __expf(sG[i] - sG[j + c]) * (f * acc[nt][half * 2 + c]) : 0.f;
        }
        if (is_q) {
          uint32_t hi, lo;
          split2(v[0], v[1], hi, lo);
          uint8_t* dst = slot + Slot::kP + i * (kC * 2) + j * 2;
          *reinterpret_cast<uint32_t*>(dst) = hi;
          *reinterpret_cast<uint32_t*>(dst + kPBytes) = lo;
        } else {
          *reinterpret_cast<float2*>(sA + i * kLd + j) = make_float2(v[0], v[1]);
        }
      }
    }
  }
  __syncthreads();

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
  // ---- the blocks below, diagonal by diagonal: T_ij = -T_ii sum_k A_ik T_kj ----
  {
    const int r = tid >> 4, c = tid & 15;
    for (int d = 1; d < 4; ++d) {
      for (int bi = d; bi < 4; ++bi) {
        const int bj = bi - d;
        float s = 0.f;
        for (int m = bj * 16; m < bi * 16; ++m) s = fmaf(sA[(bi * 16 + r) * kLd + m], sT[m * kLd + bj * 16 + c], s);
        sX[((bi - d) * 16 + r) * 17 + c] = s;
      }
      __syncthreads();
      for (int bi = d; bi < 4; ++bi) {
        float s = 0.f;
#pragma unroll
        for (int m = 0; m < 16; ++m) s = fmaf(sT[(bi * 16 + r) * kLd + bi * 16 + m], sX[((bi - d) * 16 + m) * 17 + c], s);
        sT[(bi * 16 + r) * kLd + (bi - d) * 16 + c] = -s;
      }
      __syncthreads();
    }
  }

  // ---- -W = -T diag(beta exp(G) / |k|) K (warps 0 - 3) and U0 = T diag(beta) V (4 - 7) ----
  {
    const int ti = warp & 3;
    const bool is_u = warp >= 4;
    const int dv16 = (p.dv + 15) / 16 * 16;
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
#pragma unroll
      for (int nt = 0; nt < 16; ++nt) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int row = ti * 16 + g + half * 8, col = nt * 8 + 2 * t;
          const float a = acc[nt][half * 2], c = acc[nt][half * 2 + 1];
          if (is_u) {
            if (v0 + col < dv16)
              *reinterpret_cast<float2*>(slot + Slot::kU + (static_cast<int64_t>(row) * dv16 + v0 + col) * 4) = make_float2(a, c);
          } else {
            uint32_t hi, lo;
            split2(-a, -c, hi, lo);
            uint8_t* dst = slot + Slot::kW + row * kRow + col * 2;
            *reinterpret_cast<uint32_t*>(dst) = hi;
            *reinterpret_cast<uint32_t*>(dst + kTileBytes) = lo;
          }
        }
      }
    }
  }
}

template <int BV>
struct ScanCfg {
  static constexpr int kStage = 4 * kTileBytes + 2 * kPBytes + kScalars * 4;   // W (two terms), Q, K, P (two terms), scalars
  static constexpr int kS = kD * BV * 2, kU = kC * BV * 2;                     // one term of the state, of U
  static constexpr int kSmem = 2 * kStage + 2 * kS + 4 * kU + 128;
  static_assert(kSmem <= 232448, "shared memory");
};

template <int BV>
__global__ void __launch_bounds__(kThreads, 1) gdn_scan_kernel(const PrefillParams pp) {
  using C = ScanCfg<BV>;
  constexpr int NT = BV / 8;
  const GdnRuleParams& p = pp.r;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const uint32_t base = smem_u32(smem);
  const uint32_t sS = base + 2 * C::kStage;          // two terms of the state [128][BV]
  const uint32_t sU = sS + 2 * C::kS;                // two terms of U, then of exp(G_C - G) / |k| U, [64][BV]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, ti = warp & 3;
  const bool upper = warp >= 4;                      // warps 4 - 7 form the outputs, 0 - 3 U
  const int vb = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  pdl_wait_loads();
  const int n = p.lens[b];
  const int chunks = (n + kC - 1) / kC;
  const int c_end = min(pp.chunk0 + pp.span, chunks);
  if (pp.chunk0 >= c_end) return;
  const int hk = h / (p.heads / p.k_heads);
  const int cols = min(BV, p.dv - vb * BV), dv16 = (p.dv + 15) / 16 * 16;
  const int64_t row0 = p.q_start[b];
  float* S = p.state + (static_cast<int64_t>(p.slots[b]) * p.heads + h) * p.dk * p.dv + vb * BV;
  const BF* q = static_cast<const BF*>(p.q) + static_cast<int64_t>(hk) * p.dk;
  const BF* k = static_cast<const BF*>(p.k) + static_cast<int64_t>(hk) * p.dk;

  auto slot_of = [&](int c) {
    return pp.ws + ((static_cast<int64_t>(b) * pp.span + (c - pp.chunk0)) * p.heads + h) * slot_bytes(p.dv);
  };
  auto load_stage = [&](int c) {
    const uint32_t to = base + ((c - pp.chunk0) & 1) * C::kStage;
    const uint8_t* slot = slot_of(c);
    for (int i = tid; i < 2 * kC * 16; i += kThreads) {          // both terms of W
      const int r = (i >> 4) & (kC - 1), ch = i & 15, term = i >> 10;
      cp16_zfill(to + term * kTileBytes + at128(r, ch), slot + Slot::kW + term * kTileBytes + r * kRow + ch * 16, true);
    }
    const int nv = min(kC, n - c * kC);
    for (int i = tid; i < kC * 16; i += kThreads) {
      const int r = i >> 4, ch = i & 15;
      const bool ok = r < nv && ch * 8 < p.dk;
      const int64_t row = row0 + static_cast<int64_t>(c) * kC + (ok ? r : 0);
      cp16_zfill(to + 2 * kTileBytes + at128(r, ch), q + row * p.q_ld + (ok ? ch * 8 : 0), ok);
      cp16_zfill(to + 3 * kTileBytes + at128(r, ch), k + row * p.k_ld + (ok ? ch * 8 : 0), ok);
    }
    for (int i = tid; i < 2 * kC * 8; i += kThreads) {           // both terms of P, tiles on and below the diagonal
      const int r = (i >> 3) & (kC - 1), ch = i & 7, term = i >> 9;
      if ((ch >> 1) <= (r >> 4))
        cp16_zfill(to + 4 * kTileBytes + term * kPBytes + at64(r, ch), slot + Slot::kP + term * kPBytes + r * (kC * 2) + ch * 16, true);
    }
    if (tid < kScalars / 4) cp16_zfill(to + 4 * kTileBytes + 2 * kPBytes + tid * 16, slot + Slot::kScal + tid * 16, true);
    cp_commit();
  };
  float u0[NT][4];
  auto load_u0 = [&](int c) {
    if (upper) return;
    const float* src = reinterpret_cast<const float*>(slot_of(c) + Slot::kU) + vb * BV;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int col = nt * 8 + 2 * t;
        const float2 v = vb * BV + col < dv16 ? __ldcg(reinterpret_cast<const float2*>(src + static_cast<int64_t>(ti * 16 + g + half * 8) * dv16 + col))
                                              : make_float2(0.f, 0.f);
        u0[nt][half * 2] = v.x;
        u0[nt][half * 2 + 1] = v.y;
      }
  };

  load_stage(pp.chunk0);
  load_u0(pp.chunk0);
  // the state: this warp has key features 16 warp .. 16 warp + 15
  float s[NT][4];
  const bool resume = p.has_state[b] != 0 || pp.chunk0 > 0;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = warp * 16 + g + (i >> 1) * 8, col = nt * 8 + 2 * t + (i & 1);
      s[nt][i] = resume && row < p.dk && col < cols ? S[static_cast<int64_t>(row) * p.dv + col] : 0.f;
    }

  for (int c = pp.chunk0; c < c_end; ++c) {
    const uint32_t st = base + ((c - pp.chunk0) & 1) * C::kStage;
    const float* scal = reinterpret_cast<const float*>(smem + (st - base) + 4 * kTileBytes + 2 * kPBytes);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t hi, lo;
        split2(s[nt][half * 2], s[nt][half * 2 + 1], hi, lo);
        const uint32_t to = sS + at_v<BV>(warp * 16 + g + half * 8, nt) + t * 4;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(to), "r"(hi) : "memory");
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + C::kS), "r"(lo) : "memory");
      }
    cp_wait<0>();
    __syncthreads();
    if (c + 1 < c_end) load_stage(c + 1);      // into the buffer that the chunk before has left

    // ---- U = U0 - W S0 (warps 0 - 3), Q S0 (4 - 7) ----
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt][i] = upper ? 0.f : u0[nt][i];
    {
      const uint32_t left = upper ? st + 2 * kTileBytes : st;
#pragma unroll
      for (int kk = 0; kk < kD / 16; ++kk) {
        uint32_t a[4], al[4];
        const uint32_t off = at128(ti * 16 + (lane & 15), kk * 2 + (lane >> 4));
        ldsm4(a, left + off);
        if (!upper) ldsm4(al, left + kTileBytes + off);
#pragma unroll
        for (int np = 0; np < NT / 2; ++np) {
          uint32_t w[4], wl[4];
          const uint32_t at = sS + at_v<BV>(kk * 16 + (lane & 15), np * 2 + (lane >> 4));
          ldsm4_t(w, at);
          ldsm4_t(wl, at + C::kS);
          mma_16816<BF>(acc[2 * np], a[0], a[1], a[2], a[3], w[0], w[1]);
          mma_16816<BF>(acc[2 * np + 1], a[0], a[1], a[2], a[3], w[2], w[3]);
          mma_16816<BF>(acc[2 * np], a[0], a[1], a[2], a[3], wl[0], wl[1]);
          mma_16816<BF>(acc[2 * np + 1], a[0], a[1], a[2], a[3], wl[2], wl[3]);
          if (!upper) {
            mma_16816<BF>(acc[2 * np], al[0], al[1], al[2], al[3], w[0], w[1]);
            mma_16816<BF>(acc[2 * np + 1], al[0], al[1], al[2], al[3], w[2], w[3]);
          }
        }
      }
    }
    if (c + 1 < c_end) load_u0(c + 1);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int row = ti * 16 + g + half * 8;
      const float f = scal[upper ? row : kC + row];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        float& a = acc[nt][half * 2];
        float& d = acc[nt][half * 2 + 1];
        if (upper) {
          a *= f;
          d *= f;
        } else {
          uint32_t hi, lo;
          const uint32_t to = sU + at_v<BV>(row, nt) + t * 4;
          split2(a, d, hi, lo);
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(to), "r"(hi) : "memory");
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + C::kU), "r"(lo) : "memory");
          split2(a * f, d * f, hi, lo);
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + 2 * C::kU), "r"(hi) : "memory");
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + 3 * C::kU), "r"(lo) : "memory");
        }
      }
    }
    __syncthreads();

    // ---- S = exp(G_C) S0 + K^T U' (all warps) ----
    const float carry = scal[2 * kC];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[nt][i] *= carry;
#pragma unroll
    for (int ks = 0; ks < kC / 16; ++ks) {
      uint32_t a[4];
      ldsm4_t(a, st + 3 * kTileBytes + at128(ks * 16 + (lane & 7) + ((lane >> 4) << 3), warp * 2 + ((lane >> 3) & 1)));
#pragma unroll
      for (int np = 0; np < NT / 2; ++np) {
        uint32_t w[4], wl[4];
        const uint32_t at = sU + 2 * C::kU + at_v<BV>(ks * 16 + (lane & 15), np * 2 + (lane >> 4));
        ldsm4_t(w, at);
        ldsm4_t(wl, at + C::kU);
        mma_16816<BF>(s[2 * np], a[0], a[1], a[2], a[3], w[0], w[1]);
        mma_16816<BF>(s[2 * np + 1], a[0], a[1], a[2], a[3], w[2], w[3]);
        mma_16816<BF>(s[2 * np], a[0], a[1], a[2], a[3], wl[0], wl[1]);
        mma_16816<BF>(s[2 * np + 1], a[0], a[1], a[2], a[3], wl[2], wl[3]);
      }
    }
    // ---- O = exp(G) (Q S0) + P U (warps 4 - 7) ----
    if (upper) {
#pragma unroll
      for (int ks = 0; ks < kC / 16; ++ks) {
        if (ks <= ti) {
          uint32_t a[4], al[4];
          const uint32_t off = st + 4 * kTileBytes + at64(ti * 16 + (lane & 15), ks * 2 + (lane >> 4));
          ldsm4(a, off);
          ldsm4(al, off + kPBytes);
#pragma unroll
          for (int np = 0; np < NT / 2; ++np) {
            uint32_t w[4], wl[4];
            const uint32_t at = sU + at_v<BV>(ks * 16 + (lane & 15), np * 2 + (lane >> 4));
            ldsm4_t(w, at);
            ldsm4_t(wl, at + C::kU);
            mma_16816<BF>(acc[2 * np], a[0], a[1], a[2], a[3], w[0], w[1]);
            mma_16816<BF>(acc[2 * np + 1], a[0], a[1], a[2], a[3], w[2], w[3]);
            mma_16816<BF>(acc[2 * np], a[0], a[1], a[2], a[3], wl[0], wl[1]);
            mma_16816<BF>(acc[2 * np + 1], a[0], a[1], a[2], a[3], wl[2], wl[3]);
            mma_16816<BF>(acc[2 * np], al[0], al[1], al[2], al[3], w[0], w[1]);
            mma_16816<BF>(acc[2 * np + 1], al[0], al[1], al[2], al[3], w[2], w[3]);
          }
        }
      }
      const int nv = min(kC, n - c * kC);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = ti * 16 + g + half * 8;
        BF* out = static_cast<BF*>(p.out) + ((row0 + static_cast<int64_t>(c) * kC + row) * p.heads + h) * p.dv + vb * BV;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const int col = nt * 8 + 2 * t;
          if (row < nv && col < cols) *reinterpret_cast<uint32_t*>(out + col) = pack_bf16x2(acc[nt][half * 2], acc[nt][half * 2 + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = warp * 16 + g + (i >> 1) * 8, col = nt * 8 + 2 * t + (i & 1);
      if (row < p.dk && col < cols) S[static_cast<int64_t>(row) * p.dv + col] = s[nt][i];
    }
}

constexpr int kPrepareSmem = 3 * kTileBytes + (2 * kC * kLd + 3 * 16 * 17 + 5 * kC) * 4 + 128;

template <int BV>
int launch_scan(const PrefillParams& pp, cudaStream_t s) {
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_scan_kernel<BV>), ScanCfg<BV>::kSmem) != cudaSuccess) return -3;
  const cudaError_t err = launch_pdl(gdn_scan_kernel<BV>, dim3((pp.r.dv + BV - 1) / BV, pp.r.heads, pp.r.batch), dim3(kThreads),
                                     ScanCfg<BV>::kSmem, s, pp);
  return err == cudaSuccess ? 0 : -4;
}

}  // namespace

bool gdn_prefill_covers(const GdnRuleParams& p) { return p.dt == kBF16 && !p.split_tf32 && gdn_chunk_covers(p); }

// As many chunks of all requests as `most_bytes` have room for; where not even one fits, one chunk of equal groups of requests.  The
// least is a chunk of one request.  (Groups that fill the GPU once, with longer spans, leave the scan's last CTAs of every group
// alone: 32 x 1024 tokens 1467 us instead of 1388 with 512 MB.  128 MB instead of 512: 4 x 2000 tokens 450 us instead of 432,
// 32 x 1024 1651.)
GdnPrefillPlan gdn_prefill_plan(const GdnRuleParams& p, int max_len, int64_t most_bytes) {
  const int64_t chunk = slot_bytes(p.dv) * p.heads, slots = std::max<int64_t>(1, most_bytes / chunk);
  const int64_t batch = std::max(1, p.batch), groups = (batch + slots - 1) / slots, group = (batch + groups - 1) / groups;
  const int64_t span = std::max<int64_t>(1, std::min<int64_t>((max_len + kC - 1) / kC, slots / group));
  return {static_cast<int>(group), static_cast<int>(span), group * span * chunk};
}

int launch_gdn_prefill(const GdnRuleParams& p, void* ws, const GdnPrefillPlan& plan, int max_len, int num_sms, cudaStream_t s) {
  if (p.batch <= 0 || max_len <= 0) return 0;
  if (!gdn_prefill_covers(p) || p.heads % p.k_heads != 0 || p.g == nullptr || (reinterpret_cast<uintptr_t>(p.out) & 3) != 0) return -1;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_prepare_kernel), kPrepareSmem) != cudaSuccess) return -3;
  // a wider block of value features takes a chunk's operands in fewer times and leaves fewer CTAs: the width with the least
  // waves x time of a chunk (in tenths of us)
  int best = 64, least = 1 << 30;
  const int widths[3] = {16, 32, 64}, times[3] = {12, 17, 29};
  for (int i = 0; i < 3; ++i) {
    const int64_t ctas = static_cast<int64_t>(plan.group) * p.heads * ((p.dv + widths[i] - 1) / widths[i]);
    const int64_t cost = (ctas + num_sms - 1) / num_sms * times[i];
    if (cost < least) {
      least = static_cast<int>(std::min<int64_t>(cost, 1 << 30));
      best = widths[i];
    }
  }
  const int chunks = (max_len + kC - 1) / kC;
  for (int b0 = 0; b0 < p.batch; b0 += plan.group) {
    GdnRuleParams r = p;
    r.batch = std::min(plan.group, p.batch - b0);
    r.slots += b0;
    r.lens += b0;
    r.has_state += b0;
    r.q_start += b0;
    for (int c0 = 0; c0 < chunks; c0 += plan.span) {
      PrefillParams pp{r, static_cast<uint8_t*>(ws), c0, plan.span};
      const cudaError_t err = launch_pdl(gdn_prepare_kernel, dim3(std::min(plan.span, chunks - c0), r.heads, r.batch), dim3(kThreads), kPrepareSmem, s, pp);
      note_launch();      // the pair counts as one: the rule over a span
      if (err != cudaSuccess) return -4;
      const int rc = best == 16 ? launch_scan<16>(pp, s) : best == 32 ? launch_scan<32>(pp, s) : launch_scan<64>(pp, s);
      if (rc != 0) return rc;
    }
  }
  return 0;
}

}  // namespace mb200
