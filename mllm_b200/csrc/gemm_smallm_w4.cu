// out[m, n] = x[m, k] * dequant(qweight[n, k])^T for a handful of rows (m <= 8), 4-bit weights with group scales.
//
// The decode step of a 4-bit checkpoint streams a quarter of the bytes of the 16-bit model, so it should be the
// faster one; through the tcgen05 kernel of gemm_w4a16.cu (nibbles expanded into a shared-memory operand, one
// handshake between producer, expansion warps and MMA thread per 64-wide k block) it was slower.  This is the
// register-streaming kernel of gemm_smallm.cu with the expansion done in registers between the load and the
// warp-level MMA:
//   * a unit is 8 weight rows over the whole k range; the warps of a CTA take the 128-element
//     k steps of a unit round-robin.  A lane owns 16 bytes of packed weights per step: 32 consecutive k of one row;
//   * those 16 bytes, the 4 bytes that hold the row's scale for the step's group and the 4 bytes that hold its
//     zero point travel as cp.async copies into a shared-memory slice owned by the lane alone, 6 steps ahead;
//   * per step a lane expands its four words with the exponent-bias trick (nibble | magic = 128 + q as a 16-bit
//     float, exact subtraction of 128 + zero, one multiply by the scale) and feeds each word, with the 16 bytes
//     of activations at the same k offset, to two m16n8k16 MMAs.  The words are taken in an order rotated by the
//     lane's position in its row, so that the eight lanes of a quarter warp read eight different 16-byte bank
//     groups of the activation rows;
//   * activations (8 rows) are staged once per CTA; partial sums meet in shared memory at the end of a unit as
//     in gemm_smallm.cu.  Because the packed stream needs a quarter of the copy queue, the activation rows may
//     take most of the shared memory: a second shape of CTA (16 warps, two steps in flight) serves k up to 12288.
#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "common.cuh"
#include "gemm_stream.cuh"
#include "kernels.h"

namespace mb200 {
namespace {

constexpr int kQSlot = 768;            // bytes per warp and step: 32 x 16 of weights, 32 x 4 scale words, 32 x 4 zero words
constexpr int kQRowPad = 64;
// Two shapes of CTA.  k <= 4096: 8 warps, 6 steps in flight, two CTAs of 107 KB per SM.  k <= 12288 (the MLP's
// second matrix): the activation rows alone take 197 KB, so one CTA of 16 warps with 2 steps in flight per lane.
template <int WARPS, int DEPTH, int MAXK, int BLOCKS>
struct QCfg {
  static constexpr int kWarps = WARPS, kThreads = WARPS * 32, kDepth = DEPTH, kMaxK = MAXK, kBlocks = BLOCKS;
  static constexpr int kRingBytes = WARPS * DEPTH * kQSlot;
  static constexpr int kSmemMax = kRingBytes + 8 * (2 * MAXK + kQRowPad);
};
using QSmall = QCfg<8, 6, 4096, 2>;
using QLong = QCfg<16, 2, 12288, 1>;

struct W4SmallParams {
  const uint8_t* x;
  const uint8_t* qweight;   // [n, k/8] words
  const uint8_t* scales;    // [n, k/group] 16-bit
  const uint8_t* zeros;     // [n, k/group] bytes or null (zero point 8)
  const void* bias;
  void* out;
  int m, n, k, group;
  int64_t ldx_bytes, ldq_bytes, ldc;
  int groups_per_row;
  int units, units_per_cta, steps_per_warp;
  int interleaved;
};

template <bool F16>
__device__ __forceinline__ void mma_16816_w4(float (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  if constexpr (F16) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
  }
}

// 16-bit float pair helpers on packed registers
template <bool F16>
__device__ __forceinline__ uint32_t sub_mul2(uint32_t v, uint32_t off2, uint32_t scale2) {
  if constexpr (F16) {
    __half2 a = *reinterpret_cast<const __half2*>(&v);
    a = __hmul2(__hsub2(a, *reinterpret_cast<const __half2*>(&off2)), *reinterpret_cast<const __half2*>(&scale2));
    return *reinterpret_cast<uint32_t*>(&a);
  } else {
    __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v);
    a = __hmul2(__hsub2(a, *reinterpret_cast<const __nv_bfloat162*>(&off2)),
                *reinterpret_cast<const __nv_bfloat162*>(&scale2));
    return *reinterpret_cast<uint32_t*>(&a);
  }
}
template <bool F16>
__device__ __forceinline__ uint32_t splat_f(float v) {
  if constexpr (F16) {
    __half2 r = __float2half2_rn(v);
    return *reinterpret_cast<uint32_t*>(&r);
  } else {
    __nv_bfloat162 r = __float2bfloat162_rn(v);
    return *reinterpret_cast<uint32_t*>(&r);
  }
}
template <bool F16>
__device__ __forceinline__ float half_bits_to_f(uint16_t v) {
  if constexpr (F16) return __half2float(*reinterpret_cast<const __half*>(&v));
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(&v));
}
template <bool F16>
__device__ __forceinline__ uint16_t f_to_half_bits(float v) {
  if constexpr (F16) {
    const __half h = __float2half_rn(v);
    return *reinterpret_cast<const uint16_t*>(&h);
  }
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  return *reinterpret_cast<const uint16_t*>(&h);
}

template <bool F16, typename C>
__global__ void __launch_bounds__(C::kThreads, C::kBlocks) gemm_smallm_w4_kernel(const W4SmallParams p) {
  constexpr int kQWarps = C::kWarps, kQThreads = C::kThreads, kQDepth = C::kDepth, kQRingBytes = C::kRingBytes;
  constexpr uint32_t kMagic = F16 ? 0x64006400u : 0x43004300u;   // 1024 + q / 128 + q as a 16-bit float pair
  constexpr float kBase = F16 ? 1024.f : 128.f;
  __shared__ float partial[2][kQWarps][64];
  extern __shared__ __align__(16) uint8_t smem_dyn[];
  uint8_t* ring_raw = smem_dyn;
  uint8_t* x_rows = smem_dyn + kQRingBytes;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;   // weight row inside the unit, and activation row
  const int c = lane & 3;    // which 32 k of the step's 128
  const int u0 = blockIdx.x * p.units_per_cta;
  const int u1 = min(p.units, u0 + p.units_per_cta);
  if (u0 >= u1) return;
  const int J = p.steps_per_warp;
  const int total = (u1 - u0) * J;
  const int x_pitch = 2 * p.k + kQRowPad;

  // slot s of this warp's ring: the lanes' 16 bytes of weights, then their scale words, then their zero words
  const uint32_t ring = smem_u32(ring_raw) + warp * (kQDepth * kQSlot);
  int lu = u0, lj = 0;
  auto issue = [&](int slot) {
    const int64_t row = static_cast<int64_t>(lu) * 8 + g;
    const int kstep = warp + kQWarps * lj;                 // 128-element step of the row
    const int koff = kstep * 128 + c * 32;                 // first k of this lane
    const int grp = koff / p.group;
    const uint32_t dst = ring + slot * kQSlot;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + lane * 16), "l"(p.qweight + row * p.ldq_bytes + (koff >> 1))
                 : "memory");
    const uint8_t* sc = p.scales + (row * p.groups_per_row + grp) * 2;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 512 + lane * 4),
                 "l"(reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(sc) & ~uintptr_t(3)))
                 : "memory");
    if (p.zeros != nullptr) {
      const uint8_t* zp = p.zeros + row * p.groups_per_row + grp;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 640 + lane * 4),
                   "l"(reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(zp) & ~uintptr_t(3)))
                   : "memory");
    }
    if (++lj == J) {
      lj = 0;
      ++lu;
    }
  };
  auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };
  // weights, scales and zero points are parameters: nothing in the stream writes them
#pragma unroll
  for (int s = 0; s < kQDepth; ++s) {
    if (s < total) issue(s);
    commit();
  }
  pdl_wait();
  {
    const int vec_per_row = p.k >> 3;
    for (int v = threadIdx.x; v < 8 * vec_per_row; v += kQThreads) {
      const int r = v / vec_per_row, q = v - r * vec_per_row;
      uint4 val = make_uint4(0, 0, 0, 0);
      if (r < p.m) val = __ldg(reinterpret_cast<const uint4*>(p.x + static_cast<int64_t>(r) * p.ldx_bytes) + q);
      *reinterpret_cast<uint4*>(x_rows + r * x_pitch + q * 16) = val;
    }
  }
  __syncthreads();
  const uint32_t x_lane = smem_u32(x_rows) + g * x_pitch + c * 64;

  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  int cu = u0, cj = 0, buf = 0;
  for (int base = 0; base < total; base += kQDepth) {
#pragma unroll
    for (int s = 0; s < kQDepth; ++s) {
      const int i = base + s;
      if (i < total) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kQDepth - 1) : "memory");
        const uint32_t slot = ring + s * kQSlot;
        const int kstep = warp + kQWarps * cj;
        const int grp = (kstep * 128 + c * 32) / p.group;
        // scale and zero point of (row, group): the copies fetched the aligned words that hold them
        const int64_t row = static_cast<int64_t>(cu) * 8 + g;
        const uintptr_t sc_addr = reinterpret_cast<uintptr_t>(p.scales) + (row * p.groups_per_row + grp) * 2;
        uint32_t sw, zw = 0;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sw) : "r"(slot + 512 + lane * 4) : "memory");
        const float scale = half_bits_to_f<F16>(static_cast<uint16_t>((sc_addr & 2) ? (sw >> 16) : (sw & 0xFFFFu)));
        float zero = 8.f;
        if (p.zeros != nullptr) {
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(zw) : "r"(slot + 640 + lane * 4) : "memory");
          const uintptr_t z_addr = reinterpret_cast<uintptr_t>(p.zeros) + row * p.groups_per_row + grp;
          zero = static_cast<float>((zw >> (8 * (z_addr & 3))) & 0xFFu);
        }
        const uint32_t off2 = splat_f<F16>(kBase + zero);
        const uint32_t scale2 = splat_f<F16>(scale);
        const uint32_t x_step = x_lane + kstep * 256;      // 128 k = 256 bytes of the row per step
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int jj = (t + c) & 3;                      // rotated: bank-conflict-free activation reads
          uint32_t w;
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(slot + lane * 16 + jj * 4) : "memory");
          uint4 x;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                       : "r"(x_step + jj * 16)
                       : "memory");
          uint32_t b0, b1, b2, b3;   // element pairs (0,1) (2,3) (4,5) (6,7) of the word
          if (p.interleaved) {
            b0 = sub_mul2<F16>((w & 0x000F000Fu) | kMagic, off2, scale2);
            b1 = sub_mul2<F16>(((w >> 4) & 0x000F000Fu) | kMagic, off2, scale2);
            b2 = sub_mul2<F16>(((w >> 8) & 0x000F000Fu) | kMagic, off2, scale2);
            b3 = sub_mul2<F16>(((w >> 12) & 0x000F000Fu) | kMagic, off2, scale2);
          } else {
            b0 = sub_mul2<F16>(((w & 0xFu) | ((w & 0xF0u) << 12)) | kMagic, off2, scale2);
            b1 = sub_mul2<F16>((((w >> 8) & 0xFu) | (((w >> 8) & 0xF0u) << 12)) | kMagic, off2, scale2);
            b2 = sub_mul2<F16>((((w >> 16) & 0xFu) | (((w >> 16) & 0xF0u) << 12)) | kMagic, off2, scale2);
            b3 = sub_mul2<F16>((((w >> 24) & 0xFu) | (((w >> 24) & 0xF0u) << 12)) | kMagic, off2, scale2);
          }
          mma_16816_w4<F16>(acc, x.x, x.y, b0, b1);
          mma_16816_w4<F16>(acc, x.z, x.w, b2, b3);
        }
        if (i + kQDepth < total) issue(s);   // after the loads above: the slot's old bytes are consumed
        commit();
        if (++cj == J) {
          cj = 0;
          *reinterpret_cast<float2*>(&partial[buf][warp][lane * 2]) = make_float2(acc[0], acc[1]);
          acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
          __syncthreads();
          if (threadIdx.x < 64) {
            const int tt = threadIdx.x;
            const int mrow = tt >> 3, slot_n = tt & 7;
            float v = 0.f;
#pragma unroll
            for (int w8 = 0; w8 < kQWarps; ++w8) v += partial[buf][w8][tt];
            if (mrow < p.m) {
              const int64_t col = static_cast<int64_t>(cu) * 8 + slot_n;
              if (p.bias != nullptr) v += half_bits_to_f<F16>(static_cast<const uint16_t*>(p.bias)[col]);
              static_cast<uint16_t*>(p.out)[mrow * p.ldc + col] = f_to_half_bits<F16>(v);
            }
          }
          ++cu;
          buf ^= 1;
        }
      }
    }
  }
}

template <typename C>
int launch_w4_cfg(W4SmallParams p, const W4A16Args& a, cudaStream_t s) {
  p.steps_per_warp = a.k / (128 * C::kWarps);
  const int slots = std::max(1, a.num_sms > 0 ? a.num_sms : 148) * C::kBlocks;
  p.units_per_cta = (p.units + slots - 1) / slots;
  const int grid = (p.units + p.units_per_cta - 1) / p.units_per_cta;
  const int smem = C::kRingBytes + 8 * (2 * a.k + kQRowPad);
  cudaError_t err;
  if (a.dt == kF16) {
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(gemm_smallm_w4_kernel<true, C>), C::kSmemMax) != cudaSuccess) return -3;
    err = launch_pdl(gemm_smallm_w4_kernel<true, C>, dim3(grid), dim3(C::kThreads), smem, s, p);
  } else {
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(gemm_smallm_w4_kernel<false, C>), C::kSmemMax) != cudaSuccess) return -3;
    err = launch_pdl(gemm_smallm_w4_kernel<false, C>, dim3(grid), dim3(C::kThreads), smem, s, p);
  }
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

// =====================================================================================================================
// Groups of a multiple of 128: the stream of packed weights.  Three quarters of its bytes are gone and the work per weight is not, so what
// bounds it is instructions: per 16 rows x 128 k a warp needs 24 shifts, 32 masks and 32 subtractions for the nibbles and eight MMAs,
// and shifts and masks issue at half rate.  So everything else is kept out of the loop:
//   * the rows of x are in shared memory, in the order in which the lanes take them as column operands (16 bytes a lane, no bank
//     conflicts), so that a warp needs no registers for them: 24 warps per SM in two CTAs, where x in registers allowed 16;
//   * the steps (16 weight rows x 128 k) of a CTA form one line, row block by row block, and a warp takes an equal, unbroken run of
//     it, whatever the number of row blocks.  Its sums stay in registers until the run leaves a row block, which happens once or
//     twice; the warps meet once, behind the last step.
// The rest is as in gemm_stream.cuh: copy rings of cp.async, k over a cluster where it is longer than 4096, the next kernel started at once.
//
// A nibble under an exponent's bits is base + q; one operation per pair takes base and zero point off, exactly, and the group's scale
// multiplies the fp32 sum of the group's step, so nothing of a weight is rounded.  In bf16 that operation also divides by 2048, which
// the sums get back at their end: a group's sum is then no larger than the largest x in it, and x may be as large as the type allows.
// (Taking the base off the sum, as base times the sum of x, turns an infinite x into NaN.)
//
// Before, with x in registers, 16 warps per SM and the warps of a CTA on the steps of one row block in turn, a step took 263 instructions
// a warp.  2 rows, n x k, before and now: 24576 x 4096 24.0 and 17.4 us (50 MB of weights: 7.9 us at the rate of a copy), 6144 x 4096 9.1
// and 7.2, 4096 x 12288 15.2 and 12.9, 4096 x 4096 5.7 and 5.3, 2048 x 2048 3.1 and 2.8, 5120 x 25600 53 and 28.
// =====================================================================================================================
namespace nibbles {

constexpr int kWarps = 12, kThreads = kWarps * 32;
constexpr int kDepth = 3;                     // steps in flight per warp, the one in work included
constexpr int kSlotBytes = 1024;              // 16 rows x 64 bytes
constexpr int kRingBytes = kWarps * kDepth * kSlotBytes;
constexpr int kXStep = 2048;                  // x of a step: [8 k per lane][lane], 16 bytes each
constexpr int kMaxSteps = 32;                 // of a CTA's part of k: 64 KB of x
constexpr int kPart = 128;                    // sums of a row block: [row of x][weight row]
constexpr int kHalfSm = 112 * 1024, kWholeSm = 226 * 1024;      // shared memory of a CTA where an SM holds two, and one

struct Params {
  const uint8_t* x;
  const uint8_t* w;
  const uint8_t* scales;    // [n, groups] 16-bit
  const uint8_t* zeros;     // [n, groups] bytes, or null (zero point 8)
  const void* bias;
  void* out;
  int m, n, m_log;          // 2^m_log >= m
  int steps, max_steps;     // of the whole row, of a CTA at most
  int groups, steps_per_group;
  int units_each, units_more, cluster;      // row blocks of a cluster; how many have one more
  int slots;                // row blocks that a warp's run can touch
  int64_t ldx, ldw, ldc;    // bytes, bytes, elements
};

// A pair of nibbles under the exponent's bits, base + q, to q - zero (fp16, base 1024) or (q - zero) / 2048 (bf16, base 128); both are
// exact.  `off2`: base + zero, or -(base + zero) / 2048
constexpr float kScaled = 2048.f;
template <bool F16>
__device__ __forceinline__ uint32_t expand(uint32_t v, uint32_t off2) {
  constexpr uint32_t kMagic = F16 ? 0x64006400u : 0x43004300u;
  v = (v & 0x000F000Fu) | kMagic;
  if constexpr (F16) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&off2));
    return *reinterpret_cast<const uint32_t*>(&r);
  } else {
    const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&v), __float2bfloat162_rn(1.f / kScaled),
                                     *reinterpret_cast<const __nv_bfloat162*>(&off2));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
}
// what `expand` takes off for a zero point: the bits of 1024 + zero, or of -(128 + zero) / 2048, whose last place is 2 / 2048 from
// zero points of 128 on.
template <bool F16>
__device__ __forceinline__ uint32_t zero_bits(int zero) {
  if constexpr (F16) return (0x6400u + zero) * 0x10001u;
  return (0xBD80u + zero - ((max(zero, 128) - 127) >> 1)) * 0x10001u;
}
template <bool F16>
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool F16, bool NATURAL, bool ZEROS>
__global__ void __launch_bounds__(kThreads, 2) w4_stream_kernel(const Params p) {
  extern __shared__ __align__(128) uint8_t smem[];       // x, rings, the warps' sums, (cluster) the sums of the row blocks
  __shared__ int2 touched[kWarps];                       // first and last row block of a warp's run
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int rank = p.cluster > 1 ? static_cast<int>(stream::cluster_rank()) : 0;
  const int c = static_cast<int>(blockIdx.x) / p.cluster;
  // clusters differ by one row block, and the ranks of a cluster by one step, at most
  const int u0 = c * p.units_each + min(c, p.units_more), U = p.units_each + (c < p.units_more ? 1 : 0);
  const int s0 = p.cluster > 1 ? p.steps * rank / p.cluster : 0, S = p.cluster > 1 ? p.steps * (rank + 1) / p.cluster - s0 : p.steps;
  const int line = U * S;
  const int from = line * warp / kWarps, left = line * (warp + 1) / kWarps - from;
  uint8_t* x_smem = smem;
  uint8_t* ring = smem + p.max_steps * kXStep;           // the same place in every CTA of a cluster
  float* parts = reinterpret_cast<float*>(ring + kRingBytes);
  float* unit_sums = parts + kWarps * p.slots * kPart;

  // ---- the run of this warp: where its copies are, and where its products are ----
  const int first_unit = from / S, first_step = from - first_unit * S;
  auto row_of = [&](int u) { return min((u0 + u) * 16 + g, p.n - 1); };
  auto second = [&](int row) { return min(row + 8, p.n - 1); };
  const uint32_t my_ring = smem_u32(ring) + warp * (kDepth * kSlotBytes) + lane * 16;
  int iu = first_unit, is = first_step, islot = 0, to_issue = left;
  const uint8_t *w0, *w1;
  auto weights_at = [&](int u, int step) {
    const int r = row_of(u);
    const uint8_t* at = p.w + (s0 + step) * 64 + t * 16;
    w0 = at + r * p.ldw;
    w1 = at + second(r) * p.ldw;
  };
  weights_at(iu, is);
  auto issue = [&]() {
    if (to_issue > 0) {
      const uint32_t dst = my_ring + islot * kSlotBytes;
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(w0) : "memory");
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst + 512), "l"(w1) : "memory");
      if (++islot == kDepth) islot = 0;
      w0 += 64;
      w1 += 64;
      --to_issue;
      if (++is == S && to_issue > 0) {
        is = 0;
        weights_at(++iu, 0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // parameters: no kernel in front writes them
#pragma unroll
  for (int i = 0; i < kDepth - 1; ++i) issue();

  // scales (and zero points) go into registers two steps ahead
  int fu = first_unit, fs = first_step, to_fetch = left, in_group;
  uint32_t sc0, sc1;         // which of the scales: of row g and of row g + 8
  auto scales_at = [&](int u, int step) {
    const int r = row_of(u), grp = p.steps_per_group == 1 ? s0 + step : (s0 + step) / p.steps_per_group;
    in_group = s0 + step - grp * p.steps_per_group;
    sc0 = static_cast<uint32_t>(r) * p.groups + grp;
    sc1 = static_cast<uint32_t>(second(r)) * p.groups + grp;
  };
  scales_at(fu, fs);
  struct Scale {
    uint16_t s0, s1;
    uint8_t z0, z1;
  };
  auto fetch = [&]() {
    Scale v{0, 0, 0, 0};
    if (to_fetch > 0) {
      v.s0 = __ldg(reinterpret_cast<const uint16_t*>(p.scales) + sc0);
      v.s1 = __ldg(reinterpret_cast<const uint16_t*>(p.scales) + sc1);
      if constexpr (ZEROS) {
        v.z0 = __ldg(p.zeros + sc0);
        v.z1 = __ldg(p.zeros + sc1);
      }
      --to_fetch;
      if (++in_group == p.steps_per_group) {
        in_group = 0;
        ++sc0;
        ++sc1;
      }
      if (++fs == S && to_fetch > 0) {
        fs = 0;
        scales_at(++fu, 0);
      }
    }
    return v;
  };
  Scale now = fetch(), next = fetch();
  if (lane == 0) touched[warp] = left > 0 ? make_int2(first_unit, (from + left - 1) / S) : make_int2(1, 0);
  pdl_wait_loads();

  // ---- the rows of x, as lane (g, t) takes them: k t * 32 + i * 8 of a step of row g.  What stands for the rows from m on ends up in
  // columns of the product that nobody reads ----
  {
    const int i = threadIdx.x & 3, tt = (threadIdx.x >> 2) & 3;
    const uint8_t* src = p.x + (s0 * 128 + tt * 32 + i * 8) * 2;
    uint8_t* dst = x_smem + i * 512;
    // (step, row) pairs, four loads of a thread on their way; a pair's 256 bytes lie in sixteen threads
    const int pairs = S << p.m_log;
    for (int v0 = threadIdx.x >> 4; v0 < pairs; v0 += 4 * (kThreads / 16)) {
      uint4 val[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int v = v0 + j * (kThreads / 16), r = v & ((1 << p.m_log) - 1), step = v >> p.m_log;
        if (v < pairs && r < p.m) val[j] = __ldcg(reinterpret_cast<const uint4*>(src + r * p.ldx + step * 256));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int v = v0 + j * (kThreads / 16), r = v & ((1 << p.m_log) - 1), step = v >> p.m_log;
        if (v < pairs && r < p.m) *reinterpret_cast<uint4*>(dst + step * kXStep + (((r * 4 + tt) ^ (2 * i)) << 4)) = val[j];
      }
    }
  }
  __syncthreads();

  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  int cs = first_step, slot = 0, part = 0;
  auto flush = [&]() {
    float* mine = parts + (warp * p.slots + part) * kPart;
    mine[2 * t * 16 + g] = acc[0];
    mine[(2 * t + 1) * 16 + g] = acc[1];
    mine[2 * t * 16 + g + 8] = acc[2];
    mine[(2 * t + 1) * 16 + g + 8] = acc[3];
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    ++part;
  };
  const uint8_t* xs = x_smem + cs * kXStep;
  for (int done = 0; done < left; ++done) {
    // the copies of kDepth - 1 steps are on their way; the oldest of them is this step
    asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
    const uint32_t at = my_ring + slot * kSlotBytes;
    if (++slot == kDepth) slot = 0;
    uint4 a, b;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w) : "r"(at) : "memory");
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(at + 512) : "memory");
    issue();               // into the slot of the step before, whose values are in registers
    const Scale sc = now;
    now = next;
    next = fetch();
    const uint32_t oa = ZEROS ? zero_bits<F16>(sc.z0) : zero_bits<F16>(8), ob = ZEROS ? zero_bits<F16>(sc.z1) : oa;
    float s[2][4] = {};
    const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 x = *reinterpret_cast<const uint4*>(xs + i * 512 + ((lane ^ (2 * i)) << 4));
      uint32_t ea[4], eb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if constexpr (NATURAL) {
          const uint32_t va = wa[i] >> (8 * q), vb = wb[i] >> (8 * q);
          ea[q] = expand<F16>((va & 0xFu) | ((va & 0xF0u) << 12), oa);
          eb[q] = expand<F16>((vb & 0xFu) | ((vb & 0xF0u) << 12), ob);
        } else {
          ea[q] = expand<F16>(wa[i] >> (4 * q), oa);
          eb[q] = expand<F16>(wb[i] >> (4 * q), ob);
        }
      }
      mma<F16>(s[0], ea[0], eb[0], ea[1], eb[1], x.x, x.y);
      mma<F16>(s[1], ea[2], eb[2], ea[3], eb[3], x.z, x.w);
    }
    const float f0 = stream::half_to_f<F16>(sc.s0), f1 = stream::half_to_f<F16>(sc.s1);
    acc[0] = fmaf(f0, s[0][0] + s[1][0], acc[0]);
    acc[1] = fmaf(f0, s[0][1] + s[1][1], acc[1]);
    acc[2] = fmaf(f1, s[0][2] + s[1][2], acc[2]);
    acc[3] = fmaf(f1, s[0][3] + s[1][3], acc[3]);
    xs += kXStep;
    if (++cs == S) {
      cs = 0;
      xs = x_smem;
      flush();
    }
  }
  if (cs > 0 && left > 0) flush();
  __syncthreads();

  auto finish = [&](int u, int tok, int r, float v) {
    const int64_t col = static_cast<int64_t>(u0 + u) * 16 + r;
    if (tok >= p.m || col >= p.n) return;
    if (p.bias != nullptr) v += stream::half_to_f<F16>(static_cast<const uint16_t*>(p.bias)[col]);
    static_cast<uint16_t*>(p.out)[tok * p.ldc + col] = stream::f_to_half<F16>(v);
  };
  // without a cluster only the rows that are there; with one the sums of all go to their place
  const int rows = p.cluster > 1 ? kPart : p.m * 16;
  for (int i = threadIdx.x; i < U * rows; i += kThreads) {
    const int u = i / rows, e = i - u * rows;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {           // in the order of k
      const int2 run = touched[w];
      if (u >= run.x && u <= run.y) v += parts[(w * p.slots + u - run.x) * kPart + e];
    }
    if constexpr (!F16) v *= kScaled;
    if (p.cluster > 1)
      unit_sums[i] = v;
    else
      finish(u, e >> 4, e & 15, v);
  }
  if (p.cluster > 1) {
    stream::cluster_barrier();                   // every part of every sum is in its CTA's shared memory
    const uint32_t base = smem_u32(unit_sums);
    const int cols = kPart / p.cluster;          // every CTA finishes its part of each row block
    for (int i = threadIdx.x; i < U * cols; i += kThreads) {
      const int u = i / cols, e = rank * cols + i - u * cols;
      float v = 0.f;
      for (int r = 0; r < p.cluster; ++r) v += stream::ld_peer(base + (u * kPart + e) * 4, r);      // in rank order
      finish(u, e >> 4, e & 15, v);
    }
    stream::cluster_barrier();                   // no CTA leaves while its sums are read
  }
}

template <bool F16, bool NATURAL, bool ZEROS>
int launch(Params p, int num_sms, cudaStream_t s) {
  auto kern = w4_stream_kernel<F16, NATURAL, ZEROS>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kWholeSm) != cudaSuccess) return -3;
  ensure_max_carveout(reinterpret_cast<const void*>(kern));
  if ((p.steps + 7) / 8 > kMaxSteps || static_cast<int64_t>(p.n) * p.groups >= (int64_t(1) << 31)) return 1;
  while ((1 << p.m_log) < p.m) ++p.m_log;
  p.cluster = 1;
  while ((p.steps + p.cluster - 1) / p.cluster > kMaxSteps) p.cluster *= 2;
  p.max_steps = (p.steps + p.cluster - 1) / p.cluster;
  // Two CTAs per SM, whole row blocks each, as many clusters as the device holds at once: three more of 71, behind all the others, made
  // 4096 x 12288 16.5 us instead of 12.8.  (Clusters where x fits without them, for fewer steps at most: 24576 x 4096 20.3 us, without 17.4.)
  const int all = (p.n + 15) / 16;
  int smem = 0;
  auto split = [&](int per_sm) {
    const int places = p.cluster == 1 ? per_sm * num_sms
                                      : max_clusters(p.cluster, kThreads, per_sm == 2 ? kHalfSm : kWholeSm, per_sm * num_sms / (p.cluster + 1));
    const int clusters = std::min(all, std::max(1, places));
    p.units_each = all / clusters;
    p.units_more = all % clusters;
    const int units = p.units_each + (p.units_more > 0 ? 1 : 0);
    // a run is at most ceil(units * steps / kWarps) steps: it touches one row block more than it has whole ones' worth of steps
    p.slots = std::min(units, (units + kWarps - 1) / kWarps + 1);
    smem = p.max_steps * kXStep + kRingBytes + kWarps * p.slots * kPart * 4 + (p.cluster > 1 ? units * kPart * 4 : 0);
    return clusters;
  };
  int clusters = split(2);
  if (smem > kHalfSm) {
    // sums of so many row blocks leave an SM room for one: as many clusters as run at once then, if their sums fit (2 rows, n x k, in
    // two rounds and in one: 10240 x 8192 20.6 and 17.5 us, 28672 x 8192 44.5 and 41.1, 32768 x 16384 136.8 and 96.2)
    clusters = split(1);
    if (smem > kWholeSm) clusters = split(2);
  }
  if (smem > kWholeSm) return 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * p.cluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(p.cluster);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 2 : 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, p);
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

}  // namespace nibbles

template <bool F16>
int launch_stream(const W4A16Args& a, cudaStream_t s) {
  nibbles::Params p{};
  p.x = static_cast<const uint8_t*>(a.x);
  p.w = static_cast<const uint8_t*>(a.qweight);
  p.scales = static_cast<const uint8_t*>(a.scales);
  p.zeros = a.zeros;
  p.bias = a.bias;
  p.out = a.out;
  p.m = a.m;
  p.n = a.n;
  p.steps = a.k / 128;
  p.groups = a.k / a.group;
  p.steps_per_group = a.group / 128;
  p.ldx = a.ldx * 2;
  p.ldw = a.k / 2;
  p.ldc = a.ldc;
  const int sms = a.num_sms > 0 ? a.num_sms : 148;
  if (a.zeros != nullptr)
    return a.interleaved ? nibbles::launch<F16, false, true>(p, sms, s) : nibbles::launch<F16, true, true>(p, sms, s);
  return a.interleaved ? nibbles::launch<F16, false, false>(p, sms, s) : nibbles::launch<F16, true, false>(p, sms, s);
}

}  // namespace

// Returns 0 when launched, 1 when the shape is not for this kernel (the caller goes on to the tcgen05 kernel).
int launch_w4a16_smallm(const W4A16Args& a, cudaStream_t s) {
  static const int knob = [] {
    const char* e = std::getenv("MLLM_B200_W4_SMALLM");
    return e == nullptr ? 1 : std::atoi(e);
  }();
  if (!knob || a.m > 8 || a.n < 1 || a.n % 8 != 0) return 1;
  if (a.group % 128 == 0 && a.k % a.group == 0 && a.k % 128 == 0 && (a.ldx * 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 1) == 0 &&
      ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.qweight)) & 15) == 0) {
    const int rc = a.dt == kF16 ? launch_stream<true>(a, s) : launch_stream<false>(a, s);
    if (rc <= 0) return rc;
  }
  const bool small_k = a.k <= QSmall::kMaxK && a.k % (128 * QSmall::kWarps) == 0;
  const bool long_k = a.k <= QLong::kMaxK && a.k % (128 * QLong::kWarps) == 0;
  if ((!small_k && !long_k) || a.group % 32 != 0 || a.k % a.group != 0) return 1;
  if ((a.ldx * 2) % 16 != 0 || ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.qweight)) & 15) != 0) return 1;
  if ((reinterpret_cast<uintptr_t>(a.scales) & 1) != 0) return 1;
  W4SmallParams p{};
  p.x = static_cast<const uint8_t*>(a.x);
  p.qweight = static_cast<const uint8_t*>(a.qweight);
  p.scales = static_cast<const uint8_t*>(a.scales);
  p.zeros = a.zeros;
  p.bias = a.bias;
  p.out = a.out;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.group = a.group;
  p.ldx_bytes = a.ldx * 2;
  p.ldq_bytes = static_cast<int64_t>(a.k) / 2;
  p.ldc = a.ldc;
  p.groups_per_row = a.k / a.group;
  p.units = a.n / 8;
  p.interleaved = a.interleaved;
  return small_k ? launch_w4_cfg<QSmall>(p, a, s) : launch_w4_cfg<QLong>(p, a, s);
}

}  // namespace mb200
