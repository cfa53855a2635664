// out[m, n] = x[m, k] * W[n, k]^T for up to 8 rows of x and 16-bit weights: the projections of a decode step.  (Packed 4-bit weights:
// gemm_smallm_w4.cu.)
//
// The product is a stream of the weight matrix; what costs time beside its bytes is everything that keeps the stream from
// running: the launch, the first round trip to memory, the exchange of partial sums at the end.
//   * A unit is 16 weight rows over the CTA's part of k, the row operand of warp-level MMAs (m16n8k16) whose 8 columns are
//     the rows of x.  The 8 warps take the k steps of a unit in turn (32 k: 16 bytes of row g and of row g + 8 per
//     lane).  k is permuted alike for both operands, which a dot product does not notice, so a lane's 16 bytes are its fragments as they
//     come.
//   * The rows of x are loaded once, into registers: a warp only ever meets its own k steps.  So there is nothing to stage, no
//     barrier before the first product, and the shared memory of a CTA is the copy queue alone: per lane a ring of cp.async
//     copies that the lane itself reads back, 48 KB per CTA, two CTAs per SM.
//   * k that needs more registers than that (over 4096) is cut over a cluster; its CTAs keep the sums of all their units in shared
//     memory and exchange them once, through distributed shared memory, at the end.
//   * Every kernel of the chain lets the next one start as soon as it runs itself.  With half an SM per CTA the CTAs of the next
//     product move in as these leave, and fill their rings with weights, which no kernel writes, before they wait for their
//     input: the end of one stream and the start of the next overlap.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace mb200 {
namespace stream {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kDepth = 6;                                 // k steps in flight per warp
constexpr int kSlotBytes = 1024;                          // 16 bytes of two rows per lane
constexpr int kRingBytes = kWarps * kDepth * kSlotBytes;  // 48 KB

struct Params {
  const uint8_t* x;
  const uint8_t* w;
  const void* bias;
  const void* residual;
  void* out;
  int m, n;
  int steps;                // k steps of the whole row
  int units, units_per_cluster, cluster;
  int up_rows;              // gated: rows between a gate row and its up row inside a block of gate_block rows
  int gate_block;           // gated: gate rows of a block, followed by as many up rows
  int w_static;
  float act_limit;
  int64_t ldx, ldw, ldc, ld_res;   // bytes, bytes, elements, elements
};

enum Act { kNone = 0, kSilu = 1, kGelu = 2, kRelu2 = 3, kClamped = 4 };
template <int ACT>
constexpr bool kGatedAct = ACT == kSilu || ACT == kGelu || ACT == kClamped;

template <bool F16>
__device__ __forceinline__ float half_to_f(uint16_t v) {
  if constexpr (F16) return __half2float(*reinterpret_cast<const __half*>(&v));
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(&v));
}
template <bool F16>
__device__ __forceinline__ uint16_t f_to_half(float v) {
  if constexpr (F16) {
    const __half h = __float2half_rn(v);
    return *reinterpret_cast<const uint16_t*>(&h);
  }
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  return *reinterpret_cast<const uint16_t*>(&h);
}
template <bool F16>
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_peer(uint32_t local, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// JX: k steps of one warp that the registers hold x for
template <bool F16, int ACT, int JX>
__global__ void __launch_bounds__(kThreads, 2) gemm_stream_kernel(const Params p) {
  constexpr int kStepK = 32;                             // k of a step
  constexpr int kStepBytes = 64;                         // of one weight row
  constexpr int kXRegs = kStepK / 8;                     // registers of x per step: a lane's quarter of the step, two k each
  constexpr bool kGated = kGatedAct<ACT>;
  extern __shared__ __align__(16) uint8_t smem[];        // rings, then (cluster) the sums of the units
  __shared__ float partial[2][kWarps][8][17];            // [row of x][weight row], one more column against bank conflicts
  float* unit_sums = reinterpret_cast<float*>(smem + kRingBytes);
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int rank = p.cluster > 1 ? static_cast<int>(cluster_rank()) : 0;
  const int u0 = (static_cast<int>(blockIdx.x) / p.cluster) * p.units_per_cluster;
  const int u1 = min(p.units, u0 + p.units_per_cluster);
  const int s0 = static_cast<int>(static_cast<int64_t>(p.steps) * rank / p.cluster);
  const int s1 = static_cast<int>(static_cast<int64_t>(p.steps) * (rank + 1) / p.cluster);
  const int J = (s1 - s0 + kWarps - 1) / kWarps;         // the same for every warp; a warp's last step may lie past s1
  const int total = (u1 - u0) * J;

  // first weight row of unit u that this lane's copies read (its row g), and how far on its row g + 8 is
  auto row_of = [&](int u) -> int64_t {
    if constexpr (kGated) {
      const int per = p.gate_block >> 3;
      return static_cast<int64_t>(u / per) * (2 * p.gate_block) + (u % per) * 8 + g;
    }
    return min(static_cast<int64_t>(u) * 16 + g, static_cast<int64_t>(p.n) - 1);
  };
  auto second = [&](int64_t row) -> int64_t { return kGated ? row + p.up_rows : min(row + 8, static_cast<int64_t>(p.n) - 1); };

  const uint32_t ring = smem_u32(smem) + warp * (kDepth * kSlotBytes) + lane * 16;
  int lu = u0, lj = 0, lslot = 0;
  const int lane_off = (s0 + warp) * kStepBytes + t * 16;
  const uint8_t* w0 = p.w + row_of(lu) * p.ldw + lane_off;
  const uint8_t* w1 = p.w + second(row_of(lu)) * p.ldw + lane_off;
  const int my_steps = (s1 - s0 - warp + kWarps - 1) / kWarps;     // of this warp: J, or one less
  auto issue = [&]() {
    if (lj < my_steps) {
      const uint32_t dst = ring + lslot * kSlotBytes;
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(w0) : "memory");
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst + 512), "l"(w1) : "memory");
    }
    w0 += kWarps * kStepBytes;
    w1 += kWarps * kStepBytes;
    if (++lslot == kDepth) lslot = 0;
    if (++lj == J) {
      lj = 0;
      if (++lu < u1) {
        const int64_t r = row_of(lu);
        w0 = p.w + r * p.ldw + lane_off;
        w1 = p.w + second(r) * p.ldw + lane_off;
      }
    }
  };
  auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };

  if (!p.w_static) pdl_wait_loads();
#pragma unroll
  for (int i = 0; i < kDepth - 1; ++i) {
    if (i < total) issue();
    commit();          // one group per step, empty past the end
  }
  if (p.w_static) pdl_wait_loads();

  uint32_t x[JX][kXRegs];
#pragma unroll
  for (int j = 0; j < JX; ++j) {
    const int s = s0 + j * kWarps + warp;
    const bool ok = g < p.m && s < s1;
    const uint4* src = reinterpret_cast<const uint4*>(p.x + g * p.ldx + (static_cast<int64_t>(s) * kStepK + t * (kStepK / 4)) * 2);
#pragma unroll
    for (int i = 0; i < kXRegs / 4; ++i) {
      const uint4 v = ok ? __ldcg(src + i) : make_uint4(0, 0, 0, 0);
      x[j][4 * i] = v.x;
      x[j][4 * i + 1] = v.y;
      x[j][4 * i + 2] = v.z;
      x[j][4 * i + 3] = v.w;
    }
  }

  // sum of the warps' (and the cluster's) parts of one output, activation, bias, residual, store
  auto finish = [&](int u, int tok, int r, float v, float up) {
    if (tok >= p.m) return;
    int64_t col;
    if constexpr (kGated) {
      if constexpr (ACT == kClamped) {
        if (p.bias != nullptr) {
          const int per = p.gate_block >> 3;
          const int64_t row = static_cast<int64_t>(u / per) * (2 * p.gate_block) + (u % per) * 8 + r;
          v += half_to_f<F16>(static_cast<const uint16_t*>(p.bias)[row]);
          up += half_to_f<F16>(static_cast<const uint16_t*>(p.bias)[row + p.up_rows]);
        }
        v = clamped_gate(v, up, p.act_limit);
      } else {
        v = gate_act<ACT == kGelu>(v) * up;
      }
      col = static_cast<int64_t>(u) * 8 + r;
    } else {
      col = static_cast<int64_t>(u) * 16 + r;
      if (col >= p.n) return;
      if constexpr (ACT == kRelu2) {
        v = fmaxf(v, 0.f);
        v *= v;
      }
      if (p.bias != nullptr) v += half_to_f<F16>(static_cast<const uint16_t*>(p.bias)[col]);
      if (p.residual != nullptr) v += half_to_f<F16>(__ldcg(static_cast<const uint16_t*>(p.residual) + tok * p.ld_res + col));
    }
    static_cast<uint16_t*>(p.out)[tok * p.ldc + col] = f_to_half<F16>(v);
  };

  int slot = 0, buf = 0, done = 0;
  for (int u = u0; u < u1; ++u) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < JX; ++j) {
      if (j < J) {
        // the copies of kDepth - 1 steps are on their way; the oldest of them is this step
        asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
        const uint32_t at = ring + slot * kSlotBytes;
        if (++slot == kDepth) slot = 0;
        if (j < my_steps) {
          uint4 a, b;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w) : "r"(at) : "memory");
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(at + 512) : "memory");
          mma<F16>(acc, a.x, b.x, a.y, b.y, x[j][0], x[j][1]);
          mma<F16>(acc, a.z, b.z, a.w, b.w, x[j][2], x[j][3]);
        }
        // the slot of the step before is free: its values were used by the products above it in program order
        if (done + kDepth - 1 < total) issue();
        commit();
        ++done;
      }
    }
    float(*mine)[17] = partial[buf][warp];
    mine[2 * t][g] = acc[0];
    mine[2 * t + 1][g] = acc[1];
    mine[2 * t][g + 8] = acc[2];
    mine[2 * t + 1][g + 8] = acc[3];
    __syncthreads();
    if (threadIdx.x < 128) {
      const int tok = threadIdx.x >> 4, r = threadIdx.x & 15;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += partial[buf][w][tok][r];
      if (p.cluster > 1) {
        unit_sums[(u - u0) * 128 + threadIdx.x] = v;
      } else if constexpr (kGated) {
        const float up = __shfl_down_sync(0xffffffffu, v, 8);
        if (r < 8) finish(u, tok, r, v, up);
      } else {
        finish(u, tok, r, v, 0.f);
      }
    }
    buf ^= 1;
  }
  if (p.cluster > 1) {
    cluster_barrier();                                   // every part of every sum is in its CTA's shared memory
    const uint32_t base = smem_u32(unit_sums);
    for (int u = u0 + rank; u < u1; u += p.cluster) {
      if (threadIdx.x < 128) {
        const int tok = threadIdx.x >> 4, r = threadIdx.x & 15;
        const uint32_t at = base + ((u - u0) * 128 + threadIdx.x) * 4;
        float v = 0.f;
        for (int c = 0; c < p.cluster; ++c) v += ld_peer(at, c);      // in rank order
        if constexpr (kGated) {
          const float up = __shfl_down_sync(0xffffffffu, v, 8);
          if (r < 8) finish(u, tok, r, v, up);
        } else {
          finish(u, tok, r, v, 0.f);
        }
      }
    }
    cluster_barrier();                                   // no CTA leaves while its sums are read
  }
}

// Launches the kernel for a problem whose Params hold everything but the split; 1 when the shape does not fit.
template <bool F16, int ACT>
int launch(Params p, int num_sms, cudaStream_t s) {
  constexpr int kJ = 16;
  constexpr int kMaxSmem = 110 * 1024;
  auto kern = gemm_stream_kernel<F16, ACT, kJ>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kMaxSmem) != cudaSuccess) return -3;
  ensure_max_carveout(reinterpret_cast<const void*>(kern));
  const int per_warp = (p.steps + kWarps - 1) / kWarps;
  p.cluster = 1;
  while (p.cluster < 8 && (per_warp + p.cluster - 1) / p.cluster > kJ) p.cluster *= 2;
  if (((p.steps + p.cluster - 1) / p.cluster + kWarps - 1) / kWarps > kJ) return 1;
  // two CTAs per SM, every cluster the same number of units: the stream is bound by memory, not by how many SMs pull on it
  // (n x k 5120 x 25600, 1 row: in 36 clusters of eight, of which the device holds 33 at once, 60.8 us, in 32 of them 41.4; 4096 x 12288
  // is 64 clusters of four either way)
  const int clusters =
      p.cluster == 1 ? 2 * num_sms : std::max(1, max_clusters(p.cluster, kThreads, 110 * 1024, 2 * num_sms / (p.cluster + 1)));
  p.units_per_cluster = (p.units + clusters - 1) / clusters;
  const int grid = (p.units + p.units_per_cluster - 1) / p.units_per_cluster * p.cluster;
  const int smem = kRingBytes + (p.cluster > 1 ? p.units_per_cluster * 512 : 0);
  if (smem > kMaxSmem) return 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
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

}  // namespace stream
}  // namespace mb200
