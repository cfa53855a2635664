// Grouped expert product for many tokens per expert: for every work item (expert e, chunk of 256 of its sorted rows),
// out[rows] = act[rows] * W[e]^T in 256 x 256 tiles, each by a cluster of two CTAs (tcgen05.mma.cta_group::2).  A CTA stages 128
// rows of the activations and 128 of the weights per 64-element k block: 32 KB for 512 cycles of tensor work, where the one-CTA
// kernel of moe.cu stages 48 KB (two 128-row weight tiles and 128 tokens) and is bound by what reaches shared memory from the L2
// cache.  65536 rows of 2048 features to 64 experts: gate and up 482 -> 403 us, down 350 -> 235.
//
// The rows of a tile behind the expert's last one belong to the next expert; they are multiplied and not stored.  Roles and
// barriers are those of gemm_pair_kernel (gemm_tcgen05.cu): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), warp 2
// tensor memory, warps 4 - 7 epilogue; the TMA copies of both CTAs count on the leader's barrier, commits arrive on both CTAs'
// barriers, no multicast.  All waits are bounded; a CTA that gives up raises its own and its partner's abort flag.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace mb200 {
namespace {

constexpr int kBM = 128, kBN = 256, kRowBytes = 128, kUmmaKBytes = 32, kThreads = 256;
constexpr int kStageBytes = 2 * kBM * kRowBytes;
constexpr int kStages = 6;
constexpr int kSmem = kStages * kStageBytes + 1024 + 512;

struct PairParams {
  void* out;
  int64_t ldc;
  const int* expert_offsets;
  const int2* work;
  const int* n_work;
  int* status;
  int n, k_blocks, tiles_c, out_f16;
  uint32_t idesc;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of `local` (an address in this CTA's shared memory) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_smem(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// TMA load whose completion bytes are counted on a barrier that may live in the partner CTA
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_out, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_out)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// all pair MMAs issued so far by this thread arrive on the barrier at `bar_cluster_addr` when they finish
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr)
               : "memory");
}


__device__ __forceinline__ float gelu_exact(float v) { return 0.5f * v * (1.f + erff(v * 0.70710678118654752f)); }

// ACT: 0 plain product, 1 silu(gate) * up over alternating blocks of 128 gate and 128 up rows, 2 the exact GELU
template <int ACT>
__global__ void __launch_bounds__(kThreads, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(kStages) * kStageBytes);   // leader: 1 arrival + bytes of both CTAs
  uint64_t* empty_bar = full_bar + kStages;        // per CTA: tcgen05.commit
  uint64_t* acc_full = full_bar + 2 * kStages;     // per CTA: tcgen05.commit
  uint64_t* acc_empty = acc_full + 2;              // leader: 256 epilogue threads of the pair
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 256);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
  }
  __syncthreads();
  if (warp == 2) {
    tmem_alloc_pair(tmem_holder, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  cluster_sync_all();   // both CTAs' barriers are initialised before either signals the other's
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;
  pdl_wait_loads();

  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int total = *p.n_work * p.tiles_c;
  // a pair's idx-th tile: first activation row of this CTA, one past the expert's last row, first weight row, column tile.  The
  // tiles of a chunk follow one another: its rows are read from the L2 cache by all pairs at about the same time
  auto get_tile = [&](int idx, int& row0, int& row_end, int& wrow, int& tc) -> bool {
    const int tile = pair + idx * num_pairs;
    if (tile >= total) return false;
    const int2 w = p.work[tile / p.tiles_c];
    tc = tile % p.tiles_c;
    row0 = p.expert_offsets[w.x] + w.y * kBN + static_cast<int>(rank) * kBM;
    row_end = p.expert_offsets[w.x + 1];
    wrow = w.x * p.n + tc * kBN + static_cast<int>(rank) * (kBN / 2);
    return true;
  };
  auto give_up = [&]() {
    *abort_flag = 1;
    st_cluster_u32(mapa_smem(smem_u32(const_cast<int*>(abort_flag)), rank ^ 1u), 1u);
    if (p.status != nullptr) atomicExch(p.status, kStatusPipelineTimeout);
  };
  int row0, row_end, wrow, tc;

  if (warp == 0 && elect_one()) {
    const uint32_t full_leader0 = mapa_smem(smem_u32(&full_bar[0]), 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int idx = 0; ok && get_tile(idx, row0, row_end, wrow, tc); ++idx) {
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        uint8_t* at = smem + static_cast<size_t>(stage) * kStageBytes;
        const uint32_t full = full_leader0 + static_cast<uint32_t>(stage) * 8u;
        if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * kStageBytes);
        tma_load_2d_pair(at, &tm_x, full, kb * (kRowBytes / 2), row0);
        tma_load_2d_pair(at + kBM * kRowBytes, &tm_w, full, kb * (kRowBytes / 2), wrow);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) give_up();
  } else if (warp == 1 && leader && elect_one()) {
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint64_t desc_stage0 = umma_desc_k_sw128(smem_u32(smem));
    const uint32_t empty0 = mapa_smem(smem_u32(&empty_bar[0]), 0), empty1 = mapa_smem(smem_u32(&empty_bar[0]), 1);
    for (int idx = 0; ok && get_tile(idx, row0, row_end, wrow, tc); ++idx) {
      const int acc = idx & 1;
      if (!mbar_wait(&acc_empty[acc], ((idx >> 1) & 1) ^ 1, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint64_t a_stage = desc_stage0 + static_cast<uint32_t>(stage) * (kStageBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kRowBytes / kUmmaKBytes; ++kk)
          umma_f16_pair(tmem_base + acc * kBN, a_stage + ((kk * kUmmaKBytes) >> 4), a_stage + ((kBM * kRowBytes + kk * kUmmaKBytes) >> 4), p.idesc,
                        kb > 0 || kk > 0 ? 1u : 0u);
        umma_commit_pair(empty0 + static_cast<uint32_t>(stage) * 8u);
        umma_commit_pair(empty1 + static_cast<uint32_t>(stage) * 8u);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) {
        umma_commit_pair(mapa_smem(smem_u32(&acc_full[acc]), 0));
        umma_commit_pair(mapa_smem(smem_u32(&acc_full[acc]), 1));
      }
    }
    if (!ok) give_up();
  } else if (warp >= 4) {
    const int ew = warp - 4;
    constexpr int kOutCols = ACT == 1 ? kBN / 2 : kBN;
    bool ok = true;
    for (int idx = 0; ok && get_tile(idx, row0, row_end, wrow, tc); ++idx) {
      const int acc = idx & 1;
      if (*abort_flag || !mbar_wait(&acc_full[acc], (idx >> 1) & 1, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t t_base = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + acc * kBN;
      const int64_t row = row0 + ew * 32 + lane;
      const bool row_ok = row < row_end;
      uint16_t* out = static_cast<uint16_t*>(p.out) + row * p.ldc + static_cast<int64_t>(tc) * kOutCols;
#pragma unroll 1
      for (int c = 0; c < kOutCols; c += 32) {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32(t_base + c, r0);
        if constexpr (ACT == 1) tmem_ld_32x32(t_base + kBN / 2 + c, r1);
        tmem_ld_wait();
        if (!row_ok) continue;
#pragma unroll
        for (int v8 = 0; v8 < 4; ++v8) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float f[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int at = v8 * 8 + 2 * j + q;
              f[q] = __uint_as_float(r0[at]);
              if constexpr (ACT == 1) f[q] = gate_act<false>(f[q]) * __uint_as_float(r1[at]);
              if constexpr (ACT == 2) f[q] = gelu_exact(f[q]);
            }
            if (p.out_f16) {
              const __half2 h = __floats2half2_rn(f[0], f[1]);
              w[j] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
              w[j] = pack_bf16x2(f[0], f[1]);
            }
          }
          *reinterpret_cast<uint4*>(out + c + v8 * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      tc_fence_before_sync();
      mbar_arrive_cluster(mapa_smem(smem_u32(&acc_empty[acc]), 0));
    }
    if (!ok) give_up();
  }

  pdl_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // give copies that may still be in flight time to land before the CTAs' memory is reused
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  // neither CTA may leave while its partner can still read its shared memory or signal its barriers
  cluster_sync_all();
  if (warp == 2) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <int ACT>
int launch_pair(const CUtensorMap& tx, const CUtensorMap& tw, const PairParams& p, int pairs, cudaStream_t s) {
  auto kern = moe_pair_kernel<ACT>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmem) != cudaSuccess) return -3;
  ensure_max_carveout(reinterpret_cast<const void*>(kern));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, tx, tw, p);
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

}  // namespace

// The checks of launch_moe_grouped_gemm have passed and the work items are chunks of 256 rows.
int launch_moe_pair_gemm(const MoeGemmArgs& a, cudaStream_t s) {
  if (a.n % kBN != 0) return -1;
  PairParams p{};
  p.out = a.out;
  p.ldc = a.ldc;
  p.expert_offsets = a.expert_offsets;
  p.work = reinterpret_cast<const int2*>(a.work);
  p.n_work = a.n_work;
  p.status = a.status;
  p.n = a.n;
  p.k_blocks = (a.k + 63) / 64;
  p.tiles_c = a.n / kBN;
  p.out_f16 = a.dt == kF16 ? 1 : 0;
  const uint32_t fmt = a.dt == kF16 ? 0u : 1u;
  p.idesc = umma_idesc(2 * kBM, kBN, 1u, fmt, fmt);
  CUtensorMap tx, tw;
  const int type = a.dt == kF16 ? 1 : 0;
  if (!make_tma_operand_map(&tx, a.x, a.rows_cap, a.k, a.ldx, 2, type, kBM)) return -2;
  if (!make_tma_operand_map(&tw, a.w, static_cast<int64_t>(a.experts) * a.n, a.k, a.k, 2, type, kBN / 2)) return -2;
  const int pairs = std::max(1, (a.num_sms > 0 ? a.num_sms : 148) / 2);
  if (a.gelu) return launch_pair<2>(tx, tw, p, pairs, s);
  return a.swiglu ? launch_pair<1>(tx, tw, p, pairs, s) : launch_pair<0>(tx, tw, p, pairs, s);
}

}  // namespace mb200
