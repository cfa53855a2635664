// out[m, n] = a[m, k] * b[n, k]^T where one wave of tiles is all there is: batches of 9 to 256 rows (decode steps of a serving
// batch, short prompts), and products of more rows that leave most SMs without a 256 x 256 tile (vision towers, narrow
// projections).  What costs time here is not the tensor cores but everything in front of and behind them, so:
//   * the weights are the 128-row operand and BN rows of `a` the MMA's N: a tile is small in the batch's direction, and a matrix
//     gives many of them;
//   * the k range of a tile is cut over the CTAs of a cluster until the GPU is full, and its partial sums are exchanged through
//     distributed shared memory: every CTA of the cluster finishes a slice of the columns.  (Partial sums through global memory,
//     finished by the last CTA to arrive, took 28 us for 128 rows of a 4096 x 1024 matrix and 56 us for 29 rows of a
//     24576 x 4096 one.)
//   * two CTAs share an SM where there are that many, one of them often already the next kernel's: it fills its ring with weights,
//     which no kernel writes, before it waits for its input;
//   * the sums reach the output through shared memory, eight neighbouring columns per thread: 16-byte stores, coalesced.
//
// Warp roles (192 threads): warp 0 = TMA producer, warp 1 = tensor memory and MMA issue, warps 2 - 5 = accumulators to shared
// memory; all six finish the output.  Every mbarrier wait is bounded; on expiry the status word is set and all roles drain.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace mb200 {
namespace {

constexpr int kTileRows = 128;        // weight rows of a tile
constexpr int kRowBytes = 128;        // of k per pipeline stage: one swizzle span
constexpr int kTileThreads = 192;
constexpr int kWeightBytes = kTileRows * kRowBytes;

struct TileParams {
  void* out;
  const void* bias;
  const void* residual;
  const float* a_scale;
  const float* b_scale;
  int* status;
  float act_limit;
  int m, n, k_blocks, tiles_n;
  int64_t ldc, ld_res;
  int cluster, stages, out_f16, is_int8, w_static;
  uint32_t idesc;
};

template <int SWIGLU>
constexpr bool kGatedTile = SWIGLU == 1 || SWIGLU == 2 || SWIGLU == 4;

__device__ __forceinline__ uint32_t my_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void unpack8(const uint4& v, int f16, float (&f)[8]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = f16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[i])) : unpack_bf16x2(w[i]);
    f[2 * i] = x.x;
    f[2 * i + 1] = x.y;
  }
}

template <int BN, int SWIGLU>
__global__ void __launch_bounds__(kTileThreads, 2)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const TileParams p) {
  constexpr bool kGated = kGatedTile<SWIGLU>;
  constexpr int kStageBytes = kWeightBytes + BN * kRowBytes;
  constexpr int kTmemCols = BN < 32 ? 32 : BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int n_stages = p.stages;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(n_stages) * kStageBytes);
  uint64_t* empty_bar = full_bar + n_stages;
  uint64_t* acc_full = empty_bar + n_stages;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  // behind the allocation, which waits for as long as the columns are taken: CTAs of the next kernel that took them first would hold
  // them until this kernel ends
  pdl_launch_dependents();

  const int rank = p.cluster > 1 ? static_cast<int>(my_rank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / p.cluster;
  const int tn = tile % p.tiles_n, tm = tile / p.tiles_n;
  const int kb0 = p.k_blocks * rank / p.cluster, kb1 = p.k_blocks * (rank + 1) / p.cluster;
  const int k_elems = p.is_int8 ? kRowBytes : kRowBytes / 2;
  // first weight row; a gated tile has 64 gate rows and the up rows 128 behind them
  const int w_row = kGated ? (tn >> 1) * 256 + (tn & 1) * 64 : tn * kTileRows;

  // Only the producer runs ahead of the stream-order wait.  The roles that wait for its copies begin behind it, so that their limits
  // cover this kernel's own work and not the kernels in front.
  if (warp == 0) {
    if (elect_one()) {
      auto load_w = [&](int s, int kb) {
        uint8_t* at = smem + static_cast<size_t>(s) * kStageBytes;
        mbar_arrive_expect_tx(&full_bar[s], kStageBytes);
        tma_load_2d(at, &tm_w, &full_bar[s], kb * k_elems, w_row);
        if constexpr (kGated) tma_load_2d(at + kWeightBytes / 2, &tm_w, &full_bar[s], kb * k_elems, w_row + 128);
      };
      if (!p.w_static) pdl_wait_loads();
      const int early = min(n_stages, kb1 - kb0);
      for (int i = 0; i < early; ++i) load_w(i, kb0 + i);
      if (p.w_static) pdl_wait_loads();
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kb - kb0 >= early) {
          if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          load_w(s, kb);
        }
        tma_load_2d(smem + static_cast<size_t>(s) * kStageBytes + kWeightBytes, &tm_x, &full_bar[s], kb * k_elems, tm * BN);
        if (++s == n_stages) {
          s = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status != nullptr) atomicExch(p.status, kStatusPipelineTimeout);
      }
    }
  } else if (warp == 1) {
    pdl_wait_loads();
    if (elect_one()) {
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem));
      bool ok = true;
      // One thread issues everything: what stands between two products is paid four times a stage, so the type is chosen outside and
      // descriptors are moved, not made
      auto multiply = [&](auto int8_tag) {
        constexpr bool kInt8 = decltype(int8_tag)::value;
        const uint32_t idesc = p.idesc;
        int s = 0;
        uint32_t phase = 0;
        auto stage = [&](bool first) {
          const uint64_t w_desc = desc0 + static_cast<uint32_t>(s) * (kStageBytes >> 4);
          const uint64_t x_desc = w_desc + (kWeightBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint32_t accum = first && kk == 0 ? 0u : 1u;
            if constexpr (kInt8) umma_i8(tmem, w_desc + kk * 2, x_desc + kk * 2, idesc, accum);
            else umma_f16(tmem, w_desc + kk * 2, x_desc + kk * 2, idesc, accum);
          }
          umma_commit(&empty_bar[s]);
          if (++s == n_stages) {
            s = 0;
            phase ^= 1;
          }
        };
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[s], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          stage(kb == kb0);
        }
      };
      if (p.is_int8) multiply(std::true_type{});
      else multiply(std::false_type{});
      if (ok) umma_commit(acc_full);
      if (!ok) {
        *abort_flag = 1;
        if (p.status != nullptr) atomicExch(p.status, kStatusPipelineTimeout);
      }
    }
    __syncwarp();
  } else {
    pdl_wait_loads();
    if (!mbar_wait(acc_full, 0, abort_flag)) {
      *abort_flag = 1;
      if (p.status != nullptr) atomicExch(p.status, kStatusPipelineTimeout);
    }
    tc_fence_after_sync();
  }
  __syncwarp();
  pdl_wait_loads();        // the other lanes of the producer's warp too: all finish the output from what the kernels in front left
  __syncthreads();
  if (*abort_flag) {
    // copies may still be in flight: give them time to land before the ring is used for the sums
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  // ---- sums: [source][column of the slice][weight row] in the CTA that finishes the slice, where the ring was ----
  if (p.cluster > 1) cluster_meet();        // every ring of the cluster has been read
  const int cols = BN / p.cluster, cols_log = __popc(cols - 1);      // a power of two
  const uint32_t inbox = smem_u32(smem);
  if (warp >= 2) {
    const int quad = warp & 3, row = quad * 32 + lane;
    const uint32_t t_base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
      uint32_t v[16];
      tmem_ld_32x16(t_base + c0, v);
      tmem_ld_wait();
      const uint32_t at = inbox + (((rank << cols_log) * kTileRows + row) << 2);
      if (p.cluster == 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (c0 + j) * (kTileRows * 4)), "r"(v[j]) : "memory");
      } else if (cols >= 16) {      // all sixteen columns go to one CTA
        const uint32_t to = peer_addr(at, c0 >> cols_log) + (c0 & (cols - 1)) * (kTileRows * 4);
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(to + j * (kTileRows * 4)), "r"(v[j]) : "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(peer_addr(at, (c0 + j) >> cols_log) + ((c0 + j) & (cols - 1)) * (kTileRows * 4)),
                       "r"(v[j])
                       : "memory");
      }
    }
  }
  tc_fence_before_sync();
  if (p.cluster > 1)
    cluster_meet();
  else
    __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);

  // ---- finish: a thread takes eight neighbouring outputs of one row of `a` ----
  constexpr int kGroups = (kGated ? kTileRows / 2 : kTileRows) / 8;
  const float* sums = reinterpret_cast<const float*>(smem);
  for (int i = threadIdx.x; i < cols * kGroups; i += kTileThreads) {
    const int c = i / kGroups, grp = i % kGroups;
    const int row = tm * BN + rank * cols + c;
    const int64_t col = static_cast<int64_t>(tn) * (kGated ? 64 : kTileRows) + grp * 8;
    if (row >= p.m || (!kGated && col >= p.n)) continue;
    float v[8] = {}, u[8] = {};
    // in rank order; the sums of 8-bit products stay whole numbers, which 24 bits do not hold from a k of 1040 on
    auto gather = [&](auto int8_tag) {
      auto add = [](float& sum, float part) {
        if constexpr (decltype(int8_tag)::value) sum = __int_as_float(__float_as_int(sum) + __float_as_int(part));
        else sum += part;
      };
      for (int src = 0; src < p.cluster; ++src) {
        const float4* from = reinterpret_cast<const float4*>(sums + (src * cols + c) * kTileRows + grp * 8);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 x = from[q];
          add(v[4 * q], x.x);
          add(v[4 * q + 1], x.y);
          add(v[4 * q + 2], x.z);
          add(v[4 * q + 3], x.w);
          if constexpr (kGated) {
            const float4 y = from[16 + q];              // 64 weight rows on
            add(u[4 * q], y.x);
            add(u[4 * q + 1], y.y);
            add(u[4 * q + 2], y.z);
            add(u[4 * q + 3], y.w);
          }
        }
      }
    };
    if (p.is_int8) gather(std::true_type{});
    else gather(std::false_type{});
    const int64_t wr = kGated ? w_row + grp * 8 : col;
    if (p.is_int8) {
      const float sa = __ldcg(p.a_scale + row);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = static_cast<float>(__float_as_int(v[j])) * (sa * p.b_scale[wr + j]);
        if constexpr (kGated) u[j] = static_cast<float>(__float_as_int(u[j])) * (sa * p.b_scale[wr + 128 + j]);
      }
    }
    if (p.bias != nullptr) {
      float b[8];
      unpack8(__ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.bias) + wr)), p.out_f16, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += b[j];
      if constexpr (SWIGLU == 4) {
        unpack8(__ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.bias) + wr + 128)), p.out_f16, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] += b[j];
      }
    }
    if constexpr (kGated) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = SWIGLU == 4 ? clamped_gate(v[j], u[j], p.act_limit) : gate_act<SWIGLU == 2>(v[j]) * u[j];
    } else {
      if constexpr (SWIGLU == 3) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.f) * fmaxf(v[j], 0.f);
      }
      if (p.residual != nullptr) {
        float r[8];
        unpack8(__ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.residual) + row * p.ld_res + col)), p.out_f16, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += r[j];
      }
    }
    uint4 o;
    uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (p.out_f16) {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
      } else {
        w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
      }
    }
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + row * p.ldc + col) = o;
  }
}

// Clusters of 1, 2, 4 and 8 CTAs that the device holds at once, one CTA per SM or two.  A thread keeps the counts of the device that it
// launched on last: a launch asks for up to a dozen, and from the maps of max_clusters they took the host 1 us of the 12.5 per product.
struct Places {
  int of[2][4];
  int operator()(int c, int per_sm) const { return of[per_sm - 1][c == 1 ? 0 : c == 2 ? 1 : c == 4 ? 2 : 3]; }
};
const Places& places_of_device(int num_sms) {
  thread_local Places known;
  thread_local int device = -1;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev != device) {
    for (int per_sm = 1; per_sm <= 2; ++per_sm)
      for (int i = 0; i < 4; ++i)
        known.of[per_sm - 1][i] = i == 0 ? per_sm * num_sms
                                         : max_clusters(1 << i, kTileThreads, (per_sm == 2 ? 104 : 200) * 1024, per_sm * num_sms / ((1 << i) + 1));
    device = dev;
  }
  return known;
}

template <int BN, int SWIGLU>
int launch_tile(const CUtensorMap& tw, const CUtensorMap& tx, TileParams p, int grid, const Places& places, cudaStream_t s) {
  constexpr int kStageBytes = kWeightBytes + BN * kRowBytes;
  constexpr int kTail = 1024 + 512;
  // A ring for one CTA per SM, or half of it for two; deep enough for the sums, which take its place.  (One per SM, the device measured
  // holds 15 clusters of eight.  With the whole ring for 16 of them the last ran behind the others: 29 rows of 2048 x 4096 11.0 us, with
  // half of it 7.0.)
  const int budget = (grid <= places(p.cluster, 1) * p.cluster ? 200 : 104) * 1024;
  const int blocks = (p.k_blocks + p.cluster - 1) / p.cluster;
  p.stages = std::max(2, std::min(std::min((budget - kTail) / kStageBytes, 12), blocks));
  while (p.stages * kStageBytes < BN * kTileRows * 4) ++p.stages;
  const int smem = p.stages * kStageBytes + kTail;
  auto kern = gemm_tile_kernel<BN, SWIGLU>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), 208 * 1024) != cudaSuccess) return -3;
  ensure_max_carveout(reinterpret_cast<const void*>(kern));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kTileThreads);
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
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, tw, tx, p);
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

template <int SWIGLU>
int launch_bn(int bn, const CUtensorMap& tw, const CUtensorMap& tx, const TileParams& p, int grid, const Places& places, cudaStream_t s) {
  switch (bn) {
    case 16: return launch_tile<16, SWIGLU>(tw, tx, p, grid, places, s);
    case 32: return launch_tile<32, SWIGLU>(tw, tx, p, grid, places, s);
    case 64: return launch_tile<64, SWIGLU>(tw, tx, p, grid, places, s);
    default: return launch_tile<128, SWIGLU>(tw, tx, p, grid, places, s);
  }
}

}  // namespace

// The checks of launch_gemm have passed.  Returns 1 when the product has more tiles than one wave of two CTAs per SM: the
// persistent kernels, which overlap a tile's end with the next one's loads, are then the better ones.
int launch_gemm_tile(const GemmArgs& a, cudaStream_t s) {
  if (a.gate_flags != nullptr || a.rs_tp > 0 || a.norm_weight != nullptr || a.m <= 8) return 1;
  const bool gated = a.swiglu == 1 || a.swiglu == 2 || a.swiglu == 4;
  if (a.bias != nullptr && (reinterpret_cast<uintptr_t>(a.bias) & 15) != 0) return 1;
  const int sms = a.num_sms > 0 ? a.num_sms : 148;
  const int eb = a.is_int8 ? 1 : 2, k_per = kRowBytes / eb;
  TileParams p{};
  p.tiles_n = (a.n + kTileRows - 1) / kTileRows;
  p.k_blocks = (a.k + k_per - 1) / k_per;
  auto tiles = [&](int bn) { return static_cast<int64_t>(p.tiles_n) * ((a.m + bn - 1) / bn); };
  int bn = 16;
  while (bn < a.m && bn < 128) bn *= 2;
  // few weight rows: narrower tiles, until a cluster of eight per tile would fill the GPU
  while (bn > 32 && tiles(bn) * 8 <= sms) bn /= 2;
  if (tiles(bn) > 2 * sms) return 1;
  const Places& places = places_of_device(sms);
  // Clusters grow while every CTA keeps four stages (29 rows of 4096 x 1024: in clusters of eight, with two stages, 5.9 us, of four 5.1)
  // and the device holds all of them at once, one CTA per SM: 128 rows of 6144 x 4096 17.7 us in 48 clusters of
  // four, two CTAs per SM, and 15.2 in 48 of two; 29 rows of 9216 x 2560, 72 of four of which 71 fit, 15.7 and 10.7.  With up to 32
  // columns a stage is little work and what a CTA waits for is memory: two CTAs per SM in clusters of four and eight (29 rows of
  // 2048 x 4096: of four 7.5, of eight 7.0; 5120 x 5120: of two 13.4, of four 12.6).
  auto cluster_of = [&](int bn) {
    int c = 1;
    while (c < 8 && p.k_blocks >= 8 * c &&
           (tiles(bn) <= places(2 * c, 1) || (bn <= 32 && c >= 2 && tiles(bn) <= places(2 * c, 2))))
      c *= 2;
    return c;
  };
  // Short k: what a CTA exchanges grows with the tile's width, what it multiplies with its share of k.  Narrower tiles in smaller
  // clusters while the share is under bn / 8 stages (200 rows of 4096 x 1024: 128 columns in clusters of two 8.6 us, 64 without 7.6).
  while (bn > 32 && cluster_of(bn) > 1 && p.k_blocks / cluster_of(bn) * 8 < bn) bn /= 2;
  p.cluster = cluster_of(bn);
  // Whole tiles of 128 x 128, more than half a wave of them and no gate: the persistent kernel, whose epilogue stores rows of the output as
  // they come (512 rows of 4096 x 1024 9.3 us here, 8.0 there; 1024 of 2048 x 2048 12.4 and 11.1; 384 of 6144 x 4096 19.8 and 19.3; with
  // SwiGLU 11.3 and 15.5, in two rounds instead of two per SM, 192 tiles of 512 x 6144 x 4096, 29.0 and 31.6, with 8-bit operands the same).
  if (a.m > 256 && a.swiglu == 0 && !a.is_int8 && bn == 128 && tiles(bn) > places(2, 1) && tiles(bn) <= sms) return 1;
  p.out = a.out;
  p.bias = a.bias;
  p.residual = a.residual;
  p.a_scale = a.a_scale;
  p.b_scale = a.b_scale;
  p.status = a.status;
  p.act_limit = a.act_limit;
  p.m = a.m;
  p.n = a.n;
  p.ldc = a.ldc;
  p.ld_res = a.ld_res;
  p.out_f16 = a.dt == kF16 ? 1 : 0;
  p.is_int8 = a.is_int8;
  p.w_static = a.b_static;
  const uint32_t fmt = a.is_int8 ? 1u : (a.dt == kF16 ? 0u : 1u);
  p.idesc = umma_idesc(kTileRows, bn, a.is_int8 ? 2u : 1u, fmt, fmt);
  const int type = a.is_int8 ? 2 : (a.dt == kF16 ? 1 : 0);
  CUtensorMap tw, tx;
  if (!make_tma_operand_map(&tw, a.b, a.n, a.k, a.ldb, eb, type, gated ? kTileRows / 2 : kTileRows)) return -2;
  if (!make_tma_operand_map(&tx, a.a, a.m, a.k, a.lda, eb, type, bn)) return -2;
  const int grid = static_cast<int>(tiles(bn)) * p.cluster;
  switch (a.swiglu) {
    case 1: return launch_bn<1>(bn, tw, tx, p, grid, places, s);
    case 2: return launch_bn<2>(bn, tw, tx, p, grid, places, s);
    case 3: return launch_bn<3>(bn, tw, tx, p, grid, places, s);
    case 4: return launch_bn<4>(bn, tw, tx, p, grid, places, s);
    default: return launch_bn<0>(bn, tw, tx, p, grid, places, s);
  }
}

}  // namespace mb200
