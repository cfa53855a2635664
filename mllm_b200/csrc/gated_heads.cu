// What stands around attention in layers whose query projection carries an output gate: per head [query | gate], keys and values
// behind the heads of one projected row.  One pass in front (norm per head with a gain, rotation of part of a head, cache write),
// one behind (the gate).  Both are bound by memory for prompts and by the launch for decode steps; as separate element-wise
// operators they were 27 launches a layer, of 1.2 to 3 us each in a decode step, and moved a prompt's rows eleven times.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace mb200 {
namespace {

__device__ __forceinline__ int lane_of() { return threadIdx.x & 31; }

template <typename T, int E>
struct Vec;
template <typename T>
struct Vec<T, 2> {
  using type = uint32_t;
};
template <typename T>
struct Vec<T, 4> {
  using type = uint2;
};
template <typename T>
struct Vec<T, 8> {
  using type = uint4;
};
template <typename T>
__device__ __forceinline__ float rounded(float v) {
  return to_f32(from_f32<T>(v));
}

// A warp takes the heads h_first, h_first + hsplit, ... of a token; a lane has E = D / 32 neighbouring features.  Features i and
// i + half of the first 2 half turn by the token's angles, which a lane forms once for all its heads; the partner's features are
// `half / E` lanes away.
template <typename T, int E>
__global__ void __launch_bounds__(256) gated_head_prologue_kernel(const GatedHeadArgs p) {
  using V = typename Vec<T, E>::type;
  pdl_launch_dependents();
  pdl_wait_loads();
  constexpr int D = 32 * E;
  const int heads = p.hq + 2 * p.hkv;
  const int64_t warp = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  if (warp >= static_cast<int64_t>(p.tokens) * p.hsplit) return;
  const int t = static_cast<int>(warp / p.hsplit), h_first = static_cast<int>(warp % p.hsplit), lane = lane_of();
  const int64_t slot = p.loc[t];
  const bool slot_ok = slot >= 0 && slot < p.num_slots;
  if (!slot_ok && h_first == 0 && lane == 0 && p.status != nullptr) atomicExch(p.status, kStatusBadIndex);
  float cs[E], sn[E];
  const int half_lanes = p.half / E;
  const bool turns = lane < 2 * half_lanes;
  if (turns && h_first < p.hq + p.hkv) {
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int f = lane * E + i, fi = f < p.half ? f : f - p.half;
      const int axis = p.axis_map != nullptr ? p.axis_map[fi] : 0;
      sincosf(static_cast<float>(p.positions[static_cast<int64_t>(axis) * p.tokens + t]) * p.inv_freq[fi], &sn[i], &cs[i]);
      if (f < p.half) sn[i] = -sn[i];
    }
  }
  const T* row = static_cast<const T*>(p.row) + t * p.row_stride + lane * E;
  for (int h = h_first; h < heads; h += p.hsplit) {
    const bool is_q = h < p.hq, is_k = !is_q && h < p.hq + p.hkv;
    const T* src = row + (is_q ? h * 2 * D : p.hq * 2 * D + (h - p.hq) * D);
    V raw = *reinterpret_cast<const V*>(src);
    T* e = reinterpret_cast<T*>(&raw);
    if (is_q || is_k) {
      float f[E], ss = 0.f;
#pragma unroll
      for (int i = 0; i < E; ++i) {
        f[i] = to_f32(e[i]);
        ss += f[i] * f[i];
      }
      const float rstd = rsqrtf(warp_sum(ss) / static_cast<float>(D) + p.eps);
      const V wr = *reinterpret_cast<const V*>(static_cast<const T*>(is_q ? p.q_w : p.k_w) + lane * E);
      const T* w = reinterpret_cast<const T*>(&wr);
#pragma unroll
      for (int i = 0; i < E; ++i) {
        f[i] = rounded<T>(f[i] * rstd * to_f32(w[i]));
        const float partner = __shfl_xor_sync(0xffffffffu, f[i], half_lanes);
        e[i] = from_f32<T>(turns ? f[i] * cs[i] + partner * sn[i] : f[i]);
      }
    }
    if (is_q) {
      *reinterpret_cast<V*>(static_cast<T*>(p.q_out) + (static_cast<int64_t>(t) * p.hq + h) * D + lane * E) = raw;
    } else if (slot_ok) {
      T* cache = static_cast<T*>(is_k ? p.k_cache : p.v_cache);
      const int kvh = is_k ? h - p.hq : h - p.hq - p.hkv;
      *reinterpret_cast<V*>(cache + slot * p.kv_tok_stride + kvh * p.kv_head_stride + lane * E) = raw;
    }
  }
}

// x[t, h, :] *= sigmoid(gate of head h), the gates 2 D apart in the projected row, 8 features per thread
template <typename T>
__global__ void __launch_bounds__(256) gated_head_epilogue_kernel(T* x, const T* row, int64_t row_stride, int64_t total,
                                                                  int hq, int dim) {
  pdl_launch_dependents();
  pdl_wait_loads();
  const int per_row = hq * dim / 8;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / per_row;
    const int c = static_cast<int>(i - t * per_row) * 8, h = c / dim;
    uint4 xv = *reinterpret_cast<const uint4*>(x + t * hq * dim + c);
    const uint4 gv = *reinterpret_cast<const uint4*>(row + t * row_stride + h * 2 * dim + dim + (c - h * dim));
    T* xe = reinterpret_cast<T*>(&xv);
    const T* ge = reinterpret_cast<const T*>(&gv);
#pragma unroll
    for (int j = 0; j < 8; ++j) xe[j] = from_f32<T>(to_f32(xe[j]) / (1.f + __expf(-to_f32(ge[j]))));
    *reinterpret_cast<uint4*>(x + t * hq * dim + c) = xv;
  }
}

}  // namespace

int launch_gated_head_prologue(GatedHeadArgs a, int num_sms, cudaStream_t s) {
  if (a.tokens <= 0) return 0;
  const int heads = a.hq + 2 * a.hkv;
  // a warp per token once there are enough tokens to fill the GPU: the angles are then formed once per token
  a.hsplit = 1;
  while (a.hsplit < heads && static_cast<int64_t>(a.tokens) * a.hsplit < num_sms * 32) a.hsplit = std::min(heads, a.hsplit * 2);
  const dim3 grid(static_cast<unsigned>((static_cast<int64_t>(a.tokens) * a.hsplit * 32 + 255) / 256));
  cudaError_t err = cudaErrorInvalidValue;
  MB200_DISPATCH_HALF(a.dt, {
    if (a.dim == 64) err = launch_pdl(gated_head_prologue_kernel<T, 2>, grid, dim3(256), 0, s, a);
    if (a.dim == 128) err = launch_pdl(gated_head_prologue_kernel<T, 4>, grid, dim3(256), 0, s, a);
    if (a.dim == 256) err = launch_pdl(gated_head_prologue_kernel<T, 8>, grid, dim3(256), 0, s, a);
  });
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

int launch_gated_head_epilogue(void* x, const void* row, int64_t row_stride, int tokens, int hq, int dim, DType dt, int num_sms, cudaStream_t s) {
  if (tokens <= 0) return 0;
  const int64_t total = static_cast<int64_t>(tokens) * hq * dim / 8;
  const dim3 grid(static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, num_sms * 16)));
  cudaError_t err = cudaSuccess;
  MB200_DISPATCH_HALF(dt, err = launch_pdl(gated_head_epilogue_kernel<T>, grid, dim3(256), 0, s, static_cast<T*>(x), static_cast<const T*>(row),
                                           row_stride, total, hq, dim));
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

}  // namespace mb200
