// Decode attention (one query token per request) over the slot-indexed KV pool, head sizes 64, 128 and 256, 16-bit caches.
//
// A decode step reads every cached key and value once and does 4 x (query heads of a group) operations per element: it is a
// memory stream, and what bounds it is how evenly the bytes are dealt to the SMs and how many of them are on their way.
//   * Work is cut by bytes, not by request: the tokens of all (request, kv head) pairs form one line of 64-token tiles, and
//     every CTA takes an equal run of it, whatever the lengths.  A pair that lies in one CTA is written out directly; the
//     others leave at most two partial results per CTA, which a second kernel joins.  The line is laid out on the device from
//     the sequence lengths, so a captured graph serves any batch.  (A grid of requests x heads x splits, with the splits
//     taken from the longest length the host allows for, and roles that meet at mbarriers, took 87.5 us for 29 requests of 400 to
//     3400 tokens and 8 kv heads, 128 us for 64 x 2048 and 4 heads, 25.9 us for 8 x 2048 and 8 heads; dealt evenly 44.1, 53.9 and 20.7
//     us before what the next lines say, joining included; the bytes take 34, 40 and 10 us.)
//     The chain in front of the first copy (lengths, table, rows; queries and the table's row beside them; no 64-bit division) and the
//     meeting of the warps are 4 us of a CTA's time when each load waits for the one before; side by side, and four values a thread:
//     2 x 1500 (8 kv heads) 11.4 -> 9.3 us, 8 x 2048 20.9 -> 18.2, 1 x 160 7.3 -> 6.8, 29 x 1900 46.0 -> 42.2, joining included.
//   * A warp owns 16 tokens of a tile and a ring of its own that cp.async fills two tiles ahead: 128 KB are in flight per SM,
//     and no barrier stands between the arrival of a tile and its use.  Rows come by slot one by one (16 lanes a row), so
//     a page size of 1 costs what a page size of 16 does.  The TMA engine's gather fell to half the speed there.
//   * S^T = K Q^T and O^T += V^T P^T are warp-level products with tokens (features) as the 16 rows and the group's heads as
//     the 8 columns, so that a group of 4 or 8 heads fills the tile; P^T turns from accumulator to operand layout by
//     movmatrix, in registers.  A 128-row tcgen05 tile would be 94 % padding and needs the scores to pass through shared
//     memory between barriers of the whole CTA.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace mb200 {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kWarpTokens = 16;
constexpr int kTile = kWarps * kWarpTokens;   // tokens of a tile
constexpr int kNoToken = -0x7fffffff;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleThreshold = 8.0f;     // the running maximum is raised when a score passes it by 2^8

struct DecodeParams {
  const void* q;
  const void* k_cache;
  const void* v_cache;
  void* out;
  float* part_o;     // [CTAs][2][group][HD]
  float* part_lse;   // [CTAs][2][group]
  const int* req_to_token;
  const int* req_pool_indices;
  const int* seq_lens;
  const float* sink;
  int* status;
  int64_t q_stride, out_stride, rtt_stride, num_slots, kv_tok_stride, kv_head_stride;
  int batch, hkv, group, ctas;
  int window, chunk;
  float scale_log2, cap_pre, cap_post;   // cap_post 0: no soft cap
};

// first key that the query of a sequence of `len` tokens sees, rounded down to a warp's tokens
__device__ __forceinline__ int first_key(const DecodeParams& p, int len) {
  if (p.window > 0) return max(0, len - p.window);
  return p.chunk > 0 ? (len - 1) / p.chunk * p.chunk : 0;
}
__device__ __forceinline__ int tiles_of(const DecodeParams& p, int len) {
  if (len <= 0) return 0;
  const int lo = first_key(p, len) & ~(kWarpTokens - 1);
  return (len - lo + kTile - 1) / kTile;
}

// The line: request by request, a request's kv heads in turn.  A (request, kv head) pair has a unit per tile, and kStart units
// behind them that hold no work: the time that a pair costs beside its tiles (the fill of the rings, the meeting of the warps).
// Without them many short pairs are dealt to one CTA, which all others wait for: three padded rows of a batch, 24 pairs of one
// token, made 29 requests of some 1500 tokens take 77.7 us instead of 46.0; with the units 43.6.
// Returns the units of all requests in front of this thread's run of requests [first, last) and, in `total`, of all requests (per
// kv head).
constexpr int kStart = 2;
__device__ __forceinline__ int units_of(const DecodeParams& p, int b) {
  const int n = tiles_of(p, __ldcg(p.seq_lens + b));
  return n > 0 ? n + kStart : 0;
}
__device__ __forceinline__ int scan_tiles(const DecodeParams& p, int* warp_sums, int& first, int& last, int& total) {
  const int per = (p.batch + kThreads - 1) / kThreads;
  first = min(p.batch, static_cast<int>(threadIdx.x) * per);
  last = min(p.batch, first + per);
  int mine = 0;
  for (int b = first; b < last; ++b) mine += units_of(p, b);
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if ((threadIdx.x & 31) >= o) incl += v;
  }
  if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < static_cast<int>(threadIdx.x >> 5)) before += warp_sums[w];
    total += warp_sums[w];
  }
  return before + incl - mine;
}
// CTAs that share the line and where CTA c's run begins.  A CTA is worth its set-up and its place in the join from four tiles on
// (1 x 4096 tokens, 8 kv heads: 13.4 us with four, 15.1 with two; 64 x 100: 14.9 and 17.3); up to 64 CTAs two are enough, since
// a short line is bound by what one CTA does in turn (1 x 160: 8.4 us with two, 9.4 with four).
__device__ __forceinline__ int ctas_used(const DecodeParams& p, int64_t line) {
  const int64_t want = max(line / 4, min(line / 2, static_cast<int64_t>(64)));
  return static_cast<int>(min(static_cast<int64_t>(p.ctas), max(want, static_cast<int64_t>(1))));
}
__device__ __forceinline__ int64_t run_begin(int64_t line, int c, int ctas) {
  // a division of 64 bits takes some 500 cycles of the chain in front of the first copy
  if (line < 0xFFFFFFFFll / (ctas + 1)) return static_cast<uint32_t>(line) * static_cast<uint32_t>(c) / static_cast<uint32_t>(ctas);
  return line * c / ctas;
}

__device__ __forceinline__ uint32_t movmatrix(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ void cp16_l2(uint32_t dst, const void* src, bool valid) {
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}

template <int HD, int NT>
struct Cfg {
  static constexpr int kChunks = HD / 8;                         // 16-byte pieces of a row
  static constexpr int kTensorBytes = kWarpTokens * HD * 2;      // a warp's K or V rows of one tile
  static constexpr int kStages = HD == 64 ? 4 : 3;
  static constexpr int kRingBytes = kStages * 2 * kTensorBytes;  // of one warp; afterwards its partial result
  static constexpr int kOutStride = HD + 4;                      // floats between the heads of a partial result: no bank conflicts
  static constexpr int kSmem = kWarps * kRingBytes + 128;
  static constexpr int kPerSm = HD == 256 ? 1 : 2;
  static_assert(kOutStride % 4 == 0 && kRingBytes % 16 == 0, "partial results are read four values at a time");
  static_assert(NT * 8 * kOutStride * 4 <= kRingBytes, "a warp's partial result must fit its ring");
};

template <typename T, int HD, int NT>
__global__ void __launch_bounds__(kThreads, Cfg<HD, NT>::kPerSm) attn_decode_stream_kernel(const DecodeParams p) {
  using C = Cfg<HD, NT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int warp_sums[kWarps];
  __shared__ int start[5];                          // where the run begins: request, kv head, tile; its length and row of the table
  __shared__ float part_m[kWarps][NT * 8], part_l[kWarps][NT * 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = p.group;
  pdl_wait_loads();
  pdl_launch_dependents();   // the joining kernel may lay out the line while this one streams

  // What stands between here and the first copy is a chain of round trips: lengths, then the table, then the rows.  Everything else
  // (the table's row, the queries) is on its way beside them.
  int b, hk, t0, len, row;
  int64_t left;
  {
    int first, last, total;
    const int mine = min(p.batch - 1, static_cast<int>(threadIdx.x) * ((p.batch + kThreads - 1) / kThreads));
    const int my_row = __ldcg(p.req_pool_indices + mine);       // of the first of this thread's requests
    const int before = scan_tiles(p, warp_sums, first, last, total);
    const int64_t line = static_cast<int64_t>(total) * p.hkv;
    const int used = ctas_used(p, line);
    if (static_cast<int>(blockIdx.x) >= used) return;
    const int64_t begin = run_begin(line, blockIdx.x, used);
    left = run_begin(line, blockIdx.x + 1, used) - begin;
    if (left <= 0) return;
    int64_t at = static_cast<int64_t>(before) * p.hkv;
    for (int r = first; r < last; ++r) {
      const int n = units_of(p, r);
      if (begin >= at && begin < at + static_cast<int64_t>(n) * p.hkv) {
        const int in = static_cast<int>(begin - at), h = in / n;
        start[0] = r;
        start[1] = h;
        start[2] = in - h * n;
        start[3] = __ldcg(p.seq_lens + r);
        start[4] = r == first ? my_row : __ldcg(p.req_pool_indices + r);
      }
      at += static_cast<int64_t>(n) * p.hkv;
    }
    __syncthreads();
    b = start[0];
    hk = start[1];
    t0 = start[2];
    len = start[3];
    row = start[4];
  }

  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127)) + warp * C::kRingBytes;
  const uint32_t ring_addr = smem_u32(ring);
  float* my_part = reinterpret_cast<float*>(ring);
  bool bad = false;
  bool at_run_begin = true;

  while (left > 0) {
    if (!at_run_begin) {
      len = __ldcg(p.seq_lens + b);
      row = __ldcg(p.req_pool_indices + b);
    }
    const int key0 = first_key(p, len);
    const int n_all = tiles_of(p, len);
    if (t0 >= n_all) {          // behind a pair's tiles, or a request without a token
      if (n_all > 0) left -= n_all + kStart - t0;
      t0 = 0;
      if (n_all == 0 || ++hk == p.hkv) {
        hk = 0;
        ++b;
      }
      at_run_begin = false;
      continue;
    }
    const int n = static_cast<int>(min(static_cast<int64_t>(n_all - t0), left));
    const int base0 = (key0 & ~(kWarpTokens - 1)) + t0 * kTile + warp * kWarpTokens;   // first token of this warp's first tile
    const int* rtt = p.req_to_token + static_cast<int64_t>(row) * p.rtt_stride;
    const T* kbase = static_cast<const T*>(p.k_cache) + hk * p.kv_head_stride;
    const T* vbase = static_cast<const T*>(p.v_cache) + hk * p.kv_head_stride;

    auto slot_of = [&](int t) -> int {             // slot of token (lane & 15) of this warp's tile t
      const int tok = base0 + t * kTile + (lane & 15);
      return (t < n && tok < len) ? __ldcg(rtt + tok) : kNoToken;
    };
    int ahead[C::kStages - 1];              // the slots of the first tiles, in one round trip
#pragma unroll
    for (int t = 0; t < C::kStages - 1; ++t) ahead[t] = slot_of(t);
    int slot_next = slot_of(C::kStages - 1);
    // the queries of the group as the column operand: head nt * 8 + lane / 4, features 2 (lane % 4) of every 8
    uint32_t qf[HD / 16][NT][2];
    {
      const T* q = static_cast<const T*>(p.q) + b * p.q_stride + static_cast<int64_t>(hk) * g * HD;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int h = nt * 8 + (lane >> 2);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            qf[kk][nt][i] = h < g ? __ldcg(reinterpret_cast<const uint32_t*>(q + h * HD + kk * 16 + i * 8 + 2 * (lane & 3))) : 0u;
      }
    }
    auto issue = [&](int t, int s) {
      if (t < n) {
        if (s < 0 || s >= p.num_slots) {
          bad = bad || s != kNoToken;
          s = -1;
        }
        const uint32_t dst = ring_addr + (t % C::kStages) * (2 * C::kTensorBytes);
        constexpr int kRowsPerPass = 32 / C::kChunks > 0 ? 32 / C::kChunks : 1;
        constexpr int kPasses = kWarpTokens / kRowsPerPass;
        const int ch = lane % C::kChunks, r0 = lane / C::kChunks;
#pragma unroll
        for (int i = 0; i < kPasses; ++i) {
          const int row = i * kRowsPerPass + r0;
          const int rs = __shfl_sync(0xffffffffu, s, row);
          const int64_t off = static_cast<int64_t>(max(rs, 0)) * p.kv_tok_stride + ch * 8;
          const uint32_t to = dst + row * (HD * 2) + ((ch ^ (row & 7)) << 4);
          cp16_l2(to, kbase + off, rs >= 0);
          cp16_l2(to + C::kTensorBytes, vbase + off, rs >= 0);
        }
      }
      cp_commit();
    };
#pragma unroll
    for (int t = 0; t < C::kStages - 1; ++t) issue(t, ahead[t]);
    float o[HD / 16][NT][4];
    float m[NT][2], l[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      m[nt][0] = m[nt][1] = -INFINITY;
      l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
      for (int mt = 0; mt < HD / 16; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[mt][nt][i] = 0.f;
    }

    for (int t = 0; t < n; ++t) {
      cp_wait<C::kStages - 2>();
      __syncwarp();
      issue(t + C::kStages - 1, slot_next);      // into the stage of the tile before, which every lane has left
      slot_next = slot_of(t + C::kStages);
      const int base = base0 + t * kTile;
      if (base >= len) continue;
      const uint32_t sk = ring_addr + (t % C::kStages) * (2 * C::kTensorBytes);
      const uint32_t sv = sk + C::kTensorBytes;
      float s[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[nt][i] = 0.f;
      {
        const int row = lane & 15;
        const uint32_t arow = sk + row * (HD * 2);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          uint32_t a[4];
          ldsm4(a, arow + (((kk * 2 + (lane >> 4)) ^ (row & 7)) << 4));
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_16816<T>(s[nt], a[0], a[1], a[2], a[3], qf[kk][nt][0], qf[kk][nt][1]);
        }
      }
      const int tok = base + (lane >> 2);
      const bool ok0 = tok < len && tok >= key0, ok1 = tok + 8 < len && tok + 8 >= key0;
      bool raise = false;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        if (p.cap_post > 0.f) {
#pragma unroll
          for (int i = 0; i < 4; ++i) s[nt][i] = p.cap_post * tanhf(s[nt][i] * p.cap_pre);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) s[nt][i] *= p.scale_log2;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          s[nt][i] = ok0 ? s[nt][i] : -INFINITY;
          s[nt][i + 2] = ok1 ? s[nt][i + 2] : -INFINITY;
          const float top = fmaxf(s[nt][i], s[nt][i + 2]);
          raise = raise || top > m[nt][i] + kRescaleThreshold;   // the first tile always raises
        }
      }
      if (__any_sync(0xffffffffu, raise)) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float top = fmaxf(s[nt][i], s[nt][i + 2]);
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            const float now = fmaxf(m[nt][i], top);
            const float f = m[nt][i] == -INFINITY ? 0.f : fast_exp2(m[nt][i] - now);
            m[nt][i] = now;
            l[nt][i] *= f;
#pragma unroll
            for (int mt = 0; mt < HD / 16; ++mt) {
              o[mt][nt][i] *= f;
              o[mt][nt][i + 2] *= f;
            }
          }
        }
      }
      uint32_t pb[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float m0 = m[nt][0] == -INFINITY ? 0.f : m[nt][0], m1 = m[nt][1] == -INFINITY ? 0.f : m[nt][1];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float e0 = fast_exp2(s[nt][2 * i] - m0), e1 = fast_exp2(s[nt][2 * i + 1] - m1);
          uint32_t w;
          float2 back;            // the sum takes what the product takes: the rounded probabilities
          if constexpr (std::is_same<T, __half>::value) {
            const __half2 h = __floats2half2_rn(e0, e1);
            w = *reinterpret_cast<const uint32_t*>(&h);
            back = __half22float2(h);
          } else {
            w = pack_bf16x2(e0, e1);
            back = unpack_bf16x2(w);
          }
          l[nt][0] += back.x;
          l[nt][1] += back.y;
          pb[nt][i] = movmatrix(w);
        }
      }
      {
        const int row = (lane & 7) + ((lane >> 4) << 3);
        const uint32_t vrow = sv + row * (HD * 2);
#pragma unroll
        for (int mt = 0; mt < HD / 16; ++mt) {
          uint32_t a[4];
          ldsm4_t(a, vrow + (((mt * 2 + ((lane >> 3) & 1)) ^ (row & 7)) << 4));
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_16816<T>(o[mt][nt], a[0], a[1], a[2], a[3], pb[nt][0], pb[nt][1]);
        }
      }
    }
    cp_wait<0>();
    __syncwarp();

    // ---- the warps' results meet in shared memory: this warp's goes where its ring was ----
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float sum = l[nt][i];
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        const int h = nt * 8 + 2 * (lane & 3) + i;
        if (lane < 4) {
          part_m[warp][h] = m[nt][i];
          part_l[warp][h] = sum;
        }
#pragma unroll
        for (int mt = 0; mt < HD / 16; ++mt) {
          my_part[h * C::kOutStride + mt * 16 + (lane >> 2)] = o[mt][nt][i];
          my_part[h * C::kOutStride + mt * 16 + 8 + (lane >> 2)] = o[mt][nt][i + 2];
        }
      }
    }
    __syncthreads();
    const bool whole = t0 == 0 && n == n_all;
    const int64_t part = (static_cast<int64_t>(blockIdx.x) * 2 + (at_run_begin ? 0 : 1)) * g;
    const float* parts = reinterpret_cast<const float*>(ring - warp * C::kRingBytes);
    // a sum of 0: no key to be seen.  A NaN or infinite score makes it NaN, and that the result
    for (int i = threadIdx.x; i < g * (HD / 4); i += kThreads) {
      const int h = i / (HD / 4), d = i % (HD / 4) * 4;
      float top = part_m[0][h];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) top = fmaxf(top, part_m[w][h]);
      float den = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float f = part_m[w][h] == -INFINITY ? 0.f : exp2f(part_m[w][h] - top);
        const float4 v = *reinterpret_cast<const float4*>(parts + w * (C::kRingBytes / 4) + h * C::kOutStride + d);
        den += f * part_l[w][h];
        acc[0] += f * v.x;
        acc[1] += f * v.y;
        acc[2] += f * v.z;
        acc[3] += f * v.w;
      }
      if (whole) {
        if (p.sink != nullptr) den += exp2f(p.sink[hk * g + h] * kLog2e - top);
        T* out = static_cast<T*>(p.out) + b * p.out_stride + static_cast<int64_t>(hk * g + h) * HD + d;
#pragma unroll
        for (int e = 0; e < 4; ++e) out[e] = from_f32<T>(den == 0.f ? 0.f : acc[e] / den);
      } else {
        *reinterpret_cast<float4*>(p.part_o + (part + h) * HD + d) =
            den == 0.f ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(acc[0] / den, acc[1] / den, acc[2] / den, acc[3] / den);
        if (d == 0) p.part_lse[part + h] = den == 0.f ? -INFINITY : top + log2f(den);
      }
    }
    __syncthreads();
    left -= n;
    t0 += n;
    at_run_begin = false;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0 && p.status != nullptr) atomicExch(p.status, kStatusBadIndex);
}

// Joins the partial results of a (request, kv head) pair that lies in several CTAs: out = sum_s w_s O_s with
// w_s = 2^(lse_s - max) / sum; a head's sink is one more term of the sum, without a value.  A CTA has one query head.  The line
// of tiles is laid out again before the wait: its lengths were complete when the streaming kernel began.
template <typename T, int HD>
__global__ void __launch_bounds__(kThreads) attn_decode_join_kernel(const DecodeParams p) {
  __shared__ int warp_sums[kWarps];
  __shared__ int mine[2];       // units in front of the request, and its tiles
  __shared__ float weight[kThreads];
  pdl_launch_dependents();
  const int head = blockIdx.x, b = blockIdx.y, g = p.group;
  const int hk = head / g, h = head % g;
  int first, last, total;
  int before = scan_tiles(p, warp_sums, first, last, total);
  if (b >= first && b < last) {
    for (int r = first; r < b; ++r) before += units_of(p, r);
    mine[0] = before;
    mine[1] = tiles_of(p, __ldcg(p.seq_lens + b));
  }
  __syncthreads();
  const int64_t line = static_cast<int64_t>(total) * p.hkv;
  const int used = ctas_used(p, line);
  const int n = mine[1];
  const int64_t begin = static_cast<int64_t>(mine[0]) * p.hkv + static_cast<int64_t>(hk) * (n + kStart);
  T* out = static_cast<T*>(p.out) + b * p.out_stride + static_cast<int64_t>(head) * HD;
  // the last CTA whose run begins at or before x
  auto owner = [&](int64_t x) { return static_cast<int>(min(static_cast<int64_t>(used) - 1, ((x + 1) * used - 1) / line)); };
  const int c0 = n > 0 ? owner(begin) : 0, c1 = n > 0 ? owner(begin + n - 1) : 0;
  // the first of the pair's CTAs has it in its second slot where its run begins with another pair; the others in their first
  const int first_slot = c0 * 2 + (n > 0 && run_begin(line, c0, used) < begin ? 1 : 0);
  auto slot = [&](int c) { return static_cast<int64_t>(c == c0 ? first_slot : c * 2) * g + h; };
  pdl_wait_loads();
  if (n == 0) {
    for (int d = threadIdx.x; d < HD; d += kThreads) out[d] = from_f32<T>(0.f);
    return;
  }
  if (c0 == c1) return;         // one CTA had all of it and has written the output
  const float sink = p.sink != nullptr ? p.sink[head] * kLog2e : -INFINITY;
  constexpr int kPer = (HD + kThreads - 1) / kThreads, kEarly = 8;
  // the values of the first CTAs are on their way beside the sums that weigh them
  float early[kEarly][kPer];
#pragma unroll
  for (int i = 0; i < kEarly; ++i)
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int d = threadIdx.x + k * kThreads;
      early[i][k] = c0 + i <= c1 && d < HD ? __ldcg(p.part_o + slot(c0 + i) * HD + d) : 0.f;
    }
  float top = sink, den = 0.f;
  for (int c = c0 + static_cast<int>(threadIdx.x & 31); c <= c1; c += 32) top = fmaxf(top, __ldcg(p.part_lse + slot(c)));
  top = warp_max(top);
  if (p.sink != nullptr) den = exp2f(sink - top);
  float acc[kPer] = {};
  for (int at = c0; at <= c1; at += kThreads) {
    const int m = min(kThreads, c1 + 1 - at);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < m) {
      const float lse = __ldcg(p.part_lse + slot(at + threadIdx.x));
      weight[threadIdx.x] = lse == -INFINITY ? 0.f : exp2f(lse - top);
    }
    __syncthreads();
    int from = 0;
    if (at == c0) {
#pragma unroll
      for (int i = 0; i < kEarly; ++i) {
        if (i >= m) break;
        const float w = weight[i];
        den += w;
#pragma unroll
        for (int k = 0; k < kPer; ++k) acc[k] += w * early[i][k];
      }
      from = min(kEarly, m);
    }
#pragma unroll 8
    for (int i = from; i < m; ++i) {
      const float w = weight[i];
      den += w;
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int d = threadIdx.x + k * kThreads;
        if (d < HD) acc[k] += w * __ldcg(p.part_o + slot(at + i) * HD + d);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int d = threadIdx.x + k * kThreads;
    if (d < HD) out[d] = from_f32<T>(den == 0.f ? 0.f : acc[k] / den);
  }
}

template <typename T, int HD, int NT>
int launch_one(const DecodeParams& p, cudaStream_t s) {
  auto kern = attn_decode_stream_kernel<T, HD, NT>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), Cfg<HD, NT>::kSmem) != cudaSuccess) return -3;
  cudaError_t err = launch_pdl(kern, dim3(p.ctas), dim3(kThreads), Cfg<HD, NT>::kSmem, s, p);
  note_launch();
  if (err != cudaSuccess) return -4;
  err = launch_pdl(attn_decode_join_kernel<T, HD>, dim3(p.hkv * p.group, p.batch), dim3(kThreads), 0, s, p);
  note_launch();
  return err == cudaSuccess ? 0 : -4;
}

template <typename T, int HD>
int launch_size(const DecodeParams& p, cudaStream_t s) {
  if (p.group <= 8) return launch_one<T, HD, 1>(p, s);
  if (p.group <= 16) return launch_one<T, HD, 2>(p, s);
  if constexpr (HD <= 128) return launch_one<T, HD, 4>(p, s);
  return 1;
}

}  // namespace

// The streaming kernel takes every 16-bit cache with up to 32 query heads a group (16 where heads are 256 wide: more
// accumulators than registers).  Wider groups and 8-bit caches go to the single-role kernel.
bool decode_streams(int head_dim, int group, int kv_fmt) { return kv_fmt == 0 && group <= (head_dim == 256 ? 16 : 32); }

int decode_stream_ctas(int head_dim, int num_sms) { return head_dim == 256 ? num_sms : 2 * num_sms; }

int64_t decode_stream_floats(int head_dim, int group, int ctas) { return static_cast<int64_t>(ctas) * 2 * group * (head_dim + 1); }

int launch_decode_stream(const AttnArgs& a, cudaStream_t s) {
  DecodeParams p{};
  p.q = a.q;
  p.k_cache = a.k_cache;
  p.v_cache = a.v_cache;
  p.out = a.out;
  p.part_o = a.part_o;
  p.group = a.hq / a.hkv;
  p.ctas = a.num_splits;
  p.part_lse = a.part_o + static_cast<int64_t>(p.ctas) * 2 * p.group * a.head_dim;
  p.req_to_token = a.req_to_token;
  p.req_pool_indices = a.req_pool_indices;
  p.seq_lens = a.seq_lens;
  p.sink = a.sink;
  p.status = a.status;
  p.q_stride = a.q_stride;
  p.out_stride = a.out_stride > 0 ? a.out_stride : static_cast<int64_t>(a.hq) * a.head_dim;
  p.rtt_stride = a.rtt_stride;
  p.num_slots = a.num_slots;
  p.kv_tok_stride = a.kv_tok_stride;
  p.kv_head_stride = a.kv_head_stride;
  p.batch = a.batch;
  p.hkv = a.hkv;
  p.window = a.window > 0 ? a.window : 0;
  p.chunk = a.chunk > 0 ? a.chunk : 0;
  p.scale_log2 = a.scale * kLog2e;
  if (a.logit_cap > 0.f) {
    p.cap_pre = a.scale / a.logit_cap;
    p.cap_post = a.logit_cap * kLog2e;
  }
  int rc = 1;
  MB200_DISPATCH_HALF(a.dt, rc = a.head_dim == 64 ? launch_size<T, 64>(p, s) : a.head_dim == 128 ? launch_size<T, 128>(p, s)
                                                                                                  : launch_size<T, 256>(p, s));
  return rc;
}

}  // namespace mb200
