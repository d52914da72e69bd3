// Prompt attention of the decoder on the 5th-generation tensor cores, fp32 in and out (sm_100a).
//   scores * 1/sqrt(D), causal mask, softmax, P.V   mllm/Models/ds_qwen2/modeling_ds_qwen2.hpp:127-150
//   RoPE (half-split) and the cache append          mllm/Backends/Arm/Kernels/rope.cpp:20-87, Ops/KVCacheOp.cpp:15-72
//
// The two products run as tcgen05.mma kind::f16 on operands split in two, x 2^E = hi + lo with hi = fp16(x 2^E) and
// lo = fp16(x 2^E - hi).  2^E (one per query row, one per 64-position tile of K and of V, the largest magnitude at 2^13) keeps
// hi clear of fp16's range and subnormals; what is lost of x is at most 2^-22 |x|, or 2^-38 of the row's or tile's largest
// magnitude where that is more; hi hi + hi lo + lo hi drops at most 2^-22 of a product.  Every product is exact in the fp32
// accumulator; a tile's P.V leaves tensor memory after 64 positions and is added in registers, so that no sum runs through
// more than 64 (scores: D) additions on the tensor core.  Error of the output against 64 bits (2-norm, all rows, 12 heads of
// 128), this kernel / fp32 on the CUDA cores: normal q, k, v at 97, 512, 1900, 6000 tokens 2.4, 3.1, 3.3, 3.4e-7 / 2.5, 3.5,
// 4.4, 6.1e-7; eight times larger scores 4.6, 6.0, 7.5, 8.7e-7 / 8.1, 11.9, 15.6, 18.4e-7; values of one sign, which the
// truncated sums shrink, 1.6, 1.9, 2.1, 2.3e-7 / 1.2, 2.4, 4.6, 8.1e-7.
//
// One power of two for a tile ties its positions together, those included that a row must not see.  So a tile whose rows of K
// or V differ by more than 2^14 in magnitude, or that holds infinities or NaN, is marked unfit, and the CTAs that reach it
// take the fp32 arithmetic of decoder_attn_rows.cuh (512 tokens, 12 heads of 128: 500 us a layer instead of 26; the fp32
// kernel, whose grid is finer, 85).  Below that, what a position loses to its neighbours' size is at most 2^-24 of its own
// largest element, which is what fp32 itself keeps.
//
// prefill_kv_split_kernel rotates the keys, appends keys and values to the cache and leaves both as ready operands
// (canonical K-major core matrices; V transposed), 64 positions per tile.  attention_prefill_tc_kernel: a CTA owns the
// rows (token, query head of one KV head) of 128 / group consecutive tokens = the 128 lanes of tensor memory:
//   warps 0-7  softmax: warp w has lanes 32 (w % 4).. and half of the columns; query rows are rotated, split and parked
//              in tensor memory once; per tile: scores -> online softmax -> P split into tensor memory; output in registers
//   warp 8     producer: one bulk copy per K and per V tile into two rings
//   warp 9     MMA issuer and tensor-memory owner: scores of tile j + 1 run while the softmax of tile j does
// Bound by the softmax warps' instructions (about 700 per thread and tile of 128 x 64; the products take 1536 cycles of
// the tensor pipe).  Tiles are dispatched longest causal range first.
#include <cuda_fp16.h>

#include "decoder_attn_rows.cuh"
#include "decoder_state.h"
#include "device_common.cuh"
#include "tcgen05_common.cuh"

namespace mllmb200 {

constexpr int kPaKeys = 64;                   // cache positions per tile
constexpr int kPaMaxTiles = 8192 / kPaKeys;   // the decoder's largest context
constexpr int kPaThreads = 10 * 32;
constexpr float kPaPScale = 4096.0f;          // softmax weights times 2^12: the low halves of small ones stay normal
constexpr int kPsThreads = 512;

template <int D>
struct PaLayout {
  static constexpr int kOpBytes = kPaKeys * D * 2;        // one half (hi or lo) of a K or V tile
  static constexpr int kTileBytes = 4 * kOpBytes;         // K hi, K lo, V hi, V lo
  static constexpr int kStages = D == 128 ? 3 : 6;        // 192 KB of rings either way: one CTA per SM, which owns all of tensor memory
  static constexpr int kBarBytes = 256;
  static constexpr int kScaleBytes = kPaMaxTiles * 8;
  static constexpr int kRedBytes = 2 * 2 * 128 * 4;
  static constexpr int kTotal = kBarBytes + kScaleBytes + kRedBytes + kStages * kTileBytes + 1024;
  // tensor-memory columns
  static constexpr int kColQ = 0, kColS = 128, kColP = 256, kColPV = 320;  // Q: D/2 hi, D/2 lo; S: 2 x 64; P: 32 hi, 32 lo; PV: D
};

// exponent that brings a largest magnitude into [2^13, 2^14); 2^E and 2^-E are normal numbers
__device__ __forceinline__ int pa_exponent(float mx) {
  const int e = (int)((__float_as_uint(mx) >> 23) & 0xFFu) - 127;
  return mx == 0.0f ? 0 : max(-126, min(126, 13 - e));
}
__device__ __forceinline__ float pa_pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }
// two scaled numbers to their fp16 halves
__device__ __forceinline__ void pa_split(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ uint32_t pa_magnitude(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }  // orders like |x|, infinities and NaN on top
template <int LANES>
__device__ __forceinline__ uint32_t pa_row_max(uint32_t m, int lane) {  // over the LANES lanes that share a row
  return __reduce_max_sync(LANES == 32 ? 0xffffffffu : ((1u << (LANES & 31)) - 1u) << (lane & ~(LANES - 1)), m);
}
// A tile's keys or values that one power of two does not serve: rows whose largest magnitudes (bits; of the smallest non-zero
// one, less 1) are more than a factor of 2^14 apart, infinities, NaN, nothing but numbers below 2^-113.
__device__ __forceinline__ bool pa_unfit(uint32_t largest, uint32_t smallest_less_1) {
  return largest != 0 && (largest >= 0x7F800000u || largest < (14u << 23) || (smallest_less_1 >> 23) + 14 < largest >> 23);
}

// grid (tiles, kv heads): rotates 64 new keys, appends keys and values at positions 64 tile .. to the cache
// [kv_heads][max_ctx][D] and writes the tile's operands and {2^-E of K, 2^-E of V} (zeros: the tile is unfit).
template <int D>
__global__ void __launch_bounds__(kPsThreads) prefill_kv_split_kernel(
    const float* __restrict__ k_new, const float* __restrict__ v_new, int ld, int n, const float* __restrict__ sin_t,
    const float* __restrict__ cos_t, int max_ctx, float* __restrict__ cache_k, float* __restrict__ cache_v,
    uint8_t* __restrict__ tiles, float2* __restrict__ tile_scales) {
  using L = PaLayout<D>;
  constexpr int HALF = D / 2, KI = kPaKeys * HALF / 4 / kPsThreads, VI = kPaKeys * D / 4 / kPsThreads;
  pdl_launch_dependents();
  pdl_wait_prior();
  extern __shared__ __align__(16) float ps_smem[];
  float(*s_k)[D + 1] = reinterpret_cast<float(*)[D + 1]>(ps_smem);
  float(*s_v)[D + 1] = s_k + kPaKeys;
  __shared__ uint4 s_mx[kPsThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = blockIdx.x, h = blockIdx.y, p0 = tile * kPaKeys;
  float4 x0[KI], x1[KI], sn[KI], cs[KI], vv[VI];
#pragma unroll
  for (int u = 0; u < KI; ++u) {
    const int idx = tid + u * kPsThreads, j = idx / (HALF / 4), d = idx % (HALF / 4) * 4;
    x0[u] = x1[u] = sn[u] = cs[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p0 + j < n) {
      const float* kr = k_new + (size_t)(p0 + j) * ld + h * D + d;
      x0[u] = *reinterpret_cast<const float4*>(kr);
      x1[u] = *reinterpret_cast<const float4*>(kr + HALF);
      sn[u] = *reinterpret_cast<const float4*>(sin_t + (size_t)(p0 + j) * HALF + d);
      cs[u] = *reinterpret_cast<const float4*>(cos_t + (size_t)(p0 + j) * HALF + d);
    }
  }
#pragma unroll
  for (int u = 0; u < VI; ++u) {
    const int idx = tid + u * kPsThreads, j = idx / (D / 4), d = idx % (D / 4) * 4;
    vv[u] = p0 + j < n ? *reinterpret_cast<const float4*>(v_new + (size_t)(p0 + j) * ld + h * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  uint32_t mk = 0, nk = ~0u, mv = 0, nv = ~0u;  // bits of the largest and the smallest of the rows' largest magnitudes (rows of zeros aside)
#pragma unroll
  for (int u = 0; u < KI; ++u) {
    const int idx = tid + u * kPsThreads, j = idx / (HALF / 4), d = idx % (HALF / 4) * 4;
    const float a[4] = {x0[u].x, x0[u].y, x0[u].z, x0[u].w}, b[4] = {x1[u].x, x1[u].y, x1[u].z, x1[u].w};
    const float s[4] = {sn[u].x, sn[u].y, sn[u].z, sn[u].w}, c[4] = {cs[u].x, cs[u].y, cs[u].z, cs[u].w};
    float y0[4], y1[4];
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y0[i] = a[i] * c[i] - b[i] * s[i];
      y1[i] = a[i] * s[i] + b[i] * c[i];
      s_k[j][d + i] = y0[i];
      s_k[j][d + HALF + i] = y1[i];
      m = max(m, max(pa_magnitude(y0[i]), pa_magnitude(y1[i])));
    }
    if (p0 + j < n) {
      float* dst = cache_k + ((size_t)h * max_ctx + p0 + j) * D + d;
      *reinterpret_cast<float4*>(dst) = make_float4(y0[0], y0[1], y0[2], y0[3]);
      *reinterpret_cast<float4*>(dst + HALF) = make_float4(y1[0], y1[1], y1[2], y1[3]);
    }
    m = pa_row_max<HALF / 4>(m, lane);
    mk = max(mk, m), nk = min(nk, m - 1);
  }
#pragma unroll
  for (int u = 0; u < VI; ++u) {
    const int idx = tid + u * kPsThreads, j = idx / (D / 4), d = idx % (D / 4) * 4;
    const float a[4] = {vv[u].x, vv[u].y, vv[u].z, vv[u].w};
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s_v[j][d + i] = a[i];
      m = max(m, pa_magnitude(a[i]));
    }
    if (p0 + j < n) *reinterpret_cast<float4*>(cache_v + ((size_t)h * max_ctx + p0 + j) * D + d) = vv[u];
    m = pa_row_max<D / 4>(m, lane);
    mv = max(mv, m), nv = min(nv, m - 1);
  }
  mk = __reduce_max_sync(0xffffffffu, mk), nk = __reduce_min_sync(0xffffffffu, nk);
  mv = __reduce_max_sync(0xffffffffu, mv), nv = __reduce_min_sync(0xffffffffu, nv);
  if (lane == 0) s_mx[warp] = make_uint4(mk, nk, mv, nv);
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kPsThreads / 32; ++w) {
    const uint4 o = s_mx[w];
    mk = max(mk, o.x), nk = min(nk, o.y), mv = max(mv, o.z), nv = min(nv, o.w);
  }
  const int ek = pa_exponent(__uint_as_float(mk)), ev = pa_exponent(__uint_as_float(mv));
  const size_t at = (size_t)h * gridDim.x + tile;
  if (tid == 0) tile_scales[at] = pa_unfit(mk, nk) || pa_unfit(mv, nv) ? make_float2(0.0f, 0.0f) : make_float2(pa_pow2(-ek), pa_pow2(-ev));
  uint8_t* out = tiles + at * L::kTileBytes;
  const float fk = pa_pow2(ek), fv = pa_pow2(ev);
  // 16 bytes per item: 8 dimensions of one key; 8 keys of one dimension
  for (int item = tid; item < kPaKeys * D / 8; item += kPsThreads) {
    uint32_t hi[4], lo[4];
    {
      const int r = item & 7, c = (item >> 3) % (D / 8), kg = item / D;
#pragma unroll
      for (int i = 0; i < 4; ++i) pa_split(s_k[kg * 8 + r][c * 8 + 2 * i] * fk, s_k[kg * 8 + r][c * 8 + 2 * i + 1] * fk, hi[i], lo[i]);
      *reinterpret_cast<uint4*>(out + item * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(out + L::kOpBytes + item * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    {
      const int r = item & 7, kc = (item >> 3) & 7, dg = item >> 6;
#pragma unroll
      for (int i = 0; i < 4; ++i) pa_split(s_v[kc * 8 + 2 * i][dg * 8 + r] * fv, s_v[kc * 8 + 2 * i + 1][dg * 8 + r] * fv, hi[i], lo[i]);
      *reinterpret_cast<uint4*>(out + 2 * L::kOpBytes + item * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(out + 3 * L::kOpBytes + item * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// The rows [s0, end) on the CUDA cores, by 256 threads.
template <int D>
__device__ __forceinline__ void prefill_rows_fp32(PrefillAttnSmem<D>& sm, int tid, const float* q, int ldq, int s0, int end, int kvh,
                                               const float* sin_t, const float* cos_t, int max_ctx, int group, const float* cache_k,
                                               const float* cache_v, float* out, int ldo) {
  static_assert(kPfRowThreads<2> == 256 && sizeof(PrefillAttnSmem<D>) <= (size_t)PaLayout<D>::kStages * PaLayout<D>::kTileBytes, "fits the rings");
  for (int next; s0 < end; s0 = next) {
    next = min(end, (s0 / kPfRows + 1) * kPfRows);  // the tiles of attention_prefill_kernel: an infinity reaches no other rows than there
    prefill_attn_rows<D, 2>(sm, tid, [] { asm volatile("bar.sync 5, 256;" ::: "memory"); }, q, ldq, s0, next, kvh, sin_t, cos_t, 0, max_ctx,
                            group, cache_k, cache_v, out, ldo);
  }
}

// q: rows of ldq floats (token s at position s); out: rows of ldo floats.  grid: (row tiles x kv heads), 1-D.
template <int D>
__global__ void __launch_bounds__(kPaThreads, 1) attention_prefill_tc_kernel(
    const float* __restrict__ q, int ldq, int n, const float* __restrict__ sin_t, const float* __restrict__ cos_t, int group,
    int kv_heads, const uint8_t* __restrict__ tiles, const float2* __restrict__ tile_scales, int max_ctx,
    const float* __restrict__ cache_k, const float* __restrict__ cache_v, float* __restrict__ out, int ldo) {
  using L = PaLayout<D>;
  constexpr int HALF = D / 2, QD = HALF / 2, kStages = L::kStages;  // QD: rotated pairs per thread
  pdl_launch_dependents();
  pdl_wait_prior();
  extern __shared__ __align__(128) uint8_t pa_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pa_smem) + 1023) & ~uintptr_t(1023));
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* v_full = k_full + kStages;
  uint64_t* k_free = v_full + kStages;
  uint64_t* v_free = k_free + kStages;
  uint64_t* s_full = v_free + kStages;  // [2]
  uint64_t* p_ready = s_full + 2;
  uint64_t* pv_done = p_ready + 1;
  uint64_t* q_ready = pv_done + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_ready + 1);
  static_assert((4 * kStages + 5) * 8 + 4 <= L::kBarBytes, "barrier area");
  float2* s_scales = reinterpret_cast<float2*>(smem + L::kBarBytes);
  float(*s_red)[2][128] = reinterpret_cast<float(*)[2][128]>(smem + L::kBarBytes + L::kScaleBytes);  // [buffer][column half][row]
  uint8_t* ring = smem + L::kBarBytes + L::kScaleBytes + L::kRedBytes;  // K stages, then V stages

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int tokens = 128 / group, row_tiles = (int)gridDim.x / kv_heads;
  const int rt = row_tiles - 1 - (int)blockIdx.x / kv_heads, kvh = (int)blockIdx.x % kv_heads;
  const int s0 = rt * tokens, last = min(s0 + tokens, n) - 1;
  const int nt = last / kPaKeys + 1, all_tiles = (n + kPaKeys - 1) / kPaKeys;
  const float2* scales = tile_scales + (size_t)kvh * all_tiles;
  const uint8_t* my_tiles = tiles + (size_t)kvh * all_tiles * L::kTileBytes;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&k_free[s], 1);
      mbar_init(&v_free[s], 1);
    }
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    mbar_init(p_ready, 8);
    mbar_init(pv_done, 1);
    mbar_init(q_ready, 8);
    mbar_fence_init();
  }
  bool unfit = false;
  for (int i = tid; i < nt; i += kPaThreads) {
    s_scales[i] = scales[i];
    unfit = unfit || s_scales[i].x == 0.0f;
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  unfit = __syncthreads_or(unfit) != 0;
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (unfit) {
    if (warp < 8)
      prefill_rows_fp32<D>(*reinterpret_cast<PrefillAttnSmem<D>*>(ring), tid, q, ldq, s0, last + 1, kvh, sin_t, cos_t, max_ctx, group, cache_k,
                           cache_v, out, ldo);
  } else if (warp == 8) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      constexpr uint32_t kBytes = 2 * L::kOpBytes;
      for (int j = 0; j < nt; ++j) {
        const int s = j % kStages;
        const uint32_t ph = ((uint32_t)(j / kStages) & 1u) ^ 1u;
        const uint8_t* src = my_tiles + (size_t)j * L::kTileBytes;
        if (!mbar_wait_bounded(&k_free[s], ph)) break;
        mbar_arrive_expect_tx(&k_full[s], kBytes);
        bulk_g2s(ring + s * kBytes, src, kBytes, &k_full[s]);
        if (!mbar_wait_bounded(&v_free[s], ph)) break;
        mbar_arrive_expect_tx(&v_full[s], kBytes);
        bulk_g2s(ring + (kStages + s) * kBytes, src + kBytes, kBytes, &v_full[s]);
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------ MMA issuer: the whole warp runs the loop, one lane issues
    const bool issuer = elect_one_sync();
    const uint32_t idesc_s = (1u << 4) | ((uint32_t)(kPaKeys >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t idesc_pv = (1u << 4) | ((uint32_t)(D >> 3) << 17) | ((128u >> 4) << 24);
    bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(q_ready, 0));
    auto scores = [&](int j) {  // S buffer j & 1 = Q K_j^T
      const int s = j % kStages;
      ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&k_full[s], (uint32_t)(j / kStages) & 1u));
      if (!ok) return;
      tc_fence_after();
      if (issuer) {
        const uint64_t hi = make_kmajor_desc(smem_u32(ring + s * 2 * L::kOpBytes), 128, (D / 8) * 128);
        const uint64_t lo = hi + (uint64_t)(L::kOpBytes >> 4);
        const uint32_t d = tmem + L::kColS + (uint32_t)(j & 1) * kPaKeys;
#pragma unroll
        for (int t = 0; t < 3; ++t)  // hi lo, lo hi, hi hi
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            tc_mma_f16_ts(d, tmem + L::kColQ + (uint32_t)((t == 1 ? D / 2 : 0) + ks * 8), (t == 0 ? lo : hi) + (uint64_t)(ks * 16), idesc_s,
                          t + ks > 0);
        tc_commit(&s_full[j & 1]);
        tc_commit(&k_free[s]);
      }
      __syncwarp();
    };
    tc_fence_after();
    scores(0);
    if (nt > 1) scores(1);
    for (int j = 0; j < nt && ok; ++j) {
      const int s = j % kStages;
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(p_ready, (uint32_t)j & 1u)) &&
           __all_sync(0xffffffffu, mbar_wait_bounded(&v_full[s], (uint32_t)(j / kStages) & 1u));
      if (!ok) break;
      tc_fence_after();
      if (issuer) {
        const uint64_t hi = make_kmajor_desc(smem_u32(ring + (kStages + s) * 2 * L::kOpBytes), 128, (kPaKeys / 8) * 128);
        const uint64_t lo = hi + (uint64_t)(L::kOpBytes >> 4);
#pragma unroll
        for (int t = 0; t < 3; ++t)
#pragma unroll
          for (int ks = 0; ks < kPaKeys / 16; ++ks)
            tc_mma_f16_ts(tmem + L::kColPV, tmem + L::kColP + (uint32_t)((t == 1 ? kPaKeys / 2 : 0) + ks * 8), (t == 0 ? lo : hi) + (uint64_t)(ks * 16),
                          idesc_pv, t + ks > 0);
        tc_commit(pv_done);
        tc_commit(&v_free[s]);
      }
      __syncwarp();
      if (j + 2 < nt) scores(j + 2);  // its buffer was read before p_ready(j)
    }
  } else {
    // ------------------------------------------------------------ softmax: one row per thread, half of the columns
    const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
    const int tok = s0 + row / group, head = row % group;
    const bool live = row < tokens * group && tok < n;
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + quad) : "memory"); };  // the two warps of these lanes
    float q_scale;  // 1/sqrt(D) over the row's power of two
    {
      float y[2][QD];  // rotated elements half QD + i and HALF + half QD + i
      float mx = 0.0f;
#pragma unroll
      for (int i = 0; i < QD; i += 4) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, sn = a, cs = a;
        if (live) {
          const int d = half * QD + i;
          const float* qr = q + (size_t)tok * ldq + (kvh * group + head) * D + d;
          a = *reinterpret_cast<const float4*>(qr);
          b = *reinterpret_cast<const float4*>(qr + HALF);
          sn = *reinterpret_cast<const float4*>(sin_t + (size_t)tok * HALF + d);
          cs = *reinterpret_cast<const float4*>(cos_t + (size_t)tok * HALF + d);
        }
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w}, cv[4] = {cs.x, cs.y, cs.z, cs.w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          y[0][i + t] = av[t] * cv[t] - bv[t] * sv[t];
          y[1][i + t] = av[t] * sv[t] + bv[t] * cv[t];
          mx = fmaxf(mx, fmaxf(fabsf(y[0][i + t]), fabsf(y[1][i + t])));
        }
      }
      s_red[0][half][row] = mx;
      pair_sync();
      const int eq = pa_exponent(fmaxf(mx, s_red[0][half ^ 1][row]));
      pair_sync();
      const float f = pa_pow2(eq);
      q_scale = pa_pow2(-eq) * (1.0f / sqrtf((float)D));
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int c = 0; c < QD / 16; ++c) {
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) pa_split(y[u][c * 16 + 2 * t] * f, y[u][c * 16 + 2 * t + 1] * f, hi[t], lo[t]);
          const uint32_t col = lanes + L::kColQ + (uint32_t)((u * HALF + half * QD + c * 16) / 2);
          tmem_st8(col, hi);
          tmem_st8(col + D / 2, lo);
        }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_ready);
    }
    float o[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) o[i] = 0.0f;
    float m_run = -3.402823466e+38f, l_run = 0.0f, alpha_prev = 1.0f;
    auto take_pv = [&](int j) {  // o = o alpha_j + P_j V_j
      const float vs = s_scales[j].y * (1.0f / kPaPScale);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < HALF; c += 32) {
        uint32_t v[32];
        tmem_ld32(lanes + L::kColPV + (uint32_t)(half * HALF + c), v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[c + i] = fmaf(__uint_as_float(v[i]), vs, o[c + i] * alpha_prev);
      }
    };
    // A wait that ran out: no further waits, but all barriers and arrivals as usual (the other warps count on them); no output.
    bool ok = true;
    for (int j = 0; j < nt; ++j) {
      ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&s_full[j & 1], (uint32_t)(j >> 1) & 1u));
      tc_fence_after();
      uint32_t v[32];
      tmem_ld32(lanes + L::kColS + (uint32_t)((j & 1) * kPaKeys + half * 32), v);
      tmem_ld_wait();
      const float c = q_scale * s_scales[j].x;
      const int key0 = j * kPaKeys + half * 32;
      const bool diagonal = j * kPaKeys + kPaKeys - 1 > s0;  // some row of this CTA does not see all of the tile
      const int seen = diagonal ? tok - key0 + 1 : 32;       // columns [0, seen) of this thread's 32
      float mx = -3.402823466e+38f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float s = __uint_as_float(v[i]) * c;
        v[i] = __float_as_uint(s);
        if (!diagonal || i < seen) mx = fmaxf(mx, s);
      }
      s_red[j & 1][half][row] = mx;
      pair_sync();
      const float m_new = fmaxf(m_run, fmaxf(mx, s_red[j & 1][half ^ 1][row]));
      float sum = 0.0f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float p = expf(__uint_as_float(v[i]) - m_new);
        if (diagonal && i >= seen) p = 0.0f;
        sum += p;
        v[i] = __float_as_uint(p * kPaPScale);
      }
      const float alpha = expf(m_run - m_new);
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) pa_split(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]), hi[i], lo[i]);
      if (j > 0) {  // the tensor core is done with P and P.V of the tile before
        ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(pv_done, (uint32_t)(j - 1) & 1u));
        take_pv(j - 1);
      }
      tmem_st16(lanes + L::kColP + (uint32_t)(half * 16), hi);
      tmem_st16(lanes + L::kColP + (uint32_t)(kPaKeys / 2 + half * 16), lo);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      m_run = m_new;
      l_run = l_run * alpha + sum;
      alpha_prev = alpha;
    }
    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(pv_done, (uint32_t)(nt - 1) & 1u));
    take_pv(nt - 1);
    s_red[nt & 1][half][row] = l_run;
    pair_sync();
    if (ok && live) {
      const float inv = 1.0f / (l_run + s_red[nt & 1][half ^ 1][row]);
      float* dst = out + (size_t)tok * ldo + (kvh * group + head) * D + half * HALF;
#pragma unroll
      for (int i = 0; i < HALF; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

namespace {
constexpr size_t ps_smem_bytes(int head_dim) { return (size_t)2 * kPaKeys * (head_dim + 1) * sizeof(float); }
template <int D>
cudaError_t configure() {
  cudaError_t e = cudaFuncSetAttribute(prefill_kv_split_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ps_smem_bytes(D));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(attention_prefill_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, PaLayout<D>::kTotal);
}
template <int D>
cudaError_t launch(const float* q, const float* k, const float* v, int n, int q_heads, int kv_heads, const float* sin_t, const float* cos_t,
            int max_ctx, float* cache_k, float* cache_v, uint8_t* scratch, float* out, cudaStream_t s) {
  const int tiles = (n + kPaKeys - 1) / kPaKeys, group = q_heads / kv_heads, tokens = 128 / group;
  float2* scales = reinterpret_cast<float2*>(scratch);
  uint8_t* ops = scratch + (size_t)kPaMaxTiles * kv_heads * sizeof(float2);
  const cudaError_t e = launch_pdl(prefill_kv_split_kernel<D>, dim3(tiles, kv_heads), dim3(kPsThreads), ps_smem_bytes(D), s, k, v, kv_heads * D, n,
                                   sin_t, cos_t, max_ctx, cache_k, cache_v, ops, scales);
  if (e != cudaSuccess) return e;
  return launch_pdl(attention_prefill_tc_kernel<D>, dim3((n + tokens - 1) / tokens * kv_heads), dim3(kPaThreads), PaLayout<D>::kTotal, s, q,
                    q_heads * D, n, sin_t, cos_t, group, kv_heads, ops, scales, max_ctx, cache_k, cache_v, out, q_heads * D);
}
}  // namespace

// Operands of one layer's keys and values (the layers of a prompt use it one after the other), behind the tiles' scales.
size_t prefill_attention_scratch_bytes(int kv_heads, int head_dim, int max_ctx) {
  const size_t tiles = (size_t)(max_ctx + kPaKeys - 1) / kPaKeys;
  return (size_t)kPaMaxTiles * kv_heads * sizeof(float2) + tiles * kv_heads * (head_dim == 128 ? PaLayout<128>::kTileBytes : PaLayout<64>::kTileBytes);
}

cudaError_t prefill_attention_configure(int head_dim) { return head_dim == 128 ? configure<128>() : configure<64>(); }

// n tokens from position 0: keys and values into the cache, attention of all query heads into out [n, q_heads * head_dim].
cudaError_t launch_prefill_attention(const float* q, const float* k, const float* v, int n, int q_heads, int kv_heads, int head_dim,
                                     const float* sin_t, const float* cos_t, int max_ctx, float* cache_k, float* cache_v, uint8_t* scratch,
                                     float* out, cudaStream_t s) {
  return head_dim == 128
             ? launch<128>(q, k, v, n, q_heads, kv_heads, sin_t, cos_t, max_ctx, cache_k, cache_v, scratch, out, s)
             : launch<64>(q, k, v, n, q_heads, kv_heads, sin_t, cos_t, max_ctx, cache_k, cache_v, scratch, out, s);
}

}  // namespace mllmb200
