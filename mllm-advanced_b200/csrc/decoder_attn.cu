// Attention-side operators of the decoder (reference project paths):
//   RoPE, HF half-split form with precomputed tables   mllm/Backends/Arm/Kernels/rope.cpp:20-87
//   KV cache append                                    mllm/Backends/Arm/Ops/KVCacheOp.cpp:15-72
//   scores * 1/sqrt(D), causal mask, softmax, P.V      mllm/Models/ds_qwen2/modeling_ds_qwen2.hpp:127-150
//   lm_head product and greedy argmax                  modeling_ds_qwen2.hpp:209-212, mllm/Models/AutoLLM.hpp:70-105
// The reference expands grouped-query K/V heads when it writes the cache (each row stored `rep`
// times); here the cache holds each KV head once and the query heads of a group read the same rows,
// which is the same arithmetic.  fp32 KV cache, fp32 softmax with expf.
#include <cuda_fp16.h>

#include "device_common.cuh"
#include "decoder_attn_body.cuh"
#include "decoder_attn_rows.cuh"

namespace mllmb200 {

// sin/cos[pos, d] for d < D/2: theta = pos / base^(2d/D)   (rope.cpp:20-36; the upper half duplicates)
__global__ void rope_tables_kernel(float* __restrict__ sin_t, float* __restrict__ cos_t, int max_pos, int half_dim,
                                   float base) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= max_pos * half_dim) return;
  const int pos = idx / half_dim, d = idx % half_dim;
  float theta = 1.0f / powf(base, 2.0f * (float)d / (float)(2 * half_dim));
  theta *= (float)pos;
  sin_t[idx] = sinf(theta);
  cos_t[idx] = cosf(theta);
}

// grid (kv_heads, S), block D: rotate the new keys and append keys/values at positions pos0 + s.
// k_new/v_new: rows of ld floats holding [kv_heads * D]; cache: [kv_heads][max_ctx][D].
__global__ void rope_kv_append_kernel(const float* __restrict__ k_new, const float* __restrict__ v_new, int ld,
                                      const float* __restrict__ sin_t, const float* __restrict__ cos_t,
                                      const int* __restrict__ pos0_ptr, int max_ctx, float* __restrict__ cache_k,
                                      float* __restrict__ cache_v) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int h = blockIdx.x, s = blockIdx.y, d = threadIdx.x, D = blockDim.x, half = D >> 1;
  const int pos = *pos0_ptr + s;  // the position lives in device memory so that one CUDA graph serves every step
  if (pos >= max_ctx) return;
  const float* kr = k_new + (size_t)s * ld + h * D;
  const float* vr = v_new + (size_t)s * ld + h * D;
  const int dd = d < half ? d : d - half;
  const float sn = sin_t[pos * half + dd], cs = cos_t[pos * half + dd];
  const float x0 = kr[dd], x1 = kr[dd + half];
  const float y = d < half ? (x0 * cs - x1 * sn) : (x0 * sn + x1 * cs);
  cache_k[((size_t)h * max_ctx + pos) * D + d] = y;
  cache_v[((size_t)h * max_ctx + pos) * D + d] = vr[d];
}

// Prompt attention of decoder_attn_rows.cuh: grid (ceil(S / kPfRows), kv_heads).
#ifndef MLLMB200_PF_LONGEST_FIRST
#define MLLMB200_PF_LONGEST_FIRST 1
#endif
#ifndef MLLMB200_PF_HEAD_WARPS
#define MLLMB200_PF_HEAD_WARPS 4
#endif
constexpr int kPfHeadWarps = MLLMB200_PF_HEAD_WARPS;
constexpr int kPfThreads = kPfRowThreads<kPfHeadWarps>;

template <int D>
__global__ void __launch_bounds__(kPfThreads) attention_prefill_kernel(
    const float* __restrict__ q, int ldq, int S, const float* __restrict__ sin_t, const float* __restrict__ cos_t,
    const int* __restrict__ pos0_ptr, int max_ctx, int group, const float* __restrict__ cache_k,
    const float* __restrict__ cache_v, float* __restrict__ out, int ldo) {
  extern __shared__ __align__(16) uint8_t pf_smem[];
  pdl_launch_dependents();
  pdl_wait_prior();
  // CTAs are dispatched in order of blockIdx.x and a tile's work grows with its position (causal range): the last
  // tile goes first, so that the long ones start together and the short ones fill the SMs that free up
  const int tile = MLLMB200_PF_LONGEST_FIRST ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  prefill_attn_rows<D, kPfHeadWarps>(*reinterpret_cast<PrefillAttnSmem<D>*>(pf_smem), (int)threadIdx.x, [] { __syncthreads(); }, q, ldq,
                                     tile * kPfRows, S, (int)blockIdx.y, sin_t, cos_t, *pos0_ptr, max_ctx, group, cache_k, cache_v, out, ldo);
}

template __global__ void attention_prefill_kernel<64>(const float*, int, int, const float*, const float*, const int*, int, int,
                                                      const float*, const float*, float*, int);
template __global__ void attention_prefill_kernel<128>(const float*, int, int, const float*, const float*, const int*, int, int,
                                                       const float*, const float*, float*, int);
int attention_prefill_rows() { return kPfRows; }
int attention_prefill_threads() { return kPfThreads; }
size_t attention_prefill_smem_bytes(int head_dim) {
  return head_dim == 128 ? sizeof(PrefillAttnSmem<128>) : sizeof(PrefillAttnSmem<64>);
}

// Decode-step attention over context splits: the work of one CTA is attn_partial_body
// (decoder_attn_body.cuh); grid (splits, kv_heads), 256 threads.
template <int D>
__global__ void __launch_bounds__(kAttnThreads) attn_decode_partial_kernel(
    const float* __restrict__ q, const float* __restrict__ k_new, const float* __restrict__ v_new,
    const float* __restrict__ sin_t, const float* __restrict__ cos_t, const int* __restrict__ pos_ptr, int max_ctx,
    int chunk, int group, float* __restrict__ cache_k, float* __restrict__ cache_v, float* __restrict__ part_o,
    float* __restrict__ part_ml, int splits, int use_pdl) {
  __shared__ AttnSmem<D> sm;
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  const int pos = min(*pos_ptr, max_ctx - 1);
  const int split = blockIdx.x, kvh = blockIdx.y;
  if (split * chunk > pos) return;
  attn_partial_body<D>(sm, threadIdx.x, [] { __syncthreads(); }, q + (size_t)kvh * group * D, k_new + kvh * D,
                       v_new + kvh * D, sin_t + (size_t)pos * (D / 2), cos_t + (size_t)pos * (D / 2), pos, split * chunk, min((split + 1) * chunk, pos + 1), group,
                       cache_k + (size_t)kvh * max_ctx * D, cache_v + (size_t)kvh * max_ctx * D,
                       part_o + (size_t)kvh * group * splits * D, part_ml + (size_t)kvh * group * splits * 2, splits, split);
}

template __global__ void attn_decode_partial_kernel<64>(const float*, const float*, const float*, const float*, const float*,
                                                        const int*, int, int, int, float*, float*, float*, float*, int, int);
template __global__ void attn_decode_partial_kernel<128>(const float*, const float*, const float*, const float*,
                                                         const float*, const int*, int, int, int, float*, float*, float*,
                                                         float*, int, int);

// logits[v] = sum_k x[k] * W[v,k], W fp16 [V, hidden] row-major, x fp32 (one row), fp32 accumulation.
// One warp per output row, 16-byte loads; hidden a multiple of 8.  Each CTA also leaves the largest
// logit it produced and its index in best[blockIdx] (lowest index on ties), so that greedy sampling
// is a reduction over gridDim.x pairs instead of a pass over the vocabulary.
__global__ void __launch_bounds__(256) lm_head_f16_kernel(const float* __restrict__ x, const __half* __restrict__ w,
                                                          int hidden, int vocab, float* __restrict__ logits,
                                                          float2* __restrict__ best) {
  extern __shared__ float s_x[];
  __shared__ float s_bv[8];
  __shared__ int s_bi[8];
  for (int k = threadIdx.x; k < hidden; k += blockDim.x) s_x[k] = x[k];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  float bv = -3.402823466e+38f;
  int bi = 0x7fffffff;
  for (int v = blockIdx.x * wpb + warp; v < vocab; v += gridDim.x * wpb) {
    const uint4* row = reinterpret_cast<const uint4*>(w + (size_t)v * hidden);
    float acc = 0.0f;
    for (int c = lane; c < (hidden >> 3); c += 32) {
      const uint4 pk = row[c];
      const __half2* h2 = reinterpret_cast<const __half2*>(&pk);
      const float* xs = s_x + c * 8;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h2[j]);
        acc = fmaf(f.x, xs[2 * j], acc);
        acc = fmaf(f.y, xs[2 * j + 1], acc);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) logits[v] = acc;
    if (acc > bv) {  // rows come in increasing order within a warp, so a strict test keeps the lowest index
      bv = acc;
      bi = v;
    }
  }
  if (best == nullptr) return;
  if (lane == 0) {
    s_bv[warp] = bv;
    s_bi[warp] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < wpb; ++i)
      if (s_bv[i] > bv || (s_bv[i] == bv && s_bi[i] < bi)) {
        bv = s_bv[i];
        bi = s_bi[i];
      }
    best[blockIdx.x] = make_float2(bv, __int_as_float(bi));
  }
}

}  // namespace mllmb200
