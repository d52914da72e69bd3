// The decoder-layer operators around the W4A32 linears, for the Qwen2-1.5B / DeepSeek-Distill-Qwen
// forward (reference project: mllm/Models/ds_qwen2/modeling_ds_qwen2.hpp:47-54,106-155,175-215).
// Each op follows the reference's Arm operator named beside it.  Ops that feed a quantized linear
// also emit that linear's quantized activations (the records / blocks of act_quant.cu), so that in
// decode the linears launch without a separate quantization kernel in front of them.
#include "device_common.cuh"
#include "linear_blocks.h"

namespace mllmb200 {

// ---------------------------------------------------------------------------------------------
// (residual add +) RMSNorm (+ activation quantization), one CTA per row.
//   h_out = h_in (+ delta);  y = h_out * (w * rsqrt(mean(h_out^2) + eps))
// RMSNorm as in mllm/Backends/Arm/Ops/RMSNormOp.cpp:20-77 (fp32, no unit offset).
// y_out (fp32, may be null), records/hdr (may be null): 48-byte records of y as in act_quant.cu.
// The row lives in registers between the passes (hidden <= 8 * blockDim).
// ---------------------------------------------------------------------------------------------
constexpr int kNormThreads = 256;
constexpr int kNormMaxPerThread = 8;  // hidden <= 2048

__device__ __forceinline__ float block_sum(float v, float* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = lane < (blockDim.x >> 5) ? scratch[lane] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

__device__ __forceinline__ void block_minmax(float& mn, float& mx, float* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) {
    scratch[warp] = mn;
    scratch[32 + warp] = mx;
  }
  __syncthreads();
  mn = lane < nw ? scratch[lane] : 3.402823466e+38f;
  mx = lane < nw ? scratch[32 + lane] : -3.402823466e+38f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
}

// Writes the 48-byte records of one row whose values are produced by `value(k)`; every thread of the
// CTA must call it (the quad shuffles need full warps).  k_total a multiple of 8 is not required.
template <class F>
__device__ __forceinline__ void emit_records(F value, int k_total, int num_groups, const ActQuantParams& p,
                                             uint8_t* __restrict__ out) {
  const int num_items = num_groups * 4;
  for (int base = 0; base < num_items; base += blockDim.x) {
    const int item = base + threadIdx.x;
    const bool valid = item < num_items;
    const int k0 = item * 8;
    int q8[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) q8[j] = (valid && k0 + j < k_total) ? act_quant_value(value(k0 + j), p) : 0;
    const uint32_t lo = ((uint32_t)q8[0] & 0xFFu) | (((uint32_t)q8[2] & 0xFFu) << 8) | (((uint32_t)q8[4] & 0xFFu) << 16) |
                        (((uint32_t)q8[6] & 0xFFu) << 24);
    const uint32_t hi = ((uint32_t)q8[1] & 0xFFu) | (((uint32_t)q8[3] & 0xFFu) << 8) | (((uint32_t)q8[5] & 0xFFu) << 16) |
                        (((uint32_t)q8[7] & 0xFFu) << 24);
    int s = q8[0] + q8[1] + q8[2] + q8[3] + q8[4] + q8[5] + q8[6] + q8[7];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (valid) {
      const int g = item >> 2, i = item & 3;
      uint32_t* rec = reinterpret_cast<uint32_t*>(out + (size_t)g * kActRecordBytes);
      rec[i] = lo;
      rec[4 + i] = hi;
      if (i == 0) *reinterpret_cast<uint4*>(rec + 8) = make_uint4((uint32_t)(-8 * s), 0u, 0u, 0u);
    }
  }
}

__global__ void __launch_bounds__(kNormThreads) add_rmsnorm_quant_kernel(
    const float* __restrict__ h_in, const float* __restrict__ delta, const float* __restrict__ w, float eps, int hidden,
    float* __restrict__ h_out, float* __restrict__ y_out, uint8_t* __restrict__ records, float2* __restrict__ hdr,
    int use_pdl) {
  __shared__ float scratch[64];
  __shared__ float s_y[kNormThreads * kNormMaxPerThread];
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  const int m = blockIdx.x, tid = threadIdx.x;
  const float* hi = h_in + (size_t)m * hidden;
  float v[kNormMaxPerThread], wv[kNormMaxPerThread];
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int k = tid + i * kNormThreads;
    v[i] = 0.0f;
    wv[i] = k < hidden ? w[k] : 0.0f;  // requested with the row, used after the reduction
    if (k < hidden) {
      v[i] = hi[k] + (delta ? delta[(size_t)m * hidden + k] : 0.0f);
      if (h_out) h_out[(size_t)m * hidden + k] = v[i];
      ss += v[i] * v[i];
    }
  }
  const float rms = 1.0f / sqrtf(block_sum(ss, scratch) / (float)hidden + eps);
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int k = tid + i * kNormThreads;
    if (k < hidden) {
      const float y = v[i] * (wv[i] * rms);
      s_y[k] = y;
      if (y_out) y_out[(size_t)m * hidden + k] = y;
      mn = fminf(mn, y);
      mx = fmaxf(mx, y);
    }
  }
  if (records == nullptr) return;
  block_minmax(mn, mx, scratch);  // contains the __syncthreads that publishes s_y
  const ActQuantParams p = act_quant_params(mn, mx);
  if (tid == 0) hdr[m] = make_float2(p.recip_scale, __int_as_float(-p.nzp));
  const int num_groups = (hidden + kGroup - 1) / kGroup;
  emit_records([&](int k) { return s_y[k]; }, hidden, num_groups, p, records + (size_t)m * num_groups * kActRecordBytes);
}

// ---------------------------------------------------------------------------------------------
// SwiGLU activation: a = silu(gate) * up (mllm/Backends/Arm/Kernels/silu.cpp:19-55 with libm expf;
// the Arm kernel uses a fast sigmoid approximation, so only tolerance parity is meaningful there),
// optionally followed by the activation quantization for the down projection.  One CTA per row.
// ---------------------------------------------------------------------------------------------
constexpr int kSiluThreads = 512;
__global__ void __launch_bounds__(kSiluThreads) silu_mul_quant_kernel(const float* __restrict__ gate,
                                                                      const float* __restrict__ up, int inter,
                                                                      float* __restrict__ a_out,
                                                                      uint8_t* __restrict__ records,
                                                                      float2* __restrict__ hdr, int use_pdl) {
  extern __shared__ float s_a[];  // inter floats
  __shared__ float scratch[64];
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  const int m = blockIdx.x, tid = threadIdx.x;
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
  // eight gate/up pairs per thread are requested before the first is used: with one CTA per row the
  // kernel is a chain of memory round trips, not a bandwidth problem
  constexpr int kBatch = 8;
  for (int k0 = 0; k0 < inter; k0 += kSiluThreads * kBatch) {
    float g[kBatch], u[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int k = k0 + j * kSiluThreads + tid;
      g[j] = k < inter ? gate[(size_t)m * inter + k] : 0.0f;
      u[j] = k < inter ? up[(size_t)m * inter + k] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int k = k0 + j * kSiluThreads + tid;
      if (k < inter) {
        const float a = (g[j] / (1.0f + expf(-g[j]))) * u[j];
        s_a[k] = a;
        if (a_out) a_out[(size_t)m * inter + k] = a;
        mn = fminf(mn, a);
        mx = fmaxf(mx, a);
      }
    }
  }
  if (records == nullptr) return;
  block_minmax(mn, mx, scratch);
  const ActQuantParams p = act_quant_params(mn, mx);
  if (tid == 0) hdr[m] = make_float2(p.recip_scale, __int_as_float(-p.nzp));
  const int num_groups = (inter + kGroup - 1) / kGroup;
  emit_records([&](int k) { return s_a[k]; }, inter, num_groups, p, records + (size_t)m * num_groups * kActRecordBytes);
}

// ---------------------------------------------------------------------------------------------
// Merge of the context splits written by attn_decode_partial_kernel, followed by the activation
// quantization for the o projection.  One CTA, 512 threads, q_heads * D <= 2048.
//   w[h][s] = exp(m[h][s] - max_s m) / sum_s(l[h][s] * exp(m[h][s] - max_s m));  out[h][d] = sum_s w[h][s] * o[h][s][d]
// Dynamic shared memory: q_heads * splits floats.
// ---------------------------------------------------------------------------------------------
constexpr int kCombineThreads = 512;
__global__ void __launch_bounds__(kCombineThreads) attn_combine_quant_kernel(
    const float* __restrict__ part_o, const float* __restrict__ part_ml, const int* __restrict__ pos_ptr, int max_ctx,
    int chunk, int splits, int q_heads, int head_dim, float* __restrict__ attn_out, uint8_t* __restrict__ records,
    float2* __restrict__ hdr, int use_pdl) {
  extern __shared__ float s_w[];  // [q_heads][splits]
  __shared__ float scratch[64];
  __shared__ float s_y[kNormThreads * kNormMaxPerThread];
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pos = min(*pos_ptr, max_ctx - 1);
  const int nact = min(splits, pos / chunk + 1);
  for (int h = warp; h < q_heads; h += kCombineThreads / 32) {
    const float* ml = part_ml + (size_t)h * splits * 2;
    float mx = -3.402823466e+38f;
    for (int sidx = lane; sidx < nact; sidx += 32) mx = fmaxf(mx, ml[sidx * 2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float tot = 0.0f;
    for (int sidx = lane; sidx < nact; sidx += 32) {
      const float e = expf(ml[sidx * 2] - mx);
      s_w[h * splits + sidx] = e;
      tot += ml[sidx * 2 + 1] * e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const float inv = 1.0f / tot;
    for (int sidx = lane; sidx < nact; sidx += 32) s_w[h * splits + sidx] *= inv;  // same lane wrote it
  }
  __syncthreads();
  const int width = q_heads * head_dim;
  float mn = 3.402823466e+38f, mxv = -3.402823466e+38f;
  for (int idx = tid; idx < width; idx += kCombineThreads) {
    const int h = idx / head_dim, d = idx - h * head_dim;
    const float* po = part_o + (size_t)h * splits * head_dim + d;
    float acc = 0.0f;
    for (int s0 = 0; s0 < nact; s0 += 8) {  // eight partial rows requested together (no branch between the loads); summed in split order
      float pv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) pv[j] = po[(size_t)min(s0 + j, nact - 1) * head_dim];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc = fmaf(s0 + j < nact ? s_w[h * splits + s0 + j] : 0.0f, pv[j], acc);
    }
    s_y[idx] = acc;
    if (attn_out) attn_out[idx] = acc;
    mn = fminf(mn, acc);
    mxv = fmaxf(mxv, acc);
  }
  if (records == nullptr) return;
  block_minmax(mn, mxv, scratch);
  const ActQuantParams p = act_quant_params(mn, mxv);
  if (tid == 0) hdr[0] = make_float2(p.recip_scale, __int_as_float(-p.nzp));
  const int num_groups = (width + kGroup - 1) / kGroup;
  emit_records([&](int k) { return s_y[k]; }, width, num_groups, p, records);
}

// ---------------------------------------------------------------------------------------------
// The same two operators in front of a linear of several rows: their values go straight into the operand blocks that the linear reads
// (linear_blocks.h), the bits are those of the operator followed by the linear's own quantization.  One CTA per row of the
// padded blocks; a row's pieces of 16 bytes are half sectors, the neighbouring row's CTA writes the other half.
// Bound: the chain of loads, reductions and stores on short prompts, memory on documents: gate and up of 1900 tokens are 136 MB,
// which L2 is still writing back (50 us for 306 MB).  us, width 1536 and feed-forward 8960, from the end of the GEMM before to
// the last block, operator + quantization / here: silu, 1900 tokens 50 + 34.5 / 50, 512 10.2 + 9.5 / 15.7, 64 rows 4.3 + 3.4 / 5.9
// (one launch less); norm 13 + 6.5 / 18, 4.6 + 3.9 / 6.6, 3.6 + 2.1 / 4.7.
// ---------------------------------------------------------------------------------------------
// eight values of K (left of them exist) of row m
template <int FORM>
__device__ __forceinline__ void put_item(const W4Blocks& o, int num_groups, int m, int item, const float (&f)[8], int left,
                                         const ActQuantParams& p) {
  if (FORM == kW4Stream) {
    const int first = m / o.block_rows * o.block_rows, rows = min(o.block_rows, o.m_pad - first);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = i < left ? (uint32_t)act_quant_value(f[i], p) & 0xFFu : 0u;
      if (i & 1) hi |= q << (4 * (i - 1));
      else lo |= q << (4 * i);
    }
    uint8_t* at = o.blocks + ((size_t)num_groups * first + (size_t)(item >> 2) * rows) * 32 + (size_t)(m - first) * 16 + (item & 3) * 4;
    *reinterpret_cast<uint32_t*>(at) = lo;
    *reinterpret_cast<uint32_t*>(at + (size_t)rows * 16) = hi;
  } else {
    __align__(16) __half h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int q = j < left ? act_quant_value(f[j], p) - p.nzp : 0;
      h[(j < 4) ? 2 * j : 2 * (j - 4) + 1] = __int2half_rn(q);  // chunk order {0,4,1,5,2,6,3,7}
    }
    uint8_t* at = o.blocks + ((size_t)(item >> 2) * (o.m_pad >> 3) + (m >> 3)) * 512 + (m & 7) * 16 + (item & 3) * 128;
    *reinterpret_cast<uint4*>(at) = *reinterpret_cast<const uint4*>(h);
  }
}
// what the CTAs of either kernel do before and beside their row: the K-split counters, rows of padding
template <int FORM>
__device__ __forceinline__ bool blocks_row_is_padding(const W4Blocks& o, int num_groups, int m, int m_total) {
  if (m == 0)
    for (int i = threadIdx.x; i < o.clear_count; i += blockDim.x) o.clear[i] = 0;
  if (m < m_total) return false;
  const float zeros[8] = {};
  for (int item = threadIdx.x; item < num_groups * 4; item += blockDim.x) put_item<FORM>(o, num_groups, m, item, zeros, 0, ActQuantParams{});
  return true;
}

template <int FORM>
__global__ void __launch_bounds__(kNormThreads) add_rmsnorm_blocks_kernel(const float* __restrict__ h_in, const float* __restrict__ delta,
                                                                          const float* __restrict__ w, float eps, int hidden,
                                                                          float* __restrict__ h_out, int m_total, W4Blocks out, int use_pdl) {
  __shared__ float scratch[64];
  __shared__ __align__(16) float s_y[kNormThreads * kNormMaxPerThread];
  const int m = blockIdx.x, tid = threadIdx.x, num_groups = (hidden + kGroup - 1) / kGroup;
  float v[kNormMaxPerThread], wv[kNormMaxPerThread];
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int k = tid + i * kNormThreads;
    wv[i] = k < hidden ? w[k] : 0.0f;
  }
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  if (blocks_row_is_padding<FORM>(out, num_groups, m, m_total)) return;
  const float* hi = h_in + (size_t)m * hidden;
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int k = tid + i * kNormThreads;
    v[i] = 0.0f;
    if (k < hidden) {
      v[i] = hi[k] + (delta ? delta[(size_t)m * hidden + k] : 0.0f);
      if (h_out) h_out[(size_t)m * hidden + k] = v[i];
      ss += v[i] * v[i];
    }
  }
  const float rms = 1.0f / sqrtf(block_sum(ss, scratch) / (float)hidden + eps);
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int k = tid + i * kNormThreads;
    if (k < hidden) {
      const float y = v[i] * (wv[i] * rms);
      s_y[k] = y;
      mn = fminf(mn, y);
      mx = fmaxf(mx, y);
    }
  }
  block_minmax(mn, mx, scratch);  // contains the __syncthreads that publishes s_y
  const ActQuantParams p = act_quant_params(mn, mx);
  if (tid == 0) out.hdr[m] = make_float2(p.recip_scale, __int_as_float(-p.nzp));
  for (int item = tid; item < num_groups * 4; item += kNormThreads) {
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = item * 8 + j < hidden ? s_y[item * 8 + j] : 0.0f;
    put_item<FORM>(out, num_groups, m, item, f, hidden - item * 8, p);
  }
}

// A thread keeps its ITEMS items of 8 products in registers between the minimum / maximum and the blocks.  A row is one CTA, or a
// cluster of SPLIT that exchanges minima and maxima (the order of those does not matter: same bits): a row is 72 KB of gate and up and
// three items a thread at a width of 8960, and short prompts leave SMs idle.  us from the end of the GEMM before, width 8960, one CTA /
// four: 8 rows 6.4 / 4.8, 48 7.9 / 5.9, 128 8.4 / 6.0, 192 8.5 / 10.2 (no longer all at once); 4864: 24 rows 7.6 / 4.0, 128 7.7 / 6.4.
constexpr int kSiluBlockThreads = 384, kSiluSplit = 4, kSiluSplitRows = 128;
template <int FORM, int ITEMS, int SPLIT>
__global__ void __launch_bounds__(kSiluBlockThreads) silu_mul_blocks_kernel(const float* __restrict__ gate, const float* __restrict__ up,
                                                                            int inter, int m_total, W4Blocks out, int use_pdl) {
  static_assert(SPLIT == 1 || (ITEMS == 1 && SPLIT * kSiluBlockThreads / 32 <= 64), "");
  __shared__ float scratch[64], s_mn[64], s_mx[64];
  const int num_groups = (inter + kGroup - 1) / kGroup, m = blockIdx.x / SPLIT, rank = SPLIT > 1 ? cluster_ctarank() : 0;
  const int tid = rank * blockDim.x + threadIdx.x;  // of the row's
  if (SPLIT > 1) cluster_arrive_relaxed();          // (every CTA of the cluster runs when the peers write into it)
  if (use_pdl) {
    pdl_launch_dependents();
    pdl_wait_prior();
  }
  if (SPLIT > 1) cluster_wait();
  if (blocks_row_is_padding<FORM>(out, num_groups, m, m_total)) return;
  const float *g_row = gate + (size_t)m * inter, *u_row = up + (size_t)m * inter;
  const bool vec = (inter & 3) == 0;  // (the rows start on 16 bytes)
  float a[ITEMS][8], u[ITEMS][8];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int k0 = (tid + i * kSiluBlockThreads) * 8;
    if (vec && k0 + 8 <= inter) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 x = __ldcs(reinterpret_cast<const float4*>(g_row + k0) + h), y = __ldcs(reinterpret_cast<const float4*>(u_row + k0) + h);
        a[i][4 * h] = x.x, a[i][4 * h + 1] = x.y, a[i][4 * h + 2] = x.z, a[i][4 * h + 3] = x.w;
        u[i][4 * h] = y.x, u[i][4 * h + 1] = y.y, u[i][4 * h + 2] = y.z, u[i][4 * h + 3] = y.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a[i][j] = k0 + j < inter ? g_row[k0 + j] : 0.0f;
        u[i][j] = k0 + j < inter ? u_row[k0 + j] : 0.0f;
      }
    }
  }
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a[i][j] = (a[i][j] / (1.0f + expf(-a[i][j]))) * u[i][j];
      if ((tid + i * kSiluBlockThreads) * 8 + j < inter) {
        mn = fminf(mn, a[i][j]);
        mx = fmaxf(mx, a[i][j]);
      }
    }
  if (SPLIT == 1) {
    block_minmax(mn, mx, scratch);
  } else {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, all = SPLIT * nw;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane < SPLIT) {  // each warp to every CTA of the row
      st_cluster_f32(map_to_cta(s_mn + rank * nw + (threadIdx.x >> 5), lane), mn);
      st_cluster_f32(map_to_cta(s_mx + rank * nw + (threadIdx.x >> 5), lane), mx);
    }
    cluster_sync_all();
    for (int i = lane; i < all; i += 32) {
      mn = fminf(mn, s_mn[i]);
      mx = fmaxf(mx, s_mx[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
  }
  const ActQuantParams p = act_quant_params(mn, mx);
  if (tid == 0) out.hdr[m] = make_float2(p.recip_scale, __int_as_float(-p.nzp));
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int item = tid + i * kSiluBlockThreads;
    if (item < num_groups * 4) put_item<FORM>(out, num_groups, m, item, a[i], inter - item * 8, p);
  }
}

template <class K, class... A>
static cudaError_t launch_blocks_op(K kernel, int rows, int split, int threads, int use_pdl, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * split), 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (split > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)split;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (use_pdl) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, args..., use_pdl);
}
cudaError_t launch_add_rmsnorm_blocks(const float* h_in, const float* delta, const float* w, float eps, int hidden, float* h_out, int m,
                                      const W4Blocks& out, int use_pdl, cudaStream_t s) {
  return out.form == kW4Stream
             ? launch_blocks_op(add_rmsnorm_blocks_kernel<kW4Stream>, out.m_pad, 1, kNormThreads, use_pdl, s, h_in, delta, w, eps, hidden, h_out, m, out)
             : launch_blocks_op(add_rmsnorm_blocks_kernel<kW4Tile>, out.m_pad, 1, kNormThreads, use_pdl, s, h_in, delta, w, eps, hidden, h_out, m, out);
}
template <int FORM>
static cudaError_t launch_silu_form(const float* gate, const float* up, int inter, int m, const W4Blocks& out, int use_pdl, cudaStream_t s) {
  const int items = ((inter + kGroup - 1) / kGroup) * 4;
  if (out.m_pad <= kSiluSplitRows && items > kSiluBlockThreads && items <= kSiluSplit * kSiluBlockThreads)
    return launch_blocks_op(silu_mul_blocks_kernel<FORM, 1, kSiluSplit>, out.m_pad, kSiluSplit, (items + 32 * kSiluSplit - 1) / (32 * kSiluSplit) * 32,
                            use_pdl, s, gate, up, inter, m, out);
  switch ((inter + 8 * kSiluBlockThreads - 1) / (8 * kSiluBlockThreads)) {
    case 1: return launch_blocks_op(silu_mul_blocks_kernel<FORM, 1, 1>, out.m_pad, 1, kSiluBlockThreads, use_pdl, s, gate, up, inter, m, out);
    case 2: return launch_blocks_op(silu_mul_blocks_kernel<FORM, 2, 1>, out.m_pad, 1, kSiluBlockThreads, use_pdl, s, gate, up, inter, m, out);
    case 3: return launch_blocks_op(silu_mul_blocks_kernel<FORM, 3, 1>, out.m_pad, 1, kSiluBlockThreads, use_pdl, s, gate, up, inter, m, out);
    case 4: return launch_blocks_op(silu_mul_blocks_kernel<FORM, 4, 1>, out.m_pad, 1, kSiluBlockThreads, use_pdl, s, gate, up, inter, m, out);
    default: return cudaErrorInvalidValue;  // (the decoder takes widths up to 12000)
  }
}
cudaError_t launch_silu_mul_blocks(const float* gate, const float* up, int inter, int m, const W4Blocks& out, int use_pdl, cudaStream_t s) {
  return out.form == kW4Stream ? launch_silu_form<kW4Stream>(gate, up, inter, m, out, use_pdl, s)
                               : launch_silu_form<kW4Tile>(gate, up, inter, m, out, use_pdl, s);
}

// Embedding lookup: row gather (mllm/Backends/Arm/Ops/LLMEmbeddingTokenOp.cpp:23-52).
__global__ void embedding_kernel(const int* __restrict__ ids, const float* __restrict__ table, int hidden,
                                 float* __restrict__ out) {
  const int m = blockIdx.x;
  const float* src = table + (size_t)ids[m] * hidden;
  for (int k = threadIdx.x; k < hidden; k += blockDim.x) out[(size_t)m * hidden + k] = src[k];
}

}  // namespace mllmb200
