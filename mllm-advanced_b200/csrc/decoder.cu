// Qwen2-architecture decoder (DeepSeek-Distill-Qwen-1.5B, Qwen2VL-2B language tower) on top of the
// W4A32 linears: host-side orchestration behind a C ABI (include/mllmb200.h, "decoder" section).
// Mirrors the forward of the reference project's model, mllm/Models/ds_qwen2/modeling_ds_qwen2.hpp:
// 106-155 (attention), :47-54 (MLP), :175-183 (decoder layer), :202-215 (model), and its greedy
// loop mllm/Models/AutoLLM.hpp:39-65.  Batch 1, fp32 activations and KV cache, fp16 lm_head.
//
// Decode runs as ONE CUDA graph per token, replayed: the position and the current token live in
// device memory, so nothing changes between replays.  In decode every op that feeds a quantized
// linear also writes that linear's int8 activation records, so a layer is 9 launches:
//   add+rmsnorm+quant, gemv(q,k,v), attention over context splits (rotates, appends K/V),
//   merge of the splits + quant, gemv(o), add+rmsnorm+quant,
//   gemv(gate,up), silu*up+quant, gemv(down)      (the residual add of `down` is fused into the next norm)
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <vector>

#include "../../include/mllmb200.h"
#include "decoder_state.h"
#include "device_common.cuh"
#include "linear_blocks.h"

namespace mllmb200 {
// persistent decode kernel (decoder_persistent.cu)
void persistent_prepare(Decoder* d);
bool persistent_usable(Decoder* d);
cudaError_t persistent_decode(Decoder* d, int steps);
void persistent_destroy(Decoder* d);
int persistent_phase_cycles(Decoder* d, long long* out, int capacity, int* nctas, int* stamps);
// kernels defined in the other translation units
__global__ void add_rmsnorm_quant_kernel(const float*, const float*, const float*, float, int, float*, float*, uint8_t*,
                                         float2*, int);
__global__ void silu_mul_quant_kernel(const float*, const float*, int, float*, uint8_t*, float2*, int);
cudaError_t launch_add_rmsnorm_blocks(const float*, const float*, const float*, float, int, float*, int, const W4Blocks&, int, cudaStream_t);
cudaError_t launch_silu_mul_blocks(const float*, const float*, int, int, const W4Blocks&, int, cudaStream_t);
__global__ void embedding_kernel(const int*, const float*, int, float*);
__global__ void rope_tables_kernel(float*, float*, int, int, float);
template <int D>
__global__ void attn_decode_partial_kernel(const float*, const float*, const float*, const float*, const float*, const int*,
                                           int, int, int, float*, float*, float*, float*, int, int);
__global__ void attn_combine_quant_kernel(const float*, const float*, const int*, int, int, int, int, int, float*, uint8_t*,
                                          float2*, int);
__global__ void rope_kv_append_kernel(const float*, const float*, int, const float*, const float*, const int*, int,
                                      float*, float*);
template <int D>
__global__ void attention_prefill_kernel(const float*, int, int, const float*, const float*, const int*, int, int, const float*,
                                         const float*, float*, int);
size_t attention_prefill_smem_bytes(int head_dim);
int attention_prefill_rows();
int attention_prefill_threads();
// Prompts up to here keep the fp32 attention on the CUDA cores (decoder_attn_rows.cuh).  Its time grows by blocks of 32
// positions, the tensor-core kernels' by tiles of 64 from a chain of set-up, splitting and tile latencies.  A layer's two
// kernels, fp32 / tensor cores, us: 12 heads of 128 at 64 tokens 15 / 18, 96 20 / 20, 97 24 / 20, 512 87 / 31; 14 heads of 64
// at 96 13 / 14, 97 16 / 14, 512 54 / 24; 16 heads of 128 on 4 at 96 18 / 20, 97 22 / 20.
constexpr int kShortPrompt = 96;
size_t prefill_attention_scratch_bytes(int kv_heads, int head_dim, int max_ctx);
cudaError_t prefill_attention_configure(int head_dim);
cudaError_t launch_prefill_attention(const float*, const float*, const float*, int, int, int, int, const float*, const float*, int, float*,
                                     float*, uint8_t*, float*, cudaStream_t);
__global__ void lm_head_f16_kernel(const float*, const __half*, int, int, float*, float2*);
__global__ void sample_advance_kernel(const float2*, int, int*, int*, int*, int*, int);
__global__ void act_quant_records_kernel(const float*, int, int, int, uint8_t*, float2*, int, int);
cudaError_t launch_w4a32_gemv_grouped(const uint8_t*, const float2*, int, int, int, const void* const*, float* const*,
                                      const int*, const int*, int, cudaStream_t);
cudaError_t launch_act_quant_records(const float*, int, int, int, uint8_t*, float2*, int, int, cudaStream_t);
int record_cuda_failure(cudaError_t e);  // c_api.cu

__global__ void set_int_kernel(int* dst, int v) { *dst = v; }

namespace {

#define DEC_CHECK(expr)                     \
  do {                                      \
    cudaError_t e__ = (expr);               \
    if (e__ != cudaSuccess) {               \
      d->last_error = (int)e__;             \
      return MLLMB200_CUDA_ERROR;           \
    }                                       \
  } while (0)
#define DEC_ST(expr)                        \
  do {                                      \
    int s__ = (expr);                       \
    if (s__ != MLLMB200_OK) return s__;     \
  } while (0)

int gemv_group(Decoder* d, const uint8_t* rec, const float2* hdr, int k, int count, const int* which, float* const* outs,
               const Layer& L) {
  const void* tiled[4];
  int n[4], ldy[4];
  const auto& c = d->cfg;
  for (int i = 0; i < count; ++i) {
    tiled[i] = L.w[which[i]];
    switch (which[i]) {
      case kQ: case kO: n[i] = (which[i] == kQ) ? c.q_heads * c.head_dim : c.hidden; break;
      case kK: case kV: n[i] = c.kv_heads * c.head_dim; break;
      case kGate: case kUp: n[i] = c.inter; break;
      default: n[i] = c.hidden; break;
    }
    ldy[i] = n[i];
  }
  DEC_CHECK(launch_w4a32_gemv_grouped(rec, hdr, 1, k, count, tiled, outs, n, ldy, 1, d->stream));
  return MLLMB200_OK;
}

// One decode step at the position / token held in device memory.
int enqueue_decode_step(Decoder* d) {
  const auto& c = d->cfg;
  cudaStream_t s = d->stream;
  const int H = c.hidden, QD = c.q_heads * c.head_dim, I = c.inter;
  embedding_kernel<<<1, 256, 0, s>>>(d->token, d->embedding, H, d->h);
  for (int l = 0; l < c.layers; ++l) {
    const Layer& L = d->layers[l];
    DEC_CHECK(launch_pdl(add_rmsnorm_quant_kernel, dim3(1), dim3(256), 0, s, d->h, l == 0 ? nullptr : d->down, L.ln1,
                         c.eps, H, d->h, nullptr, d->rec_a, d->hdr_a, 1));
    {
      const int which[3] = {kQ, kK, kV};
      float* outs[3] = {d->q, d->k, d->v};
      DEC_ST(gemv_group(d, d->rec_a, d->hdr_a, H, 3, which, outs, L));
    }
    {
      const dim3 grid(d->attn_splits, c.kv_heads);
      const int group = c.q_heads / c.kv_heads;
      if (c.head_dim == 128)
        DEC_CHECK(launch_pdl(attn_decode_partial_kernel<128>, grid, dim3(256), 0, s, d->q, d->k, d->v, d->sin_t, d->cos_t,
                             d->pos, c.max_ctx, d->attn_chunk, group, L.cache_k, L.cache_v, d->part_o, d->part_ml,
                             d->attn_splits, 1));
      else
        DEC_CHECK(launch_pdl(attn_decode_partial_kernel<64>, grid, dim3(256), 0, s, d->q, d->k, d->v, d->sin_t, d->cos_t,
                             d->pos, c.max_ctx, d->attn_chunk, group, L.cache_k, L.cache_v, d->part_o, d->part_ml,
                             d->attn_splits, 1));
      DEC_CHECK(launch_pdl(attn_combine_quant_kernel, dim3(1), dim3(512), (size_t)c.q_heads * d->attn_splits * sizeof(float),
                           s, d->part_o, d->part_ml, d->pos, c.max_ctx, d->attn_chunk, d->attn_splits, c.q_heads, c.head_dim,
                           nullptr, d->rec_a, d->hdr_a, 1));
    }
    {
      const int which[1] = {kO};
      float* outs[1] = {d->o};
      DEC_ST(gemv_group(d, d->rec_a, d->hdr_a, QD, 1, which, outs, L));
    }
    DEC_CHECK(launch_pdl(add_rmsnorm_quant_kernel, dim3(1), dim3(256), 0, s, d->h, d->o, L.ln2, c.eps, H, d->h, nullptr,
                         d->rec_a, d->hdr_a, 1));
    {
      const int which[2] = {kGate, kUp};
      float* outs[2] = {d->gate, d->up};
      DEC_ST(gemv_group(d, d->rec_a, d->hdr_a, H, 2, which, outs, L));
    }
    DEC_CHECK(launch_pdl(silu_mul_quant_kernel, dim3(1), dim3(512), (size_t)I * sizeof(float), s, d->gate, d->up, I,
                         nullptr, d->rec_b, d->hdr_b, 1));
    {
      const int which[1] = {kDown};
      float* outs[1] = {d->down};
      DEC_ST(gemv_group(d, d->rec_b, d->hdr_b, I, 1, which, outs, L));
    }
  }
  DEC_CHECK(launch_pdl(add_rmsnorm_quant_kernel, dim3(1), dim3(256), 0, s, d->h, d->down, d->final_norm, c.eps, H, d->h,
                       d->xn, nullptr, nullptr, 1));
  lm_head_f16_kernel<<<kHeadCtas, 256, H * sizeof(float), s>>>(d->xn, d->lm_head, H, c.vocab, d->logits, d->best);
  sample_advance_kernel<<<1, 32, 0, s>>>(d->best, kHeadCtas, d->pos, d->token, d->next, d->history, c.max_ctx);
  DEC_CHECK(cudaGetLastError());
  return MLLMB200_OK;
}

}  // namespace

int check_ready(Decoder* d) {
  if (!d->embedding || !d->lm_head) return MLLMB200_INVALID_ARG;
  for (auto& L : d->layers)
    for (int i = 0; i < kNumLinears; ++i)
      if (!L.w[i]) return MLLMB200_INVALID_ARG;
  return MLLMB200_OK;
}

static cudaError_t prompt_attention_configure(int head_dim) {
  const cudaError_t e = head_dim == 128 ? cudaFuncSetAttribute(attention_prefill_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                               (int)attention_prefill_smem_bytes(128))
                                        : cudaFuncSetAttribute(attention_prefill_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                               (int)attention_prefill_smem_bytes(64));
  return e == cudaSuccess ? prefill_attention_configure(head_dim) : e;
}
// A layer's attention over a prompt of n tokens from position 0 (*zero): rotated keys and values into the cache, the
// attention's rows into out.  tensor_cores: decoder_attn_prefill.cu, else fp32 on the CUDA cores.
static cudaError_t prompt_attention(bool tensor_cores, const float* q, const float* k, const float* v, int n, int q_heads, int kv_heads,
                                    int head_dim, const float* sin_t, const float* cos_t, const int* zero, int max_ctx, float* cache_k,
                                    float* cache_v, uint8_t* scratch, float* out, cudaStream_t s) {
  if (tensor_cores)
    return launch_prefill_attention(q, k, v, n, q_heads, kv_heads, head_dim, sin_t, cos_t, max_ctx, cache_k, cache_v, scratch, out, s);
  const int QD = q_heads * head_dim, group = q_heads / kv_heads;
  const cudaError_t e = launch_pdl(rope_kv_append_kernel, dim3(kv_heads, n), dim3(head_dim), 0, s, k, v, kv_heads * head_dim, sin_t, cos_t,
                                   zero, max_ctx, cache_k, cache_v);
  if (e != cudaSuccess) return e;
  const int rows = attention_prefill_rows();  // query rows per CTA
  const dim3 grid((n + rows - 1) / rows, kv_heads), block(attention_prefill_threads());
  const size_t smem = attention_prefill_smem_bytes(head_dim);
  return head_dim == 128 ? launch_pdl(attention_prefill_kernel<128>, grid, block, smem, s, q, QD, n, sin_t, cos_t, zero, max_ctx, group,
                                      cache_k, cache_v, out, QD)
                         : launch_pdl(attention_prefill_kernel<64>, grid, block, smem, s, q, QD, n, sin_t, cos_t, zero, max_ctx, group,
                                      cache_k, cache_v, out, QD);
}

// h += delta, and the linears of the normalized rows of a prompt
static int norm_linears(Decoder* d, const float* delta, const float* w, int n, int count, const void* const* tiled, float* const* y,
                        const int* rows) {
  const auto& c = d->cfg;
  const W4Blocks b = w4a32_blocks_for(n, c.hidden, count, rows, 5, d->ws);
  if (b.form == kW4None) {
    DEC_CHECK(launch_pdl(add_rmsnorm_quant_kernel, dim3(n), dim3(256), 0, d->stream, d->h, delta, w, c.eps, c.hidden, d->h, d->xn, nullptr, nullptr, 1));
    return mllmb200_w4a32_linear_forward_grouped(d->xn, n, c.hidden, c.hidden, count, tiled, y, rows, rows, d->ws, 5 | 0x100, d->stream);
  }
  DEC_CHECK(launch_add_rmsnorm_blocks(d->h, delta, w, c.eps, c.hidden, d->h, n, b, 1, d->stream));
  DEC_CHECK(w4a32_forward_blocks(b, n, c.hidden, count, tiled, y, rows, rows, 1, d->stream));
  return MLLMB200_OK;
}

// The prompt pass of the batch-1 decoder, writing keys / values into the given per-layer caches
// ([kv_heads][max_ctx][D] each) and the sampled token and position into the given words: the decoder's own for
// mllmb200_qwen2_prefill, a sequence's for the batched decoder (decoder_batch.cu).  Exactly one of tokens_dev
// (int32 [n]) and embeds_dev (fp32 [n, hidden], rows that are already embeddings) is given.
int prefill_into(Decoder* d, const int* tokens_dev, const float* embeds_dev, int n, float* const* cache_k,
                 float* const* cache_v, int* pos, int* token, int* next, int* history) {
  if (!d || (tokens_dev == nullptr) == (embeds_dev == nullptr) || n <= 0 || n >= d->cfg.max_ctx) return MLLMB200_INVALID_ARG;
  DEC_ST(check_ready(d));
  const auto& c = d->cfg;
  cudaStream_t s = d->stream;
  const int H = c.hidden, QD = c.q_heads * c.head_dim, KD = c.kv_heads * c.head_dim, I = c.inter;
  if (tokens_dev)
    embedding_kernel<<<n, 256, 0, s>>>(tokens_dev, d->embedding, H, d->h);
  else
    DEC_CHECK(cudaMemcpyAsync(d->h, embeds_dev, (size_t)n * H * sizeof(float), cudaMemcpyDeviceToDevice, s));
  for (int l = 0; l < c.layers; ++l) {
    const Layer& L = d->layers[l];
    {  // q, k, v share one quantization of the normalized rows
      const void* tw[3] = {L.w[kQ], L.w[kK], L.w[kV]};
      float* ty[3] = {d->q, d->k, d->v};
      const int tn[3] = {QD, KD, KD};
      DEC_ST(norm_linears(d, l == 0 ? nullptr : d->down, L.ln1, n, 3, tw, ty, tn));
    }
    DEC_CHECK(prompt_attention(n > kShortPrompt, d->q, d->k, d->v, n, c.q_heads, c.kv_heads, c.head_dim, d->sin_t, d->cos_t, d->zero, c.max_ctx,
                               cache_k[l], cache_v[l], d->kv_split, d->attn, s));
    DEC_ST(mllmb200_w4a32_linear_forward_ex(d->attn, L.w[kO], d->o, d->ws, n, QD, H, QD, H, 5 | 0x100 | L.flags[kO], s));
    {  // gate and up likewise
      const void* tw[2] = {L.w[kGate], L.w[kUp]};
      float* ty[2] = {d->gate, d->up};
      const int tn[2] = {I, I};
      DEC_ST(norm_linears(d, d->o, L.ln2, n, 2, tw, ty, tn));
    }
    const W4Blocks act = w4a32_blocks_for(n, I, 1, &H, 5 | L.flags[kDown], d->ws);
    if (act.form != kW4None) {
      const void* tw[1] = {L.w[kDown]};
      DEC_CHECK(launch_silu_mul_blocks(d->gate, d->up, I, n, act, 1, s));
      DEC_CHECK(w4a32_forward_blocks(act, n, I, 1, tw, &d->down, &H, &H, 1, s));
    } else {
      DEC_CHECK(launch_pdl(silu_mul_quant_kernel, dim3(n), dim3(512), (size_t)I * sizeof(float), s, d->gate, d->up, I, d->act, nullptr,
                           nullptr, 1));
      DEC_ST(mllmb200_w4a32_linear_forward_ex(d->act, L.w[kDown], d->down, d->ws, n, I, H, I, H, 5 | 0x100 | L.flags[kDown], s));
    }
  }
  // only the last position feeds the sampler (the reference computes all rows and reads the last)
  const size_t last = (size_t)(n - 1) * H;
  add_rmsnorm_quant_kernel<<<1, 256, 0, s>>>(d->h + last, d->down + last, d->final_norm, c.eps, H, nullptr, d->xn, nullptr,
                                             nullptr, 0);
  lm_head_f16_kernel<<<kHeadCtas, 256, H * sizeof(float), s>>>(d->xn, d->lm_head, H, c.vocab, d->logits, d->best);
  set_int_kernel<<<1, 1, 0, s>>>(pos, n - 1);
  sample_advance_kernel<<<1, 32, 0, s>>>(d->best, kHeadCtas, pos, token, next, history, c.max_ctx);
  DEC_CHECK(cudaGetLastError());
  return MLLMB200_OK;
}

}  // namespace mllmb200

#include "decoder_api.inc"
