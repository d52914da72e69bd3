// Body of the decoder's fp32 prompt attention: attention_prefill_kernel (decoder_attn.cu), and the rows of the tensor-core
// kernel (decoder_attn_prefill.cu) whose keys or values are not fit for its operands.
//
// Prompt attention, fp32 on the CUDA cores, one tile of rows: R * W warps (R = kPfRows = 4 query rows, W = HEAD_WARPS
// warps per row).  The warps own R consecutive query rows of all `group` query heads that share one KV head (R * group
// <= 32 query vectors, rotated into shared memory once) and walks the cache in blocks of 32 positions up to the causal
// limit: a key/value block is read from L2 once per tile (not once per head and row), scores are formed with lane = key
// position (key rows padded to D + 1 floats: no bank conflicts), and the running softmax (max, sum, rescale) is the
// usual online form.  A block is a chain of dependent steps (stage, barrier, scores, softmax, barrier, P.V, barrier)
// whose length - not the SM's throughput - set the run time: with 8 rows and one warp per row the launch took as long as
// the tile with the longest causal range (16 blocks of ~8 us on a 512-token prompt: 134 us per layer, SMs busy half of
// the time).  Now each warp takes the heads w / R, w / R + W, .. of its row (a shorter chain per block), a tile has 4
// rows (more CTAs than SMs), and the tiles are dispatched longest first: 512-token prefill of the 1.5B model 8.3 -> 7.1 ms.
// Arithmetic: scores * 1/sqrt(D), causal mask, softmax, P.V (modeling_ds_qwen2.hpp:127-150 of the reference project).
// q: rows of ldq floats, row s at position pos0 + s; out: rows of ldo floats.
#pragma once
#include "decoder_attn_body.cuh"

namespace mllmb200 {

#ifndef MLLMB200_PF_ROWS
#define MLLMB200_PF_ROWS 4
#endif
constexpr int kPfRows = MLLMB200_PF_ROWS;  // query rows per tile
constexpr int kPfKeys = 32;                // cache positions per block
// head warps: warp w owns row w % rows and the heads w / rows, w / rows + head warps, ..
template <int HEAD_WARPS>
constexpr int kPfRowThreads = kPfRows * HEAD_WARPS * 32;

template <int D>
struct PrefillAttnSmem {
  float q[kPfRows * kAttnMaxGroup][D];
  float k[kPfKeys][D + 1];
  float v[kPfKeys][D];
  float p[kPfRows * kAttnMaxGroup][kPfKeys];
  float alpha[kPfRows * kAttnMaxGroup], lsum[kPfRows * kAttnMaxGroup];
};

// Rows s0 .. min(s0 + kPfRows, S) - 1 at positions pos0 + s0 .., called by kPfRowThreads<HEAD_WARPS> threads;
// sync() is their barrier.
template <int D, int HEAD_WARPS, class Sync>
__device__ __forceinline__ void prefill_attn_rows(PrefillAttnSmem<D>& sm, int tid, Sync sync, const float* __restrict__ q, int ldq, int s0,
                                                  int S, int kvh, const float* __restrict__ sin_t, const float* __restrict__ cos_t,
                                                  int pos0, int max_ctx, int group, const float* __restrict__ cache_k,
                                                  const float* __restrict__ cache_v, float* __restrict__ out, int ldo) {
  constexpr int kThreads = kPfRowThreads<HEAD_WARPS>, kHeadsPerWarp = (kAttnMaxGroup + HEAD_WARPS - 1) / HEAD_WARPS;
  constexpr int HALF = D / 2, NG = kThreads / (D / 4), QPT = (kPfRows * kAttnMaxGroup + NG - 1) / NG;
  const int warp = tid >> 5, lane = tid & 31;
  const int nrows = min(kPfRows, S - s0);
  const int nq = group * kPfRows;  // query vectors: index = h * kPfRows + r
  // rotated queries (rows past S stay zero)
  for (int idx = tid; idx < nq * D; idx += kThreads) {
    const int qi = idx / D, d = idx - qi * D;
    const int h = qi / kPfRows, r = qi - h * kPfRows;
    float val = 0.0f;
    if (r < nrows) {
      const int pos = min(pos0 + s0 + r, max_ctx - 1);
      const float* qr = q + (size_t)(s0 + r) * ldq + (kvh * group + h) * D;
      const int dd = d < HALF ? d : d - HALF;
      const float sn = sin_t[pos * HALF + dd], cs = cos_t[pos * HALF + dd];
      const float x0 = qr[dd], x1 = qr[dd + HALF];
      val = d < HALF ? (x0 * cs - x1 * sn) : (x0 * sn + x1 * cs);
    }
    sm.q[qi][d] = val;
  }
  const float scale = 1.0f / sqrtf((float)D);
  const float* kbase = cache_k + (size_t)kvh * max_ctx * D;
  const float* vbase = cache_v + (size_t)kvh * max_ctx * D;
  const int last_pos = min(pos0 + s0 + nrows - 1, max_ctx - 1);  // causal limit of the tile
  // running state: warp w owns query vectors w, w + 8, ... (lane-uniform copies of max and sum)
  float m_run[kHeadsPerWarp], l_run[kHeadsPerWarp];
#pragma unroll
  for (int i = 0; i < kHeadsPerWarp; ++i) m_run[i] = -3.402823466e+38f, l_run[i] = 0.0f;
  const int wr = warp % kPfRows, wh = warp / kPfRows;  // this warp's query row and first head
  // output accumulators: thread (pc, pg) holds elements 4 pc .. 4 pc + 3 of query vectors pg, pg + NG, ...
  // (a 4-wide register tile: one 16-byte value load and one 16-byte probability load feed 16 FMAs -
  // the kernel is bound by shared-memory wavefronts, not by FMAs)
  const int pc = tid % (D / 4), pg = tid / (D / 4);
  float o_acc[QPT][4];
#pragma unroll
  for (int i = 0; i < QPT; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.0f;

  // A block's key/value rows are requested into registers one block ahead (L2 round trips of ~1k
  // cycles each otherwise sit between the blocks): thread t moves chunks t, t + 256, ... of the block.
  constexpr int kLd = kPfKeys * (D / 4) / kThreads;  // 16-byte chunks per thread and matrix
  float4 kreg[kLd], vreg[kLd];
  auto fetch = [&](int b0) {
    const int nk = min(kPfKeys, last_pos + 1 - b0);
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int idx = tid + u * kThreads;
      const int j = idx / (D / 4), c = idx - j * (D / 4);
      kreg[u] = vreg[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < nk) {
        kreg[u] = *reinterpret_cast<const float4*>(kbase + (size_t)(b0 + j) * D + c * 4);
        vreg[u] = *reinterpret_cast<const float4*>(vbase + (size_t)(b0 + j) * D + c * 4);
      }
    }
  };
  fetch(0);
  for (int b0 = 0; b0 <= last_pos; b0 += kPfKeys) {
    const int nk = min(kPfKeys, last_pos + 1 - b0);
    sync();  // the previous block's k, v, p are no longer read
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int idx = tid + u * kThreads;
      const int j = idx / (D / 4), c = idx - j * (D / 4);
      sm.k[j][c * 4 + 0] = kreg[u].x, sm.k[j][c * 4 + 1] = kreg[u].y, sm.k[j][c * 4 + 2] = kreg[u].z, sm.k[j][c * 4 + 3] = kreg[u].w;
      *reinterpret_cast<float4*>(&sm.v[j][c * 4]) = vreg[u];
    }
    if (b0 + kPfKeys <= last_pos) fetch(b0 + kPfKeys);
    sync();
    // ---- scores: lane = key position, warp w takes query vectors w + 8 i
    {
      float sc[kHeadsPerWarp];
#pragma unroll
      for (int i = 0; i < kHeadsPerWarp; ++i) sc[i] = 0.0f;
#pragma unroll 4
      for (int d = 0; d < D; d += 4) {  // query elements as 16-byte broadcast loads, key elements scalar (padded rows)
        const float k0 = sm.k[lane][d], k1 = sm.k[lane][d + 1], k2 = sm.k[lane][d + 2], k3 = sm.k[lane][d + 3];
#pragma unroll
        for (int i = 0; i < kHeadsPerWarp; ++i) {
          if (wh + HEAD_WARPS * i < group) {
            const float4 q4 = *reinterpret_cast<const float4*>(&sm.q[wr + kPfRows * (wh + HEAD_WARPS * i)][d]);
            sc[i] = fmaf(q4.x, k0, sc[i]);
            sc[i] = fmaf(q4.y, k1, sc[i]);
            sc[i] = fmaf(q4.z, k2, sc[i]);
            sc[i] = fmaf(q4.w, k3, sc[i]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kHeadsPerWarp; ++i) {
        if (wh + HEAD_WARPS * i >= group) break;
        const int qi = wr + kPfRows * (wh + HEAD_WARPS * i);  // = h * kPfRows + r
        const int pos = pos0 + s0 + wr;        // position of this query row
        const bool valid = lane < nk && b0 + lane <= pos && wr < nrows;
        const float sv = valid ? sc[i] * scale : -3.402823466e+38f;
        float mx = sv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m_run[i], mx);
        const float pv = valid ? expf(sv - m_new) : 0.0f;
        float sum = pv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float alpha = expf(m_run[i] - m_new);
        m_run[i] = m_new;
        l_run[i] = l_run[i] * alpha + sum;
        sm.p[qi][lane] = pv;
        if (lane == 0) {
          sm.alpha[qi] = alpha;
          sm.lsum[qi] = l_run[i];
        }
      }
    }
    sync();
    // ---- P.V: keys outermost, so that a value row is loaded once for all query vectors of the thread
#pragma unroll
    for (int i = 0; i < QPT; ++i) {
      const int qi = pg + i * NG;
      const float al = qi < nq ? sm.alpha[qi] : 1.0f;
      o_acc[i][0] *= al, o_acc[i][1] *= al, o_acc[i][2] *= al, o_acc[i][3] *= al;
    }
#pragma unroll 2
    for (int j = 0; j < kPfKeys; j += 4) {
      float4 v4[4];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) v4[jj] = *reinterpret_cast<const float4*>(&sm.v[j + jj][pc * 4]);
#pragma unroll
      for (int i = 0; i < QPT; ++i) {
        const int qi = pg + i * NG;
        if (qi < nq) {
          const float4 p4 = *reinterpret_cast<const float4*>(&sm.p[qi][j]);
          const float pj[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            o_acc[i][0] = fmaf(pj[jj], v4[jj].x, o_acc[i][0]);
            o_acc[i][1] = fmaf(pj[jj], v4[jj].y, o_acc[i][1]);
            o_acc[i][2] = fmaf(pj[jj], v4[jj].z, o_acc[i][2]);
            o_acc[i][3] = fmaf(pj[jj], v4[jj].w, o_acc[i][3]);
          }
        }
      }
    }
  }
  sync();
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const int qi = pg + i * NG;
    if (qi < nq) {
      const int h = qi / kPfRows, r = qi - h * kPfRows;
      if (r < nrows) {
        const float inv = 1.0f / sm.lsum[qi];
        *reinterpret_cast<float4*>(out + (size_t)(s0 + r) * ldo + (kvh * group + h) * D + pc * 4) =
            make_float4(o_acc[i][0] * inv, o_acc[i][1] * inv, o_acc[i][2] * inv, o_acc[i][3] * inv);
      }
    }
  }
}

}  // namespace mllmb200
