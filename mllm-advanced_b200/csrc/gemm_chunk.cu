// tcgen05 W4A32 GEMM for M >= 65: fp16 operands, short fp32 sums in tensor memory, the rest of every sum in fp32 registers
// (sm_100a).
//
//   A[n, k] = fp16( (u[n,k] - 8) * s[n, group(k)] * 2^E[n] )      B[m, k] = fp16( a_q[m, k] + a_off[m] )
//   y[m, n] = lhs_scale[m] * 2^-E[n] * sum_k A[n,k] B[m,k] + bias[n]
//
// (reference project tests/Arm/KaiLinearTest.hpp:338-377, production call kai_linear.cpp:350-398).  B is exact: |a_q + a_off| <=
// 255.  A is exact too: (u - 8) * s has at most 3 + 8 significant bits for a bf16-encoded scale, and E brings the matrix'
// largest |scale| to [2^10, 2^11) as long as no bit of any scale then falls below fp16's last place, 2^-24, which the repack
// notes (bf16-encoded scales: largest and smallest up to 2^27 apart).  Where one does, E[n] is the row's own; rows with more
// than that between their own scales, or with an infinity or NaN among them, are summed on the CUDA cores instead
// (ck_row_sum; the tensor core's sums of such a row are not used).
// An fp16-encoded scale needs 14 bits: those matrices go through every K-tile twice, once with the scale's first 8 bits and
// once with the rest.  All products are exact in fp32; what rounds is the addition.
//
// The tensor core truncates where it adds, which shrinks a sum of 1024 values by about 5e-8 and one of 8960 by 4e-7:
// more than fp32 additions of rounded group sums are off.  So a sum stays in tensor memory for one CHUNK of K only and is
// then added to fp32 registers.
// Two forms.  NT = 256: a PAIR of CTAs (cta_group::2) makes 256 weight rows x 256 rows of x; each holds its 128 rows of the
// operand A and of the sums in tensor memory and one half of the operand B in shared memory, so that a byte of B that comes
// from L2 feeds twice the products (the traffic of B from L2 is what bounds a single CTA of this shape).  NT = 128: single
// CTAs, for launches with few tiles.  576 threads, one CTA per SM:
//   warps 0-15 dequant: thread = weight row 32 (w % 4) + lane; a turn = two K-groups of the row (32 bytes of nibbles -> 32
//              tensor-memory columns of fp16); a finished chunk is added to the registers after the turn behind it
//   warp 16    producer: bulk copies of weight cells (evict-first) and activation blocks (a pair: tensor copies of both CTAs that
//              count on the barrier of CTA 0 that its products wait for anyway)
//   warp 17    MMA issuer (one elected lane; of CTA 0 for a pair) and tensor-memory owner
// A pair multiplies four stages (256 values of K) for the first half of its columns, then for the second: while one half's
// finished chunk is fetched the other half's products run, and the next four stages are dequantized.
// Bound: the dequantization warps' chain (wait, load, ~150 instructions per two K-groups, store, arrive) and the hand-offs around
// it, next to the tensor pipe: without its tensor-core instructions a launch on 1536 x 8960 takes 51 of 54 us at M = 65 and 57
// of 63 at M = 512, without the operand's stores to tensor memory or without the sums' fetches as long as with them.
// Measured (B200, quantization of x included), the int8 tile GEMM (gemm_tc.cu) / this kernel: 8960 x 1536, M = 512 63 / 28 us;
// 28672 x 8192, M = 512 762 / 308 us, M = 2048 2848 / 995 us (967 TFLOP/s); 1536 x 8960 (single CTAs), M = 512 78 / 62 us;
// error against 64 bits (2-norm) 6.0e-8 / 5.3e-8 at K = 1536, 1.29e-7 / 9.4e-8 at K = 8192; where weights and activations
// are of one sign throughout, 1.3e-7 / 1.0e-7 at K = 1536, 3.9e-7 / 5.3e-7 at K = 8960.  M = 65, 17920 x 1536
// 33 / 24 us; the three matrices of q, k, v, M = 65 (one launch instead of three) 47 / 14 us.  At M <= 64 the streaming
// kernel (gemm_stream.cu) mostly stays ahead: it needs no 128-row tiles (1536 x 1536, M = 64: 6.2 us; here, M = 65, 13.3).
// fp16-encoded scales, us: 1536 x 1536, M = 65 19.4, 1536 x 8960, M = 512 87, 8960 x 1536, M = 512 35 (27, 110 and 47 with
// finished chunks fetched in front of every turn and a wait of the MMA issuer for either part).
#include <cuda.h>
#include <cuda_fp16.h>

#include "device_common.cuh"
#include "tcgen05_common.cuh"

namespace mllmb200 {

constexpr int kCkDqWarps = 16;
constexpr int kCkThreads = (kCkDqWarps + 2) * 32;
constexpr int kCkRows = 128;         // weight rows per CTA
constexpr int kCkPanels = kCkRows / kPanelRows;
constexpr int kCkMaxProblems = 4;
constexpr int kCkQuad = 4;           // K-groups per quad, the unit of a chunk

struct CkProblem {
  const uint8_t* tiled;
  float* y;
  int n, ldy, num_panels, tile_begin;
  size_t bias_off;
};
struct CkParams {
  const uint8_t* a_blocks;  // [num_groups][m8][512 bytes] fp16 canonical blocks (act_quant_blocks_f16_kernel)
  const float2* a_hdr;      // [m] {lhs_scale, -}
  int m, k, num_groups, m8, num_problems, use_pdl;
  int m_tiles, chunk_quads;
  CkProblem prob[kCkMaxProblems];
};

template <int NT>
struct CkSmem {
  static constexpr bool kPair = NT == 256;
  static constexpr int kRowsB = kPair ? NT / 2 : NT;   // rows of B in this CTA's shared memory
  static constexpr int kGroups = kPair ? 2 : 4;        // K-groups per stage
  static constexpr int kSpan = kPair ? 4 : 2;          // stages in which every dequant warp has one turn
  static constexpr int kRawBytes = kCkPanels * kGroups * kCellBytes;
  static constexpr int kBBytes = kGroups * kRowsB * 64;
  static constexpr int kStageBytes = kRawBytes + kBBytes;
  static constexpr int kBarBytes = 512;
  static constexpr int kHdrBytes = NT * 4;
  static constexpr int kStages = 2 * kSpan;            // ring of loaded stages, ring of operand stages: powers of two
  static constexpr int kAStages = 2 * kSpan;
  static constexpr int kSlotCols = 128;                // two slots of sums: chunks (a pair: the halves of its columns)
  static constexpr int kAccCols = 2 * kSlotCols;       // columns [0, 256): sums; [256, 512): the weight operand
  static constexpr int kACols = kGroups * 16;          // operand columns of one stage
  static constexpr int kStageOff = kBarBytes + kHdrBytes;
  static constexpr int kTotal = kStageOff + kStages * kStageBytes + 1024;
  static_assert(kAccCols + kAStages * kACols == 512, "tensor memory");
  static_assert((3 * kStages + 2 * kAStages + 4) * 8 + 8 <= kBarBytes, "barrier area");
  static_assert(!kPair || (kStageOff % 128 == 0 && kStageBytes % 128 == 0 && kRawBytes % 128 == 0), "a tensor copy's destination");
  static_assert(kTotal <= 227 * 1024, "shared memory");
};

// mbar_wait_bounded on a shared-memory address, the whole warp: one outcome.  CLUSTER: for arrivals of the other CTA
template <bool CLUSTER>
__device__ __forceinline__ bool ck_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
template <bool CLUSTER>
__device__ __noinline__ bool ck_wait_slow(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!ck_try_wait<CLUSTER>(bar, parity))
    if (clock64() - t0 > (1ll << 31)) {
      atomicOr(&g_device_status, kDevStatusTimeout);
      return false;
    }
  return true;
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool ck_wait(uint32_t bar, uint32_t parity) {
  bool ok = ck_try_wait<CLUSTER>(bar, parity);
  if (__all_sync(0xffffffffu, ok)) return true;
  ok = ok || ck_wait_slow<CLUSTER>(bar, parity);
  return __all_sync(0xffffffffu, ok);
}
// Arrival on this CTA's barrier, or (from CTA 1 of a pair) on the one of CTA 0 that has its place there.  That one is relaxed: it hands
// on tensor memory alone, which the tcgen05 waits and fences around it order between threads of a cluster.
template <bool PAIR>
__device__ __forceinline__ void ck_arrive(uint32_t bar, int rank) {
  if (PAIR && rank != 0)
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %0, 0;\n\t"
        "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar)
        : "memory");
  else
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A box of the activation blocks, [K-group][8 rows of x][512 bytes], into this CTA's shared memory; its bytes are counted on the barrier
// of CTA 0 that has bar's place there.
__device__ __forceinline__ void ck_pair_load(uint32_t dst, const CUtensorMap* map, int m8, int group, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b32 r;\n\t"
      "mapa.shared::cluster.u32 r, %4, 0;\n\t"
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%5, %2, %3}], [r];\n\t}" ::"r"(dst),
      "l"(map), "r"(m8), "r"(group), "r"(bar), "r"(0)
      : "memory");
}
// arrival once the MMAs issued so far have completed, on both CTAs' barriers for a pair
template <bool PAIR>
__device__ __forceinline__ void ck_commit(uint32_t bar) {
  if constexpr (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void ck_mma(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    tc_mma_f16_ts(d, a, b_desc, idesc, accumulate);
}
// 2^E that brings a largest |scale| (its bits) to [2^10, 2^11); 2^E and 2^-E stay normal
__device__ __forceinline__ int ck_exponent(uint32_t top) { return min(10 - ((int)(top >> 23) - 127), 126); }
// the bits of all scales times 2^E lie at 2^-24 or above: fp16 holds them and their products with u - 8
__device__ __forceinline__ bool ck_fits(uint32_t low_bit, int e) { return low_bit <= (uint32_t)(512 + 24 + e); }
// 2^E for row `lane` of a panel: the matrix' exponent, or (rare) the row's own where that one does not fit all scales.  0: nor does the row's
__device__ __forceinline__ float ck_up(const uint8_t* tiled, int panel, int lane, int num_groups, uint32_t scale_mode) {
  const TiledHeader* h = reinterpret_cast<const TiledHeader*>(tiled);
  int e = ck_exponent(h->max_scale_bits);
  if (!ck_fits(h->low_bit, e)) {
    const uint8_t* cell = tiled + sizeof(TiledHeader) + (size_t)panel * num_groups * kCellBytes + kCellNibbleBytes + lane * 2;
    uint32_t low = 0;
    float mx = 0.0f;
    for (int g = 0; g < num_groups; ++g, cell += kCellBytes) {
      const float s = fabsf(decode_scale(*reinterpret_cast<const uint16_t*>(cell), scale_mode));
      if (s <= 3.402823466e+38f) mx = fmaxf(mx, s);
      low = max(low, scale_low_bit(s));
    }
    e = ck_exponent(__float_as_uint(mx));
    if (!ck_fits(low, e)) return 0.0f;
  }
  return __uint_as_float((uint32_t)(e + 127) << 23);
}
// One sum as the reference forms it, for rows whose scales fit no common exponent (or hold infinities): the K-groups' integer
// sums, exact in fp32, times their scales.  cell: the row's 16 bytes in its panel's first cell; scale: its scale there;
// x: the row's 16 bytes in the first activation block.
__device__ __forceinline__ float ck_row_sum(const uint8_t* cell, const uint8_t* scale, const uint8_t* x, size_t x_stride, int num_groups,
                                            uint32_t scale_mode) {
  float acc = 0.0f;
#pragma unroll 1
  for (int g = 0; g < num_groups; ++g, cell += kCellBytes, scale += kCellBytes, x += x_stride) {
    float sum = 0.0f;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(cell + c * 4);
      const __half2* h = reinterpret_cast<const __half2*>(x + c * 128);  // k = 8c + {0,4}, {1,5}, {2,6}, {3,7}
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 v = __half22float2(h[t]);
        sum = fmaf((float)((int)(w >> (4 * t) & 15u) - 8), v.x, sum);
        sum = fmaf((float)((int)(w >> (4 * t + 16) & 15u) - 8), v.y, sum);
      }
    }
    acc = fmaf(sum, decode_scale(*reinterpret_cast<const uint16_t*>(scale), scale_mode), acc);
  }
  return acc;
}
// (the single-CTA form is 3 % slower with it in line, the pair form 1 % with a call: registers of the loop in front of it)
__device__ __noinline__ float ck_row_sum_call(const uint8_t* cell, const uint8_t* scale, const uint8_t* x, size_t x_stride, int num_groups,
                                            uint32_t scale_mode) {
  return ck_row_sum(cell, scale, x, x_stride, num_groups, scale_mode);
}
__device__ __forceinline__ float ck_clamp(float v) {  // clamp_flt_max: only infinities lie outside
  return fabsf(v) > 3.402823466e+38f ? copysignf(3.402823466e+38f, v) : v;
}

template <int NT>
__global__ void __launch_bounds__(kCkThreads, 1) w4a32_gemm_chunk_kernel(const __grid_constant__ CkParams p, const __grid_constant__ CUtensorMap amap) {
  using S = CkSmem<NT>;
  constexpr bool kPair = S::kPair;
  constexpr int kStages = S::kStages, kAStages = S::kAStages, kGroups = S::kGroups, kSpan = S::kSpan;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;  // (the same place in both CTAs of a pair)
  uint8_t* smem_ptr = smem_raw + (smem - smem_u32(smem_raw));
  const uint32_t raw_full = smem;                       // [kStages]  loaded data arrived
  const uint32_t raw_free = raw_full + kStages * 8;     // [kStages]  the MMAs that read a stage completed
  const uint32_t a_full = raw_free + kStages * 8;       // [kAStages] operand written (a pair: by both, in CTA 0)
  const uint32_t a_free = a_full + kAStages * 8;        // [kAStages] operand read
  const uint32_t acc_full = a_free + kAStages * 8;      // [2] a chunk's sums are complete
  const uint32_t acc_free = acc_full + 16;              // [2] ... and are in registers (a pair: both, in CTA 0)
  // A pair: the copies of x of both CTAs count on barriers of CTA 0, whose instructions read them.  Those are a_full, one wait for both
  // (another wait a stage: 15 % of the kernel); of two parts, whose operand stages come round twice as often, barriers of their own.
  const uint32_t x_own = acc_free + 16;                 // [kStages]
  const uint32_t stages = smem + S::kStageOff;
  constexpr int kXBar = 2 * kStages + 2 * kAStages + 4, kBars = kXBar + (kPair ? kStages : 0);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_ptr);
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(bars + kBars);
  float* s_scale = reinterpret_cast<float*>(smem_ptr + S::kBarBytes);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (p.use_pdl) pdl_launch_dependents();
  // Tiles that share weights (same rows of W, other rows of x) are neighbours: one reads them from DRAM, the rest from L2.
  const int tile = kPair ? (int)blockIdx.x >> 1 : (int)blockIdx.x, rank = kPair ? (int)blockIdx.x & 1 : 0;
  const int bx = tile / p.m_tiles, m0 = (tile - bx * p.m_tiles) * NT;
  int pi = 0;
#pragma unroll
  for (int i = 1; i < kCkMaxProblems; ++i)
    if (i < p.num_problems && bx >= p.prob[i].tile_begin) pi = i;
  const CkProblem pr = p.prob[pi];
  if (!tiled_header_ok_cta(pr.tiled, pr.n, p.k)) return;  // the same answer in both CTAs of a pair
  const int panel0 = ((bx - pr.tile_begin) * (kPair ? 2 : 1) + rank) * kCkPanels, n0 = panel0 * kPanelRows;
  const int k_tiles = (p.num_groups + kGroups - 1) / kGroups;
  const uint32_t scale_mode = reinterpret_cast<const TiledHeader*>(pr.tiled)->scale_mode;
  const int parts = scale_mode == 2u ? 2 : 1;  // fp16-encoded scales: every stage twice
  // With two parts a turn of the dequant warps waits for MMAs of the span before, and those of a pair for the fetch of the
  // chunk before theirs, which comes behind the turn: no chunk ends inside a span.
  const int chunk_tiles = max(p.chunk_quads, parts) * (kCkQuad / kGroups);
  static_assert(2 * kCkQuad / kGroups % kSpan == 0 && 4 * kCkQuad / kGroups % kSpan == 0 && 6 * kCkQuad / kGroups % kSpan == 0, "chunks of whole spans");
  const int m_here = min(NT, p.m - m0);

  if (tid == 0) {
    for (int i = 0; i < kBars; ++i) {
      const bool written = i >= 2 * kStages && i < 2 * kStages + kAStages;  // a_full: a warp writes two K-groups of its 32 rows
      const bool fetched = i >= kXBar - 2 && i < kXBar;                     // acc_free
      mbar_init(&bars[i], (written ? 2 * kGroups : fetched ? kCkDqWarps : 1) * ((written || fetched) && kPair ? 2 : 1) + (kPair && written && parts == 1 ? 1 : 0));
    }
    mbar_fence_init();
  }
  if (warp == kCkDqWarps + 1) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)), "r"(512u) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(tmem_base_slot, 512u);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (kPair) cluster_sync_all();  // the other CTA's barriers and tensor memory exist
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_base_slot, 0);

  const uint32_t x_full = parts == 1 ? a_full : x_own;
  static_assert(kStages == kAStages, "a stage's number is that of its operand");
  if (warp == kCkDqWarps) {
    // ------------------------------------------------------------ producer
    const int np = max(0, min(kCkPanels, pr.num_panels - panel0));
    const int b_row0 = m0 + (kPair ? rank * S::kRowsB : 0);
    const int b_bytes = max(0, min(S::kRowsB, p.m8 * 8 - b_row0)) * 64;  // per K-group; rows of B beyond feed columns nobody reads
    const uint64_t stream_once = l2_policy_evict_first();
    auto request = [&](int it, int which) {  // bit 0: weight cells (and the barrier), bit 1: activation blocks
      const int s = it % kStages, g0 = it * kGroups, ng = min(kGroups, p.num_groups - g0);
      uint8_t* st = smem_ptr + S::kStageOff + s * S::kStageBytes;
      if ((which & 1) && lane == 0) mbar_arrive_expect_tx(&bars[s], (uint32_t)(np * ng * kCellBytes + (kPair ? 0 : ng * b_bytes)));
      __syncwarp();
      if (kPair && (which & 2) && lane == kCkPanels) {  // whole boxes: what lies outside of the blocks arrives as zeros
        if (rank == 0) mbar_arrive_expect_tx(&bars[(x_full - smem) / 8 + s], 2u * S::kBBytes);
        ck_pair_load(smem_u32(st) + S::kRawBytes, &amap, b_row0 >> 3, g0, x_full + (uint32_t)s * 8);
      }
      if ((which & 1) && lane < np)
        bulk_g2s_hint(st + lane * kGroups * kCellBytes,
                      pr.tiled + sizeof(TiledHeader) + ((size_t)(panel0 + lane) * p.num_groups + g0) * kCellBytes,
                      (uint32_t)(ng * kCellBytes), &bars[s], stream_once);
      else if (!kPair && (which & 2) && lane >= kCkPanels && lane < kCkPanels + ng && b_bytes > 0)
        bulk_g2s(st + S::kRawBytes + (lane - kCkPanels) * S::kRowsB * 64,
                 p.a_blocks + ((size_t)(g0 + lane - kCkPanels) * p.m8 + (b_row0 >> 3)) * 512, (uint32_t)b_bytes, &bars[s]);
    };
    // the weights are constant, the activations come from the kernel in front: the first lap's weights go before the wait
    const int first_lap = min(k_tiles, kStages);
    for (int it = 0; it < first_lap; ++it) request(it, p.use_pdl ? 1 : 3);
    if (p.use_pdl) {
      pdl_wait_prior();
      for (int it = 0; it < first_lap; ++it) request(it, 2);
    }
    for (int it = first_lap; it < k_tiles; ++it) {
      if (!ck_wait(raw_free + (uint32_t)(it % kStages) * 8, (uint32_t)(it / kStages - 1) & 1u)) {
        // nothing in flight when the CTA leaves: 10 ms is a thousand times what a copy takes
        for (const long long t0 = clock64(); clock64() - t0 < (1ll << 24);) {
        }
        break;
      }
      request(it, 3);
    }
  } else if (warp == kCkDqWarps + 1) {
    // ------------------------------------------------------------ MMA issuer: the whole warp loops, one lane issues
    if (!kPair || rank == 0) {
      const bool issuer = elect_one_sync();
      // D = f32, A = B = f16, both K-major.  M = 128, N = the tile's rows of x rounded up to 16; a pair: M = 256, N = 128
      const uint32_t idesc = (1u << 4) | ((uint32_t)(kPair ? 16 : (m_here + 15) / 16 * 2) << 17) | ((kPair ? 16u : 8u) << 24);
      // Everything the instructions take is computed by the whole warp, outside of the elected lane's branch.
      constexpr int kStep = kPair ? 4 : 1, kHalves = kPair ? 2 : 1;
      bool ok = true;
      int c = 0, left = min(chunk_tiles, k_tiles);  // chunk, its stages still to come
      uint32_t accumulate = 0;
      for (int it = 0; it < k_tiles && ok;) {
        const int steps = min(kStep, left);
        for (int v = it * parts + parts - 1; v < (it + steps) * parts && ok; v += parts) {
          // arrived on by warps that saw raw_full complete: orders the stage's copies too.  (Of two parts the last: the
          // same warps wrote the first before it.)
          ok = ck_wait<kPair>(a_full + (uint32_t)(v % kAStages) * 8, (uint32_t)(v / kAStages) & 1u);
          if (kPair && parts > 1 && ok) ok = ck_wait(x_full + (uint32_t)(v / parts % kStages) * 8, (uint32_t)(v / parts / kStages) & 1u);
        }
        left -= steps;
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {
          const int slot = kPair ? h : c & 1, use = kPair ? c : c >> 1;
          if (ok && accumulate == 0 && use > 0) ok = ck_wait<kPair>(acc_free + (uint32_t)slot * 8, (uint32_t)(use - 1) & 1u);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem_base + (uint32_t)(slot * S::kSlotCols);
          uint32_t acc = accumulate;
          for (int part = 0; part < parts; ++part) {
            const int v0 = it * parts + part;  // operand stages v0, v0 + parts, ..
#pragma unroll
            for (int j = 0; j < kStep; ++j)
              if (j < steps) {
                const uint32_t sa = (uint32_t)(v0 + j * parts) % kAStages, s = (uint32_t)(it + j) % kStages;
                const uint32_t a = tmem_base + S::kAccCols + sa * S::kACols;
                const uint64_t b_desc = make_kmajor_desc(stages + s * S::kStageBytes + S::kRawBytes + (uint32_t)h * 64 * 64, 128, 512);
                const int ng = min(kGroups, p.num_groups - (it + j) * kGroups);
                if (issuer) {
#pragma unroll
                  for (int g = 0; g < kGroups; ++g)
                    if (g < ng) {
                      ck_mma<kPair>(d, a + (uint32_t)(g * 16), b_desc + (uint64_t)((g * S::kRowsB * 64) >> 4), idesc, g == 0 ? acc : 1u);
                      ck_mma<kPair>(d, a + (uint32_t)(g * 16 + 8), b_desc + (uint64_t)((g * S::kRowsB * 64 + 256) >> 4), idesc, 1u);
                    }
                  if (h + 1 == kHalves) {
                    ck_commit<kPair>(a_free + sa * 8);
                    if (part + 1 == parts) ck_commit<kPair>(raw_free + s * 8);
                  }
                }
                __syncwarp();
                acc = 1;
              }
          }
          if (left == 0 && issuer) ck_commit<kPair>(acc_full + (uint32_t)slot * 8);
          __syncwarp();
        }
        it += steps;
        accumulate = 1;
        if (left == 0) {
          ++c;
          left = min(chunk_tiles, k_tiles - it);
          accumulate = 0;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ dequant and sums
    const int rset = warp & 3, turn = warp >> 2;  // 32 weight rows = tensor-memory lanes 32 (warp % 4)..
    const bool have_panel = panel0 + rset < pr.num_panels;
    const int n = n0 + rset * 32 + lane;
    const float up = have_panel ? ck_up(pr.tiled, panel0 + rset, lane, p.num_groups, scale_mode) : 1.0f;
    const uint32_t lane_base = tmem_base + ((uint32_t)(rset * 32) << 16);
    constexpr int kSlotWarpCols = 32, kCols = NT / 4;  // columns of this warp: 32 in each slot (a pair: of each half)
    float seg[kCols];
#pragma unroll
    for (int i = 0; i < kCols; ++i) seg[i] = 0.0f;
    bool ok = true;
    int drained = 0, drained_end = min(chunk_tiles, k_tiles);  // chunks fetched; stages up to the end of the next one
    // first row of x of the warp's columns in slot j of a pair: columns [0, 64) of a half are rows 64 j.. of CTA 0's
    // half of B, [64, 128) of CTA 1's
    auto first_col = [&](int j) { return kPair ? (turn >> 1) * 128 + j * 64 + (turn & 1) * 32 : turn * 32; };
    auto drain = [&]() {  // the next finished chunk: tensor memory -> registers
      const uint32_t c = (uint32_t)drained++;
      drained_end = min(drained_end + chunk_tiles, k_tiles);
#pragma unroll
      for (int h = 0; h < (kPair ? 2 : 1); ++h) {
        const uint32_t slot = kPair ? (uint32_t)h : c & 1u;
        ok = ok && ck_wait(acc_full + slot * 8, (kPair ? c : c >> 1) & 1u);
        if (!ok) return;
        tc_fence_after();
#pragma unroll
        for (int i0 = 0; i0 < kSlotWarpCols; i0 += 16) {
          uint32_t v[16];
          tmem_ld16(lane_base + slot * S::kSlotCols + (uint32_t)(turn * kSlotWarpCols + i0), v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) seg[h * kSlotWarpCols + i0 + i] += __uint_as_float(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) ck_arrive<kPair>(acc_free + slot * 8, rank);
      }
    };
    const int own = kPair ? turn : turn >> 1, half = kPair ? 0 : turn & 1;  // stage of a span, pair of its K-groups
    const uint32_t raw_off = (uint32_t)((rset * kGroups + half * 2) * kCellBytes);
    for (int span = 0; span < k_tiles && ok; span += kSpan) {
      // chunks that ended before this span are fetched behind this span's turn: the MMA issuer has work meanwhile
      const int it = span + own;
      if (it < k_tiles) {
        const uint32_t s = (uint32_t)it % kStages;
        ok = ok && ck_wait(raw_full + s * 8, (uint32_t)(it / kStages) & 1u);
        const int ng = p.num_groups - it * kGroups - half * 2;  // K-groups of this turn
        const uint8_t* raw = smem_ptr + S::kStageOff + s * S::kStageBytes + raw_off;
        for (int part = 0; part < parts && ok; ++part) {
          const uint32_t vt = (uint32_t)(it * parts + part), sa = vt % kAStages;
          if (vt >= kAStages) ok = ck_wait(a_free + sa * 8, (vt / kAStages - 1) & 1u);
          if (!ok) break;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint4 w = make_uint4(0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u);
            uint32_t sc16 = 0;
            if (have_panel && g < ng) {
              w = *reinterpret_cast<const uint4*>(raw + g * kCellBytes + lane * 16);
              sc16 = *reinterpret_cast<const uint16_t*>(raw + g * kCellBytes + kCellNibbleBytes + lane * 2);
            }
            const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
            uint32_t areg[16];  // column c * 4 + t = chunk c (k 8c .. 8c + 7), nibbles t and t + 4
            if (parts == 1) {
              // the nibble in mantissa bits 6..9 of 0x4400 reads x = 4 + u / 4; (u - 8) s = x (4 s) - 24 s in one fused
              // multiply-add whose operands and result all fit fp16
              const float s_up = __uint_as_float(sc16 << 16) * up;  // a power-of-two multiple of the scale: exact
              const __half2 s4 = __float2half2_rn(4.0f * s_up), c24 = __float2half2_rn(-24.0f * s_up);
#pragma unroll
              for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  const uint32_t moved = t == 0 ? ws[c] << 6 : t == 1 ? ws[c] << 2 : t == 2 ? ws[c] >> 2 : ws[c] >> 6;
                  const uint32_t bits = (moved & 0x03C003C0u) | 0x44004400u;
                  const __half2 v = __hfma2(*reinterpret_cast<const __half2*>(&bits), s4, c24);
                  areg[c * 4 + t] = *reinterpret_cast<const uint32_t*>(&v);
                }
            } else {
              // the scale's first 8 bits in the first part, the up to 3 that are left in the second: as above
              const float s = decode_scale(sc16, 2u), top = __uint_as_float(__float_as_uint(s) & 0xFFFF0000u);
              const float s_up = (part == 0 ? top : s - top) * up;
              const __half2 s4 = __float2half2_rn(4.0f * s_up), c24 = __float2half2_rn(-24.0f * s_up);
#pragma unroll
              for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  const uint32_t moved = t == 0 ? ws[c] << 6 : t == 1 ? ws[c] << 2 : t == 2 ? ws[c] >> 2 : ws[c] >> 6;
                  const uint32_t bits = (moved & 0x03C003C0u) | 0x44004400u;
                  const __half2 v = __hfma2(*reinterpret_cast<const __half2*>(&bits), s4, c24);
                  areg[c * 4 + t] = *reinterpret_cast<const uint32_t*>(&v);
                }
            }
            tmem_st16(lane_base + S::kAccCols + sa * S::kACols + (uint32_t)((half * 2 + g) * 16), areg);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) ck_arrive<kPair>(a_full + sa * 8, rank);
        }
      }
      while (ok && drained_end <= span) drain();
    }
    // the rows' scales (and nobody reads the old y any more): requested before the last sums are waited for
    if (p.use_pdl) pdl_wait_prior();
    float x_scale = 0.0f;
    if (tid < m_here) x_scale = p.a_hdr[m0 + tid].x;
    const bool live = n < pr.n;
    const float bs = live ? reinterpret_cast<const float*>(pr.tiled + pr.bias_off)[n] : 0.0f;
    const int chunks = (k_tiles + chunk_tiles - 1) / chunk_tiles;
    while (drained < chunks && ok) drain();
    if (tid < m_here) s_scale[tid] = x_scale;
    asm volatile("bar.sync 1, %0;" ::"n"(kCkDqWarps * 32) : "memory");
    const float down = __uint_as_float((254u << 23) - __float_as_uint(up));  // 1 / up
    if (ok && live && up == 0.0f) {
      const uint8_t* cell = pr.tiled + sizeof(TiledHeader) + (size_t)(panel0 + rset) * p.num_groups * kCellBytes;
#pragma unroll 1
      for (int i = 0; i < kCols; ++i) {
        const int col = first_col(i / kSlotWarpCols) + i % kSlotWarpCols, m = m0 + col;
        if (col >= m_here) continue;
        const float sum = (kPair ? ck_row_sum : ck_row_sum_call)(cell + lane * 16, cell + kCellNibbleBytes + lane * 2, p.a_blocks + (size_t)(m >> 3) * 512 + (m & 7) * 16,
                                     (size_t)p.m8 * 512, p.num_groups, scale_mode);
        pr.y[(size_t)m * pr.ldy + n] = ck_clamp(fmaf(sum, s_scale[col], bs));
      }
    } else if (ok && live) {
#pragma unroll
      for (int j = 0; j < kCols / kSlotWarpCols; ++j) {
        const int col0 = first_col(j);
        float* yp = pr.y + (size_t)(m0 + col0) * pr.ldy + n;
        // (a store through a generic pointer may alias shared memory: all scales first, then all stores)
#pragma unroll
        for (int i = 0; i < kSlotWarpCols; ++i)
          seg[j * kSlotWarpCols + i] = ck_clamp(fmaf(seg[j * kSlotWarpCols + i] * down, s_scale[col0 + i], bs));
        if (col0 + kSlotWarpCols <= m_here) {
#pragma unroll
          for (int i = 0; i < kSlotWarpCols; ++i) yp[(size_t)i * pr.ldy] = seg[j * kSlotWarpCols + i];
        } else {
#pragma unroll
          for (int i = 0; i < kSlotWarpCols; ++i)
            if (col0 + i < m_here) yp[(size_t)i * pr.ldy] = seg[j * kSlotWarpCols + i];
        }
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if constexpr (kPair) cluster_sync_all();  // nobody frees tensor memory or leaves while the other still uses it
  else __syncthreads();
  if (warp == kCkDqWarps + 1) {
    tc_fence_after();
    if constexpr (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    else tmem_dealloc(tmem_base, 512u);
  }
}

// The activation blocks as a tensor [num_groups][m8][128 words], in boxes of a stage's K-groups and a CTA's half of 256 rows
static cudaError_t ck_encode(CUtensorMap* map, const CkParams& prm) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    cudaDriverEntryPointQueryResult q;
    void* f = nullptr;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess ? reinterpret_cast<Encode>(f) : nullptr;
  }();
  if (!encode) return cudaErrorSymbolNotFound;
  using S = CkSmem<256>;
  const cuuint64_t dims[3] = {128, (cuuint64_t)prm.m8, (cuuint64_t)prm.num_groups}, strides[2] = {512, (cuuint64_t)prm.m8 * 512};
  const cuuint32_t box[3] = {128, S::kRowsB / 8, S::kGroups}, one[3] = {1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t*>(prm.a_blocks), dims, strides, box, one,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int NT>
static cudaError_t ck_launch_t(const CkParams& prm, int tiles, cudaStream_t stream) {
  using S = CkSmem<NT>;
  static bool configured[64] = {};  // function attributes are per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!(dev >= 0 && dev < 64 && configured[dev])) {
    e = cudaFuncSetAttribute(w4a32_gemm_chunk_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * prm.m_tiles * (S::kPair ? 2 : 1)), 1, 1);
  cfg.blockDim = dim3(kCkThreads, 1, 1);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  if (S::kPair) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = 2;
    attrs[na].val.clusterDim.y = attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  if (prm.use_pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  CUtensorMap amap = {};
  if (S::kPair && (e = ck_encode(&amap, prm)) != cudaSuccess) return e;
  return cudaLaunchKernelEx(&cfg, w4a32_gemm_chunk_kernel<NT>, prm, amap);
}

// blocks / hdr: output of launch_act_quant_blocks_f16 for the same m and k with rows padded to a multiple of 8.  Up to four
// matrices that share them.
cudaError_t launch_w4a32_gemm_chunk(const uint8_t* blocks, const float2* hdr, int m, int k, int count, const void* const* tiled,
                                    float* const* y, const int* n, const int* ldy, int use_pdl, cudaStream_t stream) {
  if (count < 1 || count > kCkMaxProblems || m < 1 || k < 1) return cudaErrorInvalidValue;
  CkParams prm = {};
  prm.a_blocks = blocks;
  prm.a_hdr = hdr;
  prm.m = m, prm.k = k;
  prm.num_groups = (k + kGroup - 1) / kGroup;
  prm.m8 = (m + 7) / 8;
  prm.num_problems = count;
  prm.use_pdl = use_pdl;
  // Chunks depend on K alone, so that a row shard or a group of matrices gives the bits of the whole matrix or the single
  // call.  As long as the error stays below that of int32 group sums: 128 values for a short K (which has few additions to
  // begin with), then longer: every chunk costs a fetch.
  const int quads = (prm.num_groups + kCkQuad - 1) / kCkQuad;
  prm.chunk_quads = quads < 8 ? 1 : quads < 16 ? 2 : quads < 64 ? 4 : 6;
  long long pairs = 0;
  for (int i = 0; i < count; ++i) pairs += (n[i] + 2 * kCkRows - 1) / (2 * kCkRows);
  const int nt = pairs * ((m + 255) / 256) < 50 ? 128 : 256;  // pairs from two thirds of a wave on
  const int rows = nt == 256 ? 2 * kCkRows : kCkRows;
  int tiles = 0;
  for (int i = 0; i < count; ++i) {
    const TiledHeader th = make_tiled_header(n[i], k, 0, 0);
    CkProblem& q = prm.prob[i];
    q.tiled = static_cast<const uint8_t*>(tiled[i]);
    q.y = y[i];
    q.n = n[i], q.ldy = ldy[i];
    q.num_panels = (int)th.num_panels;
    q.tile_begin = tiles;
    q.bias_off = th.bias_off;
    tiles += (n[i] + rows - 1) / rows;
  }
  prm.m_tiles = (m + nt - 1) / nt;
  return nt == 128 ? ck_launch_t<128>(prm, tiles, stream) : ck_launch_t<256>(prm, tiles, stream);
}

}  // namespace mllmb200
