// Streaming W4A32 GEMM for small batches (5 <= M <= 64 activation rows; up to 192 by the "fastest" policy), sm_100a.
//
//   y[m,n] = lhs_scale[m] * ( sum_b float(sum_{k in b} a_q[m,k] * w[n,k]) * s[n,b]  +  a_off[m] * zsum[n] ) + bias[n]
//
// the expression of the GEMV (gemv_stream.cu; reference project tests/Arm/KaiLinearTest.hpp:338-377, production call
// mllm/Backends/Arm/Kernels/kai_linear.cpp:350-398): exact int32 sums per K-group, one fp32 FMA with the group
// scale per (row, column, group).
//
// At these batch sizes the linear is a weight stream like the GEMV - every weight byte is read once and used for
// at most 64 rows - but 64 times the integer work of the GEMV does not fit the CUDA cores, and the tile GEMMs
// (128 weight rows x all of K per CTA) fill a fraction of the SMs: 12 CTAs for a 1536 x 1536 matrix.  Here the
// cells of the weight matrix (layout.h: [panel of 32 rows][K-group] x 576 bytes) are spread over all SMs as in the
// GEMV and the per-group integer products run on the tensor cores:
//   * a cluster of S CTAs keeps one block of at most 32 rows of x (33 rows and more: blocks of even size) and walks
//     panels; work unit = panel x block.  CTA rank r takes K-groups [r G / S, (r + 1) G / S) of every unit.  Two blocks read
//     the weights twice from L2, but 1536 x 1536 becomes 96 units on 148 SMs instead of 48 (M = 64: 9.2 -> 6.2 us with the
//     quantization, in a chain of dependent launches).  S, KS and with them the bits follow from M and K alone: a matrix has
//     the same bits by itself and in a group.
//   * a producer warp streams the unit's cells through a ring of stages (cp.async.bulk + full / empty
//     mbarriers, weights marked evict-first in L2); under programmatic dependent launch the first stages are
//     requested before griddepcontrol.wait, the activations after it.  A stage is 32 K-groups, two trips of a warp between waits,
//     where three of those fit beside the activations, else 16 (us, chain of dependent launches, 16 / 32: M = 8 1536 -> 8960 6.4 /
//     6.0, 2048 -> 17920 10.5 / 9.6, 4096 -> 17920 16.4 / 14.3, 8192 -> 28672 46 / 38; M = 48 8960 -> 1536 17.1 / 16.1; M = 64 8192 ->
//     28672 130 / 116; a stage may be cut anywhere between K-groups, the bits are the same).  The activations are one copy: in four parts,
//     of which the first lets the products start, a call of 8 rows takes 0.1 to 0.2 us longer.
//   * 8 compute warps: warp ks takes the K-groups ks, ks + 8 of a stage.  A cell: one ldmatrix.x4 = the words of four rows
//     per lane; two LOP3 and a shift make the A fragments of two mma.sync.m16n8k32 (s8: 16 (nibble - 8) in the high half
//     of each byte, so no zero-point term per group; low nibbles are k 0..15, high nibbles k 16..31 of the instruction, the
//     byte order of the activation blocks).  The accumulator starts at the bits of 786432.0f, whose last place is 1/16: the
//     s32 result read as a float is 786432 + group sum exactly (|16 sum| <= 2^19 < 2^22).  One packed add and one packed
//     FMA (two columns each) fold it into the fp32 sums.
//   * at the end of a unit the warps' sums meet in shared memory, [slice][column][row], and are added in pairs.  Three
//     epilogue warps do that beside the next unit's products; where no cluster has a second unit, the compute warps do it
//     themselves (eight are faster than three: 0.4 us).  With S > 1 ranks 1.. leave theirs in a double-buffered slot of
//     their own shared memory, signal rank 0 through an mbarrier in ITS shared memory, and rank 0 adds them in rank order
//     through distributed-shared-memory loads: deterministic.  Rank 0 (or the only CTA) applies zero-point term, row scale
//     and bias and stores four rows of a column at a time.
// What bounds it (M = 64, K = 1536, cycles of an SM): a cell takes 115, of which its tensor instructions need 32 and its
// packed FP32 instructions 32; the rest is issue (about 80 slots) and dependences.  More warps (16), registers filled one
// stage ahead and 64 columns per warp were each as slow or slower.  With u8 nibbles, a zero-point term per group, scalar
// FP32 and 32-bit loads a cell took 150.  us a call with its quantization, that form -> now, chain of dependent launches:
//   1536 -> 17920  M = 8 10.6 -> 8.5, 24 15.7 -> 12.1, 48 22.7 -> 18.9, 64 26.0 -> 21.5
//   8960 -> 1536   M = 8 12.7 -> 10.3, 24 19.3 -> 10.9, 48 24.0 -> 16.2, 64 30.7 -> 19.6
//   8192 -> 28672  M = 8 46.4 -> 38.2, 24 90 -> 54, 64 295 -> 116
//   2048 -> 4096   M = 8 5.57 -> 4.96; 2048 -> 17920 M = 8 11.9 -> 9.6
// Every wait is bounded; a cluster leaves together (one cluster barrier at the end) so that no CTA's shared memory
// disappears under a peer.
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"

namespace mllmb200 {

constexpr int kMsCWarps = 8;                  // compute warps
constexpr int kMsEWarps = 3;                  // epilogue warps; with the producer warp between them 12 warps, 3 per scheduler
constexpr int kMsThreads = (kMsCWarps + 1 + kMsEWarps) * 32;
constexpr int kMsStageGroups = 32, kMsSmallStageGroups = 16;  // K-groups per ring stage, where three of 32 fit and else
constexpr int kMsMaxStages = 6, kMsMinStages = 3;
constexpr int kMsMaxProblems = 4;
constexpr int kMsMaxCluster = 8;
constexpr int kMsActRowBytes = 32;            // per activation row and K-group: 16 + 16 bytes of int8
constexpr int kMsMaxM = 192, kMsNamedMaxM = 64;  // of a launch; of kernel 7 by name and by default
constexpr int kMsMaxTiles = 4;                // tiles of 8 rows that a CTA multiplies a cell with
constexpr int kMsRedCol = 36;                 // floats per column of a panel's sums (32 rows; 36 keep the stores free of bank conflicts)
constexpr size_t kMsSmemMax = 227 * 1024;
// Asked for at least: more than half of an SM's 228 KB, so that an SM holds one CTA.  A launch has at most one CTA an SM to give; where two
// fit (one tile of rows, K below 4064), those of a dependent launch go two by two to the SMs that the launch before it leaves first, and
// others stay idle.  us, M = 8, two CTAs an SM / one: chain of dependent launches 1536 -> 1536 4.71 / 4.34, 1536 -> 17920 10.3 / 8.6,
// 3584 -> 18944 17.9 / 13.5 (twice that N in a group 31.7 / 22.7), ordinary launches 5.73 / 5.72, 11.5 / 10.5, 19.7 / 15.3.
constexpr size_t kMsSmemMin = 114 * 1024;

struct MsProblem {
  const uint8_t* tiled;  // TiledHeader at offset 0
  float* y;
  int n, ldy, panel_begin;  // first panel of the launch
  size_t zsum_off, bias_off;
};
struct MsParams {
  const uint8_t* acts;   // per block of rows: [num_groups][ rows x 16 (low words) | rows x 16 (high words) ]
  const float2* a_hdr;   // [m] {lhs_scale, a_off bits}
  int m, m_pad, k, num_groups;
  int num_blocks;  // blocks of 8 NT rows (the last may have fewer)
  int cluster_size, num_clusters, total_panels, num_problems, stages, one_unit, use_pdl;  // one_unit: no cluster has more than one panel
  MsProblem prob[kMsMaxProblems];
};

struct MsSmem {
  size_t bars, hdr, flags, acts, ring, red, psum, total;
};
__host__ __device__ inline MsSmem ms_smem_layout(int rows, int groups_per_rank, int cluster_size, int stages, int stage_groups) {
  MsSmem L;
  size_t off = 0;
  L.bars = off;
  off += 256;  // full[6], empty[6], act, peer_full[2], peer_free[2], red_full, red_free
  L.hdr = off;
  off += (size_t)rows * 8;
  L.flags = off;
  off += 32;
  L.acts = off;
  off += (size_t)groups_per_rank * rows * kMsActRowBytes;
  off = (off + 127) & ~(size_t)127;
  L.ring = off;
  off += (size_t)stages * stage_groups * kCellBytes;
  L.red = off;
  off += (size_t)kMsCWarps * rows * kMsRedCol * 4;
  L.psum = off;
  if (cluster_size > 1) off += (size_t)2 * rows * 32 * 4;
  L.total = off;
  return L;
}

__device__ __forceinline__ void ms_ldsm4(uint32_t (&v)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(a));
}
__device__ __forceinline__ void ms_ldsm2(uint32_t& v0, uint32_t& v1, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(v0), "=r"(v1) : "r"(a));
}
__device__ __forceinline__ uint32_t ms_lds16(uint32_t a) {
  uint32_t v;
  asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 ms_ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// arrive on the same-named mbarrier of CTA `rank`; orders this CTA's earlier writes before it at cluster scope
__device__ __forceinline__ void ms_mbar_arrive_remote(uint64_t* local_bar, uint32_t rank) {
  const uint32_t addr = map_to_cta(local_bar, rank);
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ bool ms_mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool ms_mbar_wait_cluster_bounded(uint64_t* bar, uint32_t parity) {
  if (ms_mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  while (!ms_mbar_try_wait_cluster(bar, parity)) {
    if (clock64() - t0 > (1ll << 31)) {
      atomicOr(&g_device_status, kDevStatusTimeout);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ uint64_t ms_pack(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ void ms_unpack(uint64_t v, uint32_t& lo, uint32_t& hi) { asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t ms_add2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ void ms_fma2(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
constexpr uint32_t kMsMagic = 0x49400000u;                      // 786432.0f
constexpr uint64_t kMsMinusMagic2 = 0xC9400000C9400000ull;      // -786432.0f twice
// D (s32, 16 x 8) = A (s8, 16 x 32, row-major) * B (s8, 32 x 8, column-major) + c (the bits of 786432.0f)
__device__ __forceinline__ void ms_mma_s8(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const uint32_t (&c)[4]) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

// NT: 8-column tiles of a block of the batch; SG: K-groups of a ring stage
template <int NT, int SG>
__global__ void __launch_bounds__(kMsThreads, 1) w4a32_gemm_stream_kernel(const __grid_constant__ MsParams p) {
  constexpr int KS = kMsCWarps, ROWS = NT * 8;  // (KS: warps that share the K-groups of a stage)
  extern __shared__ __align__(128) uint8_t ms_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = p.cluster_size, G = p.num_groups;
  const uint32_t rank = S > 1 ? cluster_ctarank() : 0u;
  // a cluster keeps one block of the batch's rows and walks panels
  const int cluster = (int)blockIdx.x / S, blk = cluster % p.num_blocks;
  const int first_row = blk * ROWS, n_tiles = min(NT, (p.m_pad >> 3) - blk * NT), rows = n_tiles * 8, m_here = min(rows, p.m - first_row);
  const int g_lo = (int)(((long long)rank * G) / S), g_hi = (int)(((long long)(rank + 1) * G) / S);
  const int ng = g_hi - g_lo;
  constexpr int kStageBytes = SG * kCellBytes;
  const int NST = p.stages, panel_step = p.num_clusters / p.num_blocks;
  const MsSmem Lo = ms_smem_layout(ROWS, (G + S - 1) / S, S, NST, SG);
  uint64_t* full = reinterpret_cast<uint64_t*>(ms_smem + Lo.bars);
  uint64_t* empty = full + kMsMaxStages;
  uint64_t* act_bar = empty + kMsMaxStages;
  uint64_t* peer_full = act_bar + 1;   // [2] rank 0: the other ranks' partial sums of a unit are in place
  uint64_t* peer_free = peer_full + 2; // [2] ranks 1..: rank 0 has read the slot
  uint64_t* red_full = peer_free + 2;  // the warps' sums of a unit are in place
  uint64_t* red_free = red_full + 1;   // ... and have been read
  float2* s_hdr = reinterpret_cast<float2*>(ms_smem + Lo.hdr);
  volatile int* flags = reinterpret_cast<volatile int*>(ms_smem + Lo.flags);  // bad header, -, start value, -, scale encodings
  uint8_t* acts = ms_smem + Lo.acts;
  uint8_t* ring = ms_smem + Lo.ring;
  float* red = reinterpret_cast<float*>(ms_smem + Lo.red);
  float* psum = reinterpret_cast<float*>(ms_smem + Lo.psum);
  const size_t group_bytes = (size_t)rows * kMsActRowBytes;
  const uint8_t* acts_from = p.acts + (size_t)G * first_row * kMsActRowBytes;

  if (p.use_pdl) pdl_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], kMsCWarps);
    }
    mbar_init(act_bar, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&peer_full[i], (uint32_t)max(S - 1, 1));
      mbar_init(&peer_free[i], 1);
    }
    mbar_init(red_full, kMsCWarps);
    mbar_init(red_free, kMsEWarps);
    mbar_fence_init();
    flags[2] = (int)kMsMagic;
  }
  if (warp == 1) {
    // tile headers: checked before a single byte of a matrix is requested
    int bad = 0;
    if (lane < p.num_problems) {
      const uint4* at = reinterpret_cast<const uint4*>(p.prob[lane].tiled);
      const uint4 h = at[0], h2 = at[1];  // magic, version, n, k; groups, panels, scale mode, bias
      bad = h.x != kTiledMagic || h.z != (uint32_t)p.prob[lane].n || h.w != (uint32_t)p.k;
      flags[4 + lane] = h2.z == 2u;
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
      if (bad) atomicOr(&g_device_status, kDevStatusBadHeader);
      flags[0] = bad;  // 1: nothing is done
    }
  }
  __syncthreads();
  if (S > 1) cluster_sync_all();  // every CTA of the cluster runs and has its barriers initialised
  const bool run = flags[0] == 0;
  const int first_panel = run ? cluster / p.num_blocks : p.total_panels;

  auto problem_of = [&](int u) {
    int pi = 0;
#pragma unroll
    for (int i = 1; i < kMsMaxProblems; ++i)
      if (i < p.num_problems && u >= p.prob[i].panel_begin) pi = i;
    return pi;
  };

  // A unit's outputs from the warps' sums, by THREADS threads (t: this one's number; a multiple of 8, so a thread's tasks are
  // the same 4 rows of the panel in different columns).  sums: waits for them; read: they may be overwritten.
  auto finish = [&](auto threads, int t, int u, int unit_index, bool& ok, auto sums, auto read) {
    constexpr int THREADS = decltype(threads)::value, TRIPS = (ROWS * 8 + THREADS - 1) / THREADS;
    const MsProblem& pr = p.prob[problem_of(u)];
    // the rows' constants are requested now and used behind the unit
    const int n = (u - pr.panel_begin) * kPanelRows + 4 * (t & 7), n_end = pr.n, ldy = pr.ldy;
    float* const y = pr.y + n + (size_t)first_row * ldy;
    float4 zs = make_float4(0.0f, 0.0f, 0.0f, 0.0f), bs = zs;
    if (rank == 0) {
      zs = *reinterpret_cast<const float4*>(pr.tiled + pr.zsum_off + (size_t)n * 4);
      bs = *reinterpret_cast<const float4*>(pr.tiled + pr.bias_off + (size_t)n * 4);
    }
    const int buf = unit_index & 1;
    ok = sums() && ok;
    float4 v[TRIPS];
#pragma unroll
    for (int i = 0; i < TRIPS; ++i) {
      const int col = (t + i * THREADS) >> 3;
      if (col < m_here) {
        const float* from = red + (size_t)col * kMsRedCol + 4 * (t & 7);
        float4 o[KS];
#pragma unroll
        for (int r = 0; r < KS; ++r) o[r] = *reinterpret_cast<const float4*>(from + (size_t)r * ROWS * kMsRedCol);
#pragma unroll
        for (int d = 1; d < KS; d *= 2)  // pairs, pairs of pairs ..: less rounding than one after the other
#pragma unroll
          for (int r = 0; r < KS; r += 2 * d) o[r].x += o[r + d].x, o[r].y += o[r + d].y, o[r].z += o[r + d].z, o[r].w += o[r + d].w;
        v[i] = o[0];
      }
    }
    read();
    // ranks 1..: the slot written two units ago must have been read by rank 0
    if (S > 1 && rank != 0 && unit_index >= 2 && ok)
      ok = ms_mbar_wait_cluster_bounded(&peer_free[buf], (uint32_t)((unit_index >> 1) - 1) & 1u);
    if (S > 1 && rank == 0 && ok) ok = ms_mbar_wait_cluster_bounded(&peer_full[buf], (uint32_t)(unit_index >> 1) & 1u);
#pragma unroll
    for (int i = 0; i < TRIPS; ++i) {
      const int col = (t + i * THREADS) >> 3;
      if (col < m_here) {
        float* slot = psum + ((size_t)(buf * ROWS + col) * 8 + (t & 7)) * 4;
        if (S > 1 && rank != 0) *reinterpret_cast<float4*>(slot) = v[i];
        else if (ok) {
          for (uint32_t r = 1; r < (uint32_t)S; ++r) {
            const float4 o = ms_ld_cluster_f32x4(map_to_cta(slot, r));
            v[i].x += o.x, v[i].y += o.y, v[i].z += o.z, v[i].w += o.w;
          }
          const float2 hc = s_hdr[col];
          const float off = (float)__float_as_int(hc.y);
          v[i].x = clamp_flt_max(fmaf(fmaf(off, zs.x, v[i].x), hc.x, bs.x));
          v[i].y = clamp_flt_max(fmaf(fmaf(off, zs.y, v[i].y), hc.x, bs.y));
          v[i].z = clamp_flt_max(fmaf(fmaf(off, zs.z, v[i].z), hc.x, bs.z));
          v[i].w = clamp_flt_max(fmaf(fmaf(off, zs.w, v[i].w), hc.x, bs.w));
          float* to = y + (size_t)col * ldy;
          if (n + 4 <= n_end && (reinterpret_cast<uintptr_t>(to) & 15u) == 0) *reinterpret_cast<float4*>(to) = v[i];
          else {
            if (n < n_end) to[0] = v[i].x;
            if (n + 1 < n_end) to[1] = v[i].y;
            if (n + 2 < n_end) to[2] = v[i].z;
            if (n + 3 < n_end) to[3] = v[i].w;
          }
        }
      }
    }
    if (S > 1) {
      asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
      if (t == 0) {
        if (rank != 0) ms_mbar_arrive_remote(&peer_full[buf], 0);  // our partial sums of this unit are in place
        else
          for (uint32_t r = 1; r < (uint32_t)S; ++r) ms_mbar_arrive_remote(&peer_free[buf], r);
      }
    }
  };

  if (warp == kMsCWarps) {
    // =============================== producer warp (one lane) ===============================
    if (lane == 0 && ng > 0) {
      const uint64_t stream_once = l2_policy_evict_first();
      int st = 0, issued = 0;
      uint32_t ph = 0;
      bool acts_requested = false;
      auto request_acts = [&] {
        if (p.use_pdl) pdl_wait_prior();  // the activation blocks come from the kernel before this one
        const uint32_t bytes = (uint32_t)((size_t)ng * group_bytes);
        mbar_arrive_expect_tx(act_bar, bytes);
        bulk_g2s(acts, acts_from + (size_t)g_lo * group_bytes, bytes, act_bar);
        acts_requested = true;
      };
      bool ok = true;
      for (int u = first_panel; u < p.total_panels && ok; u += panel_step) {
        const MsProblem& pr = p.prob[problem_of(u)];
        const uint8_t* cells = pr.tiled + sizeof(TiledHeader) + (size_t)(u - pr.panel_begin) * G * kCellBytes;
        for (int b = g_lo; b < g_hi; b += SG) {
          if (issued == NST && !acts_requested) request_acts();  // the ring is full of weights: now the activations
          if (issued >= NST) {
            if (!mbar_wait_bounded(&empty[st], ph ^ 1u)) {
              ok = false;
              break;
            }
          }
          const uint32_t bytes = (uint32_t)(min(SG, g_hi - b) * kCellBytes);
          mbar_arrive_expect_tx(&full[st], bytes);
          bulk_g2s_hint(ring + (size_t)st * kStageBytes, cells + (size_t)b * kCellBytes, bytes, &full[st], stream_once);
          ++issued;
          if (++st == NST) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      if (!acts_requested && run) request_acts();
    }
    __syncwarp();
  } else if (warp < kMsCWarps) {
    // =============================== compute warps ===============================
    const int ks = warp, g8 = lane >> 2;
    bool ok = true;
    if (p.one_unit) {  // these warps write the outputs themselves
      if (p.use_pdl) pdl_wait_prior();
      for (int i = tid; i < m_here; i += kMsCWarps * 32) s_hdr[i] = p.a_hdr[first_row + i];
    }
    const uint32_t ring_s = smem_u32(ring), acts_s = smem_u32(acts), red_s = smem_u32(red);
    // matrices of an ldmatrix.x4 of the activations: low and high words of tile t, low and high words of tile t + 1
    const uint32_t b_lane = (uint32_t)(((lane >> 4) * 8 + (lane & 7)) * 16 + ((lane >> 3) & 1) * rows * 16);

    uint64_t acc[2][NT][2];  // pairs of columns: [half][tile][row g8, row g8 + 8]
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[h][t][0] = acc[h][t][1] = 0ull;
    // the start value of a product, in registers of which the compiler does not know the value: as a constant it would be
    // written into four registers anew for every product
    uint32_t magic[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) magic[i] = (uint32_t)flags[2];

    int st = 0, unit_index = 0;
    uint32_t ph = 0;
    for (int u = first_panel; u < p.total_panels; u += panel_step, ++unit_index) {
      const bool f16 = flags[4 + problem_of(u)] != 0;
      for (int b = g_lo; b < g_hi && ok; b += SG) {
        if (unit_index == 0 && b == g_lo) ok = mbar_wait_bounded(act_bar, 0);
        if (!ok || !mbar_wait_bounded(&full[st], ph)) {
          ok = false;
          break;
        }
        const int cnt = min(SG, g_hi - b);
        // Two cells per trip (K-groups j and j + KS of the stage), their loads and tensor-core products interleaved:
        // with two warps per scheduler the dependent chain of a single cell would leave the pipes idle.
        for (int j = ks; j < cnt; j += 2 * KS) {
          const bool two = j + KS < cnt;
          uint32_t cell[2], act[2];
          cell[0] = ring_s + (uint32_t)st * kStageBytes + (uint32_t)j * kCellBytes;
          cell[1] = two ? cell[0] + (uint32_t)KS * kCellBytes : cell[0];
          act[0] = acts_s + (uint32_t)(b - g_lo + j) * (uint32_t)group_bytes;
          act[1] = two ? act[0] + (uint32_t)KS * (uint32_t)group_bytes : act[0];
          // weights: rows g8, g8 + 8 of either 16-row half; 4 bytes = 8 nibbles = k {4 c4 .. 4 c4 + 3} low and high
          uint32_t w[2][4], v[2][4], x[2][NT > 2 ? 2 : 1][4];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            ms_ldsm4(w[c], cell[c] + (uint32_t)lane * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[c][i] = ms_lds16(cell[c] + kCellNibbleBytes + (uint32_t)(g8 + 8 * i) * 2);
            // (what lies behind the last tile of an odd number of them - bytes of the next group or of the ring - is not used)
#pragma unroll
            for (int t = 0; t < NT; t += 2) {
              if (NT > 1) ms_ldsm4(x[c][t / 2], act[c] + b_lane + (uint32_t)t * 128);
              else ms_ldsm2(x[c][0][0], x[c][0][1], act[c] + b_lane);
            }
          }
          if (f16) {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 4; ++i) v[c][i] = __float_as_uint(__half2float(__ushort_as_half((unsigned short)v[c][i])));
          } else {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 4; ++i) v[c][i] <<= 16;
          }
          uint64_t sc[2][4];
          uint32_t a[2][2][4];
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (c == 1 && !two) v[c][i] = 0u;  // the second cell of an odd trip repeats the first with scale 0
              sc[c][i] = ms_pack(v[c][i], v[c][i]);
              a[c][i >> 1][i & 1] = ((w[c][i] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
              a[c][i >> 1][2 + (i & 1)] = (w[c][i] & 0xF0F0F0F0u) ^ 0x80808080u;
            }
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            if (t < n_tiles) {
              uint32_t d[2][2][4];
#pragma unroll
              for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 2; ++c) ms_mma_s8(d[c][h], a[c][h], x[c][t / 2][2 * (t & 1)], x[c][t / 2][2 * (t & 1) + 1], magic);
#pragma unroll
              for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                  for (int i = 0; i < 2; ++i)
                    ms_fma2(acc[h][t][i], ms_add2(ms_pack(d[c][h][2 * i], d[c][h][2 * i + 1]), kMsMinusMagic2), sc[c][2 * h + i]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
        if (++st == NST) {
          st = 0;
          ph ^= 1u;
        }
      }
      // ---- end of the unit: the K-slices of the warps meet in shared memory, [slice][column][row].  Where more units follow,
      // the epilogue warps add them while this warp goes on.
      if (ok && unit_index > 0) ok = mbar_wait_bounded(red_free, (uint32_t)(unit_index - 1) & 1u);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          if (t < n_tiles) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t v0, v1;  // columns 8 t + 2 (lane % 4) (+ 1) of row 16 h + 8 i + g8
              ms_unpack(acc[h][t][i], v0, v1);
              const uint32_t at = red_s + (uint32_t)((ks * ROWS + 8 * t + 2 * (lane & 3)) * kMsRedCol + 16 * h + 8 * i + g8) * 4;
              asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v0) : "memory");
              asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + kMsRedCol * 4), "r"(v1) : "memory");
            }
          }
          acc[h][t][0] = acc[h][t][1] = 0ull;
        }
      if (p.one_unit) {
        finish(std::integral_constant<int, kMsCWarps * 32>(), tid, u, 0, ok,
               [] {
                 asm volatile("bar.sync 1, %0;" ::"n"(kMsCWarps * 32) : "memory");
                 return true;
               },
               [] {});
        break;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(red_full);
      if (!ok) break;
    }
  } else {
    // =============================== epilogue warps ===============================
    constexpr int kEThreads = kMsEWarps * 32;
    const int et = tid - (kMsCWarps + 1) * 32;
    bool ok = true;
    if (!p.one_unit) {
      if (p.use_pdl) pdl_wait_prior();
      for (int i = et; i < m_here; i += kEThreads) s_hdr[i] = p.a_hdr[first_row + i];
      asm volatile("bar.sync 1, %0;" ::"n"(kEThreads) : "memory");
      int unit_index = 0;
      for (int u = first_panel; u < p.total_panels; u += panel_step, ++unit_index)  // (to the end also when a wait ran out: the barriers)
        finish(std::integral_constant<int, kEThreads>(), et, u, unit_index, ok, [&] { return ok && mbar_wait_bounded(red_full, (uint32_t)unit_index & 1u); },
               [&] {
                 __syncwarp();
                 if (lane == 0) mbar_arrive(red_free);
               });
    }
  }
  // Leave together: ranks 1.. hold partial sums that rank 0 reads, rank 0 holds the barriers they arrive on.
  __syncthreads();
  if (S > 1) cluster_sync_all();
}

// Rows of x are cut into blocks of at most four tiles of 8, as even as that goes
static int ms_block_tiles(int m) {
  const int tiles = (m + 7) / 8, blocks = (tiles + kMsMaxTiles - 1) / kMsMaxTiles;
  return (tiles + blocks - 1) / blocks;
}

int w4a32_gemm_stream_block_rows(int m) { return ms_block_tiles(m) * 8; }

// ------------------------------------------------------------------------------------------------ activations
// Per-row int8 quantization (the arithmetic of act_quant_records_kernel) into the layout above: for K-group g
// and row m the four low words (even k of each 8-value item) at [g][m][0..16), the four high words (odd k) at
// [g][rows + m] of its block of rows.  One CTA per row of the padded batch; padding rows are zeros.  A thread keeps its ITEMS items of 8
// values in registers between minimum / maximum and quantization (all loads in flight at once).  Rows that are longer (ITEMS 0) or not
// 16-byte aligned are read twice, the former 16 bytes at a time: 14336 -> 4096 with its quantization, us, single floats / so,
// M = 8 18.0 / 17.0, 16 24.4 / 24.0, 32 30.9 / 28.9, 56 49.5 / 47.9.  (An instance of its own: in the one for up to 12288 values the
// branch costs 0.1 us at K = 8960.)
constexpr int kMsQuantThreads = 512;
template <int ITEMS>
__global__ void __launch_bounds__(kMsQuantThreads) act_quant_mma_kernel(const float* __restrict__ x, int m_total, int m_pad, int block_rows,
                                                                        int k, int ldx, int num_groups,
                                                                        uint8_t* __restrict__ acts, float2* __restrict__ hdr) {
  __shared__ float scratch[64];
  pdl_launch_dependents();  // the GEMM behind this kernel is always a dependent launch
  pdl_wait_prior();  // x may be the previous kernel's output, and that kernel may still read the blocks we overwrite
  const int m = blockIdx.x, tid = threadIdx.x;
  const bool live = m < m_total;
  const float* row = x + (size_t)(live ? m : 0) * ldx;
  const int num_items = num_groups * 4;
  const int first = m / block_rows * block_rows, rows = min(block_rows, m_pad - first);  // the block that holds this row
  acts += (size_t)num_groups * first * kMsActRowBytes + (size_t)(m - first) * 16;
  auto store = [&](int item, uint32_t lo, uint32_t hi) {
    const int g = item >> 2, i = item & 3;
    uint8_t* at = acts + (size_t)g * rows * kMsActRowBytes;
    reinterpret_cast<uint32_t*>(at)[i] = lo;
    reinterpret_cast<uint32_t*>(at + (size_t)rows * 16)[i] = hi;
  };
  if (!live) {
    for (int item = tid; item < num_items; item += kMsQuantThreads) store(item, 0u, 0u);
    return;
  }
  auto value = [&](int at) { return at < k ? row[at] : 0.0f; };
  const bool aligned = (reinterpret_cast<uintptr_t>(row) & 15u) == 0, keep = ITEMS > 0 && aligned;
  float v[ITEMS > 0 ? ITEMS : 1][8];
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
  if (keep) {
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int k0 = (tid + j * kMsQuantThreads) * 8;
      if (k0 + 8 <= k) {
        const float4 a = *reinterpret_cast<const float4*>(row + k0);
        const float4 b = *reinterpret_cast<const float4*>(row + k0 + 4);
        v[j][0] = a.x, v[j][1] = a.y, v[j][2] = a.z, v[j][3] = a.w;
        v[j][4] = b.x, v[j][5] = b.y, v[j][6] = b.z, v[j][7] = b.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j][i] = value(k0 + i);
      }
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int k0 = (tid + j * kMsQuantThreads) * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (k0 + i < k) {
          mn = fminf(mn, v[j][i]);
          mx = fmaxf(mx, v[j][i]);
        }
    }
    const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
      scratch[warp] = mn;
      scratch[32 + warp] = mx;
    }
    __syncthreads();
    mn = scratch[lane & 15];
    mx = scratch[32 + (lane & 15)];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
  } else {
    block_row_minmax(row, k, scratch, mn, mx);
  }
  const ActQuantParams qp = act_quant_params(mn, mx);
  if (tid == 0) hdr[m] = make_float2(qp.recip_scale, __int_as_float(-qp.nzp));
  auto emit = [&](int item, const float (&f)[8]) {
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = item * 8 + i < k ? (uint32_t)act_quant_value(f[i], qp) & 0xFFu : 0u;
      if (i & 1) hi |= q << (4 * (i - 1));
      else lo |= q << (4 * i);
    }
    store(item, lo, hi);
  };
  if (keep) {
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (tid + j * kMsQuantThreads < num_items) emit(tid + j * kMsQuantThreads, v[j]);
  } else {
    for (int item = tid; item < num_items; item += kMsQuantThreads) {
      float f[8];
      if (ITEMS == 0 && aligned && item * 8 + 8 <= k) {
        const float4 a = *reinterpret_cast<const float4*>(row + item * 8), b = *reinterpret_cast<const float4*>(row + item * 8 + 4);
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
        f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = value(item * 8 + i);
      }
      emit(item, f);
    }
  }
}

// ------------------------------------------------------------------------------------------------ host side
struct MsPlan {
  int m_pad, block_tiles, num_blocks, cluster_size, groups_per_rank, stages, stage_groups, total_panels;
};

template <int NT, int SG>
static cudaError_t ms_configure() {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < 64 && configured[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(w4a32_gemm_stream_kernel<NT, SG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMsSmemMax);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < 64) configured[dev] = true;
  return cudaSuccess;
}

// clusters of `s` CTAs of this kernel that the current device runs at once (148 / s without a device)
template <int NT, int SG>
static int ms_cluster_capacity(int s, size_t smem) {
  if (s <= 1) return 148;
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(s * 148), 1, 1);
  cfg.blockDim = dim3(kMsThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)s;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (ms_configure<NT, SG>() != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, w4a32_gemm_stream_kernel<NT, SG>, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    n = 148 / s;
  }
  return n;
}

// Nothing here but the number of panels depends on N: a matrix has the same bits whether it is launched alone or grouped.
// The limit of K is that of 36 bytes per row and group (as workspaces are sized) in eight shares of 112 KB.
// The smallest cluster whose shared memory holds the activations, a power of two (us, 8960 -> 1536, M = 16, an earlier form of
// the kernel: sizes 2 / 3 / 4 / 5 10.4 / 15.4 / 13.0 / 13.3); two from K = 4480 on, where one CTA would walk a unit for longer
// than the exchange takes (8960 -> 1536, M = 16: 12.7 alone, 10.1; 4864 -> 896, M = 24: 9.8, 8.7), but for a single tile of
// rows (8192 -> 28672, M = 8: 46 alone, 60).
static bool ms_shape_plan(int m, int k, int count, const int* n, MsPlan* plan) {
  if (m < 1 || m > kMsMaxM || count < 1 || count > kMsMaxProblems || k < 1) return false;
  const int G = (k + kGroup - 1) / kGroup;
  plan->m_pad = (m + 7) / 8 * 8;
  plan->block_tiles = ms_block_tiles(m);
  plan->num_blocks = (plan->m_pad / 8 + plan->block_tiles - 1) / plan->block_tiles;
  if (m <= kMsNamedMaxM && (size_t)((G + kMsMaxCluster - 1) / kMsMaxCluster) * plan->m_pad * 36 > 112 * 1024) return false;
  plan->stages = 0;
  for (int s = G >= 140 && plan->m_pad > 8 ? 2 : 1; s <= kMsMaxCluster && plan->stages == 0; s *= 2) {
    plan->cluster_size = s;
    plan->groups_per_rank = (G + s - 1) / s;
    const auto fits = [&](int stages, int groups) { return ms_smem_layout(plan->block_tiles * 8, plan->groups_per_rank, s, stages, groups).total <= kMsSmemMax; };
    if (!fits(kMsMinStages, kMsSmallStageGroups)) continue;
    plan->stages = kMsMinStages;
    plan->stage_groups = fits(kMsMinStages, kMsStageGroups) ? kMsStageGroups : kMsSmallStageGroups;
    while (plan->stages < (plan->stage_groups == kMsStageGroups ? 4 : kMsMaxStages) && fits(plan->stages + 1, plan->stage_groups)) ++plan->stages;
  }
  long long panels = 0;
  for (int i = 0; i < count; ++i) {
    if (n[i] < 1) return false;
    panels += (n[i] + kPanelRows - 1) / kPanelRows;
  }
  if (panels >= (1ll << 30)) return false;
  plan->total_panels = (int)panels;
  return plan->stages != 0;
}

bool w4a32_gemm_stream_supported(int m, int k, int count, const int* n) {
  MsPlan plan;
  return m >= 1 && m <= kMsNamedMaxM && ms_shape_plan(m, k, count, n, &plan);
}

// Where the "fastest" policy (5) takes this kernel above 64 rows: matrices, or groups, of at most 4096 rows, whose 128-row tiles
// would leave most SMs of the tile GEMMs idle, up to 192 rows of x, in blocks of 32, and as long as a CTA has few K-groups to walk
// through: its time grows with those (0.03 to 0.05 us each), that of the tile GEMMs with K alone.  The lines lie where 243 timings below 128
// rows and 450 above cross (256 to 4096 weight rows, K = 896 to 14336): what is taken is at most 3% slower than the tile GEMM that policy
// took.  us with the quantization, that / this kernel: M = 65 (gemm_chunk.cu) 1536 -> 1536 13.3 / 7.8, 8960 -> 1536 50.1 / 19.6,
// 4864 -> 896 30.0 / 12.7; M = 127 14.7 / 9.2, 54.0 / 26.9, 32.1 / 14.3; M = 192 (gemm_tcf16.cu) 15.9 / 10.8, 33.7 / 33.1, 23.0 / 16.6, 2048 -> 3072
// 18.2 / 16.9; beyond the lines 896 -> 4096 12.8 / 15.4, 4096 -> 4096 23.3 / 33.1, 14336 -> 4096 51 / 119; M = 256 1536 -> 1536 16.8 / 13.5,
// 8960 -> 1536 35.2 / 43.5.  Error against 64 bits, the same: K = 8960 9.7e-8 / 6.9e-8 (M = 65) and 4.3e-7 / 6.9e-8 (M = 192), K = 1536
// 5.2e-8 / 5.1e-8 and 7.8e-8 / 5.2e-8, K = 896 4.3e-8 / 4.5e-8 and 9.5e-8 / 4.6e-8: short K below 128 rows stays where it was.
bool w4a32_gemm_stream_preferred(int m, int k, int count, const int* n) {
  MsPlan plan;
  if (m <= kMsNamedMaxM || (m < 128 && k < 1024) || !ms_shape_plan(m, k, count, n, &plan) || plan.total_panels > 4096 / kPanelRows) return false;
  const int G = (k + kGroup - 1) / kGroup, S = plan.cluster_size, per_block = std::max(1, 148 / S / plan.num_blocks);
  const int walk = (plan.total_panels + per_block - 1) / per_block * plan.groups_per_rank;
  if (m < 128) return walk <= 180 + 16 * G / 5;
  return walk <= (G < 32 ? 3 * G : S <= 2 ? 170 + 17 * G / 10 : 7 * G / 4);
}

// bytes of the activation blocks for m rows of k values (rows padded to a multiple of 8): 32 a row and K-group are written; workspaces, and
// the limit of K above, go by 36
size_t w4a32_gemm_stream_act_bytes(int m, int k) {
  return (size_t)((k + kGroup - 1) / kGroup) * (size_t)((m + 7) / 8 * 8) * 36;
}

cudaError_t launch_act_quant_mma(const float* x, int m, int k, int ldx, uint8_t* acts, float2* hdr, int use_pdl,
                                 cudaStream_t stream) {
  const int m_pad = (m + 7) / 8 * 8, num_groups = (k + kGroup - 1) / kGroup;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)m_pad, 1, 1);
  cfg.blockDim = dim3(kMsQuantThreads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  if (use_pdl) {
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
  const auto kernel = num_groups * 4 <= kMsQuantThreads       ? act_quant_mma_kernel<1>
                      : num_groups * 4 <= 3 * kMsQuantThreads ? act_quant_mma_kernel<3>
                                                              : act_quant_mma_kernel<0>;
  return cudaLaunchKernelEx(&cfg, kernel, x, m, m_pad, ms_block_tiles(m) * 8, k, ldx, num_groups, acts, hdr);
}

template <int NT, int SG>
static cudaError_t ms_launch_t(MsParams& prm, const MsPlan& plan, cudaStream_t stream) {
  cudaError_t e = ms_configure<NT, SG>();
  if (e != cudaSuccess) return e;
  const int S = plan.cluster_size;
  static int capacity[64][kMsMaxCluster + 1] = {};  // per device and cluster size (the largest shared-memory need is assumed)
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (capacity[dev][S] == 0) capacity[dev][S] = ms_cluster_capacity<NT, SG>(S, kMsSmemMax);
  const int per_block = std::max(1, std::min(capacity[dev][S], 148 / S) / plan.num_blocks);
  prm.num_clusters = std::min(per_block, plan.total_panels) * plan.num_blocks;
  prm.one_unit = plan.total_panels <= per_block;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(prm.num_clusters * S), 1, 1);
  cfg.blockDim = dim3(kMsThreads, 1, 1);
  cfg.dynamicSmemBytes = std::max(kMsSmemMin, ms_smem_layout(plan.block_tiles * 8, plan.groups_per_rank, S, plan.stages, plan.stage_groups).total);
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  if (S > 1) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = (unsigned)S;
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  if (prm.use_pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, w4a32_gemm_stream_kernel<NT, SG>, prm);
}

template <int NT>
static cudaError_t ms_launch_tiles(MsParams& prm, const MsPlan& plan, cudaStream_t stream) {
  return plan.stage_groups == kMsStageGroups ? ms_launch_t<NT, kMsStageGroups>(prm, plan, stream)
                                             : ms_launch_t<NT, kMsSmallStageGroups>(prm, plan, stream);
}

// acts / a_hdr: output of launch_act_quant_mma for the same m and k.  Up to four matrices that share them.
cudaError_t launch_w4a32_gemm_stream(const uint8_t* acts, const float2* a_hdr, int m, int k, int count,
                                     const void* const* tiled, float* const* y, const int* n, const int* ldy, int use_pdl,
                                     cudaStream_t stream) {
  MsPlan plan;
  if (!ms_shape_plan(m, k, count, n, &plan)) return cudaErrorInvalidValue;
  MsParams prm = {};
  prm.acts = acts;
  prm.a_hdr = a_hdr;
  prm.m = m;
  prm.m_pad = plan.m_pad;
  prm.k = k;
  prm.num_groups = (k + kGroup - 1) / kGroup;
  prm.cluster_size = plan.cluster_size;
  prm.num_blocks = plan.num_blocks;
  prm.stages = plan.stages;
  prm.total_panels = plan.total_panels;
  prm.num_problems = count;
  prm.use_pdl = use_pdl;
  int begin = 0;
  for (int i = 0; i < count; ++i) {
    const TiledHeader th = make_tiled_header(n[i], k, 0, 0);
    prm.prob[i].tiled = static_cast<const uint8_t*>(tiled[i]);
    prm.prob[i].y = y[i];
    prm.prob[i].n = n[i];
    prm.prob[i].ldy = ldy[i];
    prm.prob[i].panel_begin = begin;
    prm.prob[i].zsum_off = th.zsum_off;
    prm.prob[i].bias_off = th.bias_off;
    begin += (int)th.num_panels;
  }
  switch (plan.block_tiles) {
    case 1: return ms_launch_tiles<1>(prm, plan, stream);
    case 2: return ms_launch_tiles<2>(prm, plan, stream);
    case 3: return ms_launch_tiles<3>(prm, plan, stream);
    default: return ms_launch_tiles<4>(prm, plan, stream);
  }
}

}  // namespace mllmb200
