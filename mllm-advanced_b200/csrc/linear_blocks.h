// How a W4A32 linear of more than four rows wants its activations: quantized into the operand blocks of the kernel that will run.
// The entry points quantize x themselves; an operator that produces x may write the blocks instead (decoder_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mllmb200 {

enum W4Form : int {
  kW4None = 0,  // no blocks: the linear takes x itself
  kW4Stream,    // int8 words, gemm_stream.cu
  kW4Tile,      // fp16 blocks, gemm_tcf16.cu (its K-split counters are cleared by whoever writes the blocks)
  kW4Chunk,     // fp16 blocks, gemm_chunk.cu
};
struct W4Blocks {
  int form;
  int m_pad;       // rows of the blocks, a multiple of 8; rows behind x are zeros
  int block_rows;  // kW4Stream: rows of a block of its layout
  uint8_t* blocks;
  float2* hdr;     // [m] {row scale, zero-point offset}
  int* clear;
  int clear_count;
};

// What linear_forward_ex (count 1) or linear_forward_grouped with policy 0 or 5 (and the flag of fp16-encoded scales) runs for these
// shapes, with its places in a workspace of workspace_size(M, K) bytes.
W4Blocks w4a32_blocks_for(int M, int K, int count, const int* N, int policy_and_flags, void* ws);
// The places of kernel 4 by name (gemm_tcf16.cu).
W4Blocks w4a32_tile_blocks(int M, int K, int N, void* ws);
// The launch behind the blocks.
cudaError_t w4a32_forward_blocks(const W4Blocks& b, int M, int K, int count, const void* const* tiled, float* const* y, const int* N,
                                 const int* ldy, int use_pdl, cudaStream_t stream);

}  // namespace mllmb200
