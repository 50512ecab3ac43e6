// Tensor maps and launch attributes shared by the files with tcgen05 kernels (defined in chunkwise_sm100.cu).
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace mlstm {

// token tensors (q, k, v, deltaH, and the gradients): one slab of S rows per (batch, head), so that a box hanging over the
// end of a sequence (ragged last chunk) reads zeros instead of the next head's tokens, and a store is clipped there
bool tok_map(CUtensorMap* m, const void* base, const ChunkwiseDims& d, int cols, int box_rows = 128);
// per-chunk states: one slab of DHQK x DHHV per (batch, head, chunk boundary), so that a tile hanging over the edge of
// a head dim reads zeros (and is clipped on the way out) instead of touching the next slab
bool state_map(CUtensorMap* m, const void* base, const ChunkwiseDims& d, int box_rows);

// cudaFuncSetAttribute once per kernel and device instead of on every call
template <typename K>
int set_smem_once(K kern, int bytes, bool (&done)[64]) {
  int dev = 0;
  MLSTM_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !done[dev]) {
    MLSTM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  return MLSTM_OK;
}

}  // namespace mlstm
