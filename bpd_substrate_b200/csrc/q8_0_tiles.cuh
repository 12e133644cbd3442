// Q8_0 weights re-tiled for tcgen05 (the layout is described in gemm_q8_0_tiles.cu) and the products on them.
#pragma once
#include "bpdq_common.cuh"

namespace bpdq {

constexpr int kTileRows = 128;
constexpr int kTileQuants = kTileRows * 32;              // 4096
constexpr int kTileUnit = kTileRows * BPDQ_Q80_BYTES;    // 4352

// gemm_q8_0_wide.cu: up to three matrices that read the same activations.  kWideRefused: nothing was launched, the caller goes to
// the narrow kernel (few tokens, scratch that holds only the narrow kernel's activations).
constexpr int kWideMatrices = 3, kWideRefused = 1, kWideMinTokens = 17;
int gemm_q8_0_wide(int n, const uint8_t* const* tiles, float* const* outs, const int* Ns, const float* X, int M, int K, cudaStream_t s,
                   Workspace* ws);

}  // namespace bpdq
