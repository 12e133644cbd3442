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
// With `up`, X is a gate: the activations are silu(X) * up, formed as they are quantized.
int gemm_q8_0_wide(int n, const uint8_t* const* tiles, float* const* outs, const int* Ns, const float* X, int M, int K, cudaStream_t s,
                   Workspace* ws, const float* up = nullptr);

#ifdef __CUDACC__
// The reference's libm returns the correctly rounded fp32 value of expf / cosf / sinf for all but
// a fraction of a percent of arguments; the device's fp32 versions are 1-2 ulp off for about half of
// them.  Such last-bit differences are harmless by themselves, but every product that follows
// re-quantizes its input to int8, where a last-bit difference now and then flips a rounding and
// becomes a 1e-3 difference.  So the small steps between products evaluate in binary64 and round once.
__device__ __forceinline__ float exp_rounded(float x) { return (float)exp((double)x); }
__device__ __forceinline__ float cos_rounded(float x) { return (float)cos((double)x); }
__device__ __forceinline__ float sin_rounded(float x) { return (float)sin((double)x); }
// silu(g) * u, bench/bpd_cpu.c:5504-5507 of the reference
__device__ __forceinline__ float swiglu_rounded(float g, float u) { return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, exp_rounded(-g))), u); }
#endif

}  // namespace bpdq
