// Rotary angles and turns of the Llama (NORM pairing).
#pragma once
#include "q8_0_tiles.cuh"

namespace bpdq {

// theta is reached as the reference reaches it, by repeated multiplication from (float)pos, so that the angle has the same bits.
__device__ __forceinline__ void rope_angle(int pair, int pos, const float* __restrict__ freq_factors, float theta_scale, float& c, float& s)
{
    float theta = (float)pos;
    for (int i = 0; i < pair; i++) theta = __fmul_rn(theta, theta_scale);
    const float ff = freq_factors ? freq_factors[pair] : 1.0f;
    const float te = __fdiv_rn(theta, ff);
    c = cos_rounded(te);
    s = sin_rounded(te);
}
// The cosine alone, or the sine.
__device__ __forceinline__ void rope_angle(int pair, int pos, const float* __restrict__ freq_factors, float theta_scale, bool cosine, float& c, float& s)
{
    float theta = (float)pos;
    for (int i = 0; i < pair; i++) theta = __fmul_rn(theta, theta_scale);
    const float ff = freq_factors ? freq_factors[pair] : 1.0f;
    const float te = __fdiv_rn(theta, ff);
    if (cosine) c = cos_rounded(te);
    else s = sin_rounded(te);
}
__device__ __forceinline__ void rope_turn(float x0, float x1, float c, float s, float& y0, float& y1)
{
    y0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
    y1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
}

}  // namespace bpdq
