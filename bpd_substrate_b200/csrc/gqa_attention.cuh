// Grouped-query attention of the Q8_0 Llama over contexts longer than a few keys (gqa_attention.cu).
#pragma once
#include "bpdq_common.cuh"

namespace bpdq {

struct GqaShape {
    int n_q, n_kv, heads, kv_heads, dim;
    float scale;
    int kv_offset;      // query t stands at kv_offset + t and sees keys 0 .. kv_offset + t, below n_kv
    int f16;            // caches are fp16 (else fp32)
};
// Runs the product on one of this file's kernels, or returns 1 if the shape or the pointers are not theirs.
int gqa_attention(const GqaShape& p, const float* q, const void* k, const void* v, float* dst, cudaStream_t s);

}  // namespace bpdq
