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
// What one query's q/k/v products left: q is turned as it is read, the key turned and stored with the value in cache row *pos (beyond max_seq_len: nothing is
// stored, code 20 is recorded), by the steps of k_rope_qk_store_kv (llama_forward.cu).
struct GqaNew {
    const float *k, *v;         // [kv_heads][dim]
    const int32_t* pos;
    const float* freq_factors;  // or null
    int n_dims, max_seq_len;
    float theta_scale;
    int* err;
};
// The same as gqa_attention behind those steps, for one query; q is not written.  1, and nothing is launched, where the split kernel does not take it.
int gqa_attention_new(const GqaShape& p, const GqaNew& in, const float* q, void* k, void* v, float* dst, cudaStream_t s);
// Runs the product on one of this file's kernels, or returns 1 if the shape or the pointers are not theirs.
int gqa_attention(const GqaShape& p, const float* q, const void* k, const void* v, float* dst, cudaStream_t s);

}  // namespace bpdq
