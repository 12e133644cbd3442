// The largest value of a row.
#pragma once
#include "bpdq_common.cuh"

namespace bpdq {

// By the 1024 threads of a CTA; the largest value wins, the lowest index among equals (v > best in index order).  Thread 0 holds the result.
__device__ __forceinline__ int argmax_of_row(const float* row, int n)
{
    __shared__ float s_v[32];
    __shared__ int s_i[32];
    float best = row[0];
    int bi = 0;
    auto better = [](float v, int k, float& bv, int& bk) {
        if (v > bv || (v == bv && k < bk)) { bv = v; bk = k; }
    };
    for (int k0 = threadIdx.x; k0 < n; k0 += 8 * 1024) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = k0 + 1024 * j < n ? row[k0 + 1024 * j] : row[0];
#pragma unroll
        for (int j = 0; j < 8; j++) better(v[j], k0 + 1024 * j < n ? k0 + 1024 * j : 0, best, bi);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        const int i = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        better(v, i, best, bi);
    }
    if ((threadIdx.x & 31) == 0) { s_v[threadIdx.x >> 5] = best; s_i[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x < 32) {
        best = s_v[threadIdx.x];
        bi = s_i[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            const int i = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
            better(v, i, best, bi);
        }
    }
    return bi;
}

}  // namespace bpdq
