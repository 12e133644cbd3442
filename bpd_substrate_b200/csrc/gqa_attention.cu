// Grouped-query attention of the Q8_0 Llama (bench/bpd_cpu.c:5370-5433 of the reference) for contexts of more than kShortKeys
// keys; shorter ones, and short prompts of unshared fp32 heads, stay on k_gqa_attn (llama_forward.cu), which adds in the reference's order.
//
//   k_gqa_split   a few queries: keys dealt to the CTAs of a cluster, fp32 multiply-adds, parts joined through distributed
//                 shared memory (no scratch memory, so a call can be captured without a warm-up)
//   k_gqa_tile    prompts on fp16 caches: tiles of 64 (token, head) rows x 64 keys on mma.sync, fp32 operands as the sum of two
//                 fp16 numbers
//
// Both read a key head's rows once for all query heads that share it and hold scores, weights and sums in fp32.
#include "gqa_attention.cuh"
#include "cluster_device.cuh"
#include "gqa_split.h"
#include "launch.cuh"
#include "mma_device.cuh"
#include "rope_device.cuh"
#include "../../include/bpdq.h"

#include <cuda_fp16.h>

namespace bpdq {

constexpr int kShortKeys = 64;
constexpr float kLowest = -1e38f;      // where the reference's running maximum starts

// exp(x) for x <= 0: argument reduction in two steps (Cody and Waite), then the Taylor polynomial of degree 7 on |r| <= ln(2)/2
// (remainder 5e-9).  Below -87 it is 0 (the smallest normal number is exp(-87.3)).  NaN stays NaN.
__device__ __forceinline__ float exp_below(float x)
{
    const float t = fmaf(x, 1.44269504088896341f, 12582912.0f);      // the integer part sits in t's low bits
    const float n = t - 12582912.0f;
    float r = fmaf(n, -0.693359375f, x);
    r = fmaf(n, 2.12194440e-4f, r);
    float p = 1.0f / 5040.0f;
    p = fmaf(p, r, 1.0f / 720.0f);
    p = fmaf(p, r, 1.0f / 120.0f);
    p = fmaf(p, r, 1.0f / 24.0f);
    p = fmaf(p, r, 1.0f / 6.0f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    const float e = __int_as_float(__float_as_int(p) + (__float_as_int(t) << 23));
    return x >= -87.0f ? e : (x < -87.0f ? 0.0f : x);
}

// ------------------------------------------------------------------ a few queries

// Sums NV values over groups of 2 M neighbouring lanes, halving what a lane holds at every step while it holds more than one:
// lane l ends with the sums of values first(l), first(l) + 1, ...
template <int NV, int M, int N>
__device__ __forceinline__ void sum_over_lanes(float (&v)[N], int lane)
{
    if constexpr (M > 0) {
        if constexpr (NV > 1) {
            const bool up = lane & M;
#pragma unroll
            for (int i = 0; i < NV / 2; i++) {
                const float give = up ? v[i] : v[i + NV / 2], keep = up ? v[i + NV / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, M);
            }
            sum_over_lanes<NV / 2, M / 2>(v, lane);
        } else {
            v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], M);
            sum_over_lanes<1, M / 2>(v, lane);
        }
    }
}
template <int NV, int M>
__device__ __forceinline__ int first_of_lane(int lane)
{
    if constexpr (M > 0 && NV > 1) return ((lane & M) ? NV / 2 : 0) + first_of_lane<NV / 2, M / 2>(lane);
    else return 0;
}

template <int F16>
__device__ __forceinline__ void unpack16(const uint4& w, float (&f)[F16 ? 8 : 4])
{
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if constexpr (F16) {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&ww[i]));
            f[2 * i] = v.x;
            f[2 * i + 1] = v.y;
        } else {
            f[i] = __uint_as_float(ww[i]);
        }
    }
}


// What bounds it: the read of the cache rows (4001 keys of 8 heads of 128: 16.4 MB, 2.5 us), and below about 1000 keys the launch.
// One CTA per (token, head) took 202 us there, most of it in the sums that one thread added in order; 12 us now (65 keys: 9.2,
// 8.8; 16001 keys: 905, 31 us, 2.1 TB/s).  Error against 64 bits 1.7e-6 before, 2.8e-7 now (sums over lanes, warps and CTAs).
//
// A cluster along y = one query token x R query heads of one key head; its CTAs take consecutive stretches of `stretch` keys.
// A lane holds 16 bytes of a key row, so a load of the warp covers 32 lanes / (row / 16 bytes) keys; eight such loads are in
// flight.  Scores go to shared memory; maximum, weights and their sum per CTA; values the same way as keys; the cluster then
// weighs its CTAs' sums by exp(m_i - m).
//
// NEW: a decoded token's rotation and cache row, which were a launch of their own (4 us of a layer's 80 at 4000 keys), are part of it.  The angles take one
// thread per pair; the CTA whose stretch holds the new row writes it and reads it back, for every cluster of a key head alike.
template <int F16, int D, int R, bool NEW>
__global__ void __launch_bounds__(kSplitThreads) k_gqa_split(GqaShape p, GqaNew in, const float* q, const void* kc, const void* vc, float* dst, int stretch)
{
    constexpr int E = F16 ? 8 : 4;              // elements of a load
    constexpr int L = D / E, P = 32 / L;        // lanes per key, keys per load
    constexpr int NV = 8 * R, NR = NV / L > 0 ? NV / L : 1;
    pdl_launch_dependents();
    if (!NEW) pdl_wait();
    extern __shared__ __align__(16) float sh[];
    float* s_out = sh;                          // [R][D] this CTA's sums
    float* s_part = s_out + R * D;              // [warps][R][D]
    float* s_p = s_part + kSplitWarps * R * D;  // [stretch][R] scores, then weights
    __shared__ float s_red[kSplitWarps][R], s_m[R], s_l[R];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rep = p.heads / p.kv_heads, groups = (rep + R - 1) / R;
    const int kvh = blockIdx.x / groups, h0 = (blockIdx.x % groups) * R, qt = blockIdx.z;
    const int rank = (int)cluster_rank(), ranks = (int)cluster_size();
    const int sees = min(p.n_kv, p.kv_offset + qt + 1);
    const int first = min(rank * stretch, sees), n = min(sees - first, stretch);
    const size_t row = (size_t)p.kv_heads * D * (F16 ? 2 : 4);
    const char* kbase = reinterpret_cast<const char*>(kc) + (size_t)first * row + ((size_t)kvh * D + (lane % L) * E) * (F16 ? 2 : 4);
    const char* vbase = reinterpret_cast<const char*>(vc) + (size_t)first * row + ((size_t)kvh * D + (lane % L) * E) * (F16 ? 2 : 4);
    auto head = [&](int r) { return kvh * rep + min(h0 + r, rep - 1); };      // a last group of fewer heads repeats one
    __shared__ float2 s_turn[NEW ? D / 2 : 1];      // cosine and sine of a pair
    uint4 kw[8];                                    // the warp's first keys
    auto key_of = [&](int b, int j) { return min(b + j * P + lane / L, n - 1); };
    auto fetch_keys = [&](int b) {
#pragma unroll
        for (int j = 0; j < 8; j++)         // cache rows may have been written by the launch before: not the read-only path
            kw[j] = __ldcg(reinterpret_cast<const uint4*>(kbase + (size_t)key_of(b, j) * row));
    };
    if constexpr (NEW) {
        // Position, angles and keys do not depend on the products of this token: a forward's first launch waits for everything ahead of it, and no launch
        // of it but this one writes rows of this layer's cache, the new one.
        const int pos = *in.pos;
        if (warp * 8 * P < n) fetch_keys(warp * 8 * P);
        if (tid % (D) < in.n_dims / 2 && tid < 2 * D) {      // cosines by the first D threads, sines by the next
            float c, sn;
            rope_angle(tid % D, pos, in.freq_factors, in.theta_scale, tid < D, c, sn);
            if (tid < D) s_turn[tid].x = c;
            else s_turn[tid - D].y = sn;
        }
        pdl_wait();
        __syncthreads();
        if (pos < 0 || pos >= in.max_seq_len) {
            if (tid == 0 && rank == 0 && in.err) atomicCAS(in.err, 0, 20);
        } else if (pos >= first && pos < first + n ? true : rank == 0 && pos >= sees) {
            if (tid < D) {
                const int i = tid % (D / 2);
                const float2 x = *reinterpret_cast<const float2*>((tid < D / 2 ? in.k : in.v) + (size_t)kvh * D + 2 * i);
                float y0 = x.x, y1 = x.y;
                if (tid < D / 2 && i < in.n_dims / 2) rope_turn(x.x, x.y, s_turn[i].x, s_turn[i].y, y0, y1);
                const size_t at = ((size_t)pos * p.kv_heads + kvh) * D + 2 * i;
                void* cache = const_cast<void*>(tid < D / 2 ? kc : vc);
                if (F16) {
                    reinterpret_cast<__half*>(cache)[at] = __float2half_rn(y0);
                    reinterpret_cast<__half*>(cache)[at + 1] = __float2half_rn(y1);
                } else {
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(cache) + at) = make_float2(y0, y1);
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (warp * 8 * P < n && first + key_of(warp * 8 * P, j) == pos) kw[j] = __ldcg(reinterpret_cast<const uint4*>(kbase + (size_t)(pos - first) * row));
        }
    }
    // scores
    {
        float qv[R][E];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float4* src = reinterpret_cast<const float4*>(q + ((size_t)qt * p.heads + head(r)) * D + (lane % L) * E);
#pragma unroll
            for (int i = 0; i < E / 4; i++) *reinterpret_cast<float4*>(&qv[r][4 * i]) = src[i];
            if constexpr (NEW) {
#pragma unroll
                for (int i = 0; i < E / 2; i++) {
                    const int pair = (lane % L) * (E / 2) + i;
                    const float2 turn = s_turn[min(pair, max(in.n_dims / 2 - 1, 0))];
                    float y0, y1;
                    rope_turn(qv[r][2 * i], qv[r][2 * i + 1], turn.x, turn.y, y0, y1);
                    if (pair < in.n_dims / 2) {
                        qv[r][2 * i] = y0;
                        qv[r][2 * i + 1] = y1;
                    }
                }
            }
        }
        const int at = first_of_lane<NV, L / 2>(lane);
        const bool writes = NV >= L || (lane % L) % (L / (NV < L ? NV : L)) == 0;
        for (int b = warp * 8 * P; b < n; b += kSplitWarps * 8 * P) {
            if (!NEW || b != warp * 8 * P) fetch_keys(b);
            float s[NV];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float f[E];
                unpack16<F16>(kw[j], f);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    float t = 0.0f;
#pragma unroll
                    for (int i = 0; i < E; i++) t = fmaf(qv[r][i], f[i], t);
                    s[j * R + r] = t;
                }
            }
            sum_over_lanes<NV, L / 2>(s, lane);
#pragma unroll
            for (int i = 0; i < NR; i++) {
                const int key = b + (at + i) / R * P + lane / L;
                if (writes && key < n) s_p[key * R + (at + i) % R] = s[i] * p.scale;
            }
        }
    }
    // the warp's first values are requested ahead of the softmax
    uint4 vw[8];
    if (warp * 8 * P < n) {
#pragma unroll
        for (int j = 0; j < 8; j++) vw[j] = __ldcg(reinterpret_cast<const uint4*>(vbase + (size_t)min(warp * 8 * P + j * P + lane / L, n - 1) * row));
    }
    __syncthreads();
    // thread t: head t % R
    float m = kLowest;
    for (int i = tid; i < n * R; i += kSplitThreads) m = fmaxf(m, s_p[i]);
#pragma unroll
    for (int o = 16; o >= R; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (lane < R) s_red[warp][lane] = m;
    __syncthreads();
    m = s_red[0][tid % R];
#pragma unroll
    for (int w = 1; w < kSplitWarps; w++) m = fmaxf(m, s_red[w][tid % R]);
    __syncthreads();
    float l = 0.0f;
    for (int i = tid; i < n * R; i += kSplitThreads) {
        const float e = exp_below(s_p[i] - m);
        s_p[i] = e;
        l += e;
    }
#pragma unroll
    for (int o = 16; o >= R; o >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
    if (lane < R) s_red[warp][lane] = l;
    __syncthreads();
    if (tid < R) {
        l = 0.0f;
#pragma unroll
        for (int w = 0; w < kSplitWarps; w++) l += s_red[w][tid];
        s_m[tid] = m;
        s_l[tid] = l;
    }
    // values
    {
        float acc[R][E];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int i = 0; i < E; i++) acc[r][i] = 0.0f;
        for (int b = warp * 8 * P; b < n; b += kSplitWarps * 8 * P) {
            uint4 w[8];
#pragma unroll
            for (int j = 0; j < 8; j++) w[j] = vw[j];
            const int next = b + kSplitWarps * 8 * P;
            if (next < n) {
#pragma unroll
                for (int j = 0; j < 8; j++) vw[j] = __ldcg(reinterpret_cast<const uint4*>(vbase + (size_t)min(next + j * P + lane / L, n - 1) * row));
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int key = b + j * P + lane / L;
                if (key < n) {
                    float f[E];
                    unpack16<F16>(w[j], f);
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const float e = s_p[key * R + r];
#pragma unroll
                        for (int i = 0; i < E; i++) acc[r][i] = fmaf(e, f[i], acc[r][i]);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int i = 0; i < E; i++) {
#pragma unroll
                for (int o = L; o < 32; o <<= 1) acc[r][i] += __shfl_xor_sync(0xFFFFFFFFu, acc[r][i], o);
            }
        if (lane < L) {
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int i = 0; i < E; i += 4)
                    *reinterpret_cast<float4*>(&s_part[(warp * R + r) * D + lane * E + i]) = make_float4(acc[r][i], acc[r][i + 1], acc[r][i + 2], acc[r][i + 3]);
        }
    }
    __syncthreads();
    for (int i = tid; i < R * D; i += kSplitThreads) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < kSplitWarps; w++) t += s_part[w * R * D + i];
        s_out[i] = t;
    }
    // the cluster's CTAs: each finishes a slice of the results
    cluster_arrive();
    cluster_wait();
    const int slice = (R * D + ranks - 1) / ranks;
    if (ranks >= 8 && slice <= 32) {
        // few results per CTA: a warp takes some of the CTAs, a lane a result (one thread for a result, 16 CTAs: 2.0 us of 17).  Sums per warp, then over the
        // warps: last bits differ from one thread's
        __shared__ float s_join[3][kSplitWarps][32];
        const int i = rank * slice + lane;
        const bool own = lane < slice && i < R * D;
        float top = kLowest, sum = 0.0f, out = 0.0f;
        constexpr int kEach = (kMaxCluster + kSplitWarps - 1) / kSplitWarps;
        float pm[kEach], pl[kEach], po[kEach];
#pragma unroll
        for (int c = 0; c < kEach; c++) {
            const int from = warp + c * kSplitWarps;
            const bool there = own && from < ranks;
            pm[c] = there ? load_peer(&s_m[i / D], from) : kLowest;
            pl[c] = there ? load_peer(&s_l[i / D], from) : 0.0f;
            po[c] = there ? load_peer(&s_out[i], from) : 0.0f;
        }
#pragma unroll
        for (int c = 0; c < kEach; c++) top = fmaxf(top, pm[c]);
#pragma unroll
        for (int c = 0; c < kEach; c++)
            if (warp + c * kSplitWarps < ranks) {
                const float f = exp_below(pm[c] - top);
                sum = fmaf(f, pl[c], sum);
                out = fmaf(f, po[c], out);
            }
        s_join[0][warp][lane] = top;
        s_join[1][warp][lane] = sum;
        s_join[2][warp][lane] = out;
        __syncthreads();
        if (warp == 0 && own) {
            const int used = min(ranks, kSplitWarps);
            float all = kLowest;
            for (int w = 0; w < used; w++) all = fmaxf(all, s_join[0][w][lane]);
            sum = out = 0.0f;
            for (int w = 0; w < used; w++) {
                const float f = exp_below(s_join[0][w][lane] - all);
                sum = fmaf(f, s_join[1][w][lane], sum);
                out = fmaf(f, s_join[2][w][lane], out);
            }
            const int r = i / D;
            if (h0 + r < rep) dst[((size_t)qt * p.heads + head(r)) * D + i % D] = out * (sum == 0.0f ? 0.0f : __fdiv_rn(1.0f, sum));
        }
    } else
    for (int i = rank * slice + tid; i < min(R * D, (rank + 1) * slice); i += kSplitThreads) {
        const int r = i / D;
        // all CTAs' loads in flight before the first is used (one after the other: 3 us of 12 with 16 CTAs)
        float pm[kMaxCluster], pl[kMaxCluster], po[kMaxCluster], top = kLowest;
#pragma unroll
        for (int c = 0; c < kMaxCluster; c++) {
            const int from = c < ranks ? c : 0;
            pm[c] = load_peer(&s_m[r], from);
            pl[c] = load_peer(&s_l[r], from);
            po[c] = load_peer(&s_out[i], from);
        }
#pragma unroll
        for (int c = 0; c < kMaxCluster; c++)
            if (c < ranks) top = fmaxf(top, pm[c]);
        float sum = 0.0f, out = 0.0f;
#pragma unroll
        for (int c = 0; c < kMaxCluster; c++)
            if (c < ranks) {
                const float f = exp_below(pm[c] - top);
                sum = fmaf(f, pl[c], sum);
                out = fmaf(f, po[c], out);
            }
        if (h0 + r < rep) dst[((size_t)qt * p.heads + head(r)) * D + i % D] = out * (sum == 0.0f ? 0.0f : __fdiv_rn(1.0f, sum));
    }
    cluster_arrive();       // nobody leaves while its shared memory is read
    cluster_wait();
}

// ------------------------------------------------------------------ prompts

constexpr int kTileThreads = 128, kTileRowsQ = 64, kTileKeys = 64;

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (v0, v1) = hi + lo, 22 bits of mantissa where lo stays above fp16's smallest number (6e-8)
__device__ __forceinline__ void split_f16(float v0, float v1, uint32_t& hi, uint32_t& lo)
{
    const __half2 h = __floats2half2_rn(v0, v1);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(v0 - f.x, v1 - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// One row by one warp, in fp32 and key after key: what a row with values that are not finite falls back to (there the tile's
// products of masked keys would spread them).
template <int D>
__device__ __noinline__ void gqa_row(const float* q, const __half* k, const __half* v, float* dst, int n, size_t row, float scale)
{
    const int lane = threadIdx.x & 31;
    auto score = [&](int key) {
        float s = 0.0f;
        for (int d = 0; d < D; d++) s = __fadd_rn(s, __fmul_rn(q[d], __half2float(k[(size_t)key * row + d])));
        return __fmul_rn(s, scale);
    };
    float m = kLowest, l = 0.0f, acc[D / 32];
    for (int i = lane; i < n; i += 32) m = fmaxf(m, score(i));
    m = warp_max(m);
    for (int i = lane; i < n; i += 32) l += expf(score(i) - m);
    l = warp_sum(l);
    const float inv = l == 0.0f ? 0.0f : __fdiv_rn(1.0f, l);
#pragma unroll
    for (int c = 0; c < D / 32; c++) acc[c] = 0.0f;
    for (int i0 = 0; i0 < n; i0 += 32) {
        const float w = i0 + lane < n ? expf(score(i0 + lane) - m) * inv : 0.0f;
        for (int j = 0; j < min(32, n - i0); j++) {
            const float e = __shfl_sync(0xFFFFFFFFu, w, j);
#pragma unroll
            for (int c = 0; c < D / 32; c++) acc[c] = __fadd_rn(acc[c], __fmul_rn(__half2float(v[(size_t)(i0 + j) * row + c * 32 + lane]), e));
        }
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < D / 32; c++) dst[c * 32 + lane] = acc[c];
}

// What bounds it: the tensor pipe of mma.sync (two products per multiplication: 16 GFLOP per layer at 1000 tokens, 32 heads of 128).
// 1000 tokens: 1824 us on one CTA per (token, head), 407 us on k_gqa_split, 65 us here; error against 64 bits 6.4e-7 before,
// 4.5e-7 now.
//
// A CTA = 64 rows of one key head, row = token * (heads that share it) + head; warp = 16 rows; keys and values in
// double-buffered tiles of 64 by cp.async.  A row of q is scaled by a power of two to below 2 and split into two fp16 numbers
// (error 2^-24 of the row's largest entry); keys and values are fp16 as they are; weights are scaled by 2^10 and split.  A
// tensor-core sum truncates where an fp32 addition rounds, so only one tile's products are added there (the small halves
// first, 4 to 8 steps of the large ones) and tiles are joined by fp32 additions.
template <int D>
__global__ void __launch_bounds__(kTileThreads, 2) k_gqa_tile(GqaShape p, const float* q, const __half* kc, const __half* vc, float* dst)
{
    constexpr int C = D / 8;                    // 16-byte pieces of a row
    constexpr float kWeightScale = 1024.0f;
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(128) uint8_t smem[];
    __half* s_k = reinterpret_cast<__half*>(smem);                  // [2][64][D], pieces of row r at piece ^ (r % 8)
    __half* s_v = s_k + 2 * kTileKeys * D;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int rep = p.heads / p.kv_heads, kvh = blockIdx.x, rows = p.n_q * rep;
    const int row0 = (int)(gridDim.y - 1 - blockIdx.y) * kTileRowsQ;        // the longest first
    const size_t row = (size_t)p.kv_heads * D;
    const __half* kbase = kc + (size_t)kvh * D;
    const __half* vbase = vc + (size_t)kvh * D;
    auto sees = [&](int r) { return min(p.n_kv, p.kv_offset + r / rep + 1); };
    const int n = sees(min(row0 + kTileRowsQ, rows) - 1), clear = sees(row0);       // keys of the CTA; keys that all its rows see
    const int tiles = (n + kTileKeys - 1) / kTileKeys;

    auto load = [&](int i) {
        __half* k = s_k + (i & 1) * kTileKeys * D;
        __half* v = s_v + (i & 1) * kTileKeys * D;
#pragma unroll
        for (int j = 0; j < kTileKeys * C / kTileThreads; j++) {
            const int u = tid + j * kTileThreads, r = u / C, c = u % C, key = i * kTileKeys + r;
            const size_t src = (size_t)min(key, n - 1) * row + c * 8;
            const int at = r * D + (c ^ (r & 7)) * 8;
            cp_async16(k + at, kbase + src, key < n);
            cp_async16(v + at, vbase + src, key < n);
        }
        cp_async_commit();
    };
    load(0);

    // this lane's two rows
    int qrow[2], lim[2];
    const float* qp[2];
    float f[2];
    uint32_t qh[D / 16][4], ql[D / 16][4];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        qrow[i] = row0 + warp * 16 + g + 8 * i;
        const int r = min(qrow[i], rows - 1);
        lim[i] = sees(r);
        qp[i] = q + ((size_t)(r / rep) * p.heads + kvh * rep + r % rep) * D;
        float top = 0.0f;
#pragma unroll
        for (int c = 0; c < D / 8; c++) {
            const float2 v = *reinterpret_cast<const float2*>(qp[i] + 8 * c + 2 * t4);
            top = fmaxf(top, fmaxf(fabsf(v.x), fabsf(v.y)));
        }
        top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
        const int e = min(max((__float_as_int(top) >> 23) - 127, -100), 100);       // 2^e <= top < 2^(e+1)
        const float down = __int_as_float((127 - e) << 23);
        f[i] = __int_as_float((127 + e) << 23) * p.scale;
#pragma unroll
        for (int c = 0; c < D / 16; c++) {
            const float2 v = *reinterpret_cast<const float2*>(qp[i] + 16 * c + 2 * t4);
            const float2 w = *reinterpret_cast<const float2*>(qp[i] + 16 * c + 8 + 2 * t4);
            split_f16(v.x * down, v.y * down, qh[c][i], ql[c][i]);
            split_f16(w.x * down, w.y * down, qh[c][2 + i], ql[c][2 + i]);
        }
    }
    float o[D / 8][4], m[2] = {kLowest, kLowest}, l[2] = {0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < D / 8; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) o[c][i] = 0.0f;

    for (int i = 0; i < tiles; i++) {
        if (i + 1 < tiles) {
            load(i + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            cp_async_wait_all();
        }
        __syncthreads();
        const __half* k = s_k + (i & 1) * kTileKeys * D;
        const __half* v = s_v + (i & 1) * kTileKeys * D;
        float s[8][4];
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float lo[4][4];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int x = 0; x < 4; x++) s[4 * half + j][x] = lo[j][x] = 0.0f;
#pragma unroll
            for (int c = 0; c < D / 16; c++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    uint32_t b[4];
                    const int r = half * 32 + j * 16 + ((lane >> 4) << 3) + (lane & 7), piece = 2 * c + ((lane >> 3) & 1);
                    ldsm4(b, reinterpret_cast<const bf16*>(k + r * D + (piece ^ (r & 7)) * 8));
                    mma_f16(lo[2 * j], ql[c], b[0], b[1]);
                    mma_f16(lo[2 * j + 1], ql[c], b[2], b[3]);
                    mma_f16(s[4 * half + 2 * j], qh[c], b[0], b[1]);
                    mma_f16(s[4 * half + 2 * j + 1], qh[c], b[2], b[3]);
                }
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int x = 0; x < 4; x++) s[4 * half + j][x] += lo[j][x];
        }
        // scale, mask, weights relative to the running maximum
        float top[2] = {m[0], m[1]};
        const bool whole = (i + 1) * kTileKeys <= clear;
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                s[j][x] *= f[x >> 1];
                if (!whole && i * kTileKeys + 8 * j + 2 * t4 + (x & 1) >= lim[x >> 1]) s[j][x] = -INFINITY;
                top[x >> 1] = fmaxf(top[x >> 1], s[j][x]);
            }
        bool moved = false;
        float down[2];
#pragma unroll
        for (int x = 0; x < 2; x++) {
            top[x] = fmaxf(top[x], __shfl_xor_sync(0xFFFFFFFFu, top[x], 1));
            top[x] = fmaxf(top[x], __shfl_xor_sync(0xFFFFFFFFu, top[x], 2));
            moved |= top[x] != m[x];
            down[x] = exp_below(m[x] - top[x]);
            m[x] = top[x];
        }
        if (__any_sync(0xFFFFFFFFu, moved)) {
#pragma unroll
            for (int x = 0; x < 2; x++) l[x] *= down[x];
#pragma unroll
            for (int c = 0; c < D / 8; c++)
#pragma unroll
                for (int x = 0; x < 4; x++) o[c][x] *= down[x >> 1];
        }
        uint32_t ph[4][4], pl[4][4];
#pragma unroll
        for (int j = 0; j < 8; j++) {
#pragma unroll
            for (int x = 0; x < 4; x++) {
                s[j][x] = exp_below(s[j][x] - m[x >> 1]);
                l[x >> 1] += s[j][x];
                s[j][x] *= kWeightScale;
            }
#pragma unroll
            for (int x = 0; x < 2; x++) split_f16(s[j][2 * x], s[j][2 * x + 1], ph[j / 2][(j & 1) * 2 + x], pl[j / 2][(j & 1) * 2 + x]);
        }
#pragma unroll
        for (int c = 0; c < D / 16; c++) {
            uint32_t b[4][4];
            float add[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = j * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), piece = 2 * c + (lane >> 4);
                ldsm4_t(b[j], reinterpret_cast<const bf16*>(v + r * D + (piece ^ (r & 7)) * 8));
                mma_f16(add[0], pl[j], b[j][0], b[j][1]);
                mma_f16(add[1], pl[j], b[j][2], b[j][3]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                mma_f16(add[0], ph[j], b[j][0], b[j][1]);
                mma_f16(add[1], ph[j], b[j][2], b[j][3]);
            }
#pragma unroll
            for (int x = 0; x < 4; x++) {
                o[2 * c][x] += add[0][x];
                o[2 * c + 1][x] += add[1][x];
            }
        }
        __syncthreads();
    }
    bool odd[2];
#pragma unroll
    for (int x = 0; x < 2; x++) {
        l[x] += __shfl_xor_sync(0xFFFFFFFFu, l[x], 1);
        l[x] += __shfl_xor_sync(0xFFFFFFFFu, l[x], 2);
        float bad = 0.0f * l[x];
#pragma unroll
        for (int c = 0; c < D / 8; c++) bad += 0.0f * o[c][2 * x] + 0.0f * o[c][2 * x + 1];      // NaN if anything is not finite
        odd[x] = !(bad == 0.0f);
        odd[x] = __shfl_xor_sync(0xFFFFFFFFu, (int)odd[x], 1) || odd[x];
        odd[x] = __shfl_xor_sync(0xFFFFFFFFu, (int)odd[x], 2) || odd[x];
        const float inv = (l[x] == 0.0f ? 0.0f : __fdiv_rn(1.0f, l[x])) * (1.0f / kWeightScale);
        if (qrow[x] < rows && !odd[x]) {
            float* out = dst + (qp[x] - q);
#pragma unroll
            for (int c = 0; c < D / 8; c++) *reinterpret_cast<float2*>(out + 8 * c + 2 * t4) = make_float2(o[c][2 * x] * inv, o[c][2 * x + 1] * inv);
        }
    }
#pragma unroll
    for (int x = 0; x < 2; x++) {
        const uint32_t todo = __ballot_sync(0xFFFFFFFFu, odd[x] && qrow[x] < rows && t4 == 0);
        for (uint32_t left = todo; left; left &= left - 1) {
            const int from = __ffs(left) - 1;
            const int r = __shfl_sync(0xFFFFFFFFu, qrow[x], from);
            const size_t at = ((size_t)(r / rep) * p.heads + kvh * rep + r % rep) * D;
            gqa_row<D>(q + at, kbase, vbase, dst + at, sees(r), row, p.scale);
        }
    }
}

// ------------------------------------------------------------------ host side

template <int F16, int D, int R, bool NEW>
static int launch_split(const GqaShape& p, const GqaNew& in, const float* q, const void* k, const void* v, float* dst, cudaStream_t s)
{
    auto kern = k_gqa_split<F16, D, R, NEW>;
    static int ready[64] = {0};       // the largest cluster of the kernel on a device
    int dev = 0;
    cudaGetDevice(&dev);
    int largest = dev >= 0 && dev < 64 ? ready[dev] : 0;
    if (!largest) {
        int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitMaxSmem));
        if (rc) return rc;
        rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        if (rc) return rc;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, kMaxCluster);
        cfg.blockDim = dim3(kSplitThreads);
        cfg.dynamicSmemBytes = kSplitMaxSmem;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = at.val.clusterDim.z = 1;
        at.val.clusterDim.y = kMaxCluster;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int fit = 0;
        rc = check_cuda(cudaOccupancyMaxActiveClusters(&fit, kern, &cfg));
        if (rc) return rc;
        largest = fit > 0 ? kMaxCluster : 8;        // 8 fits every device
        if (dev >= 0 && dev < 64) ready[dev] = largest;
    }
    const int rep = p.heads / p.kv_heads, groups = (rep + R - 1) / R;
    const int sees = p.kv_offset + p.n_q < p.n_kv ? p.kv_offset + p.n_q : p.n_kv;
    const GqaSplit split = gqa_split((long)p.kv_heads * groups * p.n_q, sees, R, D, largest, sm_count());
    if (!split.fits) return 1;
    const unsigned ranks = (unsigned)split.ranks;
    return launch_cluster(kern, dim3((unsigned)(p.kv_heads * groups), ranks, (unsigned)p.n_q), dim3(1, ranks, 1), kSplitThreads, split.smem, s, p, in, q, k, v,
                          dst, split.stretch);
}

template <bool NEW, int F16, int D>
static int launch_split_of(const GqaShape& p, const GqaNew& in, const float* q, const void* k, const void* v, float* dst, cudaStream_t s)
{
    const int rep = p.heads / p.kv_heads;
    if (rep == 1) return launch_split<F16, D, 1, NEW>(p, in, q, k, v, dst, s);
    if (rep == 2) return launch_split<F16, D, 2, NEW>(p, in, q, k, v, dst, s);
    return launch_split<F16, D, 4, NEW>(p, in, q, k, v, dst, s);
}
template <bool NEW>
static int launch_split_of(const GqaShape& p, const GqaNew& in, const float* q, const void* k, const void* v, float* dst, cudaStream_t s)
{
    if (p.f16) return p.dim == 64 ? launch_split_of<NEW, 1, 64>(p, in, q, k, v, dst, s) : launch_split_of<NEW, 1, 128>(p, in, q, k, v, dst, s);
    return p.dim == 64 ? launch_split_of<NEW, 0, 64>(p, in, q, k, v, dst, s) : launch_split_of<NEW, 0, 128>(p, in, q, k, v, dst, s);
}

template <int D>
static int launch_tile(const GqaShape& p, const float* q, const void* k, const void* v, float* dst, cudaStream_t s)
{
    constexpr int smem = 4 * kTileKeys * D * 2;
    int rc = allow_smem<k_gqa_tile<D>>(smem);
    if (rc) return rc;
    const int rows = p.n_q * (p.heads / p.kv_heads);
    return launch_ordered(k_gqa_tile<D>, dim3((unsigned)p.kv_heads, (unsigned)((rows + kTileRowsQ - 1) / kTileRowsQ)), kTileThreads, smem, s, p, q,
                          reinterpret_cast<const __half*>(k), reinterpret_cast<const __half*>(v), dst);
}

enum { kGeneral, kSplit, kTile };      // k_gqa_attn, k_gqa_split, k_gqa_tile
static int gqa_kernel(const GqaShape& p)
{
    if (p.kv_offset < 0 || (p.dim != 64 && p.dim != 128)) return kGeneral;
    const long sees = (long)p.kv_offset + p.n_q < p.n_kv ? (long)p.kv_offset + p.n_q : p.n_kv;
    const long rep = p.heads / p.kv_heads, rows = (long)p.n_q * rep, blocks = (rows + kTileRowsQ - 1) / kTileRowsQ;
    if (sees <= kShortKeys || blocks > 65535 || p.n_q > 65535) return kGeneral;
    // Time per 64 keys, fitted to 20 shapes of 1 to 2048 queries and 65 to 16001 keys: a tile CTA 0.5 + 0.014 dim us, two per SM at
    // a time, whatever few rows it has; the split kernel 0.64 + 0.011 (heads of a group) dim ns for every query and group.
    // Measured sides of the line (tile, split; us): 32/8 heads of 128, 532 keys, 32 queries 25, 18; 2128 keys, 128 queries
    // 107, 181; 32/32 heads of 64, 532 keys, 32 queries 16, 18; 16/4 heads of 64, 4032 keys, 32 queries 90, 32.
    const long group = rep > 2 ? 4 : rep, groups = (rep + group - 1) / group;
    const double tile_us = (double)((p.kv_heads * blocks + 2 * sm_count() - 1) / (2 * sm_count())) * (0.5 + 0.014 * p.dim);
    const double split_us = 1e-3 * (double)p.n_q * (double)(p.kv_heads * groups) * (0.64 + 0.011 * (double)group * p.dim);
    if (p.f16 && tile_us < split_us) return kTile;
    // fp32 heads of 64 that share nothing, short prompts: a CTA here costs 11 ns of the chip's time whatever few keys its query sees, there 0.1 ns
    // a key and 5 to 9 ns.  100 tokens of 32 heads: 29.9 us there, 35.2 here; 200: 78.7, 78.6; 65 of 16 heads: 11.4, 12.6; 10 keys further on 13.8, 12.9.
    if (!p.f16 && rep == 1 && p.dim == 64) {
        const double waves = (double)p.n_q * p.heads / (8.0 * sm_count()), line = 28.0 + 17.0 * waves;
        if (p.kv_offset + 0.5 * (p.n_q + 1) <= (line < 102.0 ? line : 102.0)) return kGeneral;
    }
    return kSplit;
}

int gqa_attention(const GqaShape& p, const float* q, const void* k, const void* v, float* dst, cudaStream_t s)
{
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dst) & 15) return 1;
    const int kernel = gqa_kernel(p);
    if (kernel == kGeneral) return 1;
    if (kernel == kTile) return p.dim == 64 ? launch_tile<64>(p, q, k, v, dst, s) : launch_tile<128>(p, q, k, v, dst, s);
    return launch_split_of<false>(p, GqaNew{}, q, k, v, dst, s);
}

int gqa_attention_new(const GqaShape& p, const GqaNew& in, const float* q, void* k, void* v, float* dst, cudaStream_t s)
{
    if (p.n_q != 1 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dst) & 15) || gqa_kernel(p) != kSplit) return 1;
    return launch_split_of<true>(p, in, q, k, v, dst, s);
}

}  // namespace bpdq

using namespace bpdq;

extern "C" {

int bpdq_gqa_attn_kernel(int n_q_tokens, int n_kv, int n_q_heads, int n_kv_heads, int head_dim, int kv_offset, int kv_is_f16)
{
    if (n_q_tokens < 1 || n_kv < 1 || n_q_heads < 1 || n_kv_heads < 1 || n_q_heads % n_kv_heads) return -1;
    return gqa_kernel(GqaShape{n_q_tokens, n_kv, n_q_heads, n_kv_heads, head_dim, 1.0f, kv_offset, kv_is_f16});
}

}  // extern "C"
