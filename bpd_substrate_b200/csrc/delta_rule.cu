// Gated delta rule.
//
//   k_delta_token       one token: a cluster of CTAs per head, each with 32 value columns; the state goes through HBM once.
//                       Unit lengths, prediction and read-out come from one pass over the state (the read-out of the written
//                       state is the read-out of the decayed one plus (k.q) u); the output's norm joins its CTAs through
//                       distributed shared memory.
//   k_delta_recurrence  token by token: a warp holds four value columns of a head, eight lanes over the keys, so that a token
//                       costs three shuffles and no barrier.  Short portions, fp32 runs.
//   k_delta_prepare, k_delta_chunks
//                       a prompt's portion in chunks of 16 tokens.  Inside a chunk with decays g, c_i = g_0 .. g_i and
//                         A_ij = beta_i k_i . (g_{j+1} .. g_i k_j)  (j < i),   P_ij = q_i . (g_{j+1} .. g_i k_j)  (j <= i)
//                       the writes solve (1 + A) u = beta (v - (c k) S), so that
//                         u = U - W S,  o = O + Q S,  S <- c_15 S + sum_j (g_{j+1} .. g_15 k_j) u_j^T
//                       with (1 + A) W = beta c k,  (1 + A) U = beta v,  Q = c q - P W,  O = P U.  The first kernel works these out for
//                       all chunks at once (fp32, threads for keys and value columns; only products of decays, which cannot
//                       overflow); the second walks the chunks with the transposed state in fp32 accumulators: two warps for
//                       the state of 16 value columns and two for its read-out, fed by bulk copies of ready-made fragments.
//                       What is fp32 enters mma.sync as the sum of two bf16 numbers, three products.
#include "delta_rule.cuh"
#include "cluster_device.cuh"
#include "launch.cuh"
#include "mma_device.cuh"
#include "../../include/bpdq.h"

namespace bpdq {

// An fp32 exponential that leans one way by a unit in the last place adds up over thousands of tokens.
template <typename A> __device__ __forceinline__ float decay_of(float log_decay) { return sizeof(A) == 4 ? (float)exp((double)log_decay) : expf(log_decay); }

// ------------------------------------------------------------------ one token

constexpr int kTokenCols = 32;

// grid (heads, value columns / 32), 256 threads: eight groups of four columns x 32 key phases.
template <typename A, int NI>
__global__ void __launch_bounds__(256) k_delta_token(DeltaRule a)
{
    __shared__ float4 red[8][8][2], red_s[8];
    __shared__ float s_part[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cg = tid & 7, phase = tid >> 3;
    const int h = blockIdx.x, g = h / (a.heads / a.groups), p = blockIdx.y * kTokenCols + 4 * cg;
    const bool live = p < a.value_pad;
    pdl_launch_dependents();
    const uint32_t parts = cluster_size();
    if (parts > 1) cluster_arrive();        // (everybody is there before anybody's shared memory is written)
    const float4 zero = make_float4(0, 0, 0, 0);
    const float4 nw = (a.norm_w && live) ? *reinterpret_cast<const float4*>(a.norm_w + (size_t)h * a.value_pad + p) : zero;
    pdl_wait();
    float* st = a.state + (size_t)h * a.key_pad * a.value_pad + p;
    const A* q = reinterpret_cast<const A*>(a.q) + g * a.key_pad;
    const A* k = reinterpret_cast<const A*>(a.k) + g * a.key_pad;
    const float* lg = a.log_decay + (size_t)h * a.key_pad;
    float4 s[NI];
    float kn[NI], qn[NI], dn[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const int n = phase + 32 * i;
        const bool in = n < a.key_pad;
        s[i] = (in && live) ? *reinterpret_cast<const float4*>(st + (size_t)n * a.value_pad) : zero;
        kn[i] = in ? act_load(k + n) : 0.0f;
        qn[i] = in ? act_load(q + n) : 0.0f;
        dn[i] = in ? lg[n] : 0.0f;
    }
    const size_t at = (size_t)h * a.value_pad + p;
    const float4 v = live ? act_load4(reinterpret_cast<const A*>(a.v) + at) : zero;
    const float4 gate = (a.norm_w && live) ? act_load4(reinterpret_cast<const A*>(a.gate) + at) : zero;
    const float beta = a.beta[h];
    float4 sk = zero, sq = zero;
    float kk = 0.0f, qq = 0.0f, kq = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const float d = decay_of<A>(dn[i]);
        s[i] = make_float4(s[i].x * d, s[i].y * d, s[i].z * d, s[i].w * d);
        sk.x = fmaf(s[i].x, kn[i], sk.x); sk.y = fmaf(s[i].y, kn[i], sk.y); sk.z = fmaf(s[i].z, kn[i], sk.z); sk.w = fmaf(s[i].w, kn[i], sk.w);
        sq.x = fmaf(s[i].x, qn[i], sq.x); sq.y = fmaf(s[i].y, qn[i], sq.y); sq.z = fmaf(s[i].z, qn[i], sq.z); sq.w = fmaf(s[i].w, qn[i], sq.w);
        kk = fmaf(kn[i], kn[i], kk);
        qq = fmaf(qn[i], qn[i], qq);
        kq = fmaf(kn[i], qn[i], kq);
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
        sk.x += __shfl_xor_sync(0xFFFFFFFFu, sk.x, o); sk.y += __shfl_xor_sync(0xFFFFFFFFu, sk.y, o);
        sk.z += __shfl_xor_sync(0xFFFFFFFFu, sk.z, o); sk.w += __shfl_xor_sync(0xFFFFFFFFu, sk.w, o);
        sq.x += __shfl_xor_sync(0xFFFFFFFFu, sq.x, o); sq.y += __shfl_xor_sync(0xFFFFFFFFu, sq.y, o);
        sq.z += __shfl_xor_sync(0xFFFFFFFFu, sq.z, o); sq.w += __shfl_xor_sync(0xFFFFFFFFu, sq.w, o);
        kk += __shfl_xor_sync(0xFFFFFFFFu, kk, o);
        qq += __shfl_xor_sync(0xFFFFFFFFu, qq, o);
        kq += __shfl_xor_sync(0xFFFFFFFFu, kq, o);
    }
    if (lane < 8) {
        red[warp][lane][0] = sk;
        red[warp][lane][1] = sq;
        if (lane == 0) red_s[warp] = make_float4(kk, qq, kq, 0.0f);
    }
    __syncthreads();
    sk = sq = zero;
    kk = qq = kq = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float4 x = red[i][cg][0], y = red[i][cg][1], z = red_s[i];
        sk.x += x.x; sk.y += x.y; sk.z += x.z; sk.w += x.w;
        sq.x += y.x; sq.y += y.y; sq.z += y.z; sq.w += y.w;
        kk += z.x; qq += z.y; kq += z.z;
    }
    const float rk = 1.0f / sqrtf(kk + a.unit_eps), rq = a.q_scale / sqrtf(qq + a.unit_eps);
    const float4 u = make_float4(beta * (v.x - sk.x * rk), beta * (v.y - sk.y * rk), beta * (v.z - sk.z * rk), beta * (v.w - sk.w * rk));
    const float c = kq * rk * rq;
    float4 o = make_float4(fmaf(c, u.x, sq.x * rq), fmaf(c, u.y, sq.y * rq), fmaf(c, u.z, sq.z * rq), fmaf(c, u.w, sq.w * rq));
    if (live) {
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int n = phase + 32 * i;
            if (n >= a.key_pad) break;
            const float f = kn[i] * rk;
            *reinterpret_cast<float4*>(st + (size_t)n * a.value_pad) =
                make_float4(fmaf(f, u.x, s[i].x), fmaf(f, u.y, s[i].y), fmaf(f, u.z, s[i].z), fmaf(f, u.w, s[i].w));
        }
    }
    if (a.norm_w) {
        float ss = o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w;      // columns beyond the head are zero
        ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 1);
        ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 2);
        ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 4);
        if (parts > 1) {
            cluster_wait();
            if (tid < (int)parts) store_peer(&s_part[cluster_rank()], tid, ss);
            cluster_arrive();
            cluster_wait();
            ss = 0.0f;
            for (uint32_t i = 0; i < parts; i++) ss += s_part[i];
        }
        const float f = 1.0f / sqrtf(ss / (float)a.value_dim + a.eps);
        o = make_float4(o.x * f * nw.x * sigmoid_act<A>(gate.x), o.y * f * nw.y * sigmoid_act<A>(gate.y), o.z * f * nw.z * sigmoid_act<A>(gate.z),
                        o.w * f * nw.w * sigmoid_act<A>(gate.w));
    }
    if (phase == 0 && live) act_store4(reinterpret_cast<A*>(a.o) + at, o);
}

template <typename A, int NI>
static int launch_token(const DeltaRule& a, cudaStream_t s)
{
    int parts = 1;
    while (parts * kTokenCols < a.value_pad) parts *= 2;
    return launch_cluster(k_delta_token<A, NI>, dim3(a.heads, parts), dim3(1, a.norm_w ? parts : 1), 256, 0, s, a);
}

template <typename A>
static int delta_token(const DeltaRule& a, cudaStream_t s)
{
    if (a.key_pad <= 32) return launch_token<A, 1>(a, s);
    if (a.key_pad <= 64) return launch_token<A, 2>(a, s);
    if (a.key_pad <= 128) return launch_token<A, 4>(a, s);
    if (a.key_pad <= 256) return launch_token<A, 8>(a, s);
    return launch_token<A, 16>(a, s);
}

bool delta_token_norms(int key_pad, int value_pad) { return key_pad <= 512 && value_pad <= 8 * kTokenCols; }

// ------------------------------------------------------------------ recurrence

// grid (heads, value columns / 32), eight warps of four columns; lane: keys 4 (lane & 7) + 32 i + j of column lane >> 3.  Tokens
// pass through shared memory in blocks of TB with unit lengths, decays and k.q worked out.
template <int NI, int TB>
struct DeltaStage {
    static constexpr int kKeys = 32 * NI, kToken = 3 * kKeys + kTokenCols + 4;
    static constexpr size_t kSmem = 2 * (size_t)TB * kToken * 4;
};

template <typename A, int NI, int TB>
__global__ void __launch_bounds__(256) k_delta_recurrence(DeltaRule a, int T)
{
    using S = DeltaStage<NI, TB>;
    extern __shared__ __align__(16) float sm[];      // [2][TB] of k, q, decay [kKeys] each, v [32], beta, k.q
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kl = 4 * (lane & 7);
    const int h = blockIdx.x, g = h / (a.heads / a.groups), c0 = blockIdx.y * kTokenCols;
    const int col = 4 * warp + (lane >> 3);
    const bool live = c0 + col < a.value_pad;
    pdl_launch_dependents();
    pdl_wait();
    float* st = a.state + (size_t)h * a.key_pad * a.value_pad + c0 + col;
    float s[4 * NI];
#pragma unroll
    for (int i = 0; i < 4 * NI; i++) {
        const int n = kl + 32 * (i >> 2) + (i & 3);
        s[i] = (live && n < a.key_pad) ? st[(size_t)n * a.value_pad] : 0.0f;
    }
    auto stage = [&](int t0, int b) {
        for (int r = warp; r < TB && t0 + r < T; r += 8) {
            const size_t t = t0 + r;
            float* dst = sm + (size_t)(b * TB + r) * S::kToken;
            const A* k = reinterpret_cast<const A*>(a.k) + t * a.ld + g * a.key_pad;
            const A* q = reinterpret_cast<const A*>(a.q) + t * a.ld + g * a.key_pad;
            const float* lg = a.log_decay + (t * a.heads + h) * a.key_pad;
            float kv[NI], qv[NI], dv[NI], kk = 0.0f, qq = 0.0f, kq = 0.0f;
#pragma unroll
            for (int i = 0; i < NI; i++) {
                const int n = lane + 32 * i;
                const bool in = n < a.key_pad;
                kv[i] = in ? act_load(k + n) : 0.0f;
                qv[i] = in ? act_load(q + n) : 0.0f;
                dv[i] = in ? lg[n] : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < NI; i++) { kk = fmaf(kv[i], kv[i], kk); qq = fmaf(qv[i], qv[i], qq); kq = fmaf(kv[i], qv[i], kq); }
            kk = warp_sum(kk);
            qq = warp_sum(qq);
            kq = warp_sum(kq);
            const float rk = 1.0f / sqrtf(kk + a.unit_eps), rq = a.q_scale / sqrtf(qq + a.unit_eps);
#pragma unroll
            for (int i = 0; i < NI; i++) {
                dst[lane + 32 * i] = kv[i] * rk;
                dst[S::kKeys + lane + 32 * i] = qv[i] * rq;
                dst[2 * S::kKeys + lane + 32 * i] = decay_of<A>(dv[i]);
            }
            dst[3 * S::kKeys + lane] = c0 + lane < a.value_pad ? act_load(reinterpret_cast<const A*>(a.v) + t * a.ld + (size_t)h * a.value_pad + c0 + lane) : 0.0f;
            if (lane == 0) {
                dst[3 * S::kKeys + kTokenCols] = a.beta[t * a.heads + h];
                dst[3 * S::kKeys + kTokenCols + 1] = kq * rk * rq;
            }
        }
    };
    stage(0, 0);
    for (int t0 = 0, b = 0; t0 < T; t0 += TB, b ^= 1) {
        __syncthreads();                    // this block is here, everybody has left the other buffer
        if (t0 + TB < T) stage(t0 + TB, b ^ 1);
        const int n_t = T - t0 < TB ? T - t0 : TB;
        for (int r = 0; r < n_t; r++) {
            const float* src = sm + (size_t)(b * TB + r) * S::kToken;
            float4 k4[NI];
            float sk = 0.0f, sq = 0.0f;
#pragma unroll
            for (int i = 0; i < NI; i++) {
                k4[i] = *reinterpret_cast<const float4*>(src + kl + 32 * i);
                const float4 q4 = *reinterpret_cast<const float4*>(src + S::kKeys + kl + 32 * i);
                const float4 d4 = *reinterpret_cast<const float4*>(src + 2 * S::kKeys + kl + 32 * i);
                s[4 * i] *= d4.x; s[4 * i + 1] *= d4.y; s[4 * i + 2] *= d4.z; s[4 * i + 3] *= d4.w;
                sk = fmaf(s[4 * i], k4[i].x, sk); sk = fmaf(s[4 * i + 1], k4[i].y, sk); sk = fmaf(s[4 * i + 2], k4[i].z, sk); sk = fmaf(s[4 * i + 3], k4[i].w, sk);
                sq = fmaf(s[4 * i], q4.x, sq); sq = fmaf(s[4 * i + 1], q4.y, sq); sq = fmaf(s[4 * i + 2], q4.z, sq); sq = fmaf(s[4 * i + 3], q4.w, sq);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                sk += __shfl_xor_sync(0xFFFFFFFFu, sk, o);
                sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
            }
            const float u = src[3 * S::kKeys + kTokenCols] * (src[3 * S::kKeys + col] - sk);
#pragma unroll
            for (int i = 0; i < NI; i++) {
                s[4 * i] = fmaf(k4[i].x, u, s[4 * i]); s[4 * i + 1] = fmaf(k4[i].y, u, s[4 * i + 1]);
                s[4 * i + 2] = fmaf(k4[i].z, u, s[4 * i + 2]); s[4 * i + 3] = fmaf(k4[i].w, u, s[4 * i + 3]);
            }
            if ((lane & 7) == 0 && live)
                reinterpret_cast<A*>(a.o)[((size_t)(t0 + r) * a.heads + h) * a.value_pad + c0 + col] =
                    act_from<A>(fmaf(src[3 * S::kKeys + kTokenCols + 1], u, sq));
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < 4 * NI; i++) {
            const int n = kl + 32 * (i >> 2) + (i & 3);
            if (n < a.key_pad) st[(size_t)n * a.value_pad] = s[i];
        }
    }
}

template <typename A, int NI, int TB>
static int launch_delta_recurrence(const DeltaRule& a, int T, cudaStream_t s)
{
    constexpr size_t smem = DeltaStage<NI, TB>::kSmem;
    int rc = allow_smem<k_delta_recurrence<A, NI, TB>>((int)smem);
    if (rc) return rc;
    return launch_ordered(k_delta_recurrence<A, NI, TB>, dim3(a.heads, (a.value_pad + kTokenCols - 1) / kTokenCols), 256, smem, s, a, T);
}

template <typename A>
static int delta_recurrence(const DeltaRule& a, int T, cudaStream_t s)
{
    if (a.key_pad <= 32) return launch_delta_recurrence<A, 1, 16>(a, T, s);
    if (a.key_pad <= 64) return launch_delta_recurrence<A, 2, 16>(a, T, s);
    if (a.key_pad <= 128) return launch_delta_recurrence<A, 4, 16>(a, T, s);
    if (a.key_pad <= 256) return launch_delta_recurrence<A, 8, 8>(a, T, s);
    return launch_delta_recurrence<A, 16, 8>(a, T, s);
}

// ------------------------------------------------------------------ chunks of 16 tokens

constexpr int kChunk = 16;
constexpr int kSegmentChunks = 64;          // chunks worked out at a time: what they need stays in L2

// Of a chunk and head, in the order in which k_delta_chunks' lanes read them: fragments of -W, Q and of the keys with the decays
// that follow them (64 bytes per key each: two bf16 numbers per value), then c_15 in fp32.
__host__ __device__ constexpr size_t fragment_bytes(int key_pad) { return (size_t)key_pad * (3 * 64 + 4); }
// U and O: [value column block of 16][U, O][lane][8]
__host__ __device__ constexpr size_t update_floats(int value_pad) { return (size_t)value_pad * 2 * kChunk; }

// v[j] of all lanes added up: lane j gets the sum of v[j].
__device__ __forceinline__ float transposed_sum(float (&v)[32], int lane)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
        }
    }
    return v[0];
}

// grid (heads, chunks); tokens t0 .. t1 - 1, those beyond count as zeros that neither decay nor write.  A thread per key (rounded up to whole warps)
// and as many again for the value columns.  Bound by latency: a CTA goes through a chain of some thousand instructions.  A and P are sums over
// the keys: a warp takes whole columns of both, four keys per lane, from k, q and the decays in shared memory, so that a column
// is added up across lanes once.  16 heads of 128 x 128, 64 tokens, with the kernel below: 15.6 us; with the sums of its own 32 keys of all columns in every
// warp and the value columns after the keys in the same threads 15.9; with lengths that scale the finished sums 15.1, but NaN where a square length
// leaves fp32.
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) k_delta_prepare(DeltaRule a, uint8_t* frags, float* updates, int t0, int t1)
{
    extern __shared__ __align__(16) uint8_t sf[];     // k, q, decays [token][key]; then the chunk's fragments
    __shared__ float4 sA[kChunk][4], sP[kChunk][4];
    __shared__ float s_norm[kThreads / 64][2 * kChunk], s_beta[kChunk];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int h = blockIdx.x, gr = h / (a.heads / a.groups), first = t0 + blockIdx.y * kChunk, left = t1 - first;
    const int D = a.key_pad, V = a.value_pad, n = tid, values = blockDim.x >> 1;      // first thread of the value columns
    const bool key = n < D;
    const bf16* pv = reinterpret_cast<const bf16*>(a.v) + (size_t)first * a.ld + (size_t)h * V;
    pdl_launch_dependents();
    pdl_wait();
    // the first half: k, q and decays of a key; the second: a value column
    float x[kChunk];
    if (tid < values) {
        float k[kChunk], q[kChunk], g[kChunk];
        const bf16* pk = reinterpret_cast<const bf16*>(a.k) + (size_t)first * a.ld + gr * D + n;
        const bf16* pq = reinterpret_cast<const bf16*>(a.q) + (size_t)first * a.ld + gr * D + n;
        const float* pd = a.log_decay + ((size_t)first * a.heads + h) * D + n;
        const int rows = key ? left : 0, step = a.heads * D;
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            k[i] = i < rows ? act_load(pk + i * a.ld) : 0.0f;
            q[i] = i < rows ? act_load(pq + i * a.ld) : 0.0f;
            g[i] = i < rows ? pd[i * step] : 0.0f;
        }
        if (tid < kChunk) s_beta[tid] = first + tid < t1 ? a.beta[(size_t)(first + tid) * a.heads + h] : 0.0f;
        // unit lengths ahead of every product: whatever a square length is, products of two unit vectors are at most 1 (an infinite one leaves zeros)
        float v[32];
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            v[i] = k[i] * k[i];
            v[kChunk + i] = q[i] * q[i];
        }
        s_norm[warp][lane] = transposed_sum(v, lane);
        float* to = reinterpret_cast<float*>(sf) + n;
#pragma unroll
        for (int i = 0; i < kChunk; i++)
            if (key) to[(2 * kChunk + i) * D] = expf(g[i]);
        named_bar_sync(1, values);
        float sum = 0.0f;
#pragma unroll
        for (int w = 0; w < kThreads / 64; w++) sum += 32 * w < values ? s_norm[w][lane] : 0.0f;
        const float unit = (lane < kChunk ? 1.0f : a.q_scale) / sqrtf(sum + a.unit_eps);      // a lane per token: of its k, of its q
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            const float ku = k[i] * __shfl_sync(0xFFFFFFFFu, unit, i), qu = q[i] * __shfl_sync(0xFFFFFFFFu, unit, kChunk + i);
            if (key) {
                to[i * D] = ku;
                to[(kChunk + i) * D] = qu;
            }
        }
    } else {
        const int p = tid - values;
#pragma unroll
        for (int i = 0; i < kChunk; i++) x[i] = i < left && p < V ? act_load(pv + i * a.ld + p) : 0.0f;
    }
    __syncthreads();
    // column m of P and A at distance d from the diagonal (A has none on it); a long column and a short one to each warp
    for (int pass = 0; pass * warps < kChunk; pass++) {
        const int m = pass * warps + (pass & 1 ? warps - 1 - warp : warp);
        if (m >= kChunk) continue;
        float v[32];
#pragma unroll
        for (int d = 0; d < 32; d++) v[d] = 0.0f;
        for (int n4 = 4 * lane; n4 < D; n4 += 128) {
            const float* col = reinterpret_cast<const float*>(sf) + m * D + n4;
            float4 r = make_float4(0, 0, 0, 0);
#pragma unroll
            for (int d = 0; d < kChunk; d++) {
                if (m + d >= kChunk) break;
                const float4 kk = *reinterpret_cast<const float4*>(col + d * D), qv = *reinterpret_cast<const float4*>(col + (kChunk + d) * D);
                if (d == 0) {
                    r = kk;
                } else {
                    const float4 f = *reinterpret_cast<const float4*>(col + (2 * kChunk + d) * D);
                    r = make_float4(r.x * f.x, r.y * f.y, r.z * f.z, r.w * f.w);
                }
                v[d] = fmaf(qv.x, r.x, v[d]); v[d] = fmaf(qv.y, r.y, v[d]); v[d] = fmaf(qv.z, r.z, v[d]); v[d] = fmaf(qv.w, r.w, v[d]);
                if (d == 0) continue;
                float& w = v[kChunk + d];
                w = fmaf(kk.x, r.x, w); w = fmaf(kk.y, r.y, w); w = fmaf(kk.z, r.z, w); w = fmaf(kk.w, r.w, w);
            }
        }
        const float sum = transposed_sum(v, lane);
        const int i = m + (lane & (kChunk - 1));
        if (i < kChunk) {
            if (lane < kChunk) reinterpret_cast<float*>(sP)[i * kChunk + m] = sum;
            else if (i > m) reinterpret_cast<float*>(sA)[i * kChunk + m] = sum * s_beta[i];
        }
    }
    float k[kChunk], q[kChunk], g[kChunk];
    if (tid < values) {
        const float* from = reinterpret_cast<const float*>(sf) + (key ? n : 0);
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            k[i] = from[i * D];
            q[i] = from[(kChunk + i) * D];
            g[i] = from[(2 * kChunk + i) * D];
        }
    }
    __syncthreads();
    // the first n entries of a row
    auto load_row = [](const float4 (&m)[kChunk][4], int i, int n, float (&r)[kChunk]) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (4 * j < n) *reinterpret_cast<float4*>(r + 4 * j) = m[i][j];
    };
    const size_t cell = (size_t)blockIdx.y * a.heads + h;
    if (key && tid < values) {
        uint32_t* fw = reinterpret_cast<uint32_t*>(sf);
        uint32_t* fq = fw + 16 * D;
        uint32_t* fk = fq + 16 * D;
        // the keys with the decays that follow them: a lane's 16 bytes are tokens 2 t, 2 t + 1 and 2 t + 8, 2 t + 9 of one key
        float z[kChunk], r = 1.0f;
#pragma unroll
        for (int i = kChunk - 1; i >= 0; i--) {
            z[i] = k[i] * r;
            r *= g[i];
        }
        reinterpret_cast<float*>(fk + 16 * D)[n] = r;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            uint4 w;
            split_bf16(z[2 * t], z[2 * t + 1], w.x, w.z);
            split_bf16(z[2 * t + 8], z[2 * t + 9], w.y, w.w);
            *reinterpret_cast<uint4*>(fk + ((n >> 3) * 32 + (n & 7) * 4 + t) * 4) = w;
        }
        // W by forward substitution, Q from it
        float w[kChunk], c = 1.0f;
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            c *= g[i];
            w[i] = s_beta[i] * k[i] * c;
            z[i] = q[i] * c;
        }
#pragma unroll
        for (int i = 0; i < kChunk; i++) {
            asm volatile("" ::: "memory");      // (rows read far ahead would be kept in local memory)
            alignas(16) float ar[kChunk], pr[kChunk];
            load_row(sA, i, i, ar);
            load_row(sP, i, i + 1, pr);
#pragma unroll
            for (int j = 0; j < i; j++) {
                w[i] = fmaf(-ar[j], w[j], w[i]);
                z[i] = fmaf(-pr[j], w[j], z[i]);
            }
            z[i] = fmaf(-pr[i], w[i], z[i]);
        }
        // keys n and n + 1 share a register: the even thread writes tokens 0 .. 7, the odd one 8 .. 15
        const unsigned live = D - (n & ~31) >= 32 ? 0xFFFFFFFFu : 0xFFFFu;
        const bool odd = n & 1;
        const int nn = (n & 15) >> 1;
        const size_t at = (((size_t)(n >> 4) * 2 + odd) * 32 + (nn & 3)) * 4 + (nn >> 2);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float pw = __shfl_xor_sync(live, odd ? w[i] : w[i + 8], 1), pz = __shfl_xor_sync(live, odd ? z[i] : z[i + 8], 1);
            const float w0 = odd ? pw : w[i], w1 = odd ? w[i + 8] : pw, z0 = odd ? pz : z[i], z1 = odd ? z[i + 8] : pz;
            uint32_t hi, lo;
            split_bf16(-w0, -w1, hi, lo);
            fw[at + 16 * i] = hi;
            fw[at + 16 * i + 2] = lo;
            split_bf16(z0, z1, hi, lo);
            fq[at + 16 * i] = hi;
            fq[at + 16 * i + 2] = lo;
        }
    } else if (tid >= values) {
        float* up = updates + cell * update_floats(V);
        for (int p = tid - values; p < V; p += values) {
            float u[kChunk], o[kChunk];
            if (p != tid - values) {
#pragma unroll
                for (int i = 0; i < kChunk; i++) x[i] = i < left ? act_load(pv + i * a.ld + p) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < kChunk; i++) {
                asm volatile("" ::: "memory");      // (rows read far ahead would be kept in local memory)
                float y = s_beta[i] * x[i], z = 0.0f;
                alignas(16) float ar[kChunk], pr[kChunk];
                load_row(sA, i, i, ar);
                load_row(sP, i, i + 1, pr);
#pragma unroll
                for (int j = 0; j < i; j++) {
                    y = fmaf(-ar[j], u[j], y);
                    z = fmaf(pr[j], u[j], z);
                }
                u[i] = y;
                o[i] = fmaf(pr[i], y, z);
            }
            float* dst = up + (size_t)(p >> 4) * 512 + (p & 7) * 32 + ((p >> 3) & 1) * 2;
#pragma unroll
            for (int t = 0; t < 4; t++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    *reinterpret_cast<float2*>(dst + t * 8 + e * 4) = make_float2(u[8 * e + 2 * t], u[8 * e + 2 * t + 1]);
                    *reinterpret_cast<float2*>(dst + 256 + t * 8 + e * 4) = make_float2(o[8 * e + 2 * t], o[8 * e + 2 * t + 1]);
                }
        }
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(frags + cell * fragment_bytes(D));
    for (int i = tid; i < (int)(fragment_bytes(D) / 16); i += blockDim.x) dst[i] = reinterpret_cast<const uint4*>(sf)[i];
}

// (Not a barrier for the compiler: loads of other shared memory may pass it; an arrival on a barrier publishes it.)
__device__ __forceinline__ void store_shared(uint32_t at, const uint32_t (&v)[4])
{
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
}

// A whole warp's wait: `ready` is what a look ahead of time said.  After a wait that ran out (`alive` is false, the code is recorded) none waits.
__device__ __forceinline__ void warp_wait(uint64_t* bar, uint32_t parity, bool ready, bool& alive, int* err, int code)
{
    if (__all_sync(0xFFFFFFFFu, ready)) return;
    if (alive) alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(bar, parity, err, code));
}

template <int NMAX, int kBlocks>
struct DeltaChunks {
    static constexpr int kStages = NMAX == 256 ? (kBlocks == 1 ? 3 : 2) : 4;
    static constexpr size_t kState = (size_t)NMAX / 16 * 1024;      // fragments of 16 columns of the state, high and low parts
    static size_t smem(int key_pad) { return kStages * (fragment_bytes(key_pad) + (size_t)kBlocks * kState); }
};

// grid (heads, value columns / (16 kBlocks)).  Of each block of 16 value columns two warps hold the state, half of the keys each, and two read it
// out, eight tokens each; the last warp feeds.  The chunks are one serial chain: 96 products of 10 cycles with and into a state of 128 keys, and what
// lies between them.  So the keys are on two warps, which exchange their parts of u, and each chunk has one wait of
// the state's warps on a barrier in memory, looked at ahead of time, and one meeting.  With a warp per block and three such waits (130 cycles each, even
// of barriers long complete) a chunk took 0.93 us, now 0.6 (16 heads of 128 x 128).
// kExact: the keys are NMAX, so that no step of the products hangs on a branch.
template <int NMAX, bool kExact, int kBlocks>
__global__ void __launch_bounds__(32 * (4 * kBlocks + 1), 1) k_delta_chunks(DeltaRule a, const uint8_t* frags, const float* updates, int t0, int t1, int chunks, int* err)
{
    using S = DeltaChunks<NMAX, kBlocks>;
    constexpr int KS = NMAX / 16, KH = KS / 2, NT = NMAX / 16;      // K steps of a read-out and of a half, the half's tiles of 8 keys
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[S::kStages], empty[S::kStages], written[kBlocks][S::kStages];
    __shared__ float4 s_part[kBlocks][2][2][2][32];                 // [block][buffer][half][..]: a half's part of u
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g4 = lane >> 2, t4 = lane & 3;
    const int h = blockIdx.x, D = kExact ? NMAX : a.key_pad, V = a.value_pad, ks_n = D / 16;
    const int left = V / 16 - kBlocks * (int)blockIdx.y, blocks = left < kBlocks ? left : kBlocks;
    const uint32_t bytes = (uint32_t)fragment_bytes(D);
    uint8_t* s_state = smem + S::kStages * (size_t)bytes;
    if (tid == 0) {
        for (int i = 0; i < S::kStages; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 4 * blocks); }
        for (int i = 0; i < kBlocks * S::kStages; i++) mbar_init(&written[0][0] + i, 1);
        mbar_init_fence();
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();
    if (warp == 4 * kBlocks) {
        if (lane == 0) {
            int c = 0;
            for (; c < chunks; c++) {
                const int s = c % S::kStages;
                if (c >= S::kStages && !mbar_wait_bounded(&empty[s], (uint32_t)(c / S::kStages - 1) & 1u, err, 61)) break;
                mbar_expect_tx(&full[s], bytes);
                bulk_g2s(smem + s * (size_t)bytes, frags + ((size_t)c * a.heads + h) * bytes, bytes, &full[s]);
            }
            for (int i = c > S::kStages ? c - S::kStages : 0; i < c; i++)      // no copy is left in flight
                if (!mbar_wait_bounded(&full[i % S::kStages], (uint32_t)(i / S::kStages) & 1u, err, 66)) break;
        }
        return;
    }
    const bool reads = warp >= 2 * kBlocks;
    const int pair = (warp >> 1) % kBlocks, half = warp & 1, block = kBlocks * blockIdx.y + pair;
    if (pair >= blocks) return;
    // a stage's state lies beside its fragments: whoever sees the next ones there knows that all warps have left both
    uint8_t* mine = s_state + (size_t)pair * S::kStages * S::kState + lane * 16;
    const float* up = updates + (size_t)h * update_floats(V) + (size_t)block * 512 + reads * 256 + lane * 8;
    const size_t next_up = (size_t)a.heads * update_floats(V);
    bool alive = true;
    int s = 0;
    uint32_t phase = 0;
    if (!reads) {
        // ---------------- the state, transposed: rows are value columns, columns are this half's keys
        const int k0 = half * KH, n0 = half * (NMAX / 2);
        float st[NT][4];
        float* gs = a.state + (size_t)h * D * V + 16 * block + g4;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int n = n0 + 8 * j + 2 * t4 + (e & 1);
                st[j][e] = n < D ? gs[(size_t)n * V + 8 * (e >> 1)] : 0.0f;
            }
        const float4 none = make_float4(0, 0, 0, 0);
        float4 u0 = half ? none : *reinterpret_cast<const float4*>(up), u1 = half ? none : *reinterpret_cast<const float4*>(up + 4);
        bool ready = false;
        for (int c = 0; c < chunks; c++) {
            const int b = c & 1;
            warp_wait(&full[s], phase, ready, alive, err, 62);
            const uint8_t* f = smem + s * (size_t)bytes;
            const uint32_t to = smem_addr(mine + s * S::kState);
            float x[2][4] = {{u0.x, u0.y, u0.z, u0.w}, {u1.x, u1.y, u1.z, u1.w}}, y[2][4] = {}, z[2][4] = {};
            if (!half && c + 1 < chunks) {
                up += next_up;
                u0 = *reinterpret_cast<const float4*>(up);
                u1 = *reinterpret_cast<const float4*>(up + 4);
            }
            const uint4* fw = reinterpret_cast<const uint4*>(f) + lane;
            const float* decay = reinterpret_cast<const float*>(f + (size_t)192 * D) + n0 + 2 * t4;
#pragma unroll
            for (int i = 0; i < KH; i++) {
                const int ks = k0 + i;
                if (ks >= ks_n) break;
                const uint4 w0 = fw[2 * ks * 32], w1 = fw[(2 * ks + 1) * 32];
                const float2 d0 = *reinterpret_cast<const float2*>(decay + 16 * i), d1 = *reinterpret_cast<const float2*>(decay + 16 * i + 8);
                uint32_t ah[4], al[4];
                split_bf16(st[2 * i][0], st[2 * i][1], ah[0], al[0]);
                split_bf16(st[2 * i][2], st[2 * i][3], ah[1], al[1]);
                split_bf16(st[2 * i + 1][0], st[2 * i + 1][1], ah[2], al[2]);
                split_bf16(st[2 * i + 1][2], st[2 * i + 1][3], ah[3], al[3]);
                store_shared(to + ks * 1024, ah);
                store_shared(to + ks * 1024 + 512, al);
                mma_bf16(x[0], ah, w0.x, w0.y);
                mma_bf16(x[1], ah, w1.x, w1.y);
                mma_bf16(y[0], ah, w0.z, w0.w);
                mma_bf16(y[1], ah, w1.z, w1.w);
                mma_bf16(z[0], al, w0.x, w0.y);
                mma_bf16(z[1], al, w1.x, w1.y);
                st[2 * i][0] *= d0.x; st[2 * i][1] *= d0.y; st[2 * i][2] *= d0.x; st[2 * i][3] *= d0.y;
                st[2 * i + 1][0] *= d1.x; st[2 * i + 1][1] *= d1.y; st[2 * i + 1][2] *= d1.x; st[2 * i + 1][3] *= d1.y;
            }
            // u: this half's part to the other half, and its part from there
#pragma unroll
            for (int e = 0; e < 2; e++) {
#pragma unroll
                for (int r = 0; r < 4; r++) x[e][r] += y[e][r] + z[e][r];
                s_part[pair][b][half][e][lane] = make_float4(x[e][0], x[e][1], x[e][2], x[e][3]);
            }
            named_bar_sync(1 + pair, 64);
            if (half == 0 && lane == 0) mbar_arrive(&written[pair][s]);
            const uint8_t* fk = f + (size_t)128 * D + (size_t)n0 * 64;
            uint32_t uh[4], ul[4];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float4 v = s_part[pair][b][half ^ 1][e][lane];
                split_bf16(x[e][0] + v.x, x[e][1] + v.y, uh[2 * e], ul[2 * e]);
                split_bf16(x[e][2] + v.z, x[e][3] + v.w, uh[2 * e + 1], ul[2 * e + 1]);
            }
            uint64_t* gone = &empty[s];
            if (++s == S::kStages) { s = 0; phase ^= 1; }
            ready = mbar_test(&full[s], phase);
            constexpr int kAtOnce = NT < 8 ? NT : 8;
#pragma unroll
            for (int j = 0; j < NT; j += kAtOnce) {
                if (n0 + 8 * j >= D) break;
                uint4 kf[kAtOnce];
#pragma unroll
                for (int i = 0; i < kAtOnce; i++)
                    kf[i] = n0 + 8 * (j + i) < D ? *reinterpret_cast<const uint4*>(fk + ((j + i) * 32 + lane) * 16) : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int i = 0; i < kAtOnce; i++) mma_bf16(st[j + i], uh, kf[i].x, kf[i].y);
#pragma unroll
                for (int i = 0; i < kAtOnce; i++) mma_bf16(st[j + i], uh, kf[i].z, kf[i].w);
#pragma unroll
                for (int i = 0; i < kAtOnce; i++) mma_bf16(st[j + i], ul, kf[i].x, kf[i].y);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(gone);
        }
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int n = n0 + 8 * j + 2 * t4 + (e & 1);
                if (n < D) gs[(size_t)n * V + 8 * (e >> 1)] = st[j][e];
            }
    } else {
        // ---------------- the read-out of tokens 8 half .. 8 half + 7
        bf16* out = reinterpret_cast<bf16*>(a.o) + (size_t)h * V + 16 * block + (g4 & ~1);
        up += 4 * half;
        float4 u = *reinterpret_cast<const float4*>(up);
        for (int c = 0; c < chunks; c++) {
            warp_wait(&written[pair][s], phase, false, alive, err, 65);      // (and so the fragments are there)
            const uint8_t* f = smem + s * (size_t)bytes + (size_t)64 * D;
            float x[4] = {u.x, u.y, u.z, u.w}, y[4] = {}, z[4] = {};
            if (c + 1 < chunks) u = *reinterpret_cast<const float4*>(up += next_up);
            const uint4* fq = reinterpret_cast<const uint4*>(f) + 32 * half + lane;
            const uint4* from = reinterpret_cast<const uint4*>(mine + s * S::kState);
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                if (ks >= ks_n) break;
                const uint4 hi = from[2 * ks * 32], lo = from[(2 * ks + 1) * 32], w = fq[2 * ks * 32];
                const uint32_t ah[4] = {hi.x, hi.y, hi.z, hi.w}, al[4] = {lo.x, lo.y, lo.z, lo.w};
                mma_bf16(x, ah, w.x, w.y);
                mma_bf16(y, ah, w.z, w.w);
                mma_bf16(z, al, w.x, w.y);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (++s == S::kStages) { s = 0; phase ^= 1; }
            // two neighbouring columns per store: lanes of even columns finish even tokens, those of odd ones odd tokens
            const bool odd = g4 & 1;
#pragma unroll
            for (int r = 0; r < 4; r += 2) {
                const float v0 = x[r] + (y[r] + z[r]), v1 = x[r + 1] + (y[r + 1] + z[r + 1]);
                const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? v0 : v1, 4);
                const int t = t0 + kChunk * c + 8 * half + 2 * t4 + odd;
                if (t < t1)
                    *reinterpret_cast<uint32_t*>(out + (size_t)t * a.heads * V + 4 * r) = odd ? pack_bf16(other, v1) : pack_bf16(v0, other);
            }
        }
    }
}

template <int NMAX, bool kExact, int kBlocks>
static int launch_walk(const DeltaRule& a, const uint8_t* frags, const float* updates, int t0, int t1, int chunks, cudaStream_t s)
{
    int rc = allow_smem<k_delta_chunks<NMAX, kExact, kBlocks>>((int)DeltaChunks<NMAX, kBlocks>::smem(NMAX));
    if (rc) return rc;
    return launch_ordered(k_delta_chunks<NMAX, kExact, kBlocks>, dim3(a.heads, (a.value_pad / 16 + kBlocks - 1) / kBlocks), 32 * (4 * kBlocks + 1),
                          DeltaChunks<NMAX, kBlocks>::smem(a.key_pad), s, a, frags, updates, t0, t1, chunks, device_error_flag());
}

template <int NMAX, bool kExact>
static int launch_chunks(const DeltaRule& a, int T, cudaStream_t s)
{
    int rc;
    constexpr auto prepare = k_delta_prepare<NMAX == 256 ? 512 : 256, NMAX == 256 ? 1 : 2>;
    if ((rc = allow_smem<prepare>((int)fragment_bytes(256)))) return rc;
    for (int t0 = 0; t0 < T; t0 += kSegmentChunks * kChunk) {
        const int t1 = T - t0 < kSegmentChunks * kChunk ? T : t0 + kSegmentChunks * kChunk, chunks = (t1 - t0 + kChunk - 1) / kChunk;
        uint8_t* frags = (uint8_t*)a.scratch;
        float* updates = (float*)(frags + (size_t)chunks * a.heads * fragment_bytes(a.key_pad));
        if ((rc = launch_ordered(prepare, dim3(a.heads, chunks), (a.key_pad + 31) / 32 * 64, fragment_bytes(a.key_pad), s, a, frags, updates, t0, t1)))
            return rc;
        // One block of value columns per CTA while every CTA has an SM of its own: 16 heads of 128 x 128, 700 tokens 62 us, with two 66; 8 of
        // 256 x 256, 95 and 128.  With more CTAs than SMs the fragments would only be read twice as often, and with few keys two blocks
        // are the faster always (16 heads of 64 x 64: 56 us, with one 64; 8 of 64 x 128, 2000 tokens: 110, 131).
        constexpr int kAlone = NMAX > 64 ? 1 : 2;
        if (a.heads * (a.value_pad / 16) <= sm_count()) rc = launch_walk<NMAX, kExact, kAlone>(a, frags, updates, t0, t1, chunks, s);
        else rc = launch_walk<NMAX, kExact, 2>(a, frags, updates, t0, t1, chunks, s);
        if (rc) return rc;
    }
    return 0;
}

// ------------------------------------------------------------------ host side

// From this many tokens on a bf16 prompt goes through the chunked kernels.
constexpr int kChunkedMinTokens = 32;
static bool takes_chunks(int key_pad, int T, bool act_bf16) { return act_bf16 && T >= kChunkedMinTokens && key_pad <= 256; }

size_t delta_scratch_bytes(int heads, int key_pad, int value_pad, int T, bool act_bf16)
{
    if (!takes_chunks(key_pad, T, act_bf16)) return 0;
    const int chunks = (T + kChunk - 1) / kChunk;
    return (size_t)(chunks < kSegmentChunks ? chunks : kSegmentChunks) * heads * (fragment_bytes(key_pad) + 4 * update_floats(value_pad));
}

int delta_rule(const DeltaRule& a, int T, bool act_bf16, cudaStream_t s)
{
    if (a.heads < 1 || a.groups < 1 || a.heads % a.groups || a.key_pad % 16 || a.value_pad % 16 || a.ld % 8 || T < 1) return latch(BPDQ_ERR_ARG);
    if (a.key_pad > 512) return latch(BPDQ_ERR_RANGE);
    if (a.norm_w && (T > 1 || !a.gate || !delta_token_norms(a.key_pad, a.value_pad))) return latch(BPDQ_ERR_ARG);
    if (T == 1) return act_bf16 ? delta_token<bf16>(a, s) : delta_token<float>(a, s);
    if (a.scratch && takes_chunks(a.key_pad, T, act_bf16)) {
        if (a.key_pad == 64) return launch_chunks<64, true>(a, T, s);
        if (a.key_pad == 128) return launch_chunks<128, true>(a, T, s);
        if (a.key_pad < 64) return launch_chunks<64, false>(a, T, s);
        if (a.key_pad < 128) return launch_chunks<128, false>(a, T, s);
        return launch_chunks<256, false>(a, T, s);
    }
    return act_bf16 ? delta_recurrence<bf16>(a, T, s) : delta_recurrence<float>(a, T, s);
}

}  // namespace bpdq

using namespace bpdq;

extern "C" {

int bpd_delta_rule_cuda(const void* q, const void* k, const void* v, int ld, const float* log_decay, const float* beta, float q_scale, float unit_eps,
                        float* state, void* o, const float* norm_w, const void* gate, float eps, int n_tokens, int heads, int groups, int key_pad,
                        int value_dim, int value_pad, int act_bf16, void* stream)
{
    if (n_tokens < 0 || heads < 1 || groups < 1 || key_pad < 16 || value_pad < 16 || value_dim < 1 || value_dim > value_pad) return latch(BPDQ_ERR_ARG);
    if (n_tokens == 0) return 0;
    if (!q || !k || !v || !log_decay || !beta || !state || !o) return latch(BPDQ_ERR_ARG);
    DeltaRule a = {};
    a.q = q; a.k = k; a.v = v;
    a.ld = ld;
    a.heads = heads; a.groups = groups; a.key_pad = key_pad; a.value_dim = value_dim; a.value_pad = value_pad;
    a.log_decay = log_decay;
    a.beta = beta;
    a.q_scale = q_scale; a.unit_eps = unit_eps;
    a.state = state;
    a.o = o;
    a.norm_w = norm_w; a.gate = gate; a.eps = eps;
    const size_t scratch = delta_scratch_bytes(heads, key_pad, value_pad, n_tokens, act_bf16 != 0);
    if (scratch) {
        int rc = 0;
        if (!(a.scratch = scratch_take(nullptr, kScratchDelta, scratch, (cudaStream_t)stream, &rc))) return rc;
    }
    return delta_rule(a, n_tokens, act_bf16 != 0, (cudaStream_t)stream);
}

}  // extern "C"
