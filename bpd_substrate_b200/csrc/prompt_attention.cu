// Attention of prompts on tcgen05 (prompt_attention.cuh).  A CTA = 128 rows of one key head, row = (token, query head that shares it), against blocks of
// 128 keys:
//   warp 0      tiled bulk copies of queries, keys and values into 128-byte-swizzled shared memory
//   warp 1      tensor memory, MMAs: scores S = Q K^T of the next block ahead of the sums O += P V of this one
//   warps 2-9   softmax: two threads per row, 64 keys each; weights go back to tensor memory over the scores they came from, as the sum of two bf16
//               numbers (two MMAs), and stay fp32 in the row's sum
// O stays in tensor memory.  It is rescaled only when a row's maximum has grown by more than 2^8 since the last time: until then weights are
// taken relative to the older maximum (at most 2^8, the same relative precision).  Capped scores need no maximum at all.
//
// What bounds it: a block's round (scores, softmax, sums) of about 1.4 us, in which the tensor pipe works about half of the time and the exponentials
// take 1024 cycles (three such units per capped score: 2.3 us).  With what comes ahead of it, us, on mma.sync and here: 16 latent heads of 128 + 64, 2048
// tokens 209, 57; 200 tokens after 1800 147, 50; 16 heads on 4 key heads of 128, 700 tokens, capped 48, 24, plain 47, 20.  Distance from 64 bits as before.
#include "prompt_attention.cuh"
#include "launch.cuh"
#include "mma_device.cuh"
#include "tcgen05_device.cuh"
#include "tensor_map.cuh"

namespace bpdq {

constexpr int kPaRows = 128, kPaKeys = 128, kPaPiece = 128 * 64 * 2;      // rows of a tile, keys of a block, bytes of 128 rows x 64 columns
constexpr int kPaSoftWarps = 8, kPaThreads = 32 * (2 + kPaSoftWarps);
constexpr float kPaLog2e = 1.44269504088896340736f;
constexpr float kPaGrowth = 8.0f;                                         // log2 of how far weights may exceed 1
// As in the kernel on mma.sync: with a sink the sum is at least e^-cap; up to this cap whatever underflows beside that is below fp32's resolution.
constexpr float kPaMaxCap = 64.0f;

struct PaShape {
    int T, groups, share, tiles;
    int pieces, pieces1;                // 64-column pieces of a query, and of its part in `keys`
    int value_dim, chunk;
    int key_col, value_col;             // columns between groups
    float f, in, out;                   // plain: log2 e * scale; capped: see softmax
    bf16* o;
};

__host__ __device__ constexpr int pa_smem(int pieces, int dv) { return 1024 + 3 * pieces * kPaPiece + 2 * (dv / 64) * kPaPiece + 4 * kPaRows * 4 + 256; }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),
          "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]),
          "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <int DV, bool kCapped>
__global__ void __launch_bounds__(kPaThreads, 1)
k_prompt_attn_tc5(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap rmap,
                  const __grid_constant__ CUtensorMap vmap, const PaShape p, const int* pos_p, int* err)
{
    constexpr int kHalves = DV / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sq = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sk = sq + p.pieces * kPaPiece;             // [2][pieces]
    uint8_t* sv = sk + 2 * p.pieces * kPaPiece;         // [2][kHalves]
    float* s_max = reinterpret_cast<float*>(sv + 2 * kHalves * kPaPiece);       // [2][2][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_max + 4 * kPaRows);
    uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 7, *s_full = bars + 9, *p_full = bars + 11,
             *o_done = bars + 13, *pair = bars + 14;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(q_full, 1);
        mbar_init(o_done, 1);
        for (int i = 0; i < 2; i++) {
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_full[i], kPaSoftWarps);
        }
        for (int i = 0; i < 4; i++) mbar_init(&pair[i], 2);      // the two warps of a quarter's rows
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, t_o = tmem + 256;         // scores and weights in columns 0 .. 127 and 128 .. 255 in turn
    pdl_launch_dependents();
    pdl_wait();
    const int pos = *pos_p;

    const int g = blockIdx.x % p.groups, tile = p.tiles - 1 - (int)blockIdx.x / p.groups;      // the longest rows first
    const int per = kPaRows / p.share, t0 = tile * per, n_t = p.T - t0 < per ? p.T - t0 : per;
    const int first = pos + t0, k_begin = p.chunk > 0 ? first / p.chunk * p.chunk : 0, k_end = first + n_t;
    const int blocks = (k_end - k_begin + kPaKeys - 1) / kPaKeys;
    const int v0 = blockIdx.y * DV;

    if (warp == 0) {
        // ---------------- copies
        if (lane == 0) {
            mbar_expect_tx(q_full, (uint32_t)(p.pieces * kPaPiece));
            for (int u = 0; u < p.pieces; u++) tma_rows_3d(sq + u * kPaPiece, &qmap, 64 * u, g * p.share, t0, q_full);
            for (int i = 0; i < blocks; i++) {
                const int b = i & 1, k0 = k_begin + i * kPaKeys;
                const uint32_t par = (uint32_t)((i >> 1) - 1) & 1u;
                if (i >= 2 && !mbar_wait_bounded(&k_empty[b], par, err, 61)) break;
                mbar_expect_tx(&k_full[b], (uint32_t)(p.pieces * kPaPiece));
                uint8_t* at = sk + b * p.pieces * kPaPiece;
                for (int u = 0; u < p.pieces; u++) {
                    if (u < p.pieces1) tma_rows_2d(at + u * kPaPiece, &kmap, g * p.key_col + 64 * u, k0, &k_full[b]);
                    else tma_rows_2d(at + u * kPaPiece, &rmap, 64 * (u - p.pieces1), k0, &k_full[b]);
                }
                if (i >= 2 && !mbar_wait_bounded(&v_empty[b], par, err, 62)) break;
                mbar_expect_tx(&v_full[b], (uint32_t)(kHalves * kPaPiece));
                for (int u = 0; u < kHalves; u++) tma_rows_2d(sv + (b * kHalves + u) * kPaPiece, &vmap, g * p.value_col + v0 + 64 * u, k0, &v_full[b]);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMAs
        if (elect_one()) {
            constexpr uint32_t fmt = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPaRows >> 4) << 24);
            constexpr uint32_t idesc_s = fmt | ((uint32_t)(kPaKeys >> 3) << 17), idesc_o = fmt | (1u << 16) | ((uint32_t)(DV >> 3) << 17);
            const uint64_t qd = swizzled_desc(smem_addr(sq));
            bool ok = mbar_wait_bounded(q_full, 0, err, 63);
            auto scores = [&](int i) {
                const int b = i & 1;
                if (!mbar_wait_bounded(&k_full[b], (uint32_t)(i >> 1) & 1u, err, 64)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t kd = swizzled_desc(smem_addr(sk + b * p.pieces * kPaPiece));
                for (int u = 0; u < p.pieces; u++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        umma_bf16_ss(tmem + 128 * b, qd + (uint64_t)(u * (kPaPiece >> 4) + 2 * k), kd + (uint64_t)(u * (kPaPiece >> 4) + 2 * k), idesc_s, u | k ? 1u : 0u);
                umma_commit(&s_full[b]);
                umma_commit(&k_empty[b]);
                return true;
            };
            ok = ok && scores(0);
            for (int i = 0; ok && i < blocks; i++) {
                const int b = i & 1;
                if (i + 1 < blocks && !scores(i + 1)) break;
                if (!mbar_wait_bounded(&v_full[b], (uint32_t)(i >> 1) & 1u, err, 65)) break;
                if (!mbar_wait_bounded(&p_full[b], (uint32_t)(i >> 1) & 1u, err, 66)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t vd = swizzled_desc_mn(smem_addr(sv + b * kHalves * kPaPiece), kPaPiece);
                // weights of keys 0 .. 63: columns 0 .. 31 and their small parts 32 .. 63; of keys 64 .. 127 from column 64 on
#pragma unroll
                for (int k = 0; k < kPaKeys / 16; k++) {
                    const uint32_t a = tmem + 128 * b + (k < 4 ? 8 * k : 32 + 8 * k);
                    umma_bf16_ts(t_o, a + 32, vd + (uint64_t)(k * 128), idesc_o, i | k ? 1u : 0u);
                    umma_bf16_ts(t_o, a, vd + (uint64_t)(k * 128), idesc_o, 1u);
                }
                umma_commit(o_done);
                umma_commit(&v_empty[b]);
            }
        }
        __syncwarp();
    } else {
        // ---------------- softmax
        const int quarter = warp & 3, half = (warp - 2) >> 2, r = 32 * quarter + lane;
        const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
        const int t = t0 + r / p.share, at = pos + t;
        const int last = t < t0 + n_t ? at : -1, lo = p.chunk > 0 ? at / p.chunk * p.chunk : 0;
        // the warp's rows need no mask between these positions
        const int r_end = t0 + (32 * quarter + 31) / p.share;
        const int w_last = pos + t0 + 32 * quarter / p.share, w_lo = p.chunk > 0 ? (pos + r_end) / p.chunk * p.chunk : 0;
        float top = -INFINITY, sum = 0.0f;
        // what the other half of a row holds; the slots alternate, so that one is read while the next is written
        uint32_t met = 0;
        auto other_half = [&](float mine, float& theirs) {
            float* slot = s_max + (met & 1) * 2 * kPaRows;
            slot[half * kPaRows + r] = mine;
            __syncwarp();
            if (lane == 0) mbar_arrive(&pair[quarter]);
            if (!mbar_wait_bounded(&pair[quarter], met & 1u, err, 70)) return false;
            met++;
            theirs = slot[(1 - half) * kPaRows + r];
            return true;
        };
        bool ok = true;
        for (int i = 0; i < blocks; i++) {
            const int b = i & 1, k0 = k_begin + i * kPaKeys + 64 * half;
            if (!mbar_wait_bounded(&s_full[b], (uint32_t)(i >> 1) & 1u, err, 67)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ts = tmem + lanes + 128 * b + 64 * half;
            float v[64];
            tmem_ld32(ts, v);
            tmem_ld32(ts + 32, v + 32);
            tmem_wait_ld();
            const bool edge = k0 + 63 > w_last || k0 < w_lo || w_last >= pos + t0 + n_t;
            float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (kCapped) {
                // tanh(z) = 1 - 2 / (1 + e^(2 z)); weights relative to the cap
#pragma unroll
                for (int j = 0; j < 64; j++) {
                    v[j] = ex2(p.out * __fdividef(1.0f, 1.0f + ex2(v[j] * p.in)));
                    if (edge && (k0 + j > last || k0 + j < lo)) v[j] = 0.0f;
                    part[j & 3] += v[j];
                }
            } else {
                if (edge) {
#pragma unroll
                    for (int j = 0; j < 64; j++)
                        if (k0 + j > last || k0 + j < lo) v[j] = -INFINITY;
                }
                float m = v[0];
#pragma unroll
                for (int j = 1; j < 64; j++) m = fmaxf(m, v[j]);
                float theirs;
                if (!other_half(m, theirs)) { ok = false; break; }
                m = fmaxf(m, theirs);
                const bool grown = (m - top) * p.f > kPaGrowth;
                if (i > 0 && __any_sync(0xFFFFFFFFu, grown)) {
                    if (!mbar_wait_bounded(o_done, (uint32_t)(i - 1) & 1u, err, 68)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const float down = grown ? ex2((top - m) * p.f) : 1.0f;
                    sum *= down;
#pragma unroll
                    for (int c = 0; c < DV / 2; c += 16) {
                        int ov[16];
                        const uint32_t ta = t_o + lanes + half * (DV / 2) + c;
                        tmem_ld(ta, ov);
                        tmem_wait_ld();
                        uint32_t st[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) st[j] = __float_as_uint(__int_as_float(ov[j]) * down);
                        tmem_st(ta, st);
                    }
                }
                if (grown) top = m;
                const float base = top == -INFINITY ? 0.0f : top * p.f;
#pragma unroll
                for (int j = 0; j < 64; j++) {
                    v[j] = ex2(fmaf(v[j], p.f, -base));
                    part[j & 3] += v[j];
                }
            }
            sum += (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t hi[16], low[16];
#pragma unroll
                for (int j = 0; j < 16; j++) split_bf16(v[32 * c + 2 * j], v[32 * c + 2 * j + 1], hi[j], low[j]);
                tmem_st(ts + 16 * c, hi);
                tmem_st(ts + 32 + 16 * c, low);
            }
            tmem_wait_st();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[b]);
        }
        if (ok && !mbar_wait_bounded(o_done, (uint32_t)(blocks - 1) & 1u, err, 69)) ok = false;
        float theirs;
        if (ok && other_half(sum, theirs)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            sum += theirs;
            if (kCapped) sum += ex2(0.5f * p.out);         // the sink: a score of 0, which is out / 2 below the cap
            const float inv = 1.0f / sum;
            bf16* dst = p.o + ((size_t)t * (p.groups * p.share) + g * p.share + r % p.share) * p.value_dim + v0 + half * (DV / 2);
#pragma unroll
            for (int c = 0; c < DV / 2; c += 16) {
                int ov[16];
                tmem_ld(t_o + lanes + half * (DV / 2) + c, ov);
                tmem_wait_ld();
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; j++) w[j] = pack_bf16(__int_as_float(ov[2 * j]) * inv, __int_as_float(ov[2 * j + 1]) * inv);
                if (last >= 0) {
                    *reinterpret_cast<uint4*>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
                    *reinterpret_cast<uint4*>(dst + c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------ host side

static int pa_value_tile(const PromptAttention& p) { return p.value_dim % 128 == 0 ? 128 : 64; }

bool prompt_attention_fits(const PromptAttention& p)
{
    if (p.T < 1 || p.context < p.T || p.share < 1 || p.share > kPaRows || kPaRows % p.share || p.dim % 64 || p.dim1 % 64 || p.dim1 < 64 || p.dim1 > p.dim || p.value_dim % 64) return false;
    if (pa_smem(p.dim / 64, pa_value_tile(p)) > 227 * 1024 || p.value_dim / 64 > 65535) return false;
    if (!(p.scale > 0.0f) || (p.cap != 0.0f && !(p.cap > 0.0f && p.cap <= kPaMaxCap))) return false;
    const uintptr_t places = (uintptr_t)p.q | (uintptr_t)p.keys | (uintptr_t)(p.dim > p.dim1 ? p.rest : p.keys) | (uintptr_t)p.values | (uintptr_t)p.o;
    return !(places & 15) && !((p.ld_q | p.ld_keys | (p.dim > p.dim1 ? p.ld_rest : 0) | p.ld_values) & 7);
}

template <int DV, bool kCapped>
static int launch_prompt(const PromptAttention& p, cudaStream_t s)
{
    const int per = kPaRows / p.share, pieces = p.dim / 64;
    CUtensorMap qmap, kmap, rmap, vmap;
    int rc;
    if ((rc = bf16_map(&qmap, p.q, p.dim, p.groups * p.share, p.dim, p.share, p.T, p.ld_q, per))) return rc;
    if ((rc = bf16_map(&kmap, p.keys, p.groups * p.dim1, p.context, p.ld_keys, kPaKeys))) return rc;
    rmap = kmap;
    if (p.dim > p.dim1 && (rc = bf16_map(&rmap, p.rest, p.dim - p.dim1, p.context, p.ld_rest, kPaKeys))) return rc;
    if ((rc = bf16_map(&vmap, p.values, p.groups * p.value_dim, p.context, p.ld_values, kPaKeys))) return rc;
    if ((rc = allow_smem<k_prompt_attn_tc5<DV, kCapped>>(227 * 1024))) return rc;
    PaShape a = {};
    a.T = p.T; a.groups = p.groups; a.share = p.share;
    a.tiles = (p.T + per - 1) / per;
    a.pieces = pieces; a.pieces1 = p.dim1 / 64;
    a.value_dim = p.value_dim; a.chunk = p.chunk;
    a.key_col = p.dim1; a.value_col = p.value_dim;
    a.f = p.scale * kPaLog2e;
    a.in = p.cap > 0.0f ? p.scale / p.cap * 2.0f * kPaLog2e : 0.0f;
    a.out = -2.0f * p.cap * kPaLog2e;
    a.o = p.o;
    return launch_ordered(k_prompt_attn_tc5<DV, kCapped>, dim3((unsigned)(a.tiles * p.groups), (unsigned)(p.value_dim / DV)), kPaThreads, (size_t)pa_smem(pieces, DV), s, qmap,
                          kmap, rmap, vmap, a, p.pos, device_error_flag());
}

int prompt_attention(const PromptAttention& p, cudaStream_t s)
{
    const bool wide = pa_value_tile(p) == 128;
    if (p.cap > 0.0f) return wide ? launch_prompt<128, true>(p, s) : launch_prompt<64, true>(p, s);
    return wide ? launch_prompt<128, false>(p, s) : launch_prompt<64, false>(p, s);
}

}  // namespace bpdq
