// Matrix products of the hybrid decoders: bf16 weights [N][K], activations bf16 or fp32, fp32 accumulation, and
// everything elementwise that follows a product as its epilogue (residual add between two dynamic-tanh norms, residual
// streams, SwiGLU of paired rows, GELU, step sizes, decays and the one-token convolution of a recurrent layer).  The
// dynamic-tanh norm needs no row statistics; an RMS norm ahead of a one-token product is taken into the product, whose
// CTAs all read the whole row anyway (the row enters times the norm's weight, the root mean square divides the sums).
//
//   k_linear_vec   one token: a warp streams two weight rows at a time with 16-byte loads, the first of them before the
//                  launch ahead has finished (weights are constant); HBM bound
//   k_linear_tc5   several tokens, bf16: tcgen05.mma kind::f16, 128 weight rows (TMEM lanes) x up to 256 tokens
//                  (TMEM columns) per tile, persistent CTAs, operands by tiled TMA into a 128-byte-swizzled ring, two
//                  accumulators so that a tile's epilogue runs under the next tile's products; large products on pairs of
//                  CTAs (cta_group::2), 256 rows per tile, each CTA fetching its rows and half of the tokens
//   k_linear_tile  several tokens, fp32: plain fp32 multiply-adds on tiles of 64 rows x 16 or 64 tokens
#include "cluster_device.cuh"
#include "decoder_device.cuh"
#include "launch.cuh"
#include "tcgen05_device.cuh"
#include "tensor_map.cuh"
#include "../../include/bpdq.h"

namespace bpdq {

// ------------------------------------------------------------------ one token

// R rows of a warp at a time: two, or one where there are not enough rows to give every warp two (16 loads in flight either way).
// What bounds it: HBM behind the latency of a group of rows. 2048 rows of 7168 with two rows each gave 1024 of 2368 warps work.  A decoded token of
// the hybrid decoder at 4000 keys: 281 us with pairs only, 272 with single rows where they fit.
template <typename A, int R>
__global__ void __launch_bounds__(256, 2) k_linear_vec(Linear l)
{
    extern __shared__ float4 xs[];      // [2][K / 8]: first and second four of every eight activations (split: twice)
    __shared__ float s_sum[8];
    constexpr int kBatch = 16 / R;      // 16-byte loads in flight per row and lane
    const int units = l.K / 8, groups = (l.N + R - 1) / R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int stride = gridDim.x * 8;
    int p = blockIdx.x + gridDim.x * warp;      // groups of rows are dealt over the CTAs first: every SM gets its share
    pdl_launch_dependents();
    uint4 w[R][kBatch];
    auto fetch = [&](int base) {
        const uint4* a = reinterpret_cast<const uint4*>(l.W + (size_t)(R * p) * l.K);
        const uint4* b = reinterpret_cast<const uint4*>(l.W + (size_t)(R * p + R - 1 < l.N ? R * p + R - 1 : R * p) * l.K);
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
            const int u = base + lane + 32 * i;
            w[0][i] = u < units ? __ldg(a + u) : make_uint4(0, 0, 0, 0);
            if (R > 1) w[R - 1][i] = u < units ? __ldg(b + u) : make_uint4(0, 0, 0, 0);
        }
    };
    if (p < groups) fetch(0);
    pdl_wait();
    float rnorm = 1.0f;
    if (l.norm_w) {
        const float* in = reinterpret_cast<const float*>(l.in);
        float sum = 0.0f;
        for (int j = threadIdx.x; j < 2 * units; j += 256) {
            float4 v = act_load4(in + 4 * j);
            const float4 w4 = act_load4(l.norm_w + 4 * j);
            sum = fmaf(v.x, v.x, sum); sum = fmaf(v.y, v.y, sum); sum = fmaf(v.z, v.z, sum); sum = fmaf(v.w, v.w, sum);
            xs[(j & 1) * units + (j >> 1)] = make_float4(v.x * w4.x, v.y * w4.y, v.z * w4.z, v.w * w4.w);
        }
        sum = warp_sum(sum);
        if (lane == 0) s_sum[warp] = sum;
        __syncthreads();
        sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) sum += s_sum[i];
        rnorm = 1.0f / sqrtf(sum / (float)l.norm_n + l.norm_eps);
    } else {
        const A* in = reinterpret_cast<const A*>(l.in);
        for (int j = threadIdx.x; j < 2 * units; j += 256) xs[(j & 1) * units + (j >> 1)] = act_load4(in + 4 * j);
        if (l.split)
            for (int j = threadIdx.x; j < 2 * units; j += 256) xs[(2 + (j & 1)) * units + (j >> 1)] = act_load4(in + l.in2 + 4 * j);
        __syncthreads();
    }
    bool have = true;
    for (; p < groups; p += stride) {
        const int row = R * p + lane;
        const float4* x = l.split && R * p >= l.split ? xs + 2 * units : xs;
        const bool residual = l.mode == kLinResidual && lane < R && row < l.N;
        const bool streams = l.mode == kLinStreams && lane < R && row < l.N;
        float xo[kMaxStreams];
        if (streams) {
#pragma unroll
            for (int i = 0; i < kMaxStreams; i++) xo[i] = i < l.streams.n ? l.x[(size_t)i * l.ld_x + row] : 0.0f;
        }
        float xr = 0, pw = 0, pb = 0, nw = 0, nb = 0;       // what the residual epilogue of row R p + lane needs, ahead of its use
        if (residual) {
            xr = l.x[row];
            pw = l.post.w[row];
            pb = l.post.b[row];
            if (l.next.w) { nw = l.next.w[row]; nb = l.next.b[row]; }
        }
        float acc[R] = {};
        for (int base = 0; base < units; base += 32 * kBatch) {
            if (!have) fetch(base);
            have = false;
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
                const int u = base + lane + 32 * i;
                if (u >= units) break;
                const float4 x0 = x[u], x1 = x[units + u];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint4 q = w[r][i];
                    acc[r] = fmaf(__uint_as_float(q.x << 16), x0.x, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.x & 0xFFFF0000u), x0.y, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.y << 16), x0.z, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.y & 0xFFFF0000u), x0.w, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.z << 16), x1.x, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.z & 0xFFFF0000u), x1.y, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.w << 16), x1.z, acc[r]);
                    acc[r] = fmaf(__uint_as_float(q.w & 0xFFFF0000u), x1.w, acc[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = warp_sum(acc[r]);
        const float v = (lane ? acc[R - 1] : acc[0]) * rnorm;
        if (l.mode == kLinSwiglu) {
            if (lane == 0) reinterpret_cast<A*>(l.out)[p] = act_from<A>(silu_act<A>(acc[0] * rnorm) * (acc[R - 1] * rnorm));
        } else if (streams) {
            float u = 0.0f;
#pragma unroll
            for (int i = 0; i < kMaxStreams; i++) {
                if (i >= l.streams.n) break;
                float r = l.streams.out[i] * v;
#pragma unroll
                for (int j = 0; j < kMaxStreams; j++)
                    if (j < l.streams.n) r = fmaf(l.streams.mix[j][i], xo[j], r);
                l.x[(size_t)i * l.ld_x + row] = r;
                u = fmaf(l.streams.next[i], r, u);
            }
            l.u[row] = u;
        } else if (residual) {
            const float r = xr + fmaf(tanhf(l.post.alpha * v), pw, pb);
            l.x[row] = r;
            if (l.next.w) reinterpret_cast<A*>(l.out)[row] = act_from<A>(fmaf(tanhf(l.next.alpha * r), nw, nb));
        } else if (l.mode != kLinResidual && l.mode != kLinStreams && lane < R && row < l.N) {
            linear_store<A>(l, 0, row, v);
        }
    }
}

// ------------------------------------------------------------------ several tokens, fp32

// 64 rows x 16 J tokens per CTA (J: 1 or 4), four rows and J tokens per thread.  Bound by the chain of slabs of 16 columns where there are few
// tiles (12 tokens of 2048 x 2048: 104 us at J = 4, 82 at J = 1), else by the multiply-adds and the loads of their operands.  The next launches
// may start only when a CTA's sums are done: waiting CTAs of several launches pile up on the SMs otherwise, and a later launch of fewer CTAs than
// SMs finds itself on some of them (64 tokens through three layers of the hybrid decoder, width 1536: 3862 us, 2467 so).
template <int J>
__global__ void __launch_bounds__(256) k_linear_tile(Linear l, int T)
{
    __shared__ __align__(16) float sw[16][68], sx[16][16 * J + 4];
    const int tid = threadIdx.x, tr = tid & 15, tt = tid >> 4;      // rows 4 tr .., tokens J tt ..
    const int n0 = blockIdx.x * 64, t0 = blockIdx.y * 16 * J;
    pdl_wait();
    const float* in = reinterpret_cast<const float*>(l.in);
    float acc[J][4] = {};
    const int row = tid >> 2, kq = (tid & 3) * 4;
    for (int k0 = 0; k0 < l.K; k0 += 16) {
        float4 a = make_float4(0, 0, 0, 0), b = a;
        if (n0 + row < l.N) a = act_load4(l.W + (size_t)(n0 + row) * l.K + k0 + kq);
        if (row < 16 * J && t0 + row < T) b = act_load4(in + (size_t)(t0 + row) * l.ld_in + k0 + kq);
        sw[kq][row] = a.x; sw[kq + 1][row] = a.y; sw[kq + 2][row] = a.z; sw[kq + 3][row] = a.w;
        if (row < 16 * J) { sx[kq][row] = b.x; sx[kq + 1][row] = b.y; sx[kq + 2][row] = b.z; sx[kq + 3][row] = b.w; }
        __syncthreads();
        float part[J][4] = {};      // a block's sum on its own: long sums then lose less
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float4 wv = *reinterpret_cast<const float4*>(&sw[k][4 * tr]);
            const float wr[4] = {wv.x, wv.y, wv.z, wv.w};
            float xr[J];
            if constexpr (J == 4) {
                const float4 xv = *reinterpret_cast<const float4*>(&sx[k][4 * tt]);
                xr[0] = xv.x; xr[1] = xv.y; xr[2] = xv.z; xr[3] = xv.w;
            } else {
                xr[0] = sx[k][tt];
            }
#pragma unroll
            for (int j = 0; j < J; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) part[j][i] = fmaf(wr[i], xr[j], part[j][i]);
        }
#pragma unroll
        for (int j = 0; j < J; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[j][i] += part[j][i];
        __syncthreads();
    }
    pdl_launch_dependents();
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int t = t0 + J * tt + j;
        if (t >= T) break;
        if (l.mode == kLinSwiglu) {
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const int n = n0 + 4 * tr + i;
                if (n < l.N) reinterpret_cast<float*>(l.out)[(size_t)t * l.ld_out + n / 2] = silu_act<float>(acc[j][i]) * acc[j][i + 1];
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (n0 + 4 * tr + i < l.N) linear_store<float>(l, t, n0 + 4 * tr + i, acc[j][i]);
        }
    }
}

// ------------------------------------------------------------------ several tokens, bf16, tensor cores

// BN: the most tokens of a tile; a launch takes bn of them, a multiple of 16 above BN / 2, and as many ring stages as fit then.
template <int BN>
struct Tc5Linear {
    // Epilogue warps: three or two per TMEM lane quarter, each a share of the columns.  What follows the sums of a launch's last tile runs under nothing:
    // 8500 cycles of fp32 rows with eight warps and 256 tokens.  700 tokens, eight warps and one warp for all copies, now (us): 2048 x 2048 11.7, 10.5;
    // 6400 x 2048 22.6, 20.9; 2048 x 10752 33.2, 31.4.  (Sixteen warps leave 96 registers, which spill: 11.5, 22.2, 32.4.)
    static constexpr int kEpiWarps = BN > 64 ? 12 : 8;
    static constexpr int kThreads = 32 * (3 + kEpiWarps);
    static constexpr int kTmemCols = 2 * BN;
};
constexpr int kTc5Rows = 128, kTc5Depth = 64;                          // weight rows per tile, K elements per ring stage
constexpr int kTc5ABytes = kTc5Rows * kTc5Depth * 2, kTc5MaxStages = 8;
__host__ __device__ constexpr int tc5_stage_bytes(int bn) { return kTc5ABytes + bn * kTc5Depth * 2; }      // a multiple of 1024: the swizzle's atom
__host__ __device__ constexpr int tc5_stages(int bn)
{
    const int fit = 200 * 1024 / tc5_stage_bytes(bn);
    return fit < kTc5MaxStages ? fit : kTc5MaxStages;
}
constexpr int tc5_smem(int bn) { return 1024 + tc5_stages(bn) * tc5_stage_bytes(bn) + 8 * (2 * kTc5MaxStages + 4) + 16; }

template <int BN, bool kPair>
__global__ void __launch_bounds__(Tc5Linear<BN>::kThreads, 1)
k_linear_tc5(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, Linear l, int T, int bn, int* err)
{
    using S = Tc5Linear<BN>;
    constexpr int kCtas = kPair ? 2 : 1, kTileRows = kCtas * kTc5Rows;
    const int own = bn / kCtas;                // tokens of a tile whose rows this CTA fetches
    const int stages = tc5_stages(own), stage_bytes = tc5_stage_bytes(own);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + (size_t)stages * stage_bytes);
    uint64_t* empty = full + kTc5MaxStages;
    uint64_t* acc_full = empty + kTc5MaxStages;      // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(&full[s], 2); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], kCtas * S::kEpiWarps); }
        mbar_init_fence();
    }
    if (warp == 1) {
        if (kPair) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(S::kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(S::kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (kPair) {        // (the leader's barriers are there before anything is counted on them)
        cluster_arrive();
        cluster_wait();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    const int rank = kPair ? (int)pair_rank() : 0, unit = (int)blockIdx.x / kCtas, units = (int)gridDim.x / kCtas;      // a unit has a tile at a time
    const int n_tiles = (l.N + kTileRows - 1) / kTileRows, t_tiles = (T + bn - 1) / bn;
    // tokens vary fastest: the CTAs at work share few rows of weights, which go through HBM once
    const int tiles = n_tiles * t_tiles, kb_all = (l.K + kTc5Depth - 1) / kTc5Depth;
    // few tiles: the CTAs of a cluster take a range of K each and join their sums through shared memory (one tile per cluster then)
    const int ranges = gridDim.y, range = blockIdx.y, kb0 = range * kb_all / ranges, kb_n = (range + 1) * kb_all / ranges - kb0;
    float* part_sums = reinterpret_cast<float*>(ring);      // [bn][128], once all products are done

    // What follows the sums of a tile: a thread owns one weight row and walks over its tokens, 16 at a time.  sums(c0, v) gives tokens c0 ..
    // of the row, next_of(c0) the step that this thread takes after c0 (bn and beyond: none); the first residual rows are fetched before ready().
    const int quarter = warp & 3, r = 32 * quarter + lane;
    auto finish = [&](int tile, int c_first, auto ready, auto sums, auto next_of) {
        const int n = (tile / t_tiles) * kTileRows + rank * kTc5Rows + r;
        const int tb = (tile % t_tiles) * bn;
        const bool live = n < l.N;
        // residual rows are fetched a step of 16 tokens ahead, the first under the tile's products
        float xv[16];
        auto fetch_x = [&](int c0) {
#pragma unroll
            for (int j = 0; j < 16; j++) xv[j] = (live && tb + c0 + j < T) ? l.x[(size_t)(tb + c0 + j) * l.ld_x + n] : 0.0f;
        };
        if (l.mode == kLinResidual && c_first < bn) fetch_x(c_first);
        if (!ready()) return false;
        DynTanh post = l.post, next = l.next;
        float pw = 0, pb = 0, nw = 0, nb = 0;
        if (l.mode == kLinResidual && live) {
            pw = post.w[n]; pb = post.b[n];
            if (next.w) { nw = next.w[n]; nb = next.b[n]; }
        } else if (l.mode == kLinLogDecay && live) {
            pw = l.neg_exp_a[n]; pb = l.dt_bias[n];
        }
        const bool is_step = l.mode == kLinMixerIn && live && n >= l.dt_row;      // (lanes of one warp may differ)
        if (is_step && l.dt_bias) pb = l.dt_bias[n - l.dt_row];
        const bool plain_f32 = l.mode == kLinF32 && l.cap == 0.0f;
        // rows of this warp that are only rounded and stored (after a GELU)
        const int n_end = (n - lane) + 32;
        const bool plain_warp = !((l.N | l.ld_out) & 1) &&
                                (l.mode == kLinAct || l.mode == kLinGelu || (l.mode == kLinMixerIn && n_end <= l.dt_row && !l.conv.w));
        auto step = [&](int c0, int c_next, int (&v)[16]) {
            const int t0 = tb + c0;
            if (t0 >= T) return;
            if (l.mode == kLinResidual) {
                float xr[16];
#pragma unroll
                for (int j = 0; j < 16; j++) xr[j] = xv[j];
                if (c_next < bn) fetch_x(c_next);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float q = xr[j] + fmaf(tanhf(post.alpha * __int_as_float(v[j])), pw, pb);
                    if (live && t0 + j < T) {
                        l.x[(size_t)(t0 + j) * l.ld_x + n] = q;
                        if (next.w)
                            reinterpret_cast<bf16*>(l.out)[(size_t)(t0 + j) * l.ld_out + n] =
                                act_from<bf16>(fmaf(tanhf(next.alpha * q), nw, nb));
                    }
                }
            } else if (l.mode == kLinSwiglu) {
                // lane pairs hold gate (even) and up (odd): the even lane finishes even tokens, the odd lane odd ones
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float keep = __int_as_float((lane & 1) ? v[j + 1] : v[j]);
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, __int_as_float((lane & 1) ? v[j] : v[j + 1]), 1);
                    const float g = (lane & 1) ? other : keep, u = (lane & 1) ? keep : other;
                    const int t = t0 + j + (lane & 1);
                    if (live && t < T) reinterpret_cast<bf16*>(l.out)[(size_t)t * l.ld_out + n / 2] = act_from<bf16>(silu_act<bf16>(g) * u);
                }
            } else if (plain_warp) {
                if (l.mode == kLinGelu)
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = __float_as_int(gelu_act<bf16>(__int_as_float(v[j])));
                // two neighbouring rows per store: the even lane finishes even tokens, the odd lane odd ones
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float keep = __int_as_float((lane & 1) ? v[j + 1] : v[j]);
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, __int_as_float((lane & 1) ? v[j] : v[j + 1]), 1);
                    const __nv_bfloat162 two = __floats2bfloat162_rn((lane & 1) ? other : keep, (lane & 1) ? keep : other);
                    const int t = t0 + j + (lane & 1);
                    if (live && t < T) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<bf16*>(l.out) + (size_t)t * l.ld_out + (n & ~1)) = two;
                }
            } else if (plain_f32) {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (live && t0 + j < T) reinterpret_cast<float*>(l.out)[(size_t)(t0 + j) * l.ld_out + n] = __int_as_float(v[j]);
            } else if (l.mode == kLinLogDecay) {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (live && t0 + j < T) l.dt[(size_t)(t0 + j) * l.ld_dt + n] = pw * softplus_act<bf16>(__int_as_float(v[j]) + pb);
            } else if (is_step) {
                float q[16];
#pragma unroll
                for (int j = 0; j < 16; j++) q[j] = l.dt_bias ? softplus_act<bf16>(__int_as_float(v[j]) + pb) : sigmoid_act<bf16>(__int_as_float(v[j]));
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (t0 + j < T) l.dt[(size_t)(t0 + j) * l.ld_dt + n - l.dt_row] = q[j];
            } else if (live) {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (t0 + j < T) linear_store<bf16>(l, t0 + j, n, __int_as_float(v[j]));
            }
        };
        for (int c0 = c_first; c0 < bn; c0 = next_of(c0)) {
            int v[16];
            sums(c0, v);
            step(c0, next_of(c0), v);
        }
        return true;
    };

    if (warp == 0 || warp == 2) {
        // ---------------- copies: a warp for the weights, which do not wait for the launch ahead, one for the tokens.  (One thread for both took 470
        // cycles between two K blocks, mostly its own chain of instructions, and bounded tiles of up to 200 tokens.  A look at the next barrier ahead of time, by
        // which the issuing thread gains, is one answer more to wait for here: 32 tokens of 1024 x 1024 5.65 us, 5.28 without; 200 of 2048 x 2048 8.15, 7.82.)
        if (lane == 0) {
            const bool tokens = warp == 2;
            const uint32_t to0 = smem_addr(ring) + (tokens ? kTc5ABytes : 0), bytes = (uint32_t)(tokens ? own * kTc5Depth * 2 : kTc5ABytes);
            const uint32_t full0 = smem_addr(full), empty0 = smem_addr(empty), lead0 = kPair ? leader_addr(full) : full0;
            const CUtensorMap* map = tokens ? &xmap : &wmap;
            if (tokens) pdl_wait();
            uint32_t s = 0, par = 1;
            bool ok = true, first = true;       // (the ring's first round waits for nothing)
            for (int tile = unit; ok && tile < tiles; tile += units) {
                const int y = tokens ? (tile % t_tiles) * bn + rank * own : (tile / t_tiles) * kTileRows + rank * kTc5Rows;
                int x = kb0 * kTc5Depth;
                for (int kb = 0; kb < kb_n; kb++, x += kTc5Depth) {
                    if (!first && !mbar_wait_at(empty0 + 8 * s, par, err, 41)) { ok = false; break; }
                    if (!kPair || rank == 0) mbar_expect_tx_at(full0 + 8 * s, kCtas * bytes);
                    if (kPair) tma_pair_rows_2d_at(to0 + s * stage_bytes, map, x, y, lead0 + 8 * s);
                    else tma_rows_2d_at(to0 + s * stage_bytes, map, x, y, full0 + 8 * s);
                    if (++s == (uint32_t)stages) { s = 0; par ^= 1u; first = false; }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
        auto mma = [&](uint32_t d, uint64_t ad, uint64_t bd, uint32_t accum) {
            if (kPair) umma_pair_bf16_ss(d, ad, bd, idesc, accum);
            else umma_bf16_ss(d, ad, bd, idesc, accum);
        };
        auto commit = [](uint32_t bar) {
            if (kPair) umma_pair_commit_at(bar);
            else umma_commit_at(bar);
        };
        if (rank == 0 && elect_one()) {
            // one thread walks the steps.  Whether the next stage is there is asked before this one's products are issued, so that the
            // answer's latency passes under them: 168 K blocks of 2048 rows took 49, 53, 70 us at 16, 80, 256 tokens a tile, now 34, 38, 68
            const uint32_t full0 = smem_addr(full), empty0 = smem_addr(empty), acc0 = smem_addr(acc_full);
            const uint64_t a0 = swizzled_desc(smem_addr(ring)), b0 = swizzled_desc(smem_addr(ring) + kTc5ABytes);
            const int steps_last = (l.K - (kb0 + kb_n - 1) * kTc5Depth) / 16;      // products of the last K block of a tile, if fewer than four
            uint32_t s = 0, full_par = 0, local = 0;
            bool ok = true, ready = false;
            for (int tile = unit; ok && tile < tiles; tile += units, local++) {
                const uint32_t a = local & 1, acc_par = ((local >> 1) - 1) & 1u;
                if (local >= 2 && !(kPair ? mbar_wait_cluster(&acc_empty[a], acc_par, err, 42) : mbar_wait_bounded(&acc_empty[a], acc_par, err, 42))) break;
                const uint32_t d = tmem_base + a * BN;
                for (int kb = 0; kb < kb_n; kb++) {
                    if (!ready && !mbar_wait_at(full0 + 8 * s, full_par, err, 43)) { ok = false; break; }
                    const uint32_t now = s, at = s * (uint32_t)(stage_bytes >> 4);
                    if (++s == (uint32_t)stages) { s = 0; full_par ^= 1u; }
                    ready = mbar_test_at(full0 + 8 * s, full_par);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = a0 + at, bd = b0 + at;
                    mma(d, ad, bd, kb ? 1u : 0u);
                    if (kb + 1 < kb_n || steps_last >= 4) {
#pragma unroll
                        for (int k = 1; k < 4; k++) mma(d, ad + 2 * k, bd + 2 * k, 1u);
                    } else {
                        for (int k = 1; k < steps_last; k++) mma(d, ad + 2 * k, bd + 2 * k, 1u);
                    }
                    commit(empty0 + 8 * now);
                }
                if (ok) commit(acc0 + 8 * a);
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue
        constexpr int kShares = S::kEpiWarps / 4;
        const int share = (warp - 3) >> 2, steps = bn / 16, c_begin = share * steps / kShares * 16, c_end = (share + 1) * steps / kShares * 16;
        int local = 0;
        pdl_wait();
        for (int tile = unit; tile < tiles; tile += units, local++) {
            const int a = local & 1;
            const uint32_t ta = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(a * BN);
            auto ready = [&]() {
                if (!mbar_wait_bounded(&acc_full[a], (uint32_t)(local >> 1) & 1u, err, 44)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return true;
            };
            auto sums = [&](int c0, int (&v)[16]) {
                tmem_ld(ta + c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            };
            if (!kPair && ranges > 1) {
                if (!ready()) break;
                for (int c0 = c_begin; c0 < c_end; c0 += 16) {
                    int v[16];
                    sums(c0, v);
#pragma unroll
                    for (int j = 0; j < 16; j++) part_sums[(c0 + j) * kTc5Rows + r] = __int_as_float(v[j]);
                }
            } else if (!finish(tile, c_begin < c_end ? c_begin : bn, ready, sums, [&](int c0) { return c0 + 16 < c_end ? c0 + 16 : bn; })) {
                break;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (kPair) mbar_arrive_leader(leader_addr(&acc_empty[a]));
                else mbar_arrive(&acc_empty[a]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (kPair) {        // nobody leaves while its operands or barriers are in use
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (warp == 1) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmemCols) : "memory");
        }
    } else if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmemCols) : "memory");
    }
    if (!kPair && ranges > 1) {
        // every CTA finishes some of the tile's steps of 16 tokens, its epilogue warps' halves taking turns; ranges are added in their order
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (warp >= 3) {
            constexpr int kShares = S::kEpiWarps / 4;
            const int turn = 16 * kShares * ranges;
            finish(blockIdx.x, 16 * (kShares * range + ((warp - 3) >> 2)), []() { return true; },
                   [&](int c0, int (&v)[16]) {
                       float t[16];
#pragma unroll
                       for (int j = 0; j < 16; j++) t[j] = load_peer(part_sums + (c0 + j) * kTc5Rows + r, 0);
                       for (int q = 1; q < ranges; q++) {
                           float u[16];
#pragma unroll
                           for (int j = 0; j < 16; j++) u[j] = load_peer(part_sums + (c0 + j) * kTc5Rows + r, q);
#pragma unroll
                           for (int j = 0; j < 16; j++) t[j] += u[j];
                       }
#pragma unroll
                       for (int j = 0; j < 16; j++) v[j] = __float_as_int(t[j]);
                   },
                   [&](int c0) { return c0 + turn; });
        }
        __syncwarp();
        cluster_arrive();       // nobody leaves while its sums are read
        cluster_wait();
    }
}

// ------------------------------------------------------------------ host side

struct Tc5Tiles { int tokens, ranges, ctas; };      // of a tile; of K; CTAs that share a tile

template <int BN, bool kPair>
static int launch_tc5(const Linear& l, int T, Tc5Tiles t, cudaStream_t s)
{
    using S = Tc5Linear<BN>;
    CUtensorMap wmap, xmap;
    int rc;
    constexpr int kCtas = kPair ? 2 : 1;
    const int own = t.tokens / kCtas;
    if ((rc = bf16_map(&wmap, l.W, l.K, l.N, l.K, kTc5Rows))) return rc;
    if ((rc = bf16_map(&xmap, l.in, l.K, T, l.ld_in, own))) return rc;
    if ((rc = allow_smem<k_linear_tc5<BN, kPair>>(227 * 1024))) return rc;
    const long tiles = (long)((l.N + kCtas * kTc5Rows - 1) / (kCtas * kTc5Rows)) * ((T + t.tokens - 1) / t.tokens);
    const long units = sm_count() / kCtas;
    const unsigned grid = (unsigned)(kCtas * (t.ranges > 1 || tiles < units ? tiles : units));
    return launch_cluster(k_linear_tc5<BN, kPair>, dim3(grid, (unsigned)t.ranges), dim3(kCtas, (unsigned)t.ranges, 1), S::kThreads, tc5_smem(own), s, wmap, xmap, l, T,
                          t.tokens, device_error_flag());
}

// Tokens of a tile (a multiple of 16), ranges of K and CTAs of a tile with the least time in cycles: waves of CTAs over the SMs times a tile's K blocks, each
// 310 + 1.3 per token; K is cut, into ranges of at least four blocks, where all its tiles' clusters run at once, and joining r ranges costs
// 3000 + 800 r + 25 per token.  168 K blocks of 2048 rows take 29.2 us at 16 tokens a tile, 30.9 at 128, 34.6 at 160, 53.6 at 256 (335, 355, 395, 615 cycles a
// block: the estimate, which was fitted to one copying thread and eight epilogue warps, is high around 128 tokens).  Over 37 shapes of 5 to 4096 tokens
// its tiles are within 5 % of the best ones, but for 128 tokens of 4096 x 4096 (12.2 us, 11.1 possible) and 400 of 1024 x 4096 (11.6, 10.8).
// 2048 rows of 10752 (us, one range, several): 48 tokens 29.6, 11.3 at six; 200 tokens 30.1, 16.6 at four; of 2048: 16 tokens 7.9, 6.7 at four; 200 tokens
// 8.2, 8.6 at two.
static Tc5Tiles tc5_tiles(const Linear& l, int T)
{
    const int n_tiles = (l.N + kTc5Rows - 1) / kTc5Rows, top = (T + 15) / 16 * 16 < 256 ? (T + 15) / 16 * 16 : 256;
    const int kb = (l.K + kTc5Depth - 1) / kTc5Depth, sms = sm_count();
    const int* clusters = active_clusters<k_linear_tc5<256, false>>(Tc5Linear<256>::kThreads, 200 * 1024);      // (a CTA has an SM to itself)
    Tc5Tiles best = {16, 1, 1};
    double least = 0.0;
    for (int bn = 16; bn <= top; bn += 16) {
        const long tiles = (long)n_tiles * ((T + bn - 1) / bn);
        for (int ranges = 1; ranges <= 8 && (ranges == 1 || (clusters && tiles <= clusters[ranges] && kb / ranges >= 4)); ranges++) {
            const long waves = ranges > 1 ? 1 : (tiles + sms - 1) / sms;
            const double time = (double)waves * ((kb + ranges - 1) / ranges) * (310.0 + 1.3 * bn) + (ranges > 1 ? 3000.0 + 800.0 * ranges + 25.0 * bn : 0.0);
            if ((bn == 16 && ranges == 1) || time <= least) { best = {bn, ranges, 1}; least = time; }
        }
    }
    // A pair has 256 rows to a tile and fetches a third less per product; a K block takes 180 + 1.65 per token (168 of 2048 rows, 700 tokens, us: 128
    // tokens a tile 36, 192 43, 256 56).  Setting it up costs more than one CTA, so only wide tiles and several waves: us, best single CTAs, pairs:
    // 2048 tokens of 10752 x 2048 81.2, 78.8; of 21504 x 2048 172, 161; 1024 of 14336 x 4096 111, 99; 2048 of 2048 x 2048 16.0, 17.9.
    const int pairs = sms / 2, row_pairs = (l.N + 2 * kTc5Rows - 1) / (2 * kTc5Rows);
    for (int bn = 192; bn <= top; bn += 32) {
        const long waves = ((long)row_pairs * ((T + bn - 1) / bn) + pairs - 1) / pairs;
        const double time = (double)waves * kb * (180.0 + 1.65 * bn) + 2500.0;
        if (waves >= 2 && time < least) { best = {bn, 1, 2}; least = time; }
    }
    return best;
}

template <typename A, int R>
static int launch_vec(const Linear& l, size_t smem, cudaStream_t s)
{
    int rc = allow_smem<k_linear_vec<A, R>>(200 * 1024);
    if (rc) return rc;
    const int want = (l.N + R - 1) / R, cap = 2 * sm_count();
    return launch_ordered(k_linear_vec<A, R>, want < cap ? want : cap, 256, smem, s, l);
}

int linear_forward(const Linear& l, int T, bool act_bf16, cudaStream_t s)
{
    if (l.K % 16 || l.K < 16 || l.N < 1 || T < 1 || l.ld_in % 8) return latch(BPDQ_ERR_ARG);
    if (T > 1 && (l.norm_w || l.split || l.mode == kLinStreams)) return latch(BPDQ_ERR_ARG);
    if (l.mode == kLinStreams && (l.streams.n < 1 || l.streams.n > kMaxStreams)) return latch(BPDQ_ERR_ARG);
    if (T == 1) {
        const size_t smem = (size_t)l.K * (l.split ? 8 : 4);
        if (smem > 200 * 1024) return latch(BPDQ_ERR_RANGE);
        // one row per warp and step as long as two would leave warps without any (a gate and its up are always two)
        const int warps = 2 * sm_count() * 8;
        const bool one = l.mode != kLinSwiglu && l.N <= warps;
        return act_bf16 ? (one ? launch_vec<bf16, 1>(l, smem, s) : launch_vec<bf16, 2>(l, smem, s))
                        : (one ? launch_vec<float, 1>(l, smem, s) : launch_vec<float, 2>(l, smem, s));
    }
    if (!act_bf16) {
        // narrow tiles while every SM has one at most (64 tokens of 2048 x 2048: 107 us wide, 83 narrow; 100 tokens: 107, 127), or two where 16
        // tokens are all there are (12 tokens of 14336 x 2048: 264, 214; of 22000 x 2048: 281, 324).  Both sides were measured with the next launches
        // started early; since then 12 tokens, back to back: narrow 14336 x 2048 144, 18944 x 2048 167; wide 19008 x 2048 221, 22000 x 2048 225
        const int n_tiles = (l.N + 63) / 64, narrow = (T + 15) / 16;
        if ((long)n_tiles * narrow <= (narrow == 1 ? 2 : 1) * sm_count()) return launch_ordered(k_linear_tile<1>, dim3(n_tiles, narrow), 256, 0, s, l, T);
        return launch_ordered(k_linear_tile<4>, dim3(n_tiles, (T + 63) / 64), 256, 0, s, l, T);
    }
    const Tc5Tiles t = tc5_tiles(l, T);
    if (t.ctas == 2) return launch_tc5<256, true>(l, T, t, s);
    if (t.tokens > 128) return launch_tc5<256, false>(l, T, t, s);
    if (t.tokens > 64) return launch_tc5<128, false>(l, T, t, s);
    if (t.tokens > 32) return launch_tc5<64, false>(l, T, t, s);
    return launch_tc5<32, false>(l, T, t, s);
}

}  // namespace bpdq

using namespace bpdq;

extern "C" {

// out[t][n] = sum_k W[n][k] x[t][k]: bf16 weights, bf16 or fp32 activations, fp32 results.  K a multiple of 16.
int bpd_linear_bf16_cuda(const uint16_t* W, const void* x, float* out, int n_tokens, int N, int K, int act_bf16, void* stream)
{
    if (n_tokens < 0 || N < 1 || K < 16 || (n_tokens > 0 && (!W || !x || !out))) return latch(BPDQ_ERR_ARG);
    if (((uintptr_t)W | (uintptr_t)x) & 15) return latch(BPDQ_ERR_ALIGN);
    if (n_tokens == 0) return 0;
    Linear l = {};
    l.W = reinterpret_cast<const bf16*>(W);
    l.in = x;
    l.N = N; l.K = K; l.ld_in = K;
    l.mode = kLinF32;
    l.out = out;
    l.ld_out = N;
    return linear_forward(l, n_tokens, act_bf16 != 0, (cudaStream_t)stream);
}

int bpdq_linear_bf16_ctas(int n_tokens, int N, int K)
{
    if (n_tokens < 2 || N < 1 || K < 16 || K % 16) return BPDQ_ERR_ARG;
    Linear l = {};
    l.N = N; l.K = K;
    return tc5_tiles(l, n_tokens).ctas;
}

int bpdq_linear_bf16_tiles(int n_tokens, int N, int K, int* tokens, int* ranges)
{
    if (n_tokens < 2 || N < 1 || K < 16 || K % 16 || !tokens || !ranges) return BPDQ_ERR_ARG;
    Linear l = {};
    l.N = N; l.K = K;
    const Tc5Tiles t = tc5_tiles(l, n_tokens);
    *tokens = t.tokens;
    *ranges = t.ranges;
    return 0;
}

// The same product followed by what a decoder's epilogues do to its sums (BPDQ_MAP_*).
int bpd_linear_map_cuda(const uint16_t* W, const void* x, void* out, int n_tokens, int N, int K, int map, const float* bias, const float* rate, float cap,
                        int act_bf16, void* stream)
{
    if (n_tokens < 0 || N < 1 || K < 16 || (n_tokens > 0 && (!W || !x || !out))) return latch(BPDQ_ERR_ARG);
    if (((uintptr_t)W | (uintptr_t)x) & 15) return latch(BPDQ_ERR_ALIGN);
    if (n_tokens == 0) return 0;
    Linear l = {};
    l.W = reinterpret_cast<const bf16*>(W);
    l.in = x;
    l.N = N; l.K = K; l.ld_in = K;
    l.out = out;
    l.ld_out = N;
    l.dt = reinterpret_cast<float*>(out);
    l.ld_dt = N;
    l.dt_bias = bias;
    l.neg_exp_a = rate;
    switch (map) {
    case BPDQ_MAP_GELU: l.mode = kLinGelu; break;
    case BPDQ_MAP_CAP:
        if (!(cap > 0.0f)) return latch(BPDQ_ERR_ARG);
        l.mode = kLinF32;
        l.cap = cap;
        break;
    case BPDQ_MAP_LOG_DECAY:
        if (!bias || !rate) return latch(BPDQ_ERR_ARG);
        l.mode = kLinLogDecay;
        break;
    case BPDQ_MAP_SIGMOID: l.mode = kLinMixerIn; l.dt_bias = nullptr; break;      // (rows from 0 on are write shares)
    default: return latch(BPDQ_ERR_ARG);
    }
    return linear_forward(l, n_tokens, act_bf16 != 0, (cudaStream_t)stream);
}

}  // extern "C"
