// Q8_0 x Q8_0 products of many tokens on re-tiled weights: the layout and the arithmetic of gemm_q8_0_tiles.cu, bit for bit.
// There an int8 MMA leaves an int32 sum per (row, token, block of 32), and five operations per sum (two of them the conversion)
// with the loads of the scales bound the kernel.  Here the tensor cores do all of it that is exact:
//   sum_j w_j a_j   the same whole numbers as fp16 operands; the fp32 sum is below 32 * 128 * 127 < 2^24, so exact in any order
//   wd * ad         an outer product: one more MMA per block whose operands are the scales (fp16, eleven bits each: exact in fp32)
// Two roundings are left per (row, token, block), sum * (wd * ad) and acc + that, both packed for two tokens, on values that the
// epilogue reads from tensor memory and nowhere else.
//
// A persistent CTA takes tiles of 128 rows x T tokens, tokens first, over up to three matrices that read the same activations:
//   warp 0        bulk copies of weight units, ahead of the launch before (weights are constant)
//   warp 1        tensor memory, MMAs: three of K = 16 per block into one of two sets of accumulators
//   warp 2        bulk copies of activation units (fp16 whole numbers and scales, written by k_quant_q8_0_wide)
//   warps 3-6     int8 weights to fp16 operands in the canonical K-major order
//   warps 7-22    epilogue: thread = row, T / 4 tokens per warp
// What bounds it: the handovers between the roles, about 530 of 680 cycles per block of 128 x 128 (MMA commit, sixteen warps that wait for it, their
// arrivals, the issuer's wait, for one block at a time and two sets of accumulators).  14336 x 4096, 1000 tokens, 319 us: with neither conversion
// nor anything in the epilogue but its barriers 252 are left; the conversion to fp16 alone adds 28, the epilogue's loads and sums 40 (its sums 15 of
// them); with one MMA per block instead of three it is 322.  Tensor pipe active 30 % of the time, issue 67 %.  In the narrow kernel 514 us
// (367 TFLOP/s here); 4096 x 14336: 484, 329.
// All waits are bounded; a role that gives up records a code and leaves, the others time out in turn, and warp 1 frees the tensor memory.
#include "bpdq_common.cuh"
#include "launch.cuh"
#include "q8_0_tiles.cuh"
#include "tcgen05_device.cuh"
#include "../../include/bpdq.h"

#include <cuda_fp16.h>

namespace bpdq {

template <int T>
struct WideShape {
    static constexpr int kSetBlocks = 128 / T;                      // blocks of 32 per accumulator set: 128 columns of sums, 128 of scales
    static constexpr int kBlocks = T == 32 ? 4 : 2;                 // blocks per ring stage
    static constexpr int kRawBytes = kBlocks * kTileUnit;           // a raw stage: weight units as they lie in memory
    static constexpr int kWUnit = kTileRows * (64 + 16);            // 128 x 32 fp16, then a K chunk with the scale and zeros
    static constexpr int kXUnit = T * (64 + 16);
    static constexpr int kOpBytes = kBlocks * (kWUnit + kXUnit);
    static constexpr int kRawStages = T == 32 ? 4 : 6;
    static constexpr int kOpStages = T == 128 ? 4 : T == 64 ? 5 : 3;
    static constexpr int kZeroBytes = 16 * kTileRows;               // a K chunk of zeros: the other half of a scale MMA's operands
    static constexpr int kExpandWarps = 4, kEpiWarps = 16;
    static constexpr int kThreads = 32 * (3 + kExpandWarps + kEpiWarps);
    static constexpr int kBarriers = 2 * kRawStages + 2 * kOpStages + 4;
    static constexpr size_t kSmem = (size_t)kRawStages * kRawBytes + (size_t)kOpStages * kOpBytes + kZeroBytes + 8 * kBarriers + 16;
    static_assert(kBlocks % kSetBlocks == 0, "a stage holds whole accumulator sets");
    static_assert(kSmem <= 227 * 1024, "shared memory of a CTA");
};

struct WideProducts {
    const uint8_t* tiles[kWideMatrices];
    float* out[kWideMatrices];
    int N[kWideMatrices], row_tile[kWideMatrices + 1];              // rows; first row tile of each matrix, one after the other
    int n, M, nb;
};

// ------------------------------------------------------------------ activations

// X fp32 [M][K] -> per (token tile, block) a unit of 80 T bytes: element (t, k) as fp16 at (k/8)*16*T + 16 t + 2 (k%8), then per token
// the fp16 scale and seven zeros.  The numbers are those of k_quant_q8_0_tiles (eight lanes per block); tokens beyond M quantize zeros.
// With `up` the numbers are silu(X) * up.  A prompt of 1000 tokens, four layers of an 8B Llama: 0.1 ms less than with that as a step ahead.
// A CTA takes 32 tokens, eight lanes per token, and kQuantBlocks blocks one after the other whose loads are in flight together.  1000 tokens of 14336 with `up`
// 42 us, of 4096 6 (one item of a strided loop per thread, placed by 64-bit divisions: 58, 9); four blocks are as fast there and slower at 300 tokens.
constexpr int kQuantBlocks = 2;
template <int T>
__global__ void __launch_bounds__(256) k_quant_q8_0_wide(const float* X, const float* up, uint8_t* acts, int M, int K)
{
    pdl_launch_dependents();
    const unsigned nb = (unsigned)K / 32, groups = (nb + kQuantBlocks - 1) / kQuantBlocks;
    const unsigned part = blockIdx.x / groups, b0 = (blockIdx.x - part * groups) * kQuantBlocks;
    const int l = threadIdx.x & 7, t = (int)(part % (T / 32)) * 32 + (threadIdx.x >> 3);
    const unsigned tile = part / (T / 32);
    const long tok = (long)tile * T + t;
    const bool live = tok < M;
    const size_t at = (size_t)tok * K + (size_t)b0 * 32 + 4 * l;
    pdl_wait();
    float4 v[kQuantBlocks];
#pragma unroll
    for (int i = 0; i < kQuantBlocks; i++)
        v[i] = live && b0 + i < nb ? *reinterpret_cast<const float4*>(X + at + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (up && live) {
        float4 u[kQuantBlocks];
#pragma unroll
        for (int i = 0; i < kQuantBlocks; i++)
            u[i] = b0 + i < nb ? *reinterpret_cast<const float4*>(up + at + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kQuantBlocks; i++)
            v[i] = make_float4(swiglu_rounded(v[i].x, u[i].x), swiglu_rounded(v[i].y, u[i].y), swiglu_rounded(v[i].z, u[i].z), swiglu_rounded(v[i].w, u[i].w));
    }
#pragma unroll
    for (int i = 0; i < kQuantBlocks; i++) {
        if (b0 + i >= nb) break;
        float amax = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
        const float mul = (amax != 0.0f) ? __fdiv_rn(127.0f, amax) : 0.0f;
        auto qz = [mul](float f) { return (float)(int8_t)__float2int_rn(__fmul_rn(f, mul)); };
        const __half2 lo = __floats2half2_rn(qz(v[i].x), qz(v[i].y)), hi = __floats2half2_rn(qz(v[i].z), qz(v[i].w));
        uint8_t* unit = acts + ((size_t)tile * nb + b0 + i) * 80 * T;
        *reinterpret_cast<uint2*>(unit + (l >> 1) * 16 * T + t * 16 + 8 * (l & 1)) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        if (l == 0) reinterpret_cast<uint4*>(unit + 64 * T)[t] = make_uint4(__half_as_ushort(__float2half_rn(__fdiv_rn(amax, 127.0f))), 0, 0, 0);
    }
}

// ------------------------------------------------------------------ the product

__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}
// four int8 -> four fp16: 1024 + (q + 128) is 0x6400 | byte, and taking 1152 off is exact
__device__ __forceinline__ uint2 four_halves(uint32_t w)
{
    const uint32_t u = w ^ 0x80808080u;
    uint32_t a = __byte_perm(u, 0x64646464u, 0x4140), b = __byte_perm(u, 0x64646464u, 0x4342);
    const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
    const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&a), off), y = __hsub2(*reinterpret_cast<const __half2*>(&b), off);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
}
__device__ __forceinline__ uint64_t pack2(float a, float b)
{
    return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32);
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// minus_zero: -0.0f, from the caller so that the compiler does not see its value.  x * y + (-0) is x * y rounded once; written as a
// multiplication, the assembler would join it with the addition that follows and round once where the reference rounds twice.
template <int T>
__global__ void __launch_bounds__(WideShape<T>::kThreads, 1)
k_gemm_q8_0_wide(const __grid_constant__ WideProducts p, const uint8_t* acts, float minus_zero, int* err)
{
    using S = WideShape<T>;
    constexpr int G = S::kBlocks, H = S::kSetBlocks;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* raw = smem;
    uint8_t* ops = smem + (size_t)S::kRawStages * S::kRawBytes;
    uint8_t* zeros = ops + (size_t)S::kOpStages * S::kOpBytes;
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(zeros + S::kZeroBytes);
    uint64_t* raw_empty = raw_full + S::kRawStages;
    uint64_t* op_full = raw_empty + S::kRawStages;      // the activation bytes and the expanding warps
    uint64_t* op_empty = op_full + S::kOpStages;        // MMA commit
    uint64_t* acc_full = op_empty + S::kOpStages;       // [2]
    uint64_t* acc_empty = acc_full + 2;                 // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < S::kRawStages; s++) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], S::kExpandWarps); }
        for (int s = 0; s < S::kOpStages; s++) { mbar_init(&op_full[s], 1 + S::kExpandWarps); mbar_init(&op_empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], S::kEpiWarps); }
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < S::kZeroBytes / 16; i += S::kThreads) reinterpret_cast<uint4*>(zeros)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the MMAs read the zeros
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    const int nb = p.nb, chunks = (nb + G - 1) / G;
    const int t_tiles = (p.M + T - 1) / T, tiles = p.row_tile[p.n] * t_tiles;
    auto blocks_in = [nb](int c) { const int g = nb - c * G; return g < G ? g : G; };
    auto matrix_of = [&](int row_tile) {
        int m = 0;
        while (m + 1 < p.n && row_tile >= p.row_tile[m + 1]) m++;
        return m;
    };

    if (warp == 0) {
        // ---------------- weights
        if (lane == 0) {
            int s = 0;
            uint32_t par = 1;           // the first round's waits pass
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                const int rt = tile / t_tiles, m = matrix_of(rt);
                const uint8_t* src = p.tiles[m] + (size_t)(rt - p.row_tile[m]) * nb * kTileUnit;
                for (int c = 0; c < chunks; c++) {
                    if (!mbar_wait_bounded(&raw_empty[s], par, err, 51)) { ok = false; break; }
                    const uint32_t bytes = (uint32_t)blocks_in(c) * kTileUnit;
                    mbar_expect_tx(&raw_full[s], bytes);
                    bulk_g2s(raw + (size_t)s * S::kRawBytes, src + (size_t)c * G * kTileUnit, bytes, &raw_full[s]);
                    if (++s == S::kRawStages) { s = 0; par ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- activations
        if (lane == 0) {
            int s = 0;
            uint32_t par = 1;
            bool ok = true;
            pdl_wait();
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                const uint8_t* src = acts + (size_t)(tile % t_tiles) * nb * S::kXUnit;
                for (int c = 0; c < chunks; c++) {
                    if (!mbar_wait_bounded(&op_empty[s], par, err, 52)) { ok = false; break; }
                    const uint32_t bytes = (uint32_t)blocks_in(c) * S::kXUnit;
                    mbar_expect_tx(&op_full[s], bytes);
                    bulk_g2s(ops + (size_t)s * S::kOpBytes + G * S::kWUnit, src + (size_t)c * G * S::kXUnit, bytes, &op_full[s]);
                    if (++s == S::kOpStages) { s = 0; par ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: fp32 sums, fp16 operands, both K-major.  One thread walks the sets; whether the next operands are
        // there is asked ahead of this set's MMAs, so that the answer's latency passes under them (4096 x 14336, 500 tokens: 198 -> 167 us).
        if (elect_one()) {
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(T >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
            const uint32_t z4 = smem_addr(zeros) >> 4;
            // K = 16 as one chunk of scales and one of zeros, wherever that lies: the distance is the descriptor's leading offset
            auto scales = [z4](uint32_t at) { return (uint64_t)((at >> 4) | ((z4 - (at >> 4)) << 16)) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46); };
            int s = 0;
            uint32_t par = 0, it = 0;
            bool ok = true, ready = false;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                for (int c = 0; ok && c < chunks; c++) {
                    if (!ready && !mbar_wait_bounded(&op_full[s], par, err, 53)) { ok = false; break; }
                    const int next = s + 1 == S::kOpStages ? 0 : s + 1;
                    const uint32_t next_par = next ? par : par ^ 1u;
                    const uint32_t w = smem_addr(ops + (size_t)s * S::kOpBytes), x = w + G * S::kWUnit;
                    const uint64_t a0 = umma_desc(w, 16 * kTileRows, 128), b0 = umma_desc(x, 16 * T, 128);
                    const int g_n = blocks_in(c);
#pragma unroll
                    for (int g = 0; g < G; g += H) {
                        if (g >= g_n) break;
                        const uint32_t a = it & 1;
                        if (it >= 2 && !mbar_wait_bounded(&acc_empty[a], ((it >> 1) - 1) & 1u, err, 54)) { ok = false; break; }
                        it++;
                        if (g + H >= g_n) ready = mbar_test(&op_full[next], next_par);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t d0 = tmem_base + a * 256;
#pragma unroll
                        for (int h = 0; h < H; h++) {
                            if (g + h >= g_n) break;
                            const uint32_t wu = (uint32_t)((g + h) * S::kWUnit), xu = (uint32_t)((g + h) * S::kXUnit);
                            umma_f16_ss(d0 + (uint32_t)(h * T), a0 + (wu >> 4), b0 + (xu >> 4), idesc, 0u);
                            umma_f16_ss(d0 + (uint32_t)(h * T), a0 + ((wu + 32 * kTileRows) >> 4), b0 + ((xu + 32 * T) >> 4), idesc, 1u);
                            umma_f16_ss(d0 + 128 + (uint32_t)(h * T), scales(w + wu + 64 * kTileRows), scales(x + xu + 64 * T), idesc, 0u);
                        }
                        umma_commit(&acc_full[a]);
                        if (g + H >= g_n) umma_commit(&op_empty[s]);
                    }
                    s = next;
                    par = next_par;
                }
            }
        }
        __syncwarp();
    } else if (warp < 3 + S::kExpandWarps) {
        // ---------------- int8 -> fp16
        const int r = tid - 96;
        int rs = 0, s = 0;
        uint32_t rpar = 0, par = 1;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            for (int c = 0; c < chunks; c++) {
                if (!mbar_wait_bounded(&raw_full[rs], rpar, err, 55)) { ok = false; break; }
                const uint8_t* from = raw + (size_t)rs * S::kRawBytes;
                uint8_t* to = ops + (size_t)s * S::kOpBytes;
                uint4 q[G][2];
                uint32_t wd[G];
#pragma unroll
                for (int g = 0; g < G; g++) {      // a short last chunk converts the rest of an older one, which no MMA reads
                    const uint8_t* at = from + g * kTileUnit;
                    q[g][0] = *reinterpret_cast<const uint4*>(at + 16 * r);
                    q[g][1] = *reinterpret_cast<const uint4*>(at + 16 * kTileRows + 16 * r);
                    wd[g] = *reinterpret_cast<const unsigned short*>(at + kTileQuants + 2 * r);
                }
                if (!mbar_wait_bounded(&op_empty[s], par, err, 56)) { ok = false; break; }
#pragma unroll
                for (int g = 0; g < G; g++) {
                    uint8_t* at = to + g * S::kWUnit + 16 * r;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint2 x = four_halves(q[g][h].x), y = four_halves(q[g][h].y), z = four_halves(q[g][h].z), w = four_halves(q[g][h].w);
                        *reinterpret_cast<uint4*>(at + (2 * h) * 16 * kTileRows) = make_uint4(x.x, x.y, y.x, y.y);
                        *reinterpret_cast<uint4*>(at + (2 * h + 1) * 16 * kTileRows) = make_uint4(z.x, z.y, w.x, w.y);
                    }
                    *reinterpret_cast<uint4*>(at + 64 * kTileRows) = make_uint4(wd[g], 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the MMAs read what was written here
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&raw_empty[rs]);
                    mbar_arrive(&op_full[s]);
                }
                if (++rs == S::kRawStages) { rs = 0; rpar ^= 1u; }
                if (++s == S::kOpStages) { s = 0; par ^= 1u; }
            }
        }
    } else {
        // ---------------- epilogue
        constexpr int kCols = T / 4, kStep = kCols < 16 ? kCols : 16;      // tokens of this warp
        const int quarter = warp & 3;                     // the TMEM lanes this warp may read: 32*(warp%4)..
        const int c0 = ((warp - 3 - S::kExpandWarps) >> 2) * kCols;
        const int r = 32 * quarter + lane;
        const uint32_t taddr0 = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)c0;
        const uint64_t nz = pack2(minus_zero, minus_zero);
        uint32_t it = 0;
        bool ok = true;
        pdl_wait();
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            uint64_t acc[kCols / 2];
#pragma unroll
            for (int t = 0; t < kCols / 2; t++) acc[t] = 0;
            for (int b = 0; b < nb; b += H, it++) {
                const uint32_t a = it & 1;
                if (!mbar_wait_bounded(&acc_full[a], (it >> 1) & 1u, err, 58)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int h = 0; h < H; h++) {
                    if (h == 0 || b + h < nb) {
#pragma unroll
                        for (int c = 0; c < kCols; c += kStep) {
                            int v[kStep], w[kStep];
                            const uint32_t ta = taddr0 + a * 256 + (uint32_t)(h * T + c);
                            tmem_ld(ta, v);
                            tmem_ld(ta + 128, w);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            if (c + kStep >= kCols && (h == H - 1 || b + h + 1 >= nb)) {      // everything is read
                                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                                __syncwarp();
                                if (lane == 0) mbar_arrive(&acc_empty[a]);
                            }
#pragma unroll
                            for (int t = 0; t < kStep / 2; t++) {
                                const uint64_t sum = pack2(__int_as_float(v[2 * t]), __int_as_float(v[2 * t + 1]));
                                const uint64_t scale = pack2(__int_as_float(w[2 * t]), __int_as_float(w[2 * t + 1]));
                                acc[c / 2 + t] = add2(acc[c / 2 + t], fma2(sum, scale, nz));
                            }
                        }
                    }
                }
            }
            const int rt = tile / t_tiles, m = matrix_of(rt);
            const long n = (long)(rt - p.row_tile[m]) * kTileRows + r;
            if (ok && n < p.N[m]) {
                const int tok0 = (tile % t_tiles) * T + c0;
                float* out = p.out[m] + (size_t)tok0 * p.N[m] + n;
#pragma unroll
                for (int t = 0; t < kCols; t++)
                    if (tok0 + t < p.M) out[(size_t)t * p.N[m]] = __uint_as_float((uint32_t)(acc[t / 2] >> (32 * (t & 1))));
            }
        }
    }
    // ---------------- teardown: everybody meets, then the allocating warp frees tensor memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------ host side

template <int T>
static int launch_wide(const WideProducts& p, const float* X, const float* up, int K, cudaStream_t s, Workspace* ws)
{
    using S = WideShape<T>;
    const long t_tiles = (p.M + T - 1) / T, tiles = t_tiles * p.row_tile[p.n];
    const size_t bytes = (size_t)t_tiles * p.nb * S::kXUnit;
    if (tiles > (1l << 30) || !scratch_fits(ws, kScratchTilesActs, bytes, s)) return kWideRefused;
    int rc = allow_smem<k_gemm_q8_0_wide<T>>((int)S::kSmem);
    if (rc) return latch(rc);
    uint8_t* acts = scratch_take(ws, kScratchTilesActs, bytes, s, &rc);
    if (!acts) return rc;
    const long parts = t_tiles * (T / 32) * ((p.nb + kQuantBlocks - 1) / kQuantBlocks);
    if ((rc = launch_ordered(k_quant_q8_0_wide<T>, (unsigned)parts, 256, 0, s, X, up, acts, p.M, K))) return latch(rc);
    rc = launch_ordered(k_gemm_q8_0_wide<T>, (unsigned)(tiles < sm_count() ? tiles : sm_count()), S::kThreads, S::kSmem, s, p, acts, -0.0f,
                        device_error_flag());
    return rc ? latch(rc) : 0;
}

// Tokens of a tile, or 0 where the narrow kernel's launches are expected to be faster: waves of CTAs over the SMs times the measured
// time of a tile of 4096 columns (us; narrow 14, 20.5 and 40 at 16, 32 and 64 tokens, here 23, 32 and 45 at 32, 64 and 128).
static int wide_tokens(const WideProducts& p)
{
    const int sms = sm_count();
    auto least = [&](long row_tiles, const int (&widths)[3], const double (&us)[3], int* width) {
        double best = 0.0;
        for (int i = 0; i < 3; i++) {
            if (i > 0 && p.M <= widths[i - 1]) break;
            const long tiles = row_tiles * ((p.M + widths[i] - 1) / widths[i]);
            const double t = (double)((tiles + sms - 1) / sms) * us[i];
            if (i == 0 || t <= best) { best = t; *width = widths[i]; }
        }
        return best;
    };
    int unused, T = 0;
    double narrow = 0.0;
    for (int i = 0; i < p.n; i++) narrow += least(p.row_tile[i + 1] - p.row_tile[i], {16, 32, 64}, {14.0, 20.5, 40.0}, &unused);
    return least(p.row_tile[p.n], {32, 64, 128}, {23.0, 32.0, 45.0}, &T) < narrow ? T : 0;
}

int gemm_q8_0_wide(int n, const uint8_t* const* tiles, float* const* outs, const int* Ns, const float* X, int M, int K, cudaStream_t s,
                   Workspace* ws, const float* up)
{
    if (n < 1 || n > kWideMatrices || M < kWideMinTokens || K < 32 || K % 32) return kWideRefused;
    WideProducts p = {};
    p.n = n;
    p.M = M;
    p.nb = K / 32;
    for (int i = 0; i < n; i++) {
        if (Ns[i] < 1 || !tiles[i] || !outs[i] || ((uintptr_t)tiles[i] & 15) || ((uintptr_t)outs[i] & 3)) return kWideRefused;
        p.tiles[i] = tiles[i];
        p.out[i] = outs[i];
        p.N[i] = Ns[i];
        p.row_tile[i + 1] = p.row_tile[i] + (Ns[i] + kTileRows - 1) / kTileRows;
    }
    if (!X || (((uintptr_t)X | (uintptr_t)up) & 15)) return kWideRefused;
    const int T = wide_tokens(p);
    return T == 128 ? launch_wide<128>(p, X, up, K, s, ws) : T == 64 ? launch_wide<64>(p, X, up, K, s, ws) : T == 32 ? launch_wide<32>(p, X, up, K, s, ws) : kWideRefused;
}

}  // namespace bpdq

using namespace bpdq;

extern "C" {

int bpdq_qmatmul_q8_0_tiles_width(int M, int N, int K)
{
    if (M < kWideMinTokens || N < 1 || K < 32 || K % 32) return 0;
    WideProducts p = {};
    p.n = 1;
    p.M = M;
    p.row_tile[1] = (N + kTileRows - 1) / kTileRows;
    return wide_tokens(p);
}

}  // extern "C"
