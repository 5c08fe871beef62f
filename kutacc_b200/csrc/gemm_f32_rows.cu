// fp32 products with 128 or 256 columns on the fifth-generation tensor cores, the activations read once and split on the way.
//
//   C[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n])         A [M, K] fp32, W [N, K] fp32 (W[out][in]), C fp32, K = 128 or 256
//
// (the four projections of the fp32 attention in one pass, its output projection, kutacc_af2_linear on fp32 tensors;
// src/attention/gating_attention.cpp:47-66,152-157; src/linear/mm.cpp:46-86.) tcgen05.mma has no fp32 input type. Every row of A and of
// W is brought to a largest element in [2^14, 2^15) by a power of two and split into an fp16 head and an fp16 tail, the tail
// times 2^11 so that it has the range of the head: x * 2^s = hi + lo * 2^-11 with 22 bits, for elements down to 2^-29 of their row's
// largest, and an error of 2^-51 of that one below. The product is
//   hi(A).hi(W) + 2^-11 (lo(A).hi(W) + hi(A).lo(W))        (lo.lo, about 2^-22 of the result, is dropped)
// with the small products in an accumulator of their own, and the powers of two are taken back in the epilogue. Against tf32
// heads and tails (gemm_tf32_tcgen05.cu, which keeps all other K) an operand has half the bytes and the tensor cores twice
// the rate, and there are half as many accumulations, each of which truncates.
//
// The activations stand still, as in gemm_proj.cu: a persistent CTA (one per SM) loads 128 rows, all K columns, as fp32; the
// epilogue warps split them where they lie (the head and tail of a row take just the bytes of its fp32 values), and the
// weights, split by a kernel of their own (a row of them is used by every CTA), stream past in slabs of 128 channels x 64 columns.
//   warp 0      producer: rows in slabs of 32 fp32 columns, weight slabs (tail and head in turn, a ring of four or eight)
//   warp 1      MMA issuer: 12 instructions a tail and head into a pair of 128 x 128 accumulators (two pairs in tensor memory;
//               128 x 64 for few rows)
//   warps 4-11  split the rows, 16 each; epilogue, 32 rows x 64 columns each: tcgen05.ld of both accumulators, scaling, bias,
//               one of two staging tiles (32 x 16), TMA store
// What bounds it: the way of the results out of the SM beside the products, and, twice per CTA at the size below, the way of a block
// into shared memory and its split, which nothing overlaps. With parts taken out of copies, 32768 x 1024 x 256: complete 96 us, without
// stores 82, without products 87, without both 57, without the split 92, with an eighth of the weights' bytes 93. 32768 rows x 256
// channels, four projections: 80 us (HBM 31, products 31); as a split of the activations and tf32 products 20 + 92. Error
// against 64 bits at K = 128 and 256 (2-norm): 2.0e-7 and 3.5e-7, before 3.4e-7 and 6.4e-7. The fp32 layer of 128 x 256 rows: 288 -> 227 us (now 214, with the
// slabs freed one by one, the second staging tile and a faster attention core).
//
// All mbarrier waits are bounded; on a timeout the roles fall through to the common tail, the TMEM allocation is
// released and the host-visible error word carries the site.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

namespace kutacc {
namespace dev {

namespace {

constexpr int BM = 128;
constexpr int SLAB_BYTES = 128 * 128;                   // 128 rows (or channels) x 32 fp32 or 64 fp16 columns
constexpr int EPI_WARPS = 8, EPI_WARP0 = 4;
constexpr int THREADS = (EPI_WARP0 + EPI_WARPS) * 32;
constexpr int STG_BYTES = 32 * 16 * 4;
constexpr float kTail = 1.0f / 2048;                    // weight of the small products

// KS: 64-column slabs of a row
template <int KS>
struct Geo {
    static constexpr int NW = KS == 4 ? 4 : 8;                                   // slabs of the weight ring
    static constexpr int OFF_A = NW * SLAB_BYTES;
    static constexpr int OFF_STG = OFF_A + 2 * KS * SLAB_BYTES;
    static constexpr int OFF_SCALE = OFF_STG + EPI_WARPS * 2 * STG_BYTES;            // of the rows of two blocks
    static constexpr int OFF_BAR = OFF_SCALE + 2 * BM * 4;
    static constexpr int NBARS = 2 * NW + 2 * KS + 5;
    static constexpr int SMEM_BYTES = OFF_BAR + 8 * NBARS + 16 + 1024;
    static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
};

struct alignas(64) RowsMaps {
    CUtensorMap a;        // A [M][K] fp32, box [32, 128], 128-byte swizzle
    CUtensorMap w[4];     // W' [N][2K] fp16 (head | tail) per segment, box [64, 128], 128-byte swizzle
    CUtensorMap out[4];   // per segment [M][N] (split rows: [M][2N]) fp32, box [16, 32], 64-byte swizzle
};

struct RowsParams {
    const float *bias[4];   // per segment, may be null
    const float *w_scale[4];
    float *out_t[4];        // kTf32SplitTransposed segments: [B][N/32][64][S]
    int layout[4];          // per segment: Tf32Layout
    int M, N, tiles;        // column tiles of all segments
    int S;                  // rows per batch row (transposed segments)
    int64_t vt_pitch;
    int whole, nsplit, units;       // as in gemm_proj.cu: blocks with all their column tiles, then parts of blocks
    int *err;
};

// exponent that brings the largest magnitude (its bits) to [2^14, 2^15), as the bits of 2^s and of 2^-s
__device__ __forceinline__ void scale_of(uint32_t max_bits, float &up, float &down)
{
    const int s = min(268 - (int)(max_bits >> 23), 253);           // biased; rows below 2^-112 keep 2^126
    up = __int_as_float(s << 23);
    down = __int_as_float((254 - s) << 23);
}
// two elements, already scaled: packed heads and packed tails
__device__ __forceinline__ void split_f16(float x0, float x1, uint32_t &hi, uint32_t &lo)
{
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((x0 - f.x) * 2048.f, (x1 - f.y) * 2048.f);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ uint32_t magnitude_bits(const float4 &v)
{
    const uint32_t a = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    return max(a, max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
}

// BN: channels of a column tile, 128 or 64
template <int KS, int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_rows_kernel(const __grid_constant__ RowsMaps maps, const __grid_constant__ RowsParams p)
{
    using T = Geo<KS>;
    constexpr int K = 64 * KS, NW = T::NW;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *gen = smem_raw + (smem - smem_u32(smem_raw));
    const uint32_t bar = smem + T::OFF_BAR;
    auto w_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto w_empty = [&](int s) { return bar + 8u * (uint32_t)(NW + s); };
    auto a_full = [&](int ks) { return bar + 8u * (uint32_t)(2 * NW + ks); };
    auto a_empty = [&](int ks) { return bar + 8u * (uint32_t)(2 * NW + KS + ks); };
    const uint32_t a_split = bar + 8u * (2 * NW + 2 * KS);
    auto acc_full = [&](int b) { return a_split + 8u + 8u * (uint32_t)b; };
    auto acc_empty = [&](int b) { return a_split + 24u + 8u * (uint32_t)b; };
    const uint32_t tmem_slot = bar + 8u * T::NBARS;
    float *const row_scale = reinterpret_cast<float *>(gen + T::OFF_SCALE);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // unit u: its block, first column tile and number of column tiles
    auto unit = [&](int u, int &block, int &t0, int &nt) {
        const int v = u - p.whole;
        block = v < 0 ? u : p.whole + v / p.nsplit;
        nt = v < 0 ? p.tiles : p.tiles / p.nsplit;
        t0 = v < 0 ? 0 : v % p.nsplit * nt;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NW; ++s) {
            mbar_init(w_full(s), 1);
            mbar_init(w_empty(s), 1);
        }
        for (int ks = 0; ks < KS; ++ks) {
            mbar_init(a_full(ks), 1);
            mbar_init(a_empty(ks), 1);
        }
        mbar_init(a_split, EPI_WARPS);
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), EPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0 && elect_one()) {                  // kernel parameters: may be fetched before the predecessor ends
        tma_prefetch_desc(&maps.a);
        for (int i = 0; i < 4; ++i) {
            tma_prefetch_desc(&maps.w[i]);
            tma_prefetch_desc(&maps.out[i]);
        }
    }
    release_successor();
    wait_for_predecessor();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0) {
        // ================= producer =================
        if (elect_one()) {
            bool ok = true;
            int s = 0, round = 0;                                      // next slab's slot, times the ring has gone round
            for (int n = 0; ok; ++n) {
                const int u = (int)blockIdx.x + n * (int)gridDim.x;
                if (u >= p.units) break;
                int block, t0, nt;
                unit(u, block, t0, nt);
                for (int ks = 0; ks < KS && ok; ++ks) {
                    if (n > 0) ok = mbar_wait(a_empty(ks), (uint32_t)((n - 1) & 1), p.err, 111);
                    if (!ok) break;
                    mbar_arrive_expect_tx(a_full(ks), 2 * SLAB_BYTES);
                    const uint32_t dst = smem + T::OFF_A + ks * 2 * SLAB_BYTES;
                    tma_load_2d(dst, &maps.a, a_full(ks), ks * 64, block * BM);
                    tma_load_2d(dst + SLAB_BYTES, &maps.a, a_full(ks), ks * 64 + 32, block * BM);
                }
                for (int j = 0; j < nt && ok; ++j) {
                    const int col = (t0 + j) * BN, seg = col / p.N;
                    for (int h = 0; h < 2 * KS; ++h) {                 // tails and heads in turn
                        if (round > 0) ok = mbar_wait(w_empty(s), (uint32_t)((round - 1) & 1), p.err, 112);
                        if (!ok) break;
                        mbar_arrive_expect_tx(w_full(s), BN * 128);
                        tma_load_2d(smem + (uint32_t)(s * SLAB_BYTES), &maps.w[seg], w_full(s), (h & 1 ? 0 : K) + (h >> 1) * 64, col % p.N);
                        if (++s == NW) {
                            s = 0;
                            ++round;
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc = make_instr_desc_f16(BM, BN);
        constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;                   // descriptor addresses count in units of 16 bytes
        const uint64_t wd0 = make_smem_desc_kmajor(smem, 128), ad0 = make_smem_desc_kmajor(smem + T::OFF_A, 128);
        bool ok = true;
        int s = 0, tc = 0;
        uint32_t par = 0;
        auto next_slab = [&]() {
            if (++s == NW) {
                s = 0;
                par ^= 1u;
            }
        };
        for (int n = 0; ok; ++n) {
            const int u = (int)blockIdx.x + n * (int)gridDim.x;
            if (u >= p.units) break;
            int block, t0, nt;
            unit(u, block, t0, nt);
            ok = mbar_wait_warp(a_split, (uint32_t)(n & 1), p.err, 113);
            for (int j = 0; j < nt && ok; ++j, ++tc) {
                const int buf = tc & 1;
                if (tc >= 2) ok = mbar_wait_warp(acc_empty(buf), (uint32_t)((tc / 2 - 1) & 1), p.err, 114);
                const uint32_t d = tmem_base + (uint32_t)(buf * 2 * BN);
                for (int ks = 0; ks < KS && ok; ++ks) {
                    // head.tail, then tail.head and head.head: each slab is freed as soon as it can be
                    ok = mbar_wait_warp(w_full(s), par, p.err, 115);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t a = ad0 + (uint32_t)(ks * 2 * SLAB16);
                    if (elect_one()) {
                        const uint64_t w = wd0 + (uint32_t)(s * SLAB16);
#pragma unroll
                        for (int k = 0; k < 4; ++k)                    // 16 columns = 32 bytes an instruction
                            tc_mma_bf16(d + BN, a + 2 * k, w + 2 * k, idesc, (ks > 0 || k > 0) ? 1u : 0u);
                        tc_commit(w_empty(s));
                    }
                    __syncwarp();
                    next_slab();
                    ok = mbar_wait_warp(w_full(s), par, p.err, 115);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t w = wd0 + (uint32_t)(s * SLAB16);
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc_mma_bf16(d + BN, a + SLAB16 + 2 * k, w + 2 * k, idesc, 1u);
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc_mma_bf16(d, a + 2 * k, w + 2 * k, idesc, (ks > 0 || k > 0) ? 1u : 0u);
                        tc_commit(w_empty(s));
                        if (j == nt - 1) tc_commit(a_empty(ks));
                        if (ks == KS - 1) tc_commit(acc_full(buf));
                    }
                    __syncwarp();
                    next_slab();
                }
            }
        }
    } else if (warp >= EPI_WARP0) {
        // ================= split, epilogue =================
        const int ew = warp - EPI_WARP0, half = ew >> 2, quad = warp & 3;
        const uint32_t stg0 = smem + T::OFF_STG + (uint32_t)(ew * 2 * STG_BYTES);
        uint32_t nstore = 0;
        bool ok = true;

        // 16 rows of the block: LPR lanes share a row, eight columns each
        constexpr int LPR = K / 8, RPP = 32 / LPR, U = 4;
        auto split_rows = [&](int n) {
            for (int ks = 0; ks < KS && ok; ++ks) ok = mbar_wait_warp(a_full(ks), (uint32_t)(n & 1), p.err, 116);
            if (!ok) return;
            const int l = lane % LPR, sub = lane / LPR;
            const uint32_t src = smem + T::OFF_A + (l >> 2) * SLAB_BYTES;           // slab of 32 columns, chunks 2 (l & 3) and + 1
            const uint32_t dst = smem + T::OFF_A + (l >> 3) * 2 * SLAB_BYTES;       // slab of 64 columns, chunk l & 7
            const int swap = (l >> 2) & 1;                                          // so that eight lanes read eight banks' worth
#pragma unroll 1
            for (int r0 = 0; r0 < 16; r0 += U * RPP) {
                float4 v[U][2];
                uint32_t mx[U];
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int row = ew * 16 + r0 + i * RPP + sub;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        v[i][j] = lds128_f32(src + (uint32_t)(row * 128 + (((2 * (l & 3) + (j ^ swap)) ^ (row & 7)) << 4)));
                    mx[i] = max(magnitude_bits(v[i][0]), magnitude_bits(v[i][1]));
                }
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < U; ++i) mx[i] = max(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int row = ew * 16 + r0 + i * RPP + sub;
                    float up, down;
                    scale_of(mx[i], up, down);
                    const float4 c0 = swap ? v[i][1] : v[i][0], c1 = swap ? v[i][0] : v[i][1];
                    uint32_t hi[4], lo[4];
                    split_f16(c0.x * up, c0.y * up, hi[0], lo[0]);
                    split_f16(c0.z * up, c0.w * up, hi[1], lo[1]);
                    split_f16(c1.x * up, c1.y * up, hi[2], lo[2]);
                    split_f16(c1.z * up, c1.w * up, hi[3], lo[3]);
                    // (the shuffles above come after every lane's loads of these rows)
                    const uint32_t d = dst + (uint32_t)(row * 128 + (((l & 7) ^ (row & 7)) << 4));
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(d), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(d + SLAB_BYTES), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3])
                                 : "memory");
                    if (l == 0) row_scale[(n & 1) * BM + row] = down;
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_split);
        };

        int tc = 0;
        for (int n = 0; ok; ++n) {
            const int u = (int)blockIdx.x + n * (int)gridDim.x;
            if (u >= p.units) break;
            int block, t0, nt;
            unit(u, block, t0, nt);
            split_rows(n);
            // the scales of the other warps' rows; every warp comes by here once per block
            if (ok) ok = mbar_wait_warp(a_split, (uint32_t)(n & 1), p.err, 118);
            if (!ok) break;
            const float a_scale = row_scale[(n & 1) * BM + quad * 32 + lane];
            const bool a_large = a_scale > 1.0f;
            const int m0 = block * BM + quad * 32, m = m0 + lane;
            for (int j = 0; j < nt; ++j, ++tc) {
                const int buf = tc & 1, col = (t0 + j) * BN + half * (BN / 2), seg = col / p.N, n0 = col % p.N;
                ok = mbar_wait_warp(acc_full(buf), (uint32_t)((tc / 2) & 1), p.err, 117);
                if (!ok) break;
                tc_fence_after();
                const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * 2 * BN + half * (BN / 2));
                uint32_t acc[BN / 64][32];
#pragma unroll
                for (int c = 0; c < BN / 64; ++c) {
                    tmem_ld_32x32(tcol + c * 32, acc[c]);
#pragma unroll
                    for (int q = 0; q < 32; q += 16) {
                        uint32_t small[16];
                        tmem_ld_32x16(tcol + BN + c * 32 + q, small);
                        tmem_ld_wait16(small);
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            acc[c][q + e] = __float_as_uint(fmaf(__uint_as_float(small[e]), kTail, __uint_as_float(acc[c][q + e])));
                    }
                }
                // everything is in registers: the accumulators may be overwritten
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(buf));
                const float *bias = p.bias[seg], *ws = p.w_scale[seg];
                const int layout = p.layout[seg];
                const CUtensorMap *omap = &maps.out[seg];
                float *tdst = nullptr;                            // transposed segments: this row's place in the first head
                if (layout == kTf32SplitTransposed) {
                    const int b = m / p.S;
                    tdst = p.out_t[seg] + ((int64_t)b * (p.N / 32) + n0 / 32) * 64 * p.vt_pitch + (m - b * p.S);
                }
#pragma unroll
                for (int c = 0; c < BN / 64; ++c) {
                    uint32_t(&r)[32] = acc[c];
                    const int nn = n0 + c * 32;
#pragma unroll
                    for (int j4 = 0; j4 < 8; ++j4) {
                        const float4 sv = __ldg(reinterpret_cast<const float4 *>(ws + nn) + j4);
                        const float4 bv = bias ? __ldg(reinterpret_cast<const float4 *>(bias + nn) + j4) : make_float4(0.f, 0.f, 0.f, 0.f);
                        const float s4[4] = {sv.x, sv.y, sv.z, sv.w}, b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            // the factor that may be large last: the powers of two of a row and a channel can be far apart
                            const float t = __uint_as_float(r[4 * j4 + e]) * (a_large ? s4[e] : a_scale);
                            r[4 * j4 + e] = __float_as_uint(fmaf(t, a_large ? a_scale : s4[e], b4[e]));
                        }
                    }
                    if (layout == kTf32SplitTransposed) {
                        // one head of 32 channels, split; the lanes of a store run along the sequence
                        if (m < p.M) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                const float v = __uint_as_float(r[e]), h = tf32_head(v);
                                tdst[e * p.vt_pitch] = h;
                                tdst[(32 + e) * p.vt_pitch] = v - h;
                            }
                        }
                        tdst += 64 * p.vt_pitch;
                        continue;
                    }
                    // rows, or rows with every 32 channels as [head | tail]
                    const bool split = layout == kTf32SplitRows;
                    for (int t = 0; t < (split ? 4 : 2); ++t) {               // 16 columns each, heads and tails in turn
                        const int hf = split ? t >> 1 : t;
                        const uint32_t stg = stg0 + (nstore++ & 1) * STG_BYTES;
                        if (lane == 0) tma_store_wait_read<1>();          // the last but one store has been read
                        __syncwarp();
#pragma unroll
                        for (int j4 = 0; j4 < 4; ++j4) {
                            float v[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                v[e] = __uint_as_float(hf ? r[16 + 4 * j4 + e] : r[4 * j4 + e]);
                                const float h = tf32_head(v[e]);
                                if (split) v[e] = (t & 1) == 0 ? h : v[e] - h;
                            }
                            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(stg + (uint32_t)(lane * 64 + ((j4 ^ ((lane >> 1) & 3)) << 4))),
                                         "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                                         : "memory");
                        }
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(omap, stg, (split ? 2 * nn + 32 * (t & 1) : nn) + 16 * hf, m0);
                            tma_store_commit();
                        }
                    }
                }
            }
        }
        if (lane == 0) tma_store_wait<0>();
    }

    // ================= common tail =================
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// Weights: a warp per row, up to eight matrices of the same shape a launch (blockIdx.y picks one). dst [rows][2K] fp16 (heads, then
// tails), then the rows' 2^-s.
struct SplitArgs {
    const float *src[8];
    __half *dst[8];
    float *scale[8];
};
template <int K>
__global__ void __launch_bounds__(256) split_weights_kernel(const SplitArgs args, int64_t src_ld, int rows)
{
    release_successor();
    wait_for_predecessor();
    const int row = (int)(blockIdx.x * 8 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float4 *src = reinterpret_cast<const float4 *>(args.src[blockIdx.y] + (int64_t)row * src_ld);
    float4 v[K / 128];
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < K / 128; ++i) {
        v[i] = __ldg(src + i * 32 + lane);
        mx = max(mx, magnitude_bits(v[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float up, down;
    scale_of(mx, up, down);
    __half *dst = args.dst[blockIdx.y] + (int64_t)row * 2 * K;
#pragma unroll
    for (int i = 0; i < K / 128; ++i) {
        uint2 hi, lo;
        split_f16(v[i].x * up, v[i].y * up, hi.x, lo.x);
        split_f16(v[i].z * up, v[i].w * up, hi.y, lo.y);
        *reinterpret_cast<uint2 *>(dst + (i * 32 + lane) * 4) = hi;
        *reinterpret_cast<uint2 *>(dst + K + (i * 32 + lane) * 4) = lo;
    }
    if (lane == 0) args.scale[blockIdx.y][row] = down;
}

template <int KS, int BN>
void launch_ks(cudaStream_t stream, const RowsMaps &maps, const RowsParams &p, int grid)
{
    static const cudaError_t attr = cudaFuncSetAttribute(gemm_f32_rows_kernel<KS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<KS>::SMEM_BYTES);
    KUTACC_CUDA(attr);
    launch_chained(gemm_f32_rows_kernel<KS, BN>, (unsigned)grid, THREADS, Geo<KS>::SMEM_BYTES, stream, maps, p);
}

}  // namespace

bool split_f32_weights(cudaStream_t stream, int count, const void *const *src, int64_t src_ld, void *const *dst, int rows, int K)
{
    if (count < 1 || count > 8 || rows <= 0 || rows > INT32_MAX / 8 || (K != 128 && K != 256) || src_ld % 4 != 0) return false;
    SplitArgs a;
    for (int i = 0; i < 8; ++i) {
        const int j = i < count ? i : 0;
        if ((((uintptr_t)src[j] | (uintptr_t)dst[j]) & 15u) != 0) return false;
        a.src[i] = (const float *)src[j];
        a.dst[i] = (__half *)dst[j];
        a.scale[i] = (float *)((char *)dst[j] + (size_t)rows * K * 4);
    }
    const dim3 grid((unsigned)((rows + 7) / 8), (unsigned)count);
    KernelTimer timer__("split_weights", stream);
    if (K == 128)
        launch_chained(split_weights_kernel<128>, grid, 256, 0, stream, a, src_ld, rows);
    else
        launch_chained(split_weights_kernel<256>, grid, 256, 0, stream, a, src_ld, rows);
    count_launch();
    return true;
}

bool tcgen05_gemm_f32_rows(cudaStream_t stream, const void *a, int64_t lda, const void *const *w_split, const float *const *bias,
                           void *const *out, int64_t ldo, int64_t M, int N, int K, int nseg, const Tf32Layout *layout, int S,
                           int64_t vt_pitch)
{
    if (nseg < 1 || nseg > 4 || M <= 0 || M > INT32_MAX / 2 || N <= 0 || N % 128 != 0 || (K != 128 && K != 256) || lda % 4 != 0 || lda < K ||
        ldo % 4 != 0 || ldo < N || (((uintptr_t)a) & 15u))
        return false;
    for (int i = 0; i < nseg; ++i)
        if ((((uintptr_t)w_split[i] | (uintptr_t)out[i] | (uintptr_t)bias[i]) & 15u) != 0) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    // Few rows: column tiles of half the width where those of four such products run at once; a product is then as long as one
    // tile's chain: fp32 layer of 8 x 48 rows 34.5 -> 32.6 us, of 8 x 130 rows 45.0 -> 39.0. The rule does not look at nseg, so that a
    // layer's projections and output run the same code: an output product alone in half tiles cost 40 x 60 rows 44.9 -> 48.9 us.
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    const int64_t blocks = (M + BM - 1) / BM;
    const int BN = blocks * (N / 64) * 4 <= sms ? 64 : 128;
    RowsMaps maps;
    RowsParams p = {};
    if (!make_tensor_map_2d(&maps.a, a, /*elem_bytes=*/4, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 32, BM, 128)) return false;
    for (int i = 0; i < 4; ++i) {
        const int j = i < nseg ? i : 0;
        p.bias[i] = bias[j];
        p.w_scale[i] = (const float *)((const char *)w_split[j] + (size_t)N * K * 4);
        p.layout[i] = layout ? layout[j] : kTf32Rows;
        p.out_t[i] = (float *)out[j];
        if (!make_tensor_map_2d(&maps.w[i], w_split[j], 2, (uint64_t)2 * K, (uint64_t)N, (uint64_t)2 * K, 64, BN, 128)) return false;
        const uint64_t cols = p.layout[i] == kTf32SplitRows ? 2 * (uint64_t)N : (uint64_t)N;
        if (p.layout[i] == kTf32SplitTransposed)
            maps.out[i] = maps.a;                            // stored directly
        else if (!make_tensor_map_2d(&maps.out[i], out[j], 4, cols, (uint64_t)M, p.layout[i] == kTf32SplitRows ? cols : (uint64_t)ldo, 16, 32, 64))
            return false;
    }
    p.M = (int)M;
    p.N = N;
    p.tiles = N / BN * nseg;
    p.S = S > 0 ? S : 1;
    p.vt_pitch = vt_pitch;
    p.err = ew.device;
    // As in gemm_proj.cu: whole blocks for all full waves, the blocks of the last one in 1 / nsplit of their column tiles each. A
    // unit costs its column tiles and about two for the way of its rows into shared memory and their split.
    const int64_t whole = blocks / sms * sms;
    double best = 1e30;
    for (int ns = 1; ns <= p.tiles; ++ns) {
        if (p.tiles % ns != 0 || (blocks - whole) * ns + whole > INT32_MAX / 2) continue;
        const int64_t last = (blocks - whole) * ns;
        const double cost = (double)((last + sms - 1) / sms) * ((double)p.tiles / ns + 2.0);
        if (cost < best * 0.999) {
            best = cost;
            p.whole = (int)whole;
            p.nsplit = ns;
            p.units = (int)(whole + last);
        }
    }
    const int grid = std::min(p.units, sms);
    KernelTimer timer__("gemm_tf32x3_tc", stream);           // the name of the fp32 tensor-memory products, whichever kernel
    if (BN == 64)
        K == 128 ? launch_ks<2, 64>(stream, maps, p, grid) : launch_ks<4, 64>(stream, maps, p, grid);
    else
        K == 128 ? launch_ks<2, 128>(stream, maps, p, grid) : launch_ks<4, 128>(stream, maps, p, grid);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
