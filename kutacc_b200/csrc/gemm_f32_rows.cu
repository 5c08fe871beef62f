// fp32 products with 128 or 256 columns on the fifth-generation tensor cores, the activations read once and split on the way.
//
//   C[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n])         A [M, K] fp32, W [N, K] fp32 (W[out][in]), C fp32, K = 128 or 256
//
// (the four projections of the fp32 attention in one pass, its output projection, kutacc_af2_linear on fp32 tensors;
// src/attention/gating_attention.cpp:47-66,152-157; src/linear/mm.cpp:46-86.) tcgen05.mma has no fp32 input type. An element is
// split into three bf16 pieces, x = x0 + x1 + x2: each has eight bits and the exponent range of fp32, together they are x itself, whatever
// the other elements of its row are. The product is
//   x0.w0 + (x0.w1 + x1.w0 + x1.w1 + x0.w2 + x2.w0)        (the other three, below 2^-22 of the first, are dropped)
// with the five small products in an accumulator of their own, which the epilogue adds: the tensor core truncates at every
// accumulation, and only K / 16 of them are at full magnitude. Against tf32 heads and tails (gemm_tf32_tcgen05.cu, which keeps all
// other K: three products at half the rate) the tensor cores have the same work, but an operand 6 bytes instead of 8, its activations
// are read once, and half as many accumulations count. (fp16 heads and tails with a power of two per row need half the
// work, three products at the full rate, but hold elements below 2^-29 of their row's largest in fewer bits and from 2^-51 on not at all.)
//
// The activations stand still, as in gemm_proj.cu: a persistent CTA (one per SM) loads 128 rows, all K columns, as fp32; the
// epilogue warps split them, the first two pieces into tensor memory, where five of the six products read them without a byte of
// shared memory, the third where the fp32 values were; and the weights, split by a kernel of their own (a row of them
// is used by every CTA), stream past in slabs of 128 channels x 64 columns.
//   warp 0      producer: rows in slabs of 32 fp32 columns, weight slabs (third, second, first pieces of 64 columns, a ring of five or eight)
//   warp 1      MMA issuer: 24 instructions of 16 columns for every 64, into two 128 x 128 accumulators (128 x 64 for few rows), of which the
//               epilogue takes the small products first: the next tile begins while it waits for the large ones
//   warps 4-11  split the rows, a thread half a row; epilogue, 32 rows x 64 columns each: tcgen05.ld of both accumulators, which frees them,
//               the split of the next block once the last tile of this one is in registers, bias, staging tile (32 x 16), TMA store
// What bounds it: the tensor cores and the power they take. 32768 rows x 1024 channels x 256 columns: 68 us, 117000 clocks of a CTA (for
// its 14 tiles of 6144 clocks of products; the first, whose rows come from HBM, is done at 14000), at 1.75 GHz under the power limit; with fp16
// pairs 65. As a split of the activations and tf32 products 20 + 92. x 128 columns 45 us. Error against 64 bits at K = 128 and 256 (2-norm):
// 1.3e-7 and 2.4e-7 (tf32 3.4e-7 and 6.4e-7, fp16 pairs 2.0e-7 and 3.5e-7). The fp32 layer of 128 x 256 rows: 290 us with tf32, 234 (fp16 pairs 217).
//
// All mbarrier waits are bounded; on a timeout the roles fall through to the common tail, the TMEM allocation is
// released and the host-visible error word carries the site.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

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

// KS: 64-column slabs of a row, BN: channels of a column tile
template <int KS, int BN>
struct Geo {
    static constexpr int NW = KS == 4 ? 5 : 8;                                   // slabs of the weight ring
    static constexpr int NSTG = KS == 4 ? 1 : 2;                                 // staging tiles of a warp
    static constexpr int ACC_COL = 64 * KS;                                      // after the first and second pieces of the rows
    static constexpr int OFF_A = NW * SLAB_BYTES;
    static constexpr int OFF_STG = OFF_A + 2 * KS * SLAB_BYTES;
    static constexpr int OFF_BAR = OFF_STG + EPI_WARPS * NSTG * STG_BYTES;
    static constexpr int NBARS = 2 * NW + 3 * KS + 4;
    static_assert(ACC_COL + 2 * BN <= 512, "tensor memory");
    static constexpr int SMEM_BYTES = OFF_BAR + 8 * NBARS + 16 + 1024;
    static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
};

struct alignas(64) RowsMaps {
    CUtensorMap a;        // A [M][K] fp32, box [32, 128], 128-byte swizzle
    CUtensorMap w[4];     // W' [N][3K] bf16 (the three pieces one after another) per segment, box [64, BN], 128-byte swizzle
    CUtensorMap out[4];   // per segment [M][N] (split rows: [M][2N]) fp32, box [16, 32], 64-byte swizzle
};

struct RowsParams {
    const float *bias[4];   // per segment, may be null
    float *out_t[4];        // kTf32SplitTransposed segments: [B][N/32][64][S]
    int layout[4];          // per segment: Tf32Layout
    int M, N, tiles;        // column tiles of all segments
    int S;                  // rows per batch row (transposed segments)
    int64_t vt_pitch;
    int whole;              // blocks with all their column tiles, full waves of them
    int rest, per, units;   // the tiles of the blocks after them, how many of these in a row are a unit, and whole blocks and units
    int *err;
};

// Two elements in three packed bf16 pieces each, x = x0 + x1 + x2: x0 the upper half of the bits, x1 the rest rounded, x2 what is left,
// which has eight bits.
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t &x0, uint32_t &x1, uint32_t &x2)
{
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    x0 = __byte_perm(ua, ub, 0x7632);
    const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
    x1 = pack_bf16x2(ra, rb);
    x2 = __byte_perm(__float_as_uint(ra - bf16lo_to_f32(x1)), __float_as_uint(rb - bf16hi_to_f32(x1)), 0x7632);
}

// BN: channels of a column tile, 128 or 64
template <int KS, int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_rows_kernel(const __grid_constant__ RowsMaps maps, const __grid_constant__ RowsParams p)
{
    using T = Geo<KS, BN>;
    constexpr int K = 64 * KS, NW = T::NW;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar = smem + T::OFF_BAR;
    auto w_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto w_empty = [&](int s) { return bar + 8u * (uint32_t)(NW + s); };
    auto a_full = [&](int ks) { return bar + 8u * (uint32_t)(2 * NW + ks); };
    auto a_empty = [&](int ks) { return bar + 8u * (uint32_t)(2 * NW + KS + ks); };
    auto a_split = [&](int ks) { return bar + 8u * (uint32_t)(2 * NW + 2 * KS + ks); };
    const uint32_t small_full = bar + 8u * (uint32_t)(2 * NW + 3 * KS), small_empty = small_full + 8u, large_full = small_full + 16u,
                   large_empty = small_full + 24u;
    const uint32_t tmem_slot = bar + 8u * T::NBARS;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // This CTA's next part of its units: a block, its first column tile and how many. u: the unit, at: tiles of it handed out
    auto next_part = [&](int &u, int &at, int &block, int &t0, int &nt) -> bool {
        if (u >= p.units) return false;
        const int v = u - p.whole, first = v * p.per, n = v < 0 ? p.tiles : min(p.per, p.rest - first);
        block = v < 0 ? u : p.whole + (first + at) / p.tiles;
        t0 = v < 0 ? 0 : (first + at) % p.tiles;
        nt = min(p.tiles - t0, n - at);
        at += nt;
        if (at == n) {
            at = 0;
            u += (int)gridDim.x;
        }
        return true;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NW; ++s) {
            mbar_init(w_full(s), 1);
            mbar_init(w_empty(s), 1);
        }
        for (int ks = 0; ks < KS; ++ks) {
            mbar_init(a_full(ks), 1);
            mbar_init(a_empty(ks), 1);
            mbar_init(a_split(ks), 4);
        }
        mbar_init(small_full, 1);
        mbar_init(small_empty, EPI_WARPS);
        mbar_init(large_full, 1);
        mbar_init(large_empty, EPI_WARPS);
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
            int s = 0, round = 0, rows_asked = 0;                      // next slab's slot, times the ring has gone round; row slabs asked for
            for (int n = 0, u = (int)blockIdx.x, at = 0; ok; ++n) {
                int block, t0, nt;
                if (!next_part(u, at, block, t0, nt)) break;
                for (int ks = 0; ks < KS && ok; ++ks) {
                    if (n > 0) ok = mbar_wait(a_empty(ks), (uint32_t)((n - 1) & 1), p.err, 111);
                    if (!ok) break;
                    ++rows_asked;
                    mbar_arrive_expect_tx(a_full(ks), 2 * SLAB_BYTES);
                    const uint32_t dst = smem + T::OFF_A + ks * 2 * SLAB_BYTES;
                    tma_load_2d(dst, &maps.a, a_full(ks), ks * 64, block * BM);
                    tma_load_2d(dst + SLAB_BYTES, &maps.a, a_full(ks), ks * 64 + 32, block * BM);
                }
                for (int j = 0; j < nt && ok; ++j) {
                    const int col = (t0 + j) * BN, seg = col / p.N;
                    for (int h = 0; h < 3 * KS; ++h) {                 // of every 64 columns the third, second, first pieces
                        if (round > 0) ok = mbar_wait(w_empty(s), (uint32_t)((round - 1) & 1), p.err, 112);
                        if (!ok) break;
                        mbar_arrive_expect_tx(w_full(s), BN * 128);
                        tma_load_2d(smem + (uint32_t)(s * SLAB_BYTES), &maps.w[seg], w_full(s), (2 - h % 3) * K + h / 3 * 64, col % p.N);
                        if (++s == NW) {
                            s = 0;
                            ++round;
                        }
                    }
                    if (j == 0) {                                      // the next block's rows on their way to L2
                        int u2 = u, at2 = at, next, nt0, nnt;
                        if (next_part(u2, at2, next, nt0, nnt))
                            for (int c = 0; c < 2 * KS; ++c) tma_prefetch_2d(&maps.a, c * 32, next * BM);
                    }
                }
            }
            // after a wait that ran out: no copy may still be on its way when the CTA exits
            if (!ok) {
                for (int i = 0; i < NW; ++i) {
                    const int last = i < s ? round : round - 1;
                    if (last >= 0) mbar_wait(w_full(i), (uint32_t)(last & 1), p.err, 120);
                }
                for (int ks = 0; ks < KS; ++ks) {
                    const int asked = (rows_asked + KS - 1 - ks) / KS;
                    if (asked > 0) mbar_wait(a_full(ks), (uint32_t)((asked - 1) & 1), p.err, 121);
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc = make_instr_desc_bf16(BM, BN);
        constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;                   // descriptor addresses count in units of 16 bytes
        const uint64_t wd0 = make_smem_desc_kmajor(smem, 128), ad0 = make_smem_desc_kmajor(smem + T::OFF_A, 128);
        bool ok = true;
        int s = 0, tc = 0;
        uint32_t par = 0;
        for (int n = 0, u = (int)blockIdx.x, at = 0; ok; ++n) {
            int block, t0, nt;
            if (!next_part(u, at, block, t0, nt)) break;
            for (int j = 0; j < nt && ok; ++j, ++tc) {
                if (tc > 0) ok = mbar_wait_warp(small_empty, (uint32_t)((tc - 1) & 1), p.err, 114);
                const uint32_t large = tmem_base + (uint32_t)T::ACC_COL, small = large + BN;
                for (int ks = 0; ks < KS && ok; ++ks) {
                    if (j == 0) ok = mbar_wait_warp(a_split(ks), (uint32_t)(n & 1), p.err, 113);
                    const uint32_t a0 = tmem_base + (uint32_t)(ks * 64), a1 = a0 + 32;
                    const uint64_t a2 = ad0 + (uint32_t)(ks * 2 * SLAB16);
#pragma unroll
                    for (int piece = 2; piece >= 0; --piece) {         // of W
                        ok = ok && mbar_wait_warp(w_full(s), par, p.err, 115);
                        if (ks == 0 && piece == 0 && tc > 0) ok = ok && mbar_wait_warp(large_empty, (uint32_t)((tc - 1) & 1), p.err, 118);
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            // 16 columns an instruction: 32 bytes, or 8 columns of tensor memory
                            const uint64_t w = wd0 + (uint32_t)(s * SLAB16);
                            if (piece > 0) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) tc_mma_bf16_ts(small, a0 + 8 * k, w + 2 * k, idesc, piece == 1 || ks > 0 || k > 0 ? 1u : 0u);
                            }
                            if (piece < 2) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) tc_mma_bf16_ts(small, a1 + 8 * k, w + 2 * k, idesc, 1u);
                            }
                            if (piece == 0) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) tc_mma_bf16(small, a2 + 2 * k, w + 2 * k, idesc, 1u);
                                if (ks == KS - 1) tc_commit(small_full);
#pragma unroll
                                for (int k = 0; k < 4; ++k) tc_mma_bf16_ts(large, a0 + 8 * k, w + 2 * k, idesc, ks > 0 || k > 0 ? 1u : 0u);
                                if (j == nt - 1) tc_commit(a_empty(ks));
                                if (ks == KS - 1) tc_commit(large_full);
                            }
                            tc_commit(w_empty(s));
                        }
                        __syncwarp();
                        if (++s == NW) {
                            s = 0;
                            par ^= 1u;
                        }
                    }
                }
            }
        }
    } else if (warp >= EPI_WARP0) {
        // ================= split, epilogue =================
        const int ew = warp - EPI_WARP0, half = ew >> 2, quad = warp & 3;
        const uint32_t stg0 = smem + T::OFF_STG + (uint32_t)(ew * T::NSTG * STG_BYTES);
        uint32_t nstore = 0;
        bool ok = true;

        // a thread's row, of every 64 columns that this half of the warps takes: the fp32 values make way for the first pieces (where
        // columns 0..31 lay) and the second pieces, the third go to tensor memory
        auto split_rows = [&](int n) {
            constexpr int CH = 8;                                      // chunks of 16 bytes (4 columns) at a time
            const int row = quad * 32 + lane;
#pragma unroll 1
            for (int ks = half * (KS / 2); ks < (half + 1) * (KS / 2); ++ks) {
                ok = mbar_wait_warp(a_full(ks), (uint32_t)(n & 1), p.err, 116);
                if (!ok) return;
                tc_fence_after();
                const uint32_t slab = smem + T::OFF_A + (uint32_t)(ks * 2 * SLAB_BYTES + row * 128);
                auto chunk = [&](int c) { return slab + (uint32_t)((c >> 3) * SLAB_BYTES + (((c & 7) ^ (row & 7)) << 4)); };
                const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(ks * 64);
#pragma unroll
                for (int c = 0; c < 16; c += CH) {                     // no chunk is written before it has been read
                    float4 v[CH];
#pragma unroll
                    for (int e = 0; e < CH; ++e) v[e] = lds128_f32(chunk(c + e));
#pragma unroll
                    for (int e = 0; e < CH; e += 4) {
                        uint32_t x0[8], x1[8], x2[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            split_bf16(v[e + i].x, v[e + i].y, x0[2 * i], x1[2 * i], x2[2 * i]);
                            split_bf16(v[e + i].z, v[e + i].w, x0[2 * i + 1], x1[2 * i + 1], x2[2 * i + 1]);
                        }
                        tmem_st_32x8(t_row + (c + e) * 2, x0);
                        tmem_st_32x8(t_row + 32 + (c + e) * 2, x1);
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(chunk((c + e) / 2 + i)), "r"(x2[4 * i]), "r"(x2[4 * i + 1]),
                                         "r"(x2[4 * i + 2]), "r"(x2[4 * i + 3])
                                         : "memory");
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(a_split(ks));
            }
        };

        int tc = 0;
        for (int n = 0, u = (int)blockIdx.x, at = 0; ok; ++n) {
            int block, t0, nt;
            if (!next_part(u, at, block, t0, nt)) break;
            if (n == 0) split_rows(0);
            if (!ok) break;
            const int m0 = block * BM + quad * 32, m = m0 + lane;
            for (int j = 0; j < nt; ++j, ++tc) {
                const int col = (t0 + j) * BN + half * (BN / 2), seg = col / p.N, n0 = col % p.N;
                const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(T::ACC_COL + half * (BN / 2));
                uint32_t acc[BN / 64][32], small[BN / 64][32];
                // out of tensor memory, so that the next tile's small products may begin, and then its large ones
                ok = mbar_wait_warp(small_full, (uint32_t)(tc & 1), p.err, 119);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < BN / 64; ++c) tmem_ld_32x32(tcol + BN + c * 32, small[c]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(small_empty);
                ok = mbar_wait_warp(large_full, (uint32_t)(tc & 1), p.err, 117);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < BN / 64; ++c) tmem_ld_32x32(tcol + c * 32, acc[c]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(large_empty);
#pragma unroll
                for (int c = 0; c < BN / 64; ++c)
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[c][e] = __float_as_uint(__uint_as_float(acc[c][e]) + __uint_as_float(small[c][e]));
                // the next block's products wait for its split
                if (j == nt - 1 && u < p.units) split_rows(n + 1);
                if (!ok) break;
                const float *bias = p.bias[seg];
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
                    if (bias) {
#pragma unroll
                        for (int j4 = 0; j4 < 8; ++j4) {
                            const float4 bv = __ldg(reinterpret_cast<const float4 *>(bias + nn) + j4);
                            r[4 * j4] = __float_as_uint(__uint_as_float(r[4 * j4]) + bv.x);
                            r[4 * j4 + 1] = __float_as_uint(__uint_as_float(r[4 * j4 + 1]) + bv.y);
                            r[4 * j4 + 2] = __float_as_uint(__uint_as_float(r[4 * j4 + 2]) + bv.z);
                            r[4 * j4 + 3] = __float_as_uint(__uint_as_float(r[4 * j4 + 3]) + bv.w);
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
                        const uint32_t stg = stg0 + nstore++ % T::NSTG * STG_BYTES;
                        if (lane == 0) tma_store_wait_read<T::NSTG - 1>();          // the store out of this tile has been read
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

// Weights: a warp per row, up to eight matrices of the same shape a launch (blockIdx.y picks one). dst [rows][3K] bf16.
struct SplitArgs {
    const float *src[8];
    __nv_bfloat16 *dst[8];
};
template <int K>
__global__ void __launch_bounds__(256) split_weights_kernel(const __grid_constant__ SplitArgs args, int64_t src_ld, int rows)
{
    release_successor();
    wait_for_predecessor();
    const int row = (int)(blockIdx.x * 8 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float4 *src = reinterpret_cast<const float4 *>(args.src[blockIdx.y] + (int64_t)row * src_ld);
    float4 v[K / 128];
#pragma unroll
    for (int i = 0; i < K / 128; ++i) v[i] = __ldg(src + i * 32 + lane);
    __nv_bfloat16 *dst = args.dst[blockIdx.y] + (int64_t)row * 3 * K + lane * 4;
#pragma unroll
    for (int i = 0; i < K / 128; ++i) {
        uint2 x[3];
        split_bf16(v[i].x, v[i].y, x[0].x, x[1].x, x[2].x);
        split_bf16(v[i].z, v[i].w, x[0].y, x[1].y, x[2].y);
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2 *>(dst + e * K + i * 128) = x[e];
    }
}

template <int KS, int BN>
void launch_ks(cudaStream_t stream, const RowsMaps &maps, const RowsParams &p, int grid)
{
    static const cudaError_t attr = cudaFuncSetAttribute(gemm_f32_rows_kernel<KS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<KS, BN>::SMEM_BYTES);
    KUTACC_CUDA(attr);
    launch_chained(gemm_f32_rows_kernel<KS, BN>, (unsigned)grid, THREADS, Geo<KS, BN>::SMEM_BYTES, stream, maps, p);
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
        a.dst[i] = (__nv_bfloat16 *)dst[j];
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
    // Few rows: column tiles of half the width while those of four such products are three for each SM. Fewer of them make a CTA wait
    // on one tile's chain: fp32 layer of 8 heads, 8 x 48 rows 33.8 -> 30.6 us, 20 x 60 38.8 -> 34.9, 24 x 130 57.8 -> 52.2; past the line 12 x 350
    // rows would be 75.6 -> 77.4, a linear layer of 32768 rows x 1024 channels x 128 columns 77 -> 88 (an instruction of 64 channels takes more than
    // half the time). The rule does not look at nseg, so that a layer's projections and output run the same code.
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    const int64_t blocks = (M + BM - 1) / BM;
    const int BN = blocks * (N / 64) * 4 <= 3 * sms ? 64 : 128;
    RowsMaps maps;
    RowsParams p = {};
    if (!make_tensor_map_2d(&maps.a, a, /*elem_bytes=*/4, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 32, BM, 128)) return false;
    for (int i = 0; i < 4; ++i) {
        const int j = i < nseg ? i : 0;
        p.bias[i] = bias[j];
        p.layout[i] = layout ? layout[j] : kTf32Rows;
        p.out_t[i] = (float *)out[j];
        if (!make_tensor_map_2d(&maps.w[i], w_split[j], 2, (uint64_t)3 * K, (uint64_t)N, (uint64_t)3 * K, 64, BN, 128)) return false;
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
    // Whole blocks for all full waves; the blocks of the last one are dealt out in equal runs of their column tiles. A run costs its
    // tiles and START tiles for every block it touches, whose rows are loaded and split.
    constexpr double START = 0.75;
    p.whole = (int)(blocks / sms * sms);
    p.rest = (int)(blocks - p.whole) * p.tiles;
    double best = 1e30;
    for (int per = p.tiles; per > 0; per = std::min(per - 1, 4096)) {
        const int units = (p.rest + per - 1) / per;
        const double cost = (double)((units + sms - 1) / sms) * (per + START * (p.tiles % per ? 2 : 1));
        if (cost < best * 0.999) {
            best = cost;
            p.per = per;
            p.units = p.whole + units;
        }
    }
    const int grid = std::min(p.units, sms);
    KernelTimer timer__("gemm_f32_rows", stream);
    if (BN == 64)
        K == 128 ? launch_ks<2, 64>(stream, maps, p, grid) : launch_ks<4, 64>(stream, maps, p, grid);
    else
        K == 128 ? launch_ks<2, 128>(stream, maps, p, grid) : launch_ks<4, 128>(stream, maps, p, grid);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
