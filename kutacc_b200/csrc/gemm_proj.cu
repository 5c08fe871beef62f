// Q/K/V/gate projection of the attention on the fifth-generation tensor cores, with the LayerNorm in front of it where the
// caller asks for one (up to 256 channels).
//
//   q, k [B, H, S, D], v^T [B, H*D, S] (row pitch a multiple of 8), gate = bf16(x.Wg + bg) [B, S, C] or bf16(sigmoid(gate))
//
// (src/attention/gating_attention.cpp:47-66; with gate_sigmoid the sigmoid of :134-147 is applied here.) The activations stand still: a
// persistent CTA (one per SM) loads a block of 256 rows once, all K columns of it, and streams the four weights past it in
// slabs of 128 channels x 64 columns, each of which serves both 128-row tiles of the block. With a 128 x 128 tile at a time
// every tile brought its own 64 to 128 KB of operands from L2, which bound the kernel: 146 us for 196608 rows x 256 channels.
//   warp 0      producer: row blocks in slabs of 64 columns (two blocks in flight up to 128 channels), weight slabs (ring)
//   warp 1      MMA issuer: 128 x 128 accumulators, two row tiles x two column tiles in tensor memory
//   warps 4-19  epilogue, eight per row tile, 32 rows x 64 columns each: tcgen05.ld, bias and sigmoid for the gate, bf16,
//               staging tile, TMA store into the destination layout
// A row tile is four groups of 32 rows, and a group never crosses a batch row: S is padded to 32, not to 128, and the TMA
// stores of a warp (32 rows) stay inside one batch row. Rows past S are zero-filled on load and clipped on store.
//
// What bounds it: at 128 channels the writes to memory (2^20 rows: 238 us without launch, the bytes alone 205); at 256
// channels the products, whose 128 x 128 instructions read 128 bytes of shared memory per clock (196608 rows: 105 us, of which
// about 60 on the tensor cores; 77 for the bytes). Before: 266 and 140 us.
//
// LayerNorm: the epilogue warps normalise the block where it lies in shared memory (statistics and arithmetic of layernorm.cu,
// one bf16 rounding), 16 rows each, before the products read it; for 128 channels the next block's turn comes after the
// first column tile of this one, so that the products do not wait for it. The normalised tensor is never written.
//
// All mbarrier waits are bounded; on a timeout the roles fall through to the common tail, the TMEM allocation is released
// and the host-visible error word carries the site.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ln_utils.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

#include <algorithm>
#include <climits>

namespace kutacc {
namespace dev {

namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int SLAB_BYTES = 128 * BK * 2;                // 16 KB: 128 rows (or output channels) x 64 columns
constexpr int NW = 4;                                   // weight ring
constexpr int EPI_WARPS = 16, EPI_WARP0 = 4;
constexpr int THREADS = (EPI_WARP0 + EPI_WARPS) * 32;
constexpr int STG_BYTES = 32 * 32 * 2;
constexpr int DIRECT_D = 8;                             // head size whose q and k are stored without a staging tile
constexpr int OFF_W = 0, OFF_A = NW * SLAB_BYTES;

// KS: 64-column slabs of a row (channels / 64)
template <int KS>
struct Geo {
    static constexpr int NBLK = KS == 4 ? 1 : 2;                     // row blocks in shared memory
    static constexpr int BLOCK_BYTES = 2 * KS * SLAB_BYTES;
    static constexpr int OFF_STG = OFF_A + NBLK * BLOCK_BYTES;
    static constexpr int OFF_VEC = OFF_STG + EPI_WARPS * STG_BYTES;  // gate bias
    static constexpr int OFF_BAR = OFF_VEC + KS * 64 * 4;
    static constexpr int NBARS = 2 * NW + NBLK * (2 * KS + 1) + 8;
    static constexpr int SMEM_BYTES = OFF_BAR + 8 * NBARS + 16 + 1024;
    static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
};

struct alignas(64) ProjMaps {
    CUtensorMap a;        // x [B][S][C], box [64, 128 or 32 rows], 128-byte swizzle
    CUtensorMap w[4];     // [C][C], box [64, 128 (64 channels: 64)], 128-byte swizzle
    CUtensorMap out[4];   // 32 x 32 staging tiles
};

struct ProjParams {
    const float *bg, *gamma, *beta;     // gamma: null without LayerNorm
    __nv_bfloat16 *qk[2];               // heads of 8: q and k without a tensor map
    float eps;
    int S, B, D;
    int s32;              // 32-row groups per batch row
    int rows128;          // S is a multiple of 128: a row tile is one box
    int whole;            // a unit of work is a block with all its column tiles, up to this unit;
    int nsplit;           // after it a unit is 1 / nsplit of a block's column tiles
    int units;
    int *err;
};

// R: row tiles per block, 1 or 2. GATE_SIGMOID: the stored gate is bf16(sigmoid(bf16(x.Wg + bg)))
template <int KS, int R, bool LN, bool GATE_SIGMOID>
__global__ void __launch_bounds__(THREADS, 1)
proj_kernel(const __grid_constant__ ProjMaps maps, const __grid_constant__ ProjParams p)
{
    using T = Geo<KS>;
    constexpr int C = KS * 64, NT = 4 * C / BN, NBLK = T::NBLK;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *gen = smem_raw + (smem - smem_u32(smem_raw));
    const uint32_t bar = smem + T::OFF_BAR;
    auto w_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto w_empty = [&](int s) { return bar + 8u * (uint32_t)(NW + s); };
    // the rows arrive and leave in slabs of 64 columns: the next block follows while the last column tile is at work
    constexpr int BAR_A = 2 * NW, BAR_ACC = BAR_A + NBLK * (2 * KS + 1);
    auto a_full = [&](int s, int ks) { return bar + 8u * (uint32_t)(BAR_A + s * (2 * KS + 1) + ks); };
    auto a_empty = [&](int s, int ks) { return bar + 8u * (uint32_t)(BAR_A + s * (2 * KS + 1) + KS + ks); };
    auto a_norm = [&](int s) { return bar + 8u * (uint32_t)(BAR_A + s * (2 * KS + 1) + 2 * KS); };
    auto acc_full = [&](int i) { return bar + 8u * (uint32_t)(BAR_ACC + i); };                  // i = 2 * buffer + row tile
    auto acc_empty = [&](int i) { return bar + 8u * (uint32_t)(BAR_ACC + 4 + i); };
    const uint32_t tmem_slot = bar + 8u * T::NBARS;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // unit u: its block, first column tile and number of column tiles
    auto unit = [&](int u, int &block, int &t0, int &nt) {
        const int v = u - p.whole;
        block = v < 0 ? u : p.whole + v / p.nsplit;
        nt = v < 0 ? NT : NT / p.nsplit;
        t0 = v < 0 ? 0 : v % p.nsplit * nt;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NW; ++s) {
            mbar_init(w_full(s), 1);
            mbar_init(w_empty(s), 1);
        }
        for (int s = 0; s < NBLK; ++s) {
            for (int ks = 0; ks < KS; ++ks) {
                mbar_init(a_full(s, ks), 1);
                mbar_init(a_empty(s, ks), 1);
            }
            mbar_init(a_norm(s), (uint32_t)(8 * R));
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(acc_full(i), 1);
            mbar_init(acc_empty(i), 8);
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
    for (int i = threadIdx.x; i < C; i += THREADS) reinterpret_cast<float *>(gen + T::OFF_VEC)[i] = p.bg[i];
    __syncthreads();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0) {
        // ================= producer =================
        if (elect_one()) {
            bool ok = true;
            int wit = 0;
            auto load_rows = [&](int n, int ks) {                      // a slab of the rows of this CTA's n-th unit
                const int u = (int)blockIdx.x + n * (int)gridDim.x, s = n % NBLK;
                if (u >= p.units || !ok) return;
                int block, t0, nt;
                unit(u, block, t0, nt);
                if (n >= NBLK) ok = mbar_wait(a_empty(s, ks), (uint32_t)((n / NBLK - 1) & 1), p.err, 101);
                if (!ok) return;
                mbar_arrive_expect_tx(a_full(s, ks), (uint32_t)(R * SLAB_BYTES));
                for (int r = 0; r < R; ++r) {
                    const int g0 = (block * R + r) * 4;
                    const uint32_t dst = smem + OFF_A + s * T::BLOCK_BYTES + (r * KS + ks) * SLAB_BYTES;
                    if (p.rows128) {
                        tma_load_3d(dst, &maps.a, a_full(s, ks), ks * BK, g0 % p.s32 * 32, g0 / p.s32);
                    } else {
                        for (int q = 0; q < 4; ++q)
                            tma_load_3d(dst + q * 4096, &maps.a, a_full(s, ks), ks * BK, (g0 + q) % p.s32 * 32, (g0 + q) / p.s32);
                    }
                }
            };
            for (int ks = 0; ks < KS && NBLK == 2; ++ks) load_rows(0, ks);
            for (int n = 0; ok; ++n) {
                const int u = (int)blockIdx.x + n * (int)gridDim.x;
                if (u >= p.units) break;
                int block, t0, nt;
                unit(u, block, t0, nt);
                for (int j = 0; j < nt && ok; ++j) {
                    for (int ks = 0; ks < KS && ok; ++ks, ++wit) {
                        if (NBLK == 1 && j == 0) load_rows(n, ks);
                        const int s = wit % NW;
                        if (wit >= NW && ok) ok = mbar_wait(w_empty(s), (uint32_t)((wit / NW - 1) & 1), p.err, 102);
                        if (!ok) break;
                        mbar_arrive_expect_tx(w_full(s), SLAB_BYTES);
                        const uint32_t dst = smem + OFF_W + s * SLAB_BYTES;
                        const int col = (t0 + j) * BN;
                        tma_load_3d(dst, &maps.w[col / C], w_full(s), ks * BK, col % C, 0);
                        if (KS == 1) tma_load_3d(dst + SLAB_BYTES / 2, &maps.w[col / C + 1], w_full(s), ks * BK, 0, 0);
                    }
                    for (int ks = 0; ks < KS && NBLK == 2 && j == 0; ++ks) load_rows(n + 1, ks);
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc = make_instr_desc_bf16(BM, BN);
        constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;                   // descriptor addresses count in units of 16 bytes
        const uint64_t wd0 = make_smem_desc_kmajor(smem + OFF_W, 128), ad0 = make_smem_desc_kmajor(smem + OFF_A, 128);
        bool ok = true;
        int wit = 0, tc = 0;
        for (int n = 0; ok; ++n) {
            const int u = (int)blockIdx.x + n * (int)gridDim.x, sa = n % NBLK;
            if (u >= p.units) break;
            int block, t0, nt;
            unit(u, block, t0, nt);
            if (LN) ok = mbar_wait_warp(a_norm(sa), (uint32_t)((n / NBLK) & 1), p.err, 103);
            const uint64_t ad = ad0 + (uint32_t)(sa * (T::BLOCK_BYTES >> 4));
            for (int j = 0; j < nt && ok; ++j, ++tc) {
                const int buf = tc & 1;
                for (int r = 0; r < R && tc >= 2 && ok; ++r)
                    ok = mbar_wait_warp(acc_empty(2 * buf + r), (uint32_t)((tc / 2 - 1) & 1), p.err, 104);
                for (int ks = 0; ks < KS && ok; ++ks, ++wit) {
                    const int s = wit % NW;
                    if (!LN && j == 0) ok = mbar_wait_warp(a_full(sa, ks), (uint32_t)((n / NBLK) & 1), p.err, 108);
                    ok = ok && mbar_wait_warp(w_full(s), (uint32_t)((wit / NW) & 1), p.err, 105);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t wd = wd0 + (uint32_t)(s * SLAB16);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const uint64_t a = ad + (uint32_t)((r * KS + ks) * SLAB16);
                            const uint32_t d = tmem_base + (uint32_t)((2 * buf + r) * BN);
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k) tc_mma_bf16(d, a + 2 * k, wd + 2 * k, idesc, (ks > 0 || k > 0) ? 1u : 0u);
                            if (ks == KS - 1) tc_commit(acc_full(2 * buf + r));
                        }
                        tc_commit(w_empty(s));
                        if (j == nt - 1) tc_commit(a_empty(sa, ks));
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= EPI_WARP0) {
        // ================= epilogue =================
        const int ew = warp - EPI_WARP0, rt = ew >> 3, half = (ew >> 2) & 1, quad = warp & 3;
        const uint32_t stg = smem + T::OFF_STG + (uint32_t)(ew * STG_BYTES), bg_a = smem + T::OFF_VEC;
        bool ok = rt < R;

        // LayerNorm of this warp's 16 rows of unit n's block, in place. LPR lanes share a row, one 16-byte chunk (8 channels) each.
        constexpr int LPR = 8 * KS, RPP = 32 / LPR, PASSES = 16 / RPP;
        float gs[8], bs[8];
        if (LN) {
            const int ch = lane % LPR * 8;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                gs[e] = p.gamma[ch + e];
                bs[e] = p.beta[ch + e];
            }
        }
        auto normalise = [&](int n) {
            if ((int)blockIdx.x + n * (int)gridDim.x >= p.units || !ok) return;
            const int sa = n % NBLK, sub = lane / LPR, l = lane % LPR;
            for (int ks = 0; ks < KS && ok; ++ks) ok = mbar_wait_warp(a_full(sa, ks), (uint32_t)((n / NBLK) & 1), p.err, 106);
            if (!ok) return;
            const uint32_t base = smem + OFF_A + sa * T::BLOCK_BYTES + (rt * KS + l / 8) * SLAB_BYTES;
            constexpr int U = 4;                                       // rows in flight per lane group
#pragma unroll 1
            for (int p0 = 0; p0 < PASSES; p0 += U) {
                uint32_t addr[U];
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int row = (ew & 7) * 16 + (p0 + i) * RPP + sub;
                    addr[i] = base + (uint32_t)(row * 128 + (((l & 7) ^ (row & 7)) << 4));
                }
                layernorm_smem_rows<LPR, U>(addr, gs, bs, p.eps);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_norm(sa));
        };

        int tc = 0;
        if (LN) normalise(0);
        for (int n = 0; ok; ++n) {
            const int u = (int)blockIdx.x + n * (int)gridDim.x;
            if (u >= p.units) break;
            int block, t0, nt;
            unit(u, block, t0, nt);
            const int G = (block * R + rt) * 4 + quad, b = G / p.s32, row0 = G % p.s32 * 32;
            for (int j = 0; j < nt; ++j, ++tc) {
                const int buf = tc & 1, col = (t0 + j) * BN + half * 64, seg = col / C;
                ok = mbar_wait_warp(acc_full(2 * buf + rt), (uint32_t)((tc / 2) & 1), p.err, 107);
                if (!ok) break;
                tc_fence_after();
                uint32_t r[2][32];
                const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)((2 * buf + rt) * BN + half * 64);
                tmem_ld_32x32(tcol, r[0]);
                tmem_ld_32x32(tcol + 32, r[1]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(2 * buf + rt));
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int nn = col % C + c * 32;                   // first channel of the segment
                    uint32_t packed[16];
                    if (seg == 3) {
#pragma unroll
                        for (int j4 = 0; j4 < 8; ++j4) {
                            const float4 bv = lds128_f32(bg_a + (uint32_t)((nn + 4 * j4) * 4));
                            float y[4] = {__uint_as_float(r[c][4 * j4]) + bv.x, __uint_as_float(r[c][4 * j4 + 1]) + bv.y,
                                          __uint_as_float(r[c][4 * j4 + 2]) + bv.z, __uint_as_float(r[c][4 * j4 + 3]) + bv.w};
                            if (GATE_SIGMOID) {
#pragma unroll
                                for (int e = 0; e < 4; ++e) y[e] = sigmoid_of_bf16(y[e]);
                            }
                            packed[2 * j4] = pack_bf16x2(y[0], y[1]);
                            packed[2 * j4 + 1] = pack_bf16x2(y[2], y[3]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) packed[i] = pack_bf16x2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1]));
                    }
                    if (seg < 2 && p.D == DIRECT_D) {
                        // Rows of 16 bytes: four stores a lane, each of a warp 512 contiguous bytes. A TMA box of such rows is slow: 256 x 384
                        // rows of 8 heads of 8, the whole call, 183 -> 176 us. (Heads of 32 the same way, in whole sectors: 196608 rows x 256
                        // channels 109 -> 116 us.)
                        if (row0 + lane < p.S && b < p.B) {
                            __nv_bfloat16 *dst = p.qk[seg] + ((((int64_t)b * C + nn) / DIRECT_D) * p.S + row0 + lane) * DIRECT_D;
#pragma unroll
                            for (int i = 0; i < 32 / DIRECT_D; ++i)
#pragma unroll
                                for (int e = 0; e < DIRECT_D / 8; ++e) {
                                    const int v = (i * DIRECT_D / 8 + e) * 4;
                                    *reinterpret_cast<uint4 *>(dst + (int64_t)i * p.S * DIRECT_D + e * 8) =
                                        make_uint4(packed[v], packed[v + 1], packed[v + 2], packed[v + 3]);
                                }
                        }
                        continue;
                    }
                    if (lane == 0) tma_store_wait_read<0>();           // the store out of the staging tile has been read
                    __syncwarp();
                    if (seg == 2) {
                        // transposed staging tile: row = channel, column = this lane's position; 64-byte swizzle
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const uint32_t addr = stg + (uint32_t)(i * 64 + (((lane >> 3) ^ ((i >> 1) & 3)) << 4) + (lane & 7) * 2);
                            const uint16_t hv = (uint16_t)((i & 1) ? (packed[i >> 1] >> 16) : (packed[i >> 1] & 0xffffu));
                            asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(addr), "h"(hv) : "memory");
                        }
                    } else {
#pragma unroll
                        for (int ch = 0; ch < 4; ++ch) {
                            // heads of 16 channels: [head][row][channel], no swizzle
                            const uint32_t off = seg == 3 || p.D >= 32 ? (uint32_t)(lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4))
                                                                       : (uint32_t)((ch >> 1) * 1024 + lane * 32 + (ch & 1) * 16);
                            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(stg + off), "r"(packed[4 * ch]),
                                         "r"(packed[4 * ch + 1]), "r"(packed[4 * ch + 2]), "r"(packed[4 * ch + 3])
                                         : "memory");
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        const CUtensorMap *omap = &maps.out[seg];
                        if (seg == 2)
                            tma_store_3d(omap, stg, row0, b * C + nn, 0);
                        else if (seg == 3)
                            tma_store_3d(omap, stg, nn, row0, b);
                        else
                            tma_store_3d(omap, stg, nn % p.D, row0, (b * C + nn) / p.D);
                        tma_store_commit();
                    }
                }
                if (LN && NBLK == 2 && j == 0) normalise(n + 1);
                if (!ok) break;
            }
            if (LN && NBLK == 1) normalise(n + 1);
        }
        if (lane == 0) tma_store_wait<0>();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int KS, int R, bool LN, bool GATE_SIGMOID>
void launch_one(cudaStream_t stream, int grid, const ProjMaps &maps, const ProjParams &p)
{
    static const cudaError_t attr =
        cudaFuncSetAttribute(proj_kernel<KS, R, LN, GATE_SIGMOID>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<KS>::SMEM_BYTES);
    KUTACC_CUDA(attr);
    launch_chained(proj_kernel<KS, R, LN, GATE_SIGMOID>, (unsigned)grid, THREADS, Geo<KS>::SMEM_BYTES, stream, maps, p);
}

template <int KS, bool GATE_SIGMOID>
bool launch_ks(cudaStream_t stream, const ProjMaps &maps, ProjParams p)
{
    // How the work is cut: blocks of 256 rows, or of 128 where that fills the chip better; whole blocks for all full waves, and
    // the blocks of the last one in 1 / nsplit of their column tiles each, whichever ends first. A unit costs its column tiles
    // plus about one for its rows: a wave of units of 256 rows x 4, 2 and 1 tiles takes 7.0, 3.8 and 2.6 us at 128 channels, of 8, 4
    // and 2 tiles 18.6, 9.7 and 5.7 us at 256. Units of 128 rows take 4.4, 2.9, 1.7 and 10.5, 6.2, 4.0 us: a block of 256 counts as
    // 1.3 of them, less than the 1.5 to 1.75 measured, which prefers it in calls of a wave or less.
    constexpr int NT = 4 * KS * 64 / BN;
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    const int64_t groups = (int64_t)p.B * p.s32;
    double best = 1e30;
    int R = 2;
    for (int r = 2; r >= 1; --r) {
        const int64_t blocks = (groups + 4 * r - 1) / (4 * r), whole = blocks / sms * sms;
        for (int ns = 1; ns <= NT; ns *= 2) {
            const int64_t last = (blocks - whole) * ns;
            const double cost = ((double)(whole / sms) * (NT + 1.0) + (double)((last + sms - 1) / sms) * ((double)NT / ns + 1.0)) *
                                (r == 2 ? 1.3 : 1.0);
            if (cost < best * 0.999) {
                best = cost;
                R = r;
                p.whole = (int)whole;
                p.nsplit = ns;
                p.units = (int)(whole + last);
            }
        }
    }
    const int grid = std::min(p.units, sms);
    KernelTimer timer__("proj_qkvg", stream);
    if (p.gamma)
        R == 2 ? launch_one<KS, 2, true, GATE_SIGMOID>(stream, grid, maps, p) : launch_one<KS, 1, true, GATE_SIGMOID>(stream, grid, maps, p);
    else
        R == 2 ? launch_one<KS, 2, false, GATE_SIGMOID>(stream, grid, maps, p) : launch_one<KS, 1, false, GATE_SIGMOID>(stream, grid, maps, p);
    count_launch();
    return true;
}

}  // namespace

bool tcgen05_proj_rows_bf16(cudaStream_t stream, const void *x, const void *wq, const void *wk, const void *wv, const void *wg,
                            const float *bg, void *q, void *k, void *vt, int64_t vt_pitch, void *gate, bool gate_sigmoid, int B, int S,
                            int H, int D, const float *ln_gamma, const float *ln_beta, float ln_eps)
{
    const int C = H * D;
    if ((C != 64 && C != 128 && C != 256) || (D != 8 && D != 16 && D != 32) || vt_pitch % 8 != 0 || vt_pitch < S) return false;
    const int64_t s32 = (S + 31) / 32;
    if (s32 * B > INT32_MAX / 8 || (int64_t)B * C > INT32_MAX / 2) return false;
    if ((((uintptr_t)x | (uintptr_t)wq | (uintptr_t)wk | (uintptr_t)wv | (uintptr_t)wg) & 15u) != 0) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    ProjParams p = {};
    p.rows128 = S % 128 == 0;
    ProjMaps maps;
    const void *w[4] = {wq, wk, wv, wg};
    void *o[2] = {q, k};
    if (!make_tensor_map_bf16_3d(&maps.a, x, C, S, B, C, (uint64_t)S * C, BK, p.rows128 ? 128 : 32, 128)) return false;
    for (int i = 0; i < 4; ++i)
        if (!make_tensor_map_bf16_3d(&maps.w[i], w[i], C, C, 1, C, (uint64_t)C * C, BK, C == 64 ? 64 : 128, 128)) return false;
    // [B*H][S][D]; a 32-channel staging tile holds one head, or two of 16 channels
    for (int i = 0; i < 2; ++i) {
        p.qk[i] = (__nv_bfloat16 *)o[i];
        maps.out[i] = maps.a;
        if (D != DIRECT_D &&
            !make_tensor_map_bf16_3d(&maps.out[i], o[i], D, S, (uint64_t)B * H, D, (uint64_t)S * D, D, 32, D < 32 ? 0 : 64, 32 / D))
            return false;
    }
    if (!make_tensor_map_bf16_3d(&maps.out[2], vt, S, (uint64_t)B * C, 1, (uint64_t)vt_pitch, (uint64_t)B * C * vt_pitch, 32, 32, 64) ||
        !make_tensor_map_bf16_3d(&maps.out[3], gate, C, S, B, C, (uint64_t)S * C, 32, 32, 64))
        return false;
    p.bg = bg;
    p.gamma = ln_gamma;
    p.beta = ln_beta;
    p.eps = ln_eps;
    p.S = S;
    p.B = B;
    p.D = D;
    p.s32 = (int)s32;
    p.err = ew.device;
    if (gate_sigmoid)                    // wide layers with heads of 32
        return C == 64 ? false : C == 128 ? launch_ks<2, true>(stream, maps, p) : launch_ks<4, true>(stream, maps, p);
    return C == 64 ? launch_ks<1, false>(stream, maps, p) : C == 128 ? launch_ks<2, false>(stream, maps, p) : launch_ks<4, false>(stream, maps, p);
}

}  // namespace dev
}  // namespace kutacc
