// Projection GEMMs on the fifth-generation tensor cores: tcgen05.mma with TMEM accumulators, operands
// staged in shared memory by TMA, results written back by TMA stores.
//
//   C[b, s, n] = sum_k X[b, s, k] * W[n, k] (+ bias[n])         X [B, S, K] bf16, W [N, K] bf16 (W[out][in])
//
// Persistent CTAs (two per SM) walk 128 x 128 output tiles (128 x 64 for 64 output channels). A row tile never crosses a
// batch row: every TMA box lies inside one [S, *] slab and rows past S are zero-filled on load and clipped on store; callers
// whose rows follow one another evenly pass them as one batch row, so that no tile ends early. Warp roles:
//   warp 0      producer: TMA loads of 128 x 64 slabs of X and W (128-byte swizzle) into a 2-stage ring
//   warp 1      MMA issuer: one elected lane issues tcgen05.mma (M = 128, N = 128, K = 16) four times per
//               slab into one of two 128-column TMEM accumulators and commits to mbarriers
//   warps 2-9   epilogue: each warp owns 32 TMEM lanes x 64 columns of the tile: two tcgen05.ld in flight,
//               bias add, bf16 rounding, swizzled 32 x 32 staging tiles in shared memory, TMA stores into
//               the destination layout
// The two accumulators let the epilogue of tile i overlap the MMAs of tile i+1; with K = 128 a tile is only
// eight MMAs, so what hides the rest of the per-tile chain (TMA in, tcgen05.ld, staging, TMA store) is the
// second CTA resident on the SM (99 KB of shared memory and half of the tensor memory each).
//
// It serves the output projection and the other linear layers, the products of the triangle multiplication (one right-hand
// matrix per batch), and the fused Q/K/V/gate projection of the layers that gemm_proj.cu does not take (more than 256
// channels, heads of 64): there the four weights are four tensor maps and the destination maps scatter straight into the
// attention kernel's layouts (q, k, v) and into [B, S, C] (gate, with the gate bias added).
//
// Replaces addmm -> kutacc_core_bgemm_ex of the reference
// (src/attention/gating_attention.cpp:47-66,152-157; src/linear/mm.cpp:46-86).
//
// All mbarrier waits are bounded; on a timeout the roles fall through to the common tail, the TMEM
// allocation is released and the host-visible error word carries the site.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

#include <algorithm>
#include <climits>
#include <utility>

namespace kutacc {
namespace dev {

namespace {

constexpr int BM = 128, BNMAX = 128, BK = 64;
constexpr int NSTAGE = 2;
constexpr int ACC_STAGES = 2;
constexpr int SLAB_BYTES = BM * BK * 2;                 // 16 KB, A and W slabs alike
constexpr int STAGE_BYTES = 2 * SLAB_BYTES;
constexpr int EPI_WARPS = 8;                            // two per TMEM lane quarter, 64 columns each
constexpr int STG_BYTES = 32 * 32 * 2;                  // one 32 x 32 bf16 staging tile
constexpr int STG_PER_WARP = 2;
static_assert(STG_PER_WARP == 2, "the epilogue alternates between staging tiles 0 and 1 of its warp");
constexpr int STG_OFF = NSTAGE * STAGE_BYTES;
constexpr int BAR_OFF = STG_OFF + EPI_WARPS * STG_PER_WARP * STG_BYTES;
constexpr int NBARS = 2 * NSTAGE + 2 * ACC_STAGES;
constexpr int SMEM_BYTES = BAR_OFF + NBARS * 8 + 16 + 1024;
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr int TMEM_COLS = ACC_STAGES * BNMAX;              // 256: half of the SM's tensor memory (two CTAs per SM)

struct alignas(64) GemmMaps {
    CUtensorMap a;        // X  [B][S][K], box [64, 128, 1], 128-byte swizzle
    CUtensorMap a2;       // F_TWO: X of segment 1
    CUtensorMap w[4];     // W  [1][N_seg][K], box [64, 128 (segments of 64 channels and 64-wide tiles: 64), 1], 128-byte swizzle
    CUtensorMap out[4];   // destination per segment, box [32, 32, 1], 64-byte swizzle; head sizes below 32: box [D, 32, 32 / D]
};

struct GemmParams {
    const float *bias[4];   // per segment, may be null
    int seg_n;              // output channels per segment (multiple of 128)
    int nseg;
    int head_dim;           // > 0: segment output is [B*H][S][D] (coords d, s, b*H + h); 0: [B][S][N_seg]
    int head_layout_mask;   // bit i set: segment i uses the head layout
    int transposed_mask;    // bit i set: segment i is stored transposed, [B * N_seg][S] (coords s, b * N_seg + n)
    int w_batched;          // non-zero: W is [B][N_seg][K], one matrix per batch row (coords k, n, b)
    int K;
    int S, B;
    int relu;               // non-zero: max(0, .) after the bias, before the bf16 rounding
    const float2 *ln_stats; // F_LN: (mean, rstd) of every row of X, [B * S]
    const float *ln_s[4];   // F_LN: rounding residue of the folded weight rows, per segment
    int rotate;             // non-zero: column tile of tile t is rotated by t / gridDim.x (see tile_of)
    int sigmoid_mask;       // bit i set: segment i stores bf16(sigmoid(bf16(y))) (the gate of the attention, whose
                            // reference rounds the gate to bf16 before the sigmoid: gating_attention.cpp:62-66,134-147)
    __nv_bfloat16 *direct;  // F_DIRECT: out[b * direct_b + n * direct_n + s]
    int64_t direct_b, direct_n;
    int *err;
};

// shared-memory matrix descriptor: K-major operand, rows of 128 bytes, 128-byte swizzle, 8-row groups
// 1024 bytes apart; `addr` is the byte address of the (1024-aligned) slab plus the K offset inside the
// swizzle atom
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);         // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                          // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                          // 128-byte swizzle
    return d;
}
// MN-major operand (rows of 64 elements = 128 bytes along M or N, one row per k, 128-byte swizzle): 8 k-rows are 1024 bytes
// apart, the next 64 elements of M or N follow one 64-row block (8 KB) later
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((64 * 128) >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Compile-time feature sets, so that each use of the kernel carries only the epilogue code it needs
// (the sigmoid and the transposed staging cost registers that the plain linear layer would spill).
// F_MNMAJOR: both operands are stored with their rows and columns exchanged, X [B][K][S] and W [B][K][N]: the tensor core
// reads them as they lie (MN-major operands), so a product of transposed matrices needs no transposed copies.
// F_DIRECT: out[b][n][s] element by element, s along the lanes of a warp (64 contiguous bytes per channel and store): for
// destinations whose strides no TMA store takes.
// F_NARROW: head sizes of 8 or 16.
// F_TWO: two linear layers of one shape in one launch, segment i reads its own X (the gate and output layers of the triangle
// multiplication: 384 x 384 x 128 27 us as two launches, 25 as one; 301 x 301 22 and 17, as one fills the last wave).
// F_PAIR64: segments of 64 channels, two of them in a column tile (a layer of one head of 64).
constexpr int F_SIGMOID = 1, F_TRANSPOSED = 2, F_RELU = 4, F_WBATCH = 8, F_LN = 16, F_NARROW = 32, F_MNMAJOR = 64,
              F_DIRECT = 128, F_PAIR64 = 256, F_TWO = 512;

// BN: width of a column tile, 128, or 64 for a product with 64 output channels
template <int FEAT, int BN>
__global__ void __launch_bounds__(THREADS, 2)
gemm_tcgen05_kernel(const __grid_constant__ GemmMaps maps, const GemmParams p)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem + BAR_OFF;
    auto full_bar = [&](int s) { return bar_base + 8u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (uint32_t)(NSTAGE + s); };
    auto acc_full = [&](int a) { return bar_base + 8u * (uint32_t)(2 * NSTAGE + a); };
    auto acc_empty = [&](int a) { return bar_base + 8u * (uint32_t)(2 * NSTAGE + ACC_STAGES + a); };
    const uint32_t tmem_slot = bar_base + 8u * NBARS;

    constexpr int COLS = BN / 2;                        // columns of an epilogue warp
    constexpr uint32_t instr_desc = make_instr_desc_bf16(BM, BN) | ((FEAT & F_MNMAJOR) ? (1u << 15) | (1u << 16) : 0u);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int s_tiles = (p.S + BM - 1) / BM;
    const int n_tiles_seg = (p.seg_n + BN - 1) / BN;    // a ragged last tile is zero-filled on load and clipped on store
    constexpr bool pair64 = (FEAT & F_PAIR64) != 0;
    const int n_tiles = pair64 ? p.nseg / 2 : n_tiles_seg * p.nseg;
    const int num_tiles = p.B * s_tiles * n_tiles;
    const int nk = (p.K + BK - 1) / BK;                 // columns past K are zero-filled by TMA
    // Tile t covers row tile t / n_tiles and column tile t % n_tiles. A CTA walks t = blockIdx.x + k * gridDim.x, so
    // when the grid size is a multiple of n_tiles it would meet the same column tile, i.e. the same segment, every
    // time, and the CTAs that only get the gate segment (a sigmoid per element) would finish long after the others.
    // With `rotate` the column tile is shifted by k, which is constant over the n_tiles tiles of a row tile (they
    // lie in one block of gridDim.x consecutive t), so the map stays one to one and every CTA meets every segment.
    auto tile_of = [&](int tile, int &m_tile, int &n_tile) {
        m_tile = tile / n_tiles;
        n_tile = tile % n_tiles;
        if (p.rotate) n_tile = (n_tile + tile / (int)gridDim.x) % n_tiles;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < ACC_STAGES; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), EPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0 && elect_one()) {                  // kernel parameters: may be fetched before the predecessor ends
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.w[0]);
        tma_prefetch_desc(&maps.out[0]);
    }
    release_successor();
    wait_for_predecessor();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);          // warp-uniform

    if (warp == 0) {
        // ================= producer =================
        if (elect_one()) {
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                int m_tile, n_tile;
                tile_of(tile, m_tile, n_tile);
                const int b = m_tile / s_tiles, s0 = (m_tile % s_tiles) * BM;
                const int seg = pair64 ? 2 * n_tile : n_tile / n_tiles_seg, n0 = pair64 ? 0 : (n_tile % n_tiles_seg) * BN;
                const CUtensorMap *wmap = &maps.w[seg], *amap = (FEAT & F_TWO) && seg == 1 ? &maps.a2 : &maps.a;
                for (int kc = 0; kc < nk; ++kc, ++it) {
                    const int s = it % NSTAGE;
                    if (it >= NSTAGE && !mbar_wait(empty_bar(s), (uint32_t)((it / NSTAGE - 1) & 1), p.err, 11)) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = smem + (uint32_t)s * STAGE_BYTES;
                    mbar_arrive_expect_tx(full_bar(s), SLAB_BYTES + BN * BK * 2);
                    if (FEAT & F_MNMAJOR) {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {            // 64 rows or columns per box
                            tma_load_3d(st + j * SLAB_BYTES / 2, &maps.a, full_bar(s), s0 + 64 * j, kc * BK, b);
                            tma_load_3d(st + SLAB_BYTES + j * SLAB_BYTES / 2, wmap, full_bar(s), n0 + 64 * j, kc * BK, b);
                        }
                        continue;
                    }
                    tma_load_3d(st, amap, full_bar(s), kc * BK, s0, b);
                    tma_load_3d(st + SLAB_BYTES, wmap, full_bar(s), kc * BK, n0, (FEAT & F_WBATCH) ? b : 0);
                    if (pair64) tma_load_3d(st + SLAB_BYTES + 64 * BK * 2, wmap + 1, full_bar(s), kc * BK, 0, 0);
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        int it = 0, tcount = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tcount) {
            const int a = tcount % ACC_STAGES;
            if (tcount >= ACC_STAGES && !mbar_wait_warp(acc_empty(a), (uint32_t)((tcount / ACC_STAGES - 1) & 1), p.err, 12)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(a * BNMAX);
            for (int kc = 0; kc < nk; ++kc, ++it) {
                const int s = it % NSTAGE;
                if (!mbar_wait_warp(full_bar(s), (uint32_t)((it / NSTAGE) & 1), p.err, 13)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t st = smem + (uint32_t)s * STAGE_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint64_t adesc = (FEAT & F_MNMAJOR) ? make_smem_desc_mn(st + k * 2048) : make_smem_desc(st + k * 32);
                        const uint64_t bdesc = (FEAT & F_MNMAJOR) ? make_smem_desc_mn(st + SLAB_BYTES + k * 2048)
                                                                  : make_smem_desc(st + SLAB_BYTES + k * 32);
                        tc_mma_bf16(d_tmem, adesc, bdesc, instr_desc, (kc > 0 || k > 0) ? 1u : 0u);
                    }
                    tc_commit(empty_bar(s));                 // slab may be overwritten once these MMAs retire
                    if (kc == nk - 1) tc_commit(acc_full(a));
                }
                __syncwarp();
            }
        }
    } else {
        // ================= epilogue =================
        const int quad = warp & 3;                            // TMEM lanes 32*quad .. 32*quad+31
        const int ew = warp - 2;
        const int half = ew >> 2;                             // which half of the tile's columns
        const uint32_t stg0 = smem + STG_OFF + (uint32_t)(ew * STG_PER_WARP) * STG_BYTES;
        int tcount = 0, nstore = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tcount) {
            int m_tile, n_tile;
            tile_of(tile, m_tile, n_tile);
            const int b = m_tile / s_tiles, s0 = (m_tile % s_tiles) * BM;
            const int seg = pair64 ? 2 * n_tile + half : n_tile / n_tiles_seg;
            const int n0 = pair64 ? 0 : (n_tile % n_tiles_seg) * BN + half * COLS;     // this warp's first channel of the segment
            const int a = tcount % ACC_STAGES;
            if (!mbar_wait_warp(acc_full(a), (uint32_t)((tcount / ACC_STAGES) & 1), p.err, 14)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const float *bias = p.bias[seg];
            const bool head_layout = (p.head_layout_mask >> seg) & 1;
            const bool transposed = (FEAT & F_TRANSPOSED) && ((p.transposed_mask >> seg) & 1);
            const bool sigmoid = (FEAT & F_SIGMOID) && ((p.sigmoid_mask >> seg) & 1);
            const bool relu = (FEAT & F_RELU) && p.relu;
            const CUtensorMap *omap = &maps.out[seg];
            const int row0 = s0 + quad * 32;                  // first row of this warp inside the batch row
            // LayerNorm-folded projection: y = rstd * (acc - mean * s[n]) + t[n] with this thread's row statistics
            float ln_a = 1.f, ln_b = 0.f;
            if (FEAT & F_LN) {
                const int rr = row0 + lane < p.S ? row0 + lane : p.S - 1;
                const float2 st = __ldg(p.ln_stats + (int64_t)b * p.S + rr);
                ln_a = st.y;
                ln_b = -st.y * st.x;
            }
            uint32_t r[COLS / 32][32];
            const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * BNMAX + half * COLS);
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) tmem_ld_32x32(tcol + c * 32, r[c]);
            tmem_ld_wait();
            // everything is in registers: the accumulator may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(a));
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                const int n = n0 + c * 32;
                uint32_t packed[16];
                if (bias) {
#pragma unroll
                    for (int j4 = 0; j4 < 8; ++j4) {
                        const float4 bv = __ldg(reinterpret_cast<const float4 *>(bias + n) + j4);
                        float y0, y1, y2, y3;
                        if (FEAT & F_LN) {
                            // two outputs per instruction on the packed fp32 pipe: y = ln_a * acc + (ln_b * s + t)
                            const float4 sv = __ldg(reinterpret_cast<const float4 *>(p.ln_s[seg] + n) + j4);
                            const uint64_t a2 = pack_f32x2(ln_a, ln_a), b2 = pack_f32x2(ln_b, ln_b);
                            const uint64_t w01 = fma_f32x2(pack_f32x2(sv.x, sv.y), b2, pack_f32x2(bv.x, bv.y));
                            const uint64_t w23 = fma_f32x2(pack_f32x2(sv.z, sv.w), b2, pack_f32x2(bv.z, bv.w));
                            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[c][4 * j4]), __uint_as_float(r[c][4 * j4 + 1])),
                                                   a2, w01), y0, y1);
                            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[c][4 * j4 + 2]),
                                                              __uint_as_float(r[c][4 * j4 + 3])), a2, w23), y2, y3);
                        } else {
                            y0 = __uint_as_float(r[c][4 * j4]) + bv.x;
                            y1 = __uint_as_float(r[c][4 * j4 + 1]) + bv.y;
                            y2 = __uint_as_float(r[c][4 * j4 + 2]) + bv.z;
                            y3 = __uint_as_float(r[c][4 * j4 + 3]) + bv.w;
                        }
                        if (relu) {
                            y0 = fmaxf(y0, 0.f);
                            y1 = fmaxf(y1, 0.f);
                            y2 = fmaxf(y2, 0.f);
                            y3 = fmaxf(y3, 0.f);
                        }
                        if (sigmoid) {
                            y0 = sigmoid_of_bf16(y0);
                            y1 = sigmoid_of_bf16(y1);
                            y2 = sigmoid_of_bf16(y2);
                            y3 = sigmoid_of_bf16(y3);
                        }
                        packed[2 * j4] = pack_bf16x2(y0, y1);
                        packed[2 * j4 + 1] = pack_bf16x2(y2, y3);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float y0 = __uint_as_float(r[c][2 * j]), y1 = __uint_as_float(r[c][2 * j + 1]);
                        if (relu) {
                            y0 = fmaxf(y0, 0.f);
                            y1 = fmaxf(y1, 0.f);
                        }
                        packed[j] = pack_bf16x2(y0, y1);
                    }
                }
                if (FEAT & F_DIRECT) {
                    __nv_bfloat16 *dst = p.direct + b * p.direct_b + n * p.direct_n + row0 + lane;
                    if (row0 + lane < p.S) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
#pragma unroll
                            for (int e = 0; e < 2; ++e)
                                if (n + 2 * j + e < p.seg_n)
                                    dst[(2 * j + e) * p.direct_n] =
                                        __ushort_as_bfloat16((unsigned short)(e ? packed[j] >> 16 : packed[j] & 0xffffu));
                        }
                    }
                    continue;
                }
                // staging tile: row = lane, 64 bytes per row, 16-byte chunks swizzled as the 64-byte TMA mode
                const uint32_t stg = stg0 + (uint32_t)(nstore & 1) * STG_BYTES;
                if (nstore >= STG_PER_WARP) {
                    if (lane == 0) tma_store_wait_read<STG_PER_WARP - 1>();
                    __syncwarp();
                }
                if (transposed) {
                    // transposed staging tile: row = channel d, column = this lane's sequence position
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int d = 2 * j + e;
                            const uint32_t addr = stg + (uint32_t)(d * 64 + (((lane >> 3) ^ ((d >> 1) & 3)) << 4) + (lane & 7) * 2);
                            const uint16_t hv = (uint16_t)(e ? (packed[j] >> 16) : (packed[j] & 0xffffu));
                            asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(addr), "h"(hv) : "memory");
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_3d(omap, stg, row0, b * p.seg_n + n, 0);
                        tma_store_commit();
                    }
                    ++nstore;
                    continue;
                }
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    // heads of 8 or 16 channels: [head][row][channel], no swizzle
                    const uint32_t off = !(FEAT & F_NARROW) || !head_layout ? (uint32_t)(lane * 64 + ((ch ^ ((lane >> 1) & 3)) << 4))
                                         : p.head_dim == 16 ? (uint32_t)((ch >> 1) * 1024 + lane * 32 + (ch & 1) * 16)
                                                            : (uint32_t)(ch * 512 + lane * 16);
                    const uint32_t addr = stg + off;
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(packed[4 * ch]),
                                 "r"(packed[4 * ch + 1]), "r"(packed[4 * ch + 2]), "r"(packed[4 * ch + 3])
                                 : "memory");
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (head_layout) {
                        const int hh = (b * p.seg_n + n) / p.head_dim;
                        tma_store_3d(omap, stg, b * p.seg_n + n - hh * p.head_dim, row0, hh);
                    } else {
                        tma_store_3d(omap, stg, n, row0, b);
                    }
                    tma_store_commit();
                }
                ++nstore;
            }
        }
        if (lane == 0) tma_store_wait<0>();
    }

    // ================= common tail =================
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int FEAT, int BN = 128>
bool launch(cudaStream_t stream, const GemmMaps &maps, const GemmParams &p, const char *name)
{
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<FEAT, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
    const int s_tiles = (p.S + BM - 1) / BM;
    const int n_tiles = (FEAT & F_PAIR64) ? p.nseg / 2 : ((p.seg_n + BN - 1) / BN) * p.nseg;
    const int64_t tiles = (int64_t)p.B * s_tiles * n_tiles;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, 2 * std::max(1, sm_count() - runtime().sm_margin));
    GemmParams q = p;
    q.rotate = (n_tiles > 1 && grid % (unsigned)n_tiles == 0) ? 1 : 0;
    KernelTimer timer__(name, stream);
    launch_chained(gemm_tcgen05_kernel<FEAT, BN>, grid, THREADS, SMEM_BYTES, stream, maps, q);
    count_launch();
    return true;
}

}  // namespace

bool tcgen05_proj_qkvg_bf16(cudaStream_t stream, const void *x, const void *wq, const void *wk, const void *wv,
                            const void *wg, const float *bg, void *q, void *k, void *v, void *gate, int B, int S,
                            int H, int D, bool v_transposed, int64_t v_pitch, bool gate_sigmoid, const void *ln_stats,
                            const float *const *ln_s, const float *const *ln_t)
{
    const int C = H * D;
    if ((C % 128 != 0 && C != 64) || (D != 8 && D != 16 && D != 32 && D != 64) || C > 256 * 64 || ((uintptr_t)bg & 15u)) return false;
    if (v_transposed && (v_pitch % 8 != 0 || v_pitch < S)) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    GemmMaps maps;
    const void *w[4] = {wq, wk, wv, wg};
    void *o[3] = {q, k, v};
    if (!make_tensor_map_bf16_3d(&maps.a, x, C, S, B, C, (uint64_t)S * C, BK, BM, 128)) return false;
    for (int i = 0; i < 4; ++i)
        if (!make_tensor_map_bf16_3d(&maps.w[i], w[i], C, C, 1, C, (uint64_t)C * C, BK, C == 64 ? 64 : BNMAX, 128)) return false;
    for (int i = 0; i < 3; ++i) {
        if (i == 2 && v_transposed) {
            // v^T: [B*H*D][S] with row pitch v_pitch (a multiple of 8 elements)
            if (!make_tensor_map_bf16_3d(&maps.out[i], o[i], S, (uint64_t)B * C, 1, (uint64_t)v_pitch, (uint64_t)B * C * v_pitch,
                                         32, 32, 64))
                return false;
            continue;
        }
        // [B*H][S][D]; a 32-channel staging tile holds one head, a part of one, or several of 8 or 16 channels
        const uint32_t box_d = D < 32 ? D : 32;
        if (!make_tensor_map_bf16_3d(&maps.out[i], o[i], D, S, (uint64_t)B * H, D, (uint64_t)S * D, box_d, 32, D < 32 ? 0 : 64,
                                     32 / box_d))
            return false;
    }
    if (!make_tensor_map_bf16_3d(&maps.out[3], gate, C, S, B, C, (uint64_t)S * C, 32, 32, 64)) return false;
    GemmParams p;
    p.bias[0] = p.bias[1] = p.bias[2] = nullptr;
    p.bias[3] = bg;
    p.ln_stats = (const float2 *)ln_stats;
    for (int i = 0; i < 4; ++i) {
        p.ln_s[i] = ln_stats ? ln_s[i] : nullptr;
        if (ln_stats) p.bias[i] = ln_t[i];
        if (ln_stats && ((((uintptr_t)ln_s[i] | (uintptr_t)ln_t[i]) & 15u) != 0)) return false;
    }
    p.seg_n = C;
    p.nseg = 4;
    p.head_dim = D;
    p.head_layout_mask = 0x7;
    p.transposed_mask = v_transposed ? 0x4 : 0;
    p.w_batched = 0;
    p.K = C;
    p.S = S;
    p.B = B;
    p.relu = 0;
    p.sigmoid_mask = gate_sigmoid ? 0x8 : 0;
    p.err = ew.device;
    // the combinations that callers use: k, v and the sigmoid of the gate for the attention core on tensor memory, with heads of 32
    // (with LayerNorm or without), the plain gate with narrower heads; everything as it is for the other core, with heads of 32 or 64
    if (gate_sigmoid != (v_transposed && D == 32) || (ln_stats && !gate_sigmoid)) return false;
    if (v_transposed) {
        if (C == 64 || D == 64) return false;                  // gemm_proj.cu; no such core
        if (D < 32) return launch<F_TRANSPOSED | F_NARROW>(stream, maps, p, "proj_qkvg");
        return ln_stats ? launch<F_TRANSPOSED | F_SIGMOID | F_LN>(stream, maps, p, "proj_qkvg_ln")
                        : launch<F_TRANSPOSED | F_SIGMOID>(stream, maps, p, "proj_qkvg");
    }
    if (D < 32) return false;
    return C == 64 ? launch<F_PAIR64>(stream, maps, p, "proj_qkvg") : launch<0>(stream, maps, p, "proj_qkvg");
}

bool tcgen05_linear_bias_bf16(cudaStream_t stream, const void *a, const void *w, const float *bias, void *out,
                              int64_t out_row_stride, int B, int S, int N, int K, bool relu, int64_t a_row_stride)
{
    if (a_row_stride <= 0) a_row_stride = K;
    // the rows of all batch rows lie evenly: one long batch row, no tile ends early
    if ((int64_t)B * S <= INT32_MAX / 2) {
        S *= B;
        B = 1;
    }
    if ((N % 128 != 0 && (N != 64 || relu)) || K % 64 != 0 || out_row_stride % 8 != 0 || a_row_stride % 8 != 0 || a_row_stride < K ||
        ((uintptr_t)out & 15u) || ((uintptr_t)a & 15u) || ((uintptr_t)w & 15u) || ((uintptr_t)bias & 15u))
        return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    // Few tiles: columns in halves, so that twice as many SMs share the epilogue, which is on the path of a small call. 4 rows x 192
    // positions x 128 channels, the whole attention call: 20.6 -> 20.3 us. Where halves would need a second wave, tiles of 128. So also for a result that lies
    // over its own rows: with 128 channels a tile has read its rows before it writes them, halves would not wait for each other.
    const int64_t rows = (int64_t)B * S;
    const bool narrow = !relu && (int64_t)B * ((S + BM - 1) / BM) * (N / BNMAX) * 2 <= sm_count() &&
                        apart(a, (size_t)((rows - 1) * a_row_stride + K) * 2, out, (size_t)((rows - 1) * out_row_stride + N) * 2);
    GemmMaps maps;
    if (!make_tensor_map_bf16_3d(&maps.a, a, K, S, B, (uint64_t)a_row_stride, (uint64_t)S * a_row_stride, BK, BM, 128))
        return false;
    if (!make_tensor_map_bf16_3d(&maps.w[0], w, K, N, 1, K, (uint64_t)N * K, BK, N == 64 || narrow ? 64 : BNMAX, 128)) return false;
    if (!make_tensor_map_bf16_3d(&maps.out[0], out, N, S, B, (uint64_t)out_row_stride, (uint64_t)S * out_row_stride, 32,
                                 32, 64))
        return false;
    for (int i = 1; i < 4; ++i) {
        maps.w[i] = maps.w[0];
        maps.out[i] = maps.out[0];
    }
    GemmParams p;
    p.bias[0] = bias;
    p.bias[1] = p.bias[2] = p.bias[3] = nullptr;
    p.seg_n = N;
    p.nseg = 1;
    p.head_dim = 0;
    p.head_layout_mask = 0;
    p.transposed_mask = 0;
    p.w_batched = 0;
    p.K = K;
    p.S = S;
    p.B = B;
    p.relu = relu ? 1 : 0;
    p.ln_stats = nullptr;
    p.ln_s[0] = p.ln_s[1] = p.ln_s[2] = p.ln_s[3] = nullptr;
    p.sigmoid_mask = 0;
    p.err = ew.device;
    if (N == 64 || narrow) return launch<0, 64>(stream, maps, p, "linear_bias");
    return relu ? launch<F_RELU>(stream, maps, p, "linear_bias_relu") : launch<0>(stream, maps, p, "linear_bias");
}

// Two linear layers of one shape in one launch: out_i = a_i . w_i^T + bias_i
bool tcgen05_linear_pair_bf16(cudaStream_t stream, const LinearOperands (&l)[2], int64_t rows, int N, int K)
{
    if (N % 128 != 0 || K % 64 != 0 || rows > INT32_MAX / 2) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    GemmMaps maps;
    GemmParams p = {};
    for (int i = 0; i < 2; ++i) {
        if (l[i].out_row_stride % 8 != 0 || l[i].a_row_stride % 8 != 0 || l[i].a_row_stride < K ||
            ((((uintptr_t)l[i].out | (uintptr_t)l[i].a | (uintptr_t)l[i].w | (uintptr_t)l[i].bias) & 15u) != 0))
            return false;
        if (!make_tensor_map_bf16_3d(i ? &maps.a2 : &maps.a, l[i].a, K, rows, 1, (uint64_t)l[i].a_row_stride, (uint64_t)rows * l[i].a_row_stride,
                                     BK, BM, 128) ||
            !make_tensor_map_bf16_3d(&maps.w[i], l[i].w, K, N, 1, K, (uint64_t)N * K, BK, BNMAX, 128) ||
            !make_tensor_map_bf16_3d(&maps.out[i], l[i].out, N, rows, 1, (uint64_t)l[i].out_row_stride, (uint64_t)rows * l[i].out_row_stride, 32, 32,
                                     64))
            return false;
        p.bias[i] = l[i].bias;
    }
    for (int i = 2; i < 4; ++i) {
        maps.w[i] = maps.w[0];
        maps.out[i] = maps.out[0];
    }
    p.seg_n = N;
    p.nseg = 2;
    p.K = K;
    p.S = (int)rows;
    p.B = 1;
    p.err = ew.device;
    return launch<F_TWO>(stream, maps, p, "linear_pair");
}

// Batched product with one right-hand matrix per batch: out[b, m, n] = sum_k a[b, m, k] * w[b, n, k], or with
// `transposed` sum_k a[b, k, m] * w[b, k, n] (a, w, out with row and batch strides in elements). The per-channel products
// of the triangle multiplication (src/attention/triangle_multiplication.cpp:75-104). An output that no TMA store takes
// (strides that are not multiples of 8 elements, n not of 8) is computed as its transpose, so that a warp's lanes run along
// the contiguous index, and stored directly.
bool tcgen05_batched_bf16(cudaStream_t stream, bool transposed, const void *a, int64_t a_row_stride, int64_t a_batch_stride,
                          const void *w, int64_t w_row_stride, int64_t w_batch_stride, void *out, int64_t out_row_stride,
                          int64_t out_batch_stride, int B, int M, int N, int K)
{
    if ((a_row_stride | a_batch_stride | w_row_stride | w_batch_stride) % 8 != 0 || a_row_stride < (transposed ? M : K) ||
        w_row_stride < (transposed ? N : K) || out_row_stride < N || ((((uintptr_t)a | (uintptr_t)w) & 15u) != 0))
        return false;
    const bool direct = (out_row_stride | out_batch_stride) % 8 != 0 || ((uintptr_t)out & 15u) != 0;
    if (direct) {
        std::swap(a, w);
        std::swap(a_row_stride, w_row_stride);
        std::swap(a_batch_stride, w_batch_stride);
        std::swap(M, N);
    }
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    GemmMaps maps;
    if (transposed) {
        if (!make_tensor_map_bf16_3d(&maps.a, a, M, K, B, (uint64_t)a_row_stride, (uint64_t)a_batch_stride, 64, BK, 128) ||
            !make_tensor_map_bf16_3d(&maps.w[0], w, N, K, B, (uint64_t)w_row_stride, (uint64_t)w_batch_stride, 64, BK, 128))
            return false;
    } else {
        if (!make_tensor_map_bf16_3d(&maps.a, a, K, M, B, (uint64_t)a_row_stride, (uint64_t)a_batch_stride, BK, BM, 128) ||
            !make_tensor_map_bf16_3d(&maps.w[0], w, K, N, B, (uint64_t)w_row_stride, (uint64_t)w_batch_stride, BK, BNMAX, 128))
            return false;
    }
    if (!direct) {
        if (!make_tensor_map_bf16_3d(&maps.out[0], out, N, M, B, (uint64_t)out_row_stride, (uint64_t)out_batch_stride, 32, 32, 64))
            return false;
    } else {
        maps.out[0] = maps.a;
    }
    for (int i = 1; i < 4; ++i) {
        maps.w[i] = maps.w[0];
        maps.out[i] = maps.out[0];
    }
    GemmParams p;
    p.bias[0] = p.bias[1] = p.bias[2] = p.bias[3] = nullptr;
    p.seg_n = N;
    p.nseg = 1;
    p.head_dim = 0;
    p.head_layout_mask = 0;
    p.transposed_mask = 0;
    p.w_batched = 1;
    p.K = K;
    p.S = M;
    p.B = B;
    p.relu = 0;
    p.ln_stats = nullptr;
    p.ln_s[0] = p.ln_s[1] = p.ln_s[2] = p.ln_s[3] = nullptr;
    p.sigmoid_mask = 0;
    p.direct = (__nv_bfloat16 *)out;
    p.direct_b = out_batch_stride;
    p.direct_n = out_row_stride;
    p.err = ew.device;
    if (direct)
        return transposed ? launch<F_WBATCH | F_MNMAJOR | F_DIRECT>(stream, maps, p, "tm_equation")
                          : launch<F_WBATCH | F_DIRECT>(stream, maps, p, "tm_equation");
    return transposed ? launch<F_WBATCH | F_MNMAJOR>(stream, maps, p, "tm_equation")
                      : launch<F_WBATCH>(stream, maps, p, "tm_equation");
}

}  // namespace dev
}  // namespace kutacc
