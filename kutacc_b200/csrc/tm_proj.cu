// Projection step of the triangle multiplication in one kernel: both products, mask and gate.
//
//   gate[n, b, s] = bf16(x[b, s, :] . Wg[n, :] + bg[n])
//   proj[n, b, s] = bf16((bf16(x[b, s, :] . Wp[n, :] + bp[n]) * mask[b, s]) * sigmoid(gate[n, b, s]))
//
// (src/attention/triangle_multiplication.cpp:38-69). Persistent CTAs, one per SM; a tile is 128 positions x 128 channels of
// BOTH products, so that the epilogue has a position's projection and gate in the same thread and nothing is read back from
// memory:
//   warp 0      TMA loads of 128 x 64 slabs of x, Wp and Wg (128-byte swizzle) into a 3-stage ring
//   warp 1      one elected lane issues both products of a slab; two pairs of accumulators fill the tensor memory
//   warps 4-19  epilogue, 32 channels x 32 positions each, two elements at a time through the packed fp32 operations
// The outputs are channel-major. Where TMA takes their strides the products are transposed (a lane of the accumulators is a
// channel): the bias is a register, a lane's positions lie side by side, and the results leave through a staging tile by TMA.
// For other strides (an odd number of residues) a lane is a position, and the 32 lanes of a 2-byte store write 64 contiguous
// bytes of a channel; storing words of two positions from staging tiles was slower (301 x 301 x 128: 30 to 34 us against 20 to 25).
// Bound by HBM (x in, two outputs; 113 MB at 384 x 384 x 128, 17 us) and by the instructions of the epilogue: with one element
// and one position per lane at a time it took 35 per element and the kernel 34.5 us; now 26. Where rows of positions follow
// one another without gaps the batch rows are one row of n_res * n_res_gather positions. The clocks of a CTA showed 2000 of a
// tile's 3700 between two tiles' arithmetic: mask and biases on their way from memory and the wait for the staging tiles, both now
// out of that path (384 x 384 x 128: 25 -> 22 us).
//
// All mbarrier waits are bounded; on a timeout the roles fall through to the common tail, the TMEM allocation is released
// and the host-visible error word carries the site.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

#include <algorithm>

namespace kutacc {
namespace dev {

namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int NSTAGE = 3;
constexpr int SLAB_BYTES = 128 * BK * 2;
constexpr int STAGE_BYTES = 3 * SLAB_BYTES;
constexpr int EPI_WARPS = 16, EPI_WARP0 = 4;
constexpr int THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
constexpr int TILE_BYTES = 32 * 32 * 2;                        // staging tile of a warp, one per output
constexpr int STG_OFF = NSTAGE * STAGE_BYTES;
constexpr int MASK_OFF = STG_OFF + EPI_WARPS * 2 * TILE_BYTES;
constexpr int BAR_OFF = MASK_OFF + EPI_WARPS * 32 * 4;
constexpr int SMEM_BYTES = BAR_OFF + 128 + 1024;
constexpr int TMEM_COLS = 4 * BM;               // two pairs of accumulators of 128 channels x 128 positions
constexpr float kLog2e = 1.4426950408889634f;

struct TmProjParams {
    const float *bias_p, *bias_g;
    const __nv_bfloat16 *mask;
    __nv_bfloat16 *proj, *gate;
    int64_t p_s0, p_s1, g_s0, g_s1, m_s0;
    int B, S, N, K;
    int *err;
};

// Two elements of the result from their rounded projections, gates and mask values:
// (proj * mask) * sigmoid(gate), in this order (triangle_multiplication.cpp:60-64)
__device__ __forceinline__ void gated(uint32_t p16, uint32_t g16, uint64_t mask2, float &y0, float &y1)
{
    float e0, e1;
    unpack_f32x2(mul_f32x2(pack_f32x2(bf16lo_to_f32(g16), bf16hi_to_f32(g16)), pack_f32x2(-kLog2e, -kLog2e)), e0, e1);
    unpack_f32x2(add_f32x2(pack_f32x2(ex2_approx(e0), ex2_approx(e1)), pack_f32x2(1.f, 1.f)), e0, e1);
    const uint64_t pm = mul_f32x2(pack_f32x2(bf16lo_to_f32(p16), bf16hi_to_f32(p16)), mask2);
    unpack_f32x2(mul_f32x2(pm, pack_f32x2(__fdividef(1.f, e0), __fdividef(1.f, e1))), y0, y1);
}

// bf16 pair of two accumulators plus their biases
__device__ __forceinline__ uint32_t biased(uint32_t a0, uint32_t a1, uint64_t bias2)
{
    float y0, y1;
    unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(a0), __uint_as_float(a1)), bias2), y0, y1);
    return pack_bf16x2(y0, y1);
}

// TMA_OUT: the strides of both outputs are multiples of 16 bytes
template <bool TMA_OUT>
__global__ void __launch_bounds__(THREADS, 1)
tm_proj_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_wp,
               const __grid_constant__ CUtensorMap tm_wg, const __grid_constant__ CUtensorMap tm_proj,
               const __grid_constant__ CUtensorMap tm_gate, const __grid_constant__ TmProjParams p)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar = smem + BAR_OFF;
    auto full_bar = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return bar + 8u * (uint32_t)(NSTAGE + s); };
    auto acc_full = [&](int i) { return bar + 8u * (uint32_t)(2 * NSTAGE + i); };
    auto acc_empty = [&](int i) { return bar + 8u * (uint32_t)(2 * NSTAGE + 2 + i); };
    const uint32_t tmem_slot = bar + 8u * (2 * NSTAGE + 4);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int s_tiles = (p.S + BM - 1) / BM, n_tiles = (p.N + BN - 1) / BN;
    const int num_tiles = p.B * s_tiles * n_tiles;
    const int nk = p.K / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full(i), 1);
            mbar_init(acc_empty(i), EPI_WARPS);
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
        tma_prefetch_desc(&tm_x);
        tma_prefetch_desc(&tm_wp);
        tma_prefetch_desc(&tm_wg);
    }
    release_successor();
    wait_for_predecessor();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0) {
        if (elect_one()) {
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                const int m_tile = tile / n_tiles, n0 = tile % n_tiles * BN;
                const int b = m_tile / s_tiles, s0 = m_tile % s_tiles * BM;
                for (int kc = 0; kc < nk; ++kc, ++it) {
                    const int s = it % NSTAGE;
                    if (it >= NSTAGE && !mbar_wait(empty_bar(s), (uint32_t)((it / NSTAGE - 1) & 1), p.err, 51)) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = smem + (uint32_t)s * STAGE_BYTES;
                    mbar_arrive_expect_tx(full_bar(s), STAGE_BYTES);
                    tma_load_3d(st, &tm_x, full_bar(s), kc * BK, s0, b);
                    tma_load_3d(st + SLAB_BYTES, &tm_wp, full_bar(s), kc * BK, n0, 0);
                    tma_load_3d(st + 2 * SLAB_BYTES, &tm_wg, full_bar(s), kc * BK, n0, 0);
                }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_instr_desc_bf16(128, 128);
        int it = 0, t = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++t) {
            if (t >= 2 && !mbar_wait_warp(acc_empty(t & 1), (uint32_t)((t / 2 - 1) & 1), p.err, 52)) break;
            const uint32_t d = tmem_base + (uint32_t)((t & 1) * 2 * BM);
            for (int kc = 0; kc < nk; ++kc, ++it) {
                const int s = it % NSTAGE;
                if (!mbar_wait_warp(full_bar(s), (uint32_t)((it / NSTAGE) & 1), p.err, 53)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t xd = make_smem_desc_kmajor(smem + (uint32_t)s * STAGE_BYTES, 128);
                    constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;        // descriptor addresses count in units of 16 bytes
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint32_t acc = (kc > 0 || k > 0) ? 1u : 0u;
                        const uint64_t x = xd + 2 * k, wp = x + SLAB16, wg = x + 2 * SLAB16;
                        tc_mma_bf16(d, TMA_OUT ? wp : x, TMA_OUT ? x : wp, idesc, acc);
                        tc_mma_bf16(d + BM, TMA_OUT ? wg : x, TMA_OUT ? x : wg, idesc, acc);
                    }
                    tc_commit(empty_bar(s));
                    if (kc == nk - 1) tc_commit(acc_full(t & 1));
                }
                __syncwarp();
            }
        }
    } else if (warp >= EPI_WARP0) {
        // 32 rows (quad) x 32 columns (grp) of both accumulators
        const int ew = warp - EPI_WARP0, quad = warp & 3, grp = ew >> 2;
        const uint32_t stg = smem + STG_OFF + (uint32_t)(ew * 2 * TILE_BYTES), mk = smem + MASK_OFF + (uint32_t)(ew * 128);
        int t = 0, b, row0, row, n;
        // where this warp's part of a tile lies, and its mask value and biases, which are loaded a tile ahead: their way from memory
        // (and the wait for the staging tiles, which comes as late as it can) was half of a tile's time
        auto place = [&](int tile) {
            const int m_tile = tile / n_tiles;
            n = tile % n_tiles * BN + (TMA_OUT ? quad : grp) * 32;
            b = m_tile / s_tiles;
            row0 = m_tile % s_tiles * BM + (TMA_OUT ? grp : quad) * 32;
            row = row0 + lane;
        };
        __nv_bfloat16 mask_next = __float2bfloat16(0.f);
        float bp = 0.f, bg = 0.f, bp_next = 0.f, bg_next = 0.f;
        auto load_next = [&](int tile) {
            if (tile >= num_tiles) return;
            place(tile);
            mask_next = row < p.S ? p.mask[b * p.m_s0 + row] : __float2bfloat16(0.f);
            if (TMA_OUT) {
                bp_next = __ldg(p.bias_p + n + lane);
                bg_next = __ldg(p.bias_g + n + lane);
            }
        };
        load_next(blockIdx.x);
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++t) {
            const float mv = __bfloat162float(mask_next);
            bp = bp_next;
            bg = bg_next;
            load_next(tile + gridDim.x);
            place(tile);
            const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)((t & 1) * 2 * BM + grp * 32);
            if (TMA_OUT) {
                asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(mk + lane * 4), "f"(mv) : "memory");
                __syncwarp();
            }
            if (!mbar_wait_warp(acc_full(t & 1), (uint32_t)((t / 2) & 1), p.err, 54)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t rp[16], rg[16];
                __syncwarp();
                tmem_ld_32x16(tcol + c * 16, rp);
                tmem_ld_32x16(tcol + BM + c * 16, rg);
                tmem_ld_wait16(rp);
                tmem_ld_wait16(rg);
                if (c == 1) {
                    // everything is in registers: the accumulators may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty(t & 1));
                }
                if (TMA_OUT) {
                    uint32_t op[8], og[8];
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const float4 m4 = lds128_f32(mk + (uint32_t)((c * 16 + j) * 4));
#pragma unroll
                        for (int h = 0; h < 4; h += 2) {
                            float y0, y1;
                            const uint32_t p16 = biased(rp[j + h], rp[j + h + 1], pack_f32x2(bp, bp));
                            const uint32_t g16 = biased(rg[j + h], rg[j + h + 1], pack_f32x2(bg, bg));
                            gated(p16, g16, h == 0 ? pack_f32x2(m4.x, m4.y) : pack_f32x2(m4.z, m4.w), y0, y1);
                            op[(j + h) >> 1] = pack_bf16x2(y0, y1);
                            og[(j + h) >> 1] = g16;
                        }
                    }
                    if (c == 0) {                                  // the staging tiles may be rewritten
                        if (lane == 0) tma_store_wait_read<0>();
                        __syncwarp();
                    }
                    // staging tile: a row of 64 bytes per channel, 64-byte swizzle
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const uint32_t at = stg + (uint32_t)(lane * 64) + ((uint32_t)((c * 2 + v) ^ ((lane >> 1) & 3)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(at), "r"(op[4 * v]), "r"(op[4 * v + 1]),
                                     "r"(op[4 * v + 2]), "r"(op[4 * v + 3])
                                     : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(at + TILE_BYTES), "r"(og[4 * v]),
                                     "r"(og[4 * v + 1]), "r"(og[4 * v + 2]), "r"(og[4 * v + 3])
                                     : "memory");
                    }
                } else if (row < p.S) {
                    uint16_t *po = reinterpret_cast<uint16_t *>(p.proj + b * p.p_s1 + (n + c * 16) * p.p_s0 + row);
                    uint16_t *go = reinterpret_cast<uint16_t *>(p.gate + b * p.g_s1 + (n + c * 16) * p.g_s0 + row);
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const float4 bp4 = __ldg(reinterpret_cast<const float4 *>(p.bias_p + n + c * 16 + j));
                        const float4 bg4 = __ldg(reinterpret_cast<const float4 *>(p.bias_g + n + c * 16 + j));
#pragma unroll
                        for (int h = 0; h < 4; h += 2) {
                            float y0, y1;
                            const uint32_t p16 = biased(rp[j + h], rp[j + h + 1], h == 0 ? pack_f32x2(bp4.x, bp4.y) : pack_f32x2(bp4.z, bp4.w));
                            const uint32_t g16 = biased(rg[j + h], rg[j + h + 1], h == 0 ? pack_f32x2(bg4.x, bg4.y) : pack_f32x2(bg4.z, bg4.w));
                            gated(p16, g16, pack_f32x2(mv, mv), y0, y1);
                            const uint32_t y16 = pack_bf16x2(y0, y1);
                            po[0] = (uint16_t)y16;
                            go[0] = (uint16_t)g16;
                            po[p.p_s0] = (uint16_t)(y16 >> 16);
                            go[p.g_s0] = (uint16_t)(g16 >> 16);
                            po += 2 * p.p_s0;
                            go += 2 * p.g_s0;
                        }
                    }
                }
            }
            if (TMA_OUT) {
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    tma_store_3d(&tm_proj, stg, row0, n, b);
                    tma_store_3d(&tm_gate, stg + TILE_BYTES, row0, n, b);
                    tma_store_commit();
                }
            }
        }
        if (TMA_OUT && lane == 0) tma_store_wait<0>();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace

bool tcgen05_tm_proj_bf16(cudaStream_t stream, const void *x, const void *wp, const float *bp, const void *wg, const float *bg,
                          const void *mask, int64_t m_s0, void *proj, int64_t p_s0, int64_t p_s1, void *gate, int64_t g_s0,
                          int64_t g_s1, int B, int S, int N, int K)
{
    if (N % 128 != 0 || K % 64 != 0 ||
        ((((uintptr_t)x | (uintptr_t)wp | (uintptr_t)wg | (uintptr_t)bp | (uintptr_t)bg) & 15u) != 0))
        return false;
    if (p_s1 == S && g_s1 == S && m_s0 == S && (int64_t)B * S <= INT32_MAX / 2) {
        S *= B;
        B = 1;
    }
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    CUtensorMap tx, tp, tg, op = {}, og = {};
    if (!make_tensor_map_bf16_3d(&tx, x, K, S, B, K, (uint64_t)S * K, BK, BM, 128) ||
        !make_tensor_map_bf16_3d(&tp, wp, K, N, 1, K, (uint64_t)N * K, BK, BN, 128) ||
        !make_tensor_map_bf16_3d(&tg, wg, K, N, 1, K, (uint64_t)N * K, BK, BN, 128))
        return false;
    TmProjParams p = {};
    p.bias_p = bp;
    p.bias_g = bg;
    p.mask = (const __nv_bfloat16 *)mask;
    p.proj = (__nv_bfloat16 *)proj;
    p.gate = (__nv_bfloat16 *)gate;
    p.p_s0 = p_s0;
    p.p_s1 = p_s1;
    p.g_s0 = g_s0;
    p.g_s1 = g_s1;
    p.m_s0 = m_s0;
    p.B = B;
    p.S = S;
    p.N = N;
    p.K = K;
    p.err = ew.device;
    // batch rows of one: any stride that TMA takes
    const int64_t pb = B == 1 ? (int64_t)N * p_s0 : p_s1, gb = B == 1 ? (int64_t)N * g_s0 : g_s1;
    const bool tma_out = (p_s0 | g_s0 | pb | gb) % 8 == 0 && (((uintptr_t)proj | (uintptr_t)gate) & 15u) == 0 &&
                         make_tensor_map_bf16_3d(&op, proj, S, N, B, p_s0, pb, 32, 32, 64) &&
                         make_tensor_map_bf16_3d(&og, gate, S, N, B, g_s0, gb, 32, 32, 64);
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(tm_proj_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        KUTACC_CUDA(cudaFuncSetAttribute(tm_proj_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
    const int64_t tiles = (int64_t)B * ((S + BM - 1) / BM) * (N / BN);
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, std::max(1, sm_count() - runtime().sm_margin));
    KernelTimer timer__("tm_proj", stream);
    launch_chained(tma_out ? tm_proj_kernel<true> : tm_proj_kernel<false>, grid, THREADS, SMEM_BYTES, stream, tx, tp, tg, op, og, p);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
