// Projection step of the triangle multiplication in one kernel: both products, mask and gate.
//
//   gate[n, b, s] = bf16(x[b, s, :] . Wg[n, :] + bg[n])
//   proj[n, b, s] = bf16((bf16(x[b, s, :] . Wp[n, :] + bp[n]) * mask[b, s]) * sigmoid(gate[n, b, s]))
//
// (src/attention/triangle_multiplication.cpp:38-69). Persistent CTAs, two per SM; a tile is 128 positions x 128 channels
// of BOTH products, whose accumulators fill 256 columns of tensor memory, so that the epilogue has a position's
// projection and gate in the same thread and nothing is read back from memory:
//   warp 0      TMA loads of 128 x 64 slabs of x, Wp and Wg (128-byte swizzle) into a 2-stage ring
//   warp 1      one elected lane issues both products of a slab
//   warps 2-9   epilogue, 32 positions x 64 channels each. A lane is a position and the outputs are channel-major, so
//               the 32 lanes of a store write 64 contiguous bytes of one channel: coalesced whatever the strides are, which
//               a TMA store (multiples of 16 bytes) or vector stores would not take for an odd number of residues.
// Bound by HBM (x in, two outputs; 113 MB at 384 x 384 x 128). Where rows of positions follow one another without gaps the
// batch rows are one row of n_res * n_res_gather positions.
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
constexpr int NSTAGE = 2;
constexpr int SLAB_BYTES = 128 * BK * 2;
constexpr int STAGE_BYTES = 3 * SLAB_BYTES;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr int BAR_OFF = NSTAGE * STAGE_BYTES;
constexpr int SMEM_BYTES = BAR_OFF + 64 + 1024;
constexpr int TMEM_COLS = 2 * BN;               // half of the SM's tensor memory (two CTAs per SM)
constexpr float kLog2e = 1.4426950408889634f;

struct TmProjParams {
    const float *bias_p, *bias_g;
    const __nv_bfloat16 *mask;
    __nv_bfloat16 *proj, *gate;
    int64_t p_s0, p_s1, g_s0, g_s1, m_s0;
    int B, S, N, K;
    int *err;
};

__global__ void __launch_bounds__(THREADS, 2)
tm_proj_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_wp,
               const __grid_constant__ CUtensorMap tm_wg, const TmProjParams p)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar = smem + BAR_OFF;
    auto full_bar = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return bar + 8u * (uint32_t)(NSTAGE + s); };
    const uint32_t acc_full = bar + 8u * (2 * NSTAGE), acc_empty = acc_full + 8, tmem_slot = acc_full + 16;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int s_tiles = (p.S + BM - 1) / BM, n_tiles = (p.N + BN - 1) / BN;
    const int num_tiles = p.B * s_tiles * n_tiles;
    const int nk = p.K / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, EPI_WARPS);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
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
        constexpr uint32_t idesc = make_instr_desc_bf16(BM, BN);
        int it = 0, t = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++t) {
            if (t > 0 && !mbar_wait_warp(acc_empty, (uint32_t)((t - 1) & 1), p.err, 52)) break;
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
                        tc_mma_bf16(tmem_base, xd + 2 * k, xd + SLAB16 + 2 * k, idesc, acc);
                        tc_mma_bf16(tmem_base + BN, xd + 2 * k, xd + 2 * SLAB16 + 2 * k, idesc, acc);
                    }
                    tc_commit(empty_bar(s));
                    if (kc == nk - 1) tc_commit(acc_full);
                }
                __syncwarp();
            }
        }
    } else {
        const int quad = warp & 3, half = (warp - 2) >> 2;
        int t = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++t) {
            const int m_tile = tile / n_tiles, n0 = tile % n_tiles * BN + half * 64;
            const int b = m_tile / s_tiles, row = m_tile % s_tiles * BM + quad * 32 + lane;
            const bool live = row < p.S;
            const float mv = live ? __bfloat162float(p.mask[b * p.m_s0 + row]) : 0.f;
            __nv_bfloat16 *pr = p.proj + b * p.p_s1 + row, *gr = p.gate + b * p.g_s1 + row;
            if (!mbar_wait_warp(acc_full, (uint32_t)(t & 1), p.err, 54)) break;
            tc_fence_after();
            const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 64);
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                uint32_t rp[16], rg[16];
                __syncwarp();
                tmem_ld_32x16(tcol + c * 16, rp);
                tmem_ld_32x16(tcol + BN + c * 16, rg);
                tmem_ld_wait16(rp);
                tmem_ld_wait16(rg);
                if (c == 3) {
                    // everything is in registers: the next tile may overwrite the accumulators
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty);
                }
                const int n = n0 + c * 16;
                if (!live || n >= p.N) continue;
#pragma unroll
                for (int j4 = 0; j4 < 4; ++j4) {
                    const float4 bp = __ldg(reinterpret_cast<const float4 *>(p.bias_p + n) + j4);
                    const float4 bg = __ldg(reinterpret_cast<const float4 *>(p.bias_g + n) + j4);
                    const float bps[4] = {bp.x, bp.y, bp.z, bp.w}, bgs[4] = {bg.x, bg.y, bg.z, bg.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int64_t ch = n + j4 * 4 + e;
                        const float pv = round_to_bf16_f32(__uint_as_float(rp[j4 * 4 + e]) + bps[e]);
                        const __nv_bfloat16 g16 = __float2bfloat16_rn(__uint_as_float(rg[j4 * 4 + e]) + bgs[e]);
                        // (proj * mask) * sigmoid(gate), in this order (triangle_multiplication.cpp:60-64)
                        const float sg = __fdividef(1.0f, 1.0f + ex2_approx(-__bfloat162float(g16) * kLog2e));
                        gr[ch * p.g_s0] = g16;
                        pr[ch * p.p_s0] = __float2bfloat16_rn((pv * mv) * sg);
                    }
                }
            }
        }
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
    CUtensorMap tx, tp, tg;
    if (!make_tensor_map_bf16_3d(&tx, x, K, S, B, K, (uint64_t)S * K, BK, BM, 128) ||
        !make_tensor_map_bf16_3d(&tp, wp, K, N, 1, K, (uint64_t)N * K, BK, BN, 128) ||
        !make_tensor_map_bf16_3d(&tg, wg, K, N, 1, K, (uint64_t)N * K, BK, BN, 128))
        return false;
    TmProjParams p;
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
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(tm_proj_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
    const int64_t tiles = (int64_t)B * ((S + BM - 1) / BM) * (N / BN);
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, 2 * std::max(1, sm_count() - runtime().sm_margin));
    KernelTimer timer__("tm_proj", stream);
    launch_chained(tm_proj_kernel, grid, THREADS, SMEM_BYTES, stream, tx, tp, tg, p);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
