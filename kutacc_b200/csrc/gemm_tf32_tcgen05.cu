// fp32 projections on the fifth-generation tensor cores with fp32-level accuracy.
//
//   C[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n])         A [M, K] fp32, W [N, K] fp32 (W[out][in]), C fp32
//
// tcgen05.mma has no fp32 input type; its tf32 kind keeps 11 significant bits of each operand. Every operand is
// therefore split beforehand (split_tf32_kernel) into a tf32 head and a tail, x = hi + lo with |lo| <= 2^-11 |x|,
// stored side by side as one row [hi(0..K) | lo(0..K)] of 2K floats, and the product is taken as
//   lo(A).hi(W) + hi(A).lo(W) + hi(A).hi(W)        (lo.lo, about 2^-22 of the result, is dropped)
// accumulated in fp32 in tensor memory, the small products in an accumulator of their own that the epilogue adds: the tensor
// core truncates at every accumulation, and with all three products in one accumulator there are three times as many of them
// at full magnitude (2-norm error at K = 256: 1.7e-6, this way 6.4e-7). Persistent CTAs, one per SM, walk 128 x 256 output tiles (128 x 128 where there are too
// few of the wide ones to go round or the columns do not divide):
//   warp 0      producer: per 32-column slab of K one stage with the heads AND tails of A' and W' (TMA, 128-byte swizzle), so
//               that the three products read each slab from L2 once
//   warp 1      MMA issuer: one elected lane issues the 12 tcgen05.mma kind::tf32 (K = 8) of a stage into a pair of TMEM
//               accumulators (two pairs of 128 columns each, or one of 256) and commits to mbarriers
//   warps 2-9   epilogue: each warp owns 32 TMEM lanes x half of the columns: tcgen05.ld of both accumulators into
//               registers, which frees them, then bias add, staging tile (32 x 32), TMA store
// Up to four weight matrices share one pass over A (the fused Q/K/V/gate projection of the fp32 attention).
// What bounds it: the way of the operands from L2. Loading the slab pair of each product by itself with 128 x 128 tiles
// moves 1.6 GB for 32768 x 1024 x 256 (10 TB/s at its 160 us); sharing the slabs halves that.
//
// Replaces addmm -> kutacc_core_bgemm_ex of the reference for fp32 tensors
// (src/attention/gating_attention.cpp:47-66,152-157; src/linear/mm.cpp:46-86).
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

constexpr int BM = 128, BK = 32;                        // BK floats = one 128-byte swizzle row
constexpr int SLAB_BYTES = 128 * BK * 4;                // 16 KB: 128 rows of A', or of W'
constexpr int EPI_WARPS = 8;
constexpr int STG_BYTES = 32 * 32 * 4;                  // one staging tile per epilogue warp
constexpr int THREADS = 32 * (2 + EPI_WARPS);

template <int BN>
struct Geo {
    static constexpr int NB = BN / 128;                              // 128-column blocks of a tile
    static constexpr int STAGE_BYTES = 2 * (1 + NB) * SLAB_BYTES;    // heads and tails of A' and W'
    static constexpr int NSTAGE = BN == 256 ? 2 : 3;
    static constexpr int ACC_STAGES = 256 / BN;                      // pairs of accumulators (hi.hi; the two small products)
    static constexpr int STG_OFF = NSTAGE * STAGE_BYTES;
    static constexpr int BAR_OFF = STG_OFF + EPI_WARPS * STG_BYTES;
    static constexpr int NBARS = 2 * NSTAGE + 2 * ACC_STAGES;
    static constexpr int SMEM_BYTES = BAR_OFF + NBARS * 8 + 16 + 1024;
    static constexpr int TMEM_COLS = ACC_STAGES * 2 * BN;
    static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
};

struct alignas(64) Tf32Maps {
    CUtensorMap a;        // A' [M][2K] fp32, box [32, 128], 128-byte swizzle
    CUtensorMap w[4];     // W' [N][2K] fp32 per segment, box [32, 128], 128-byte swizzle
    CUtensorMap out[4];   // per segment [M][N] (split rows: [M][2N]), box [32, 32], 128-byte swizzle
};

struct Tf32Params {
    const float *bias[4];   // per segment, may be null
    float *out_t[4];        // kTf32SplitTransposed segments: [B][N/32][64][S]
    int layout[4];          // per segment: Tf32Layout
    int M, N, K, nseg;
    int S;                  // rows per batch row (transposed segments)
    int64_t vt_pitch;
    int *err;
};

__device__ __forceinline__ void tc_mma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tf32x3_tc_kernel(const __grid_constant__ Tf32Maps maps, const __grid_constant__ Tf32Params p)
{
    using T = Geo<BN>;
    constexpr int NSTAGE = T::NSTAGE, ACC_STAGES = T::ACC_STAGES;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem + T::BAR_OFF;
    auto full_bar = [&](int s) { return bar_base + 8u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (uint32_t)(NSTAGE + s); };
    auto acc_full = [&](int a) { return bar_base + 8u * (uint32_t)(2 * NSTAGE + a); };
    auto acc_empty = [&](int a) { return bar_base + 8u * (uint32_t)(2 * NSTAGE + ACC_STAGES + a); };
    const uint32_t tmem_slot = bar_base + 8u * T::NBARS;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int m_tiles = (p.M + BM - 1) / BM;
    const int n_tiles = p.N * p.nseg / BN;
    const int num_tiles = m_tiles * n_tiles;
    const int nk = p.K / BK;

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
        tmem_alloc(tmem_slot, T::TMEM_COLS);
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
        // ================= producer =================
        if (elect_one()) {
            tma_prefetch_desc(&maps.a);
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                const int m0 = (tile / n_tiles) * BM, c0 = tile % n_tiles * BN;
                for (int kc = 0; kc < nk; ++kc, ++it) {
                    const int s = it % NSTAGE;
                    if (it >= NSTAGE && !mbar_wait(empty_bar(s), (uint32_t)((it / NSTAGE - 1) & 1), p.err, 41)) {
                        ok = false;
                        break;
                    }
                    // [A head | A tail | W heads | W tails]
                    const uint32_t st = smem + (uint32_t)s * T::STAGE_BYTES;
                    mbar_arrive_expect_tx(full_bar(s), T::STAGE_BYTES);
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const int col = t * p.K + kc * BK;
                        tma_load_2d(st + t * SLAB_BYTES, &maps.a, full_bar(s), col, m0);
#pragma unroll
                        for (int j = 0; j < T::NB; ++j) {
                            const int c = c0 + j * 128;
                            tma_load_2d(st + (2 + t * T::NB + j) * SLAB_BYTES, &maps.w[c / p.N], full_bar(s), col, c % p.N);
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc = make_instr_desc_tf32(BM, BN);
        constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;        // descriptor addresses count in units of 16 bytes
        int it = 0, tcount = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tcount) {
            const int a = tcount % ACC_STAGES;
            if (tcount >= ACC_STAGES && !mbar_wait_warp(acc_empty(a), (uint32_t)((tcount / ACC_STAGES - 1) & 1), p.err, 42)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(a * 2 * BN);
            for (int kc = 0; kc < nk; ++kc, ++it) {
                const int s = it % NSTAGE;
                if (!mbar_wait_warp(full_bar(s), (uint32_t)((it / NSTAGE) & 1), p.err, 43)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t ad = make_smem_desc_kmajor(smem + (uint32_t)s * T::STAGE_BYTES, 128), wd = ad + 2 * SLAB16;
#pragma unroll
                    for (int pr = 0; pr < 3; ++pr)                   // tail.head, head.tail, head.head
#pragma unroll
                        for (int k = 0; k < BK / 8; ++k)             // 8 tf32 = 32 bytes per instruction
                            tc_mma_tf32(d_tmem + (pr < 2 ? BN : 0), ad + (pr == 0 ? SLAB16 : 0u) + 2 * k,
                                        wd + (pr == 1 ? T::NB * SLAB16 : 0u) + 2 * k, idesc, (kc > 0 || pr == 1 || k > 0) ? 1u : 0u);
                    tc_commit(empty_bar(s));                 // the stage may be overwritten once these MMAs retire
                    if (kc == nk - 1) tc_commit(acc_full(a));
                }
                __syncwarp();
            }
        }
    } else {
        // ================= epilogue =================
        constexpr int COLS = BN / 2;
        const int quad = warp & 3;                            // TMEM lanes 32*quad .. 32*quad+31
        const int ew = warp - 2, half = ew >> 2;              // which half of the tile's columns
        const uint32_t stg = smem + T::STG_OFF + (uint32_t)ew * STG_BYTES;
        int tcount = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++tcount) {
            const int m0 = (tile / n_tiles) * BM + quad * 32, c0 = tile % n_tiles * BN + half * COLS;
            const int seg = c0 / p.N, n0 = c0 % p.N;
            const int a = tcount % ACC_STAGES;
            if (!mbar_wait_warp(acc_full(a), (uint32_t)((tcount / ACC_STAGES) & 1), p.err, 44)) break;
            tc_fence_after();
            const float *bias = p.bias[seg];
            const int layout = p.layout[seg], m = m0 + lane;
            const CUtensorMap *omap = &maps.out[seg];
            float *tdst = nullptr;                            // transposed segments: this row's place in the first head
            if (layout == kTf32SplitTransposed) {
                const int b = m / p.S;
                tdst = p.out_t[seg] + ((int64_t)b * (p.N / 32) + n0 / 32) * 64 * p.vt_pitch + (m - b * p.S);
            }
            const uint32_t tcol = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * 2 * BN + half * COLS);
            uint32_t acc[COLS / 32][32];
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                tmem_ld_32x32(tcol + c * 32, acc[c]);
#pragma unroll
                for (int q = 0; q < 32; q += 16) {
                    uint32_t small[16];
                    tmem_ld_32x16(tcol + BN + c * 32 + q, small);
                    tmem_ld_wait16(small);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[c][q + j] = __float_as_uint(__uint_as_float(acc[c][q + j]) + __uint_as_float(small[j]));
                }
            }
            // everything is in registers: the accumulators may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(a));
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                uint32_t(&r)[32] = acc[c];
                const int n = n0 + c * 32;
                if (bias) {
#pragma unroll
                    for (int j4 = 0; j4 < 8; ++j4) {
                        const float4 bv = __ldg(reinterpret_cast<const float4 *>(bias + n) + j4);
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
                        for (int j = 0; j < 32; ++j) {
                            const float v = __uint_as_float(r[j]), h = tf32_head(v);
                            tdst[j * p.vt_pitch] = h;
                            tdst[(32 + j) * p.vt_pitch] = v - h;
                        }
                    }
                    tdst += 64 * p.vt_pitch;
                    continue;
                }
                // rows, or rows with every 32 channels as [head | tail]
                const bool split = layout == kTf32SplitRows;
                for (int t = 0; t < (split ? 2 : 1); ++t) {
                    if (lane == 0) tma_store_wait_read<0>();          // the store out of the staging tile has been read
                    __syncwarp();
#pragma unroll
                    for (int j4 = 0; j4 < 8; ++j4) {
                        float4 v = make_float4(__uint_as_float(r[4 * j4]), __uint_as_float(r[4 * j4 + 1]),
                                               __uint_as_float(r[4 * j4 + 2]), __uint_as_float(r[4 * j4 + 3]));
                        if (split) {
                            const float4 h = make_float4(tf32_head(v.x), tf32_head(v.y), tf32_head(v.z), tf32_head(v.w));
                            v = t == 0 ? h : make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
                        }
                        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(stg + (uint32_t)(lane * 128 + ((j4 ^ (lane & 7)) << 4))),
                                     "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                                     : "memory");
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(omap, stg, split ? 2 * n + 32 * t : n, m0);
                        tma_store_commit();
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
        tmem_dealloc(tmem_base, T::TMEM_COLS);
    }
}

// up to eight matrices of the same shape per launch (blockIdx.y picks one): the five weights of an attention call
struct SplitArgs {
    const float *src[8];
    float *dst[8];
};

// dst[r, 0..K) = tf32 head of src[r, :], dst[r, K..2K) = src - head (fp32, at most 12 significant bits)
__global__ void __launch_bounds__(256) split_tf32_kernel(const SplitArgs args, int64_t src_ld, int64_t rows, int K)
{
    release_successor();
    wait_for_predecessor();
    const float *__restrict__ src = args.src[blockIdx.y];
    float *__restrict__ dst = args.dst[blockIdx.y];
    const uint32_t kv = (uint32_t)K / 4, total = (uint32_t)rows * kv, step = gridDim.x * blockDim.x;
    constexpr int U = 4;                                     // loads in flight per thread
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < total; i0 += U * step) {
        float4 v[U];
        uint32_t r[U], c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = i0 + u * step < total ? i0 + u * step : i0;
            r[u] = i / kv;
            c[u] = i % kv * 4;
            v[u] = __ldg(reinterpret_cast<const float4 *>(src + (int64_t)r[u] * src_ld + c[u]));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u * step >= total) continue;
            const float4 h = make_float4(tf32_head(v[u].x), tf32_head(v[u].y), tf32_head(v[u].z), tf32_head(v[u].w));
            float *d = dst + (int64_t)r[u] * 2 * K + c[u];
            *reinterpret_cast<float4 *>(d) = h;
            *reinterpret_cast<float4 *>(d + K) = make_float4(v[u].x - h.x, v[u].y - h.y, v[u].z - h.z, v[u].w - h.w);
        }
    }
}

}  // namespace

bool launch_split_tf32_many(cudaStream_t stream, int count, const void *const *src, int64_t src_ld, void *const *dst,
                            int64_t rows, int K)
{
    if (count < 1 || count > 8 || rows <= 0 || K <= 0 || K % 4 != 0 || src_ld % 4 != 0 || rows * (K / 4) > INT32_MAX / 2) return false;
    SplitArgs a;
    for (int i = 0; i < 8; ++i) {
        const int j = i < count ? i : 0;
        if ((((uintptr_t)src[j] | (uintptr_t)dst[j]) & 15u) != 0) return false;
        a.src[i] = (const float *)src[j];
        a.dst[i] = (float *)dst[j];
    }
    const int64_t total = rows * (K / 4);
    const unsigned gx = (unsigned)std::min<int64_t>((total + 1023) / 1024, (int64_t)sm_count() * 8);
    KernelTimer timer__("split_tf32", stream);
    launch_chained(split_tf32_kernel, dim3(gx, (unsigned)count), 256, 0, stream, a, src_ld, rows, K);
    count_launch();
    return true;
}

bool launch_split_tf32(cudaStream_t stream, const void *src, int64_t src_ld, void *dst, int64_t rows, int K)
{
    return launch_split_tf32_many(stream, 1, &src, src_ld, &dst, rows, K);
}

bool tcgen05_gemm_tf32x3(cudaStream_t stream, const void *a_split, const void *const *w_split, const float *const *bias,
                         void *const *out, int64_t ldo, int64_t M, int N, int K, int nseg, const Tf32Layout *layout, int S,
                         int64_t vt_pitch)
{
    if (nseg < 1 || nseg > 4 || M <= 0 || M > INT32_MAX / 2 || N % 128 != 0 || K % BK != 0 || K <= 0 || ldo % 4 != 0 ||
        ldo < N || (((uintptr_t)a_split) & 15u))
        return false;
    for (int i = 0; i < nseg; ++i)
        if ((((uintptr_t)w_split[i] | (uintptr_t)out[i] | (uintptr_t)bias[i]) & 15u) != 0) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    Tf32Maps maps;
    Tf32Params p;
    if (!make_tensor_map_2d(&maps.a, a_split, /*elem_bytes=*/4, (uint64_t)2 * K, (uint64_t)M, (uint64_t)2 * K, BK, BM, 128))
        return false;
    for (int i = 0; i < 4; ++i) {
        const int j = i < nseg ? i : 0;
        p.bias[i] = bias[j];
        p.layout[i] = layout ? layout[j] : kTf32Rows;
        p.out_t[i] = (float *)out[j];
        if (!make_tensor_map_2d(&maps.w[i], w_split[j], 4, (uint64_t)2 * K, (uint64_t)N, (uint64_t)2 * K, BK, 128, 128))
            return false;
        const uint64_t cols = p.layout[i] == kTf32SplitRows ? 2 * (uint64_t)N : (uint64_t)N;
        if (p.layout[i] == kTf32SplitTransposed)
            maps.out[i] = maps.a;                            // stored directly
        else if (!make_tensor_map_2d(&maps.out[i], out[j], 4, cols, (uint64_t)M,
                                     p.layout[i] == kTf32SplitRows ? cols : (uint64_t)ldo, 32, 32, 128))
            return false;
    }
    p.M = (int)M;
    p.N = N;
    p.K = K;
    p.nseg = nseg;
    p.S = S > 0 ? S : 1;
    p.vt_pitch = vt_pitch;
    p.err = ew.device;
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(gemm_tf32x3_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<128>::SMEM_BYTES));
        KUTACC_CUDA(cudaFuncSetAttribute(gemm_tf32x3_tc_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<256>::SMEM_BYTES));
        configured = true;
    }
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    const int64_t blocks = ((M + BM - 1) / BM) * (int64_t)(N / 128) * nseg;      // 128 x 128
    const bool wide = (int64_t)N * nseg % 256 == 0 && blocks / 2 >= sms;
    const int64_t tiles = wide ? blocks / 2 : blocks;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, sms);
    KernelTimer timer__("gemm_tf32x3_tc", stream);
    if (wide)
        launch_chained(gemm_tf32x3_tc_kernel<256>, grid, THREADS, Geo<256>::SMEM_BYTES, stream, maps, p);
    else
        launch_chained(gemm_tf32x3_tc_kernel<128>, grid, THREADS, Geo<128>::SMEM_BYTES, stream, maps, p);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
