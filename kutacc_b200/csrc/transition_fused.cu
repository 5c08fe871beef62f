// Transition MLP in one kernel: out = relu(x . W1^T + b1) . W2^T + b2, the hidden activations never leave the SM.
//
// (src/attention/transition.cpp:21-61; hidden is a bf16 tensor there, and is rounded to bf16 here.) A CTA works on two
// 128-row tiles at a time (128 channels; one tile with 256 channels) and walks the hidden channels in chunks of 128:
//   S = x . W1_chunk^T                    128 fp32 columns of tensor memory
//   P = bf16(relu(S + b1))                written back over S, read by the tensor core from tensor memory
//   O += P . W2_chunk^T                   128 (256) columns
// Two chains of this kind run side by side (the two row tiles, or even and odd chunks of one row tile), so that the tensor
// core works on one while the warps convert the other's logits of the hidden layer:
//   warp 0      TMA producer: x tiles, and the weights as a stream of 128 x 64 slabs through a 7-slab ring
//   warp 1      MMA issuer
//   warps 2-3   idle (they keep the register split by warps even)
//   warps 4-19  four groups of four warps, one row and 64 columns per thread: hidden epilogue of chain 0 / 1, output
//               epilogue (bias, bf16, staging tile, TMA store). With one group of four warps per chain the conversion of a
//               chunk took longer than the other chain's products (53 against 50 us at 147456 rows)
// Two row tiles share every weight slab: the weights stream from L2 once per 256 rows (302 MB instead of 604 MB at 147456
// rows x 128 channels). Bound by the chain product, conversion, product and by the operands' way through shared memory (tensor
// pipe 40 % busy) where the two-kernel version was bound by the round trip of the hidden tensor (302 MB through L2 and HBM):
// 90 -> 42 us there, 0.92 PFLOP/s.
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

constexpr int BM = 128, BH = 128, BK = 64;      // rows of a tile, hidden channels of a chunk, k columns of a slab
constexpr int RING_SLABS = 7;
constexpr int SLAB_BYTES = 128 * BK * 2;
constexpr int X_BYTES = 4 * SLAB_BYTES;         // two tiles of 128 channels or one of 256
constexpr int STG_TILE = 128 * 64;              // output staging, 128 rows x 32 channels per group
constexpr int STG_BYTES = 4 * STG_TILE;
constexpr int MAX_HIDDEN = 2048;
constexpr int OFF_RING = X_BYTES, OFF_STG = OFF_RING + RING_SLABS * SLAB_BYTES, OFF_BAR = OFF_STG + STG_BYTES;
constexpr int OFF_BIAS = OFF_BAR + 256;
constexpr int SMEM_BYTES = OFF_BIAS + (MAX_HIDDEN + 256) * 4 + 1024;
constexpr int THREADS = 20 * 32;
constexpr int S_COL = 0, O_COL = 256;           // S of chain c at 128 c, O (of tile r at 128 r) from 256
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");

struct MlpParams {
    const float *b1, *b2;
    int M, hidden;
    int tiles;              // row tiles per CTA and step (128 channels: 1 or 2)
    int *err;
};

// relu of a NaN is 0, as in the epilogue of the two-product path (max.bf16x2 takes the operand that is a number; cvt.relu
// would keep the NaN)
__device__ __forceinline__ uint32_t pack_relu_bf16x2(float lo, float hi)
{
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;\n" : "=r"(r) : "r"(pack_bf16x2(lo, hi)), "r"(0u));
    return r;
}
__device__ __forceinline__ void group_bar(int g) { asm volatile("bar.sync %0, 128;\n" ::"r"(g + 1) : "memory"); }

template <int CO>
__global__ void __launch_bounds__(THREADS, 1)
transition_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w1,
                  const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_out, const MlpParams p)
{
    // The weight ring counts in units of SPU slabs. With 128 channels a chunk of W1 or W2 is two slabs that come and go together: half
    // the waits and commits on the issuing warp's path (160000 rows x 512 hidden: 56.3 -> 52.3 us). With 256 channels it is four, and
    // a ring that moves in twos is too short for them (160000 rows x 1024: 189 us by single slabs, 196 in twos).
    constexpr int SPU = CO == 128 ? 2 : 1, NUNIT = RING_SLABS / SPU;
    constexpr int KX = CO / BK;                 // slabs of an x tile, and of a chunk of W1
    constexpr int NO = CO / 128;                // 128-row blocks of W2
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem_gen = smem_raw + (smem - smem_u32(smem_raw));
    const uint32_t bar = smem + OFF_BAR;
    auto w_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto w_empty = [&](int s) { return bar + 8u * (uint32_t)(NUNIT + s); };
    auto x_full = [&](int r) { return bar + 8u * (uint32_t)(2 * NUNIT + r); };
    auto x_empty = [&](int r) { return bar + 8u * (uint32_t)(2 * NUNIT + 2 + r); };
    auto s_full = [&](int c) { return bar + 8u * (uint32_t)(2 * NUNIT + 4 + c); };
    auto p_full = [&](int c) { return bar + 8u * (uint32_t)(2 * NUNIT + 6 + c); };
    auto o_full = [&](int r) { return bar + 8u * (uint32_t)(2 * NUNIT + 8 + r); };
    const uint32_t o_free = bar + 8u * (2 * NUNIT + 10), tmem_slot = o_free + 8;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int R = CO == 128 ? p.tiles : 1;
    const int nch = p.hidden / BH;
    const int steps = (p.M + BM * R - 1) / (BM * R);            // groups of R row tiles
    const int mine = (int)blockIdx.x < steps ? (steps - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    float *bias1 = reinterpret_cast<float *>(smem_gen + OFF_BIAS), *bias2 = bias1 + MAX_HIDDEN;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NUNIT; ++s) {
            mbar_init(w_full(s), 1);
            mbar_init(w_empty(s), 1);
        }
        for (int r = 0; r < 2; ++r) {
            mbar_init(x_full(r), 1);
            mbar_init(x_empty(r), 1);
            mbar_init(s_full(r), 1);
            mbar_init(p_full(r), 8);
            mbar_init(o_full(r), 1);
        }
        mbar_init(o_free, 16);
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
        tma_prefetch_desc(&tm_x);
        tma_prefetch_desc(&tm_w1);
        tma_prefetch_desc(&tm_w2);
        tma_prefetch_desc(&tm_out);
    }
    release_successor();
    wait_for_predecessor();
    for (int i = threadIdx.x; i < p.hidden; i += THREADS) bias1[i] = p.b1[i];
    for (int i = threadIdx.x; i < CO; i += THREADS) bias2[i] = p.b2[i];
    __syncthreads();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0) {
        // ================= producer =================
        if (elect_one()) {
            int unit = 0;                                          // asked for so far (a count and its remainder: with a slot and a
                                                                   // round 51925 rows of 256 channels take 60.4 us, so 59.6)
            bool ok = true;
            int filled = 0;                                        // slabs of the unit that have been asked for
            auto slab = [&](const CUtensorMap *map, int c0, int c1) {
                const int s = unit % NUNIT;
                if (filled == 0) {
                    if (unit >= NUNIT && ok) ok = mbar_wait(w_empty(s), (uint32_t)((unit / NUNIT - 1) & 1), p.err, 61);
                    if (!ok) return;
                    mbar_arrive_expect_tx(w_full(s), SPU * SLAB_BYTES);
                }
                if (!ok) return;
                tma_load_3d(smem + OFF_RING + (s * SPU + filled) * SLAB_BYTES, map, w_full(s), c0, c1, 0);
                if (++filled < SPU) return;
                filled = 0;
                ++unit;
            };
            auto load_w1 = [&](int j) {
                for (int k = 0; k < KX; ++k) slab(&tm_w1, k * BK, j * BH);
            };
            auto load_w2 = [&](int j) {
                for (int k = 0; k < BH / BK; ++k)
                    for (int o = 0; o < NO; ++o) slab(&tm_w2, j * BH + k * BK, o * 128);
            };
            auto load_x = [&](int t) {                             // t counts this CTA's steps
                const int row0 = ((int)blockIdx.x + t * (int)gridDim.x) * BM * R;
                for (int r = 0; r < R && ok; ++r) {
                    if (t > 0) ok = mbar_wait(x_empty(r), (uint32_t)((t - 1) & 1), p.err, 62);
                    if (!ok) return;
                    mbar_arrive_expect_tx(x_full(r), KX * SLAB_BYTES);
                    for (int k = 0; k < KX; ++k)
                        tma_load_3d(smem + (r * KX + k) * SLAB_BYTES, &tm_x, x_full(r), k * BK, row0 + r * BM, 0);
                }
                // the next rows come into L2 meanwhile: their load is on the path from one step to the next
                if (t + 1 < mine)
                    for (int r = 0; r < R; ++r)
                        for (int k = 0; k < KX; ++k)
                            tma_prefetch_3d(&tm_x, k * BK, row0 + (int)gridDim.x * BM * R + r * BM, 0);
            };
            // the weights in the order in which the MMA issuer takes them
            const int total = mine * nch;
            if (total > 0) {
                load_x(0);
                load_w1(0);
                if (CO == 256 && total > 1) {
                    if (nch == 1) load_x(1);
                    load_w1(1 % nch);
                }
                constexpr int AHEAD = CO == 256 ? 2 : 1;
                for (int c = 0; c < total && ok; ++c) {
                    load_w2(c % nch);
                    const int n = c + AHEAD;                       // the chunk whose first product follows
                    if (n < total) {
                        if (n % nch == 0) load_x(n / nch);
                        load_w1(n % nch);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        constexpr uint32_t idesc_h = make_instr_desc_bf16(BM, BH);
        constexpr uint32_t SLAB16 = SLAB_BYTES >> 4;               // descriptor addresses count in units of 16 bytes
        const uint64_t xd = make_smem_desc_kmajor(smem, 128), wd = make_smem_desc_kmajor(smem + OFF_RING, 128);
        bool ok = true;
        // place of a unit in the ring; its barrier's parity
        struct Pos {
            int s;
            uint32_t par;
        };
        auto advance = [](Pos q, int n) {
            q.s += n;
            if (q.s >= NUNIT) {
                q.s -= NUNIT;
                q.par ^= 1u;
            }
            return q;
        };
        Pos it = {0, 0};
        auto wait_units = [&](Pos q, int n) {
            for (int i = 0; i < n && ok; ++i, q = advance(q, 1)) ok = mbar_wait_warp(w_full(q.s), q.par, p.err, 63);
        };
        auto free_units = [&](Pos q, int n) {                      // by the elected lane
            for (int i = 0; i < n; ++i, q = advance(q, 1)) tc_commit(w_empty(q.s));
        };
        // descriptor of the i-th slab from the unit `q` on
        auto slab_desc = [&](Pos q, int i) {
            q = advance(q, i / SPU);
            return wd + (uint32_t)((q.s * SPU + i % SPU) * SLAB16);
        };
        // S_c = x_r . W1_chunk^T with the units from `q` on
        auto mma1 = [&](int c, int r, Pos q) {
#pragma unroll
            for (int k = 0; k < KX; ++k) {
                const uint64_t a = xd + (uint32_t)((r * KX + k) * SLAB16), b = slab_desc(q, k);
#pragma unroll
                for (int e = 0; e < BK / 16; ++e)
                    tc_mma_bf16(tmem_base + S_COL + c * BH, a + 2 * e, b + 2 * e, idesc_h, (k > 0 || e > 0) ? 1u : 0u);
            }
            tc_commit(s_full(c));
        };
        // O_r += P_c . W2_chunk^T
        auto mma2 = [&](int c, int r, Pos q, bool fresh) {
#pragma unroll
            for (int k = 0; k < BH / BK; ++k)
#pragma unroll
                for (int o = 0; o < NO; ++o) {
                    const uint64_t b = slab_desc(q, k * NO + o);
#pragma unroll
                    for (int e = 0; e < BK / 16; ++e)
                        tc_mma_bf16_ts(tmem_base + O_COL + (r * NO + o) * 128, tmem_base + S_COL + c * BH + k * 64 + e * 8, b + 2 * e,
                                       idesc_h, (!fresh || k > 0 || e > 0) ? 1u : 0u);
                }
        };
        const int total = mine * nch;
        constexpr int W1N = KX / SPU, W2N = BH / BK * NO / SPU;
        if constexpr (CO == 128) {
            if (total > 0) {
                for (int r = 0; r < R && ok; ++r) ok = mbar_wait_warp(x_full(r), 0, p.err, 64);
                wait_units(it, W1N);
                tc_fence_after();
                if (ok && elect_one()) {
                    for (int r = 0; r < R; ++r) {
                        mma1(r, r, it);
                        if (nch == 1) tc_commit(x_empty(r));
                    }
                    free_units(it, W1N);
                }
                __syncwarp();
                it = advance(it, W1N);
            }
            for (int c = 0; c < total && ok; ++c) {
                const int j = c % nch, n = c + 1;                  // chunk c with its W2, then chunk n with its W1
                const bool more = n < total;
                wait_units(it, W2N);
                for (int r = 0; r < R && ok; ++r) {
                    ok = ok && mbar_wait_warp(p_full(r), (uint32_t)(c & 1), p.err, 65);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        mma2(r, r, it, j == 0);
                        if (j == nch - 1) tc_commit(o_full(r));
                        if (r == R - 1) free_units(it, W2N);
                    }
                    __syncwarp();
                    if (!more) continue;
                    if (r == 0) wait_units(advance(it, W2N), W1N);
                    if (n % nch == 0) ok = ok && mbar_wait_warp(x_full(r), (uint32_t)((n / nch) & 1), p.err, 64);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        mma1(r, r, advance(it, W2N));                      // overwrites P: the products run in the order of issue
                        if (n % nch == nch - 1) tc_commit(x_empty(r));
                        if (r == R - 1) free_units(advance(it, W2N), W1N);
                    }
                    __syncwarp();
                }
                it = advance(it, W2N);
                if (more) it = advance(it, W1N);
            }
        } else {
            auto first_product = [&](int n, Pos first) {           // chunk n into chain n & 1
                wait_units(first, W1N);
                if (ok && n % nch == 0) ok = mbar_wait_warp(x_full(0), (uint32_t)((n / nch) & 1), p.err, 64);
                if (!ok) return;
                tc_fence_after();
                if (elect_one()) {
                    mma1(n & 1, 0, first);
                    if (n % nch == nch - 1) tc_commit(x_empty(0));
                    free_units(first, W1N);
                }
                __syncwarp();
            };
            for (int n = 0; n < 2 && n < total && ok; ++n, it = advance(it, W1N)) first_product(n, it);
            for (int c = 0; c < total && ok; ++c) {
                const int j = c % nch, t = c / nch;
                wait_units(it, W2N);
                // the first product into O of a tile: both groups have read the tile before
                if (ok && j == 0 && t > 0) ok = mbar_wait_warp(o_free, (uint32_t)((t - 1) & 1), p.err, 66);
                ok = ok && mbar_wait_warp(p_full(c & 1), (uint32_t)((c >> 1) & 1), p.err, 65);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    mma2(c & 1, 0, it, j == 0);
                    if (j == nch - 1) tc_commit(o_full(0));
                    free_units(it, W2N);
                }
                __syncwarp();
                it = advance(it, W2N);
                if (c + 2 < total) {
                    first_product(c + 2, it);
                    it = advance(it, W1N);
                }
            }
        }
    } else if (warp >= 4) {
        // ================= epilogues =================
        // group = chain and 64-column half of its 128 columns
        const int grp = (warp - 4) >> 2, chain = grp >> 1, col = (grp & 1) * 64, quad = warp & 3, row = quad * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t stg = smem + OFF_STG + grp * STG_TILE;
        bool ok = true;
        // P = bf16(relu(S + b1)) of this group's chain, chunk j; u counts the chain's chunks. P of a half lies in the first
        // columns of its own half of S, so that the two groups of a chain need not wait for each other.
        auto hidden_chunk = [&](int j, int u) {
            ok = mbar_wait_warp(s_full(chain), (uint32_t)(u & 1), p.err, 67);
            if (!ok) return;
            tc_fence_after();
            const uint32_t ts = t_lane + S_COL + chain * BH + col;
            const uint32_t b1a = smem + OFF_BIAS + (uint32_t)((j * BH + col) * 4);
            uint32_t a[2][32];
            tmem_ld_32x32(ts, a[0]);
            tmem_ld_32x32(ts + 32, a[1]);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 bv = lds128_f32(b1a + c * 128 + i * 16);
                    const uint32_t *r = &a[c][4 * i];
                    float y0, y1, y2, y3;
                    unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(r[0]), __uint_as_float(r[1])), pack_f32x2(bv.x, bv.y)), y0, y1);
                    unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(r[2]), __uint_as_float(r[3])), pack_f32x2(bv.z, bv.w)), y2, y3);
                    pk[2 * i] = pack_relu_bf16x2(y0, y1);
                    pk[2 * i + 1] = pack_relu_bf16x2(y2, y3);
                }
                tmem_st_32x16(ts + c * 16, pk);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(chain));
        };
        // out rows of tile `row0`: this group's 64 columns of O, channels n0 + col on
        auto output_tile = [&](int ob, int row0, int n0, int t) {
            ok = mbar_wait_warp(o_full(ob), (uint32_t)(t & 1), p.err, 68);
            if (!ok) return;
            tc_fence_after();
            const uint32_t to = t_lane + O_COL + chain * 128 + col;
            uint32_t a[2][32];
            tmem_ld_32x32(to, a[0]);
            tmem_ld_32x32(to + 32, a[1]);
            tmem_ld_wait();
            tc_fence_before();
            if (CO == 256) {
                __syncwarp();
                if (lane == 0) mbar_arrive(o_free);
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                // the store out of the staging tile has been read
                if (quad == 0 && lane == 0) tma_store_wait_read<0>();
                group_bar(grp);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pk[4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float4 bv = lds128_f32(smem + OFF_BIAS + (uint32_t)((MAX_HIDDEN + n0 + col + c * 32 + q * 8 + i * 4) * 4));
                        const uint32_t *r = &a[c][q * 8 + i * 4];
                        pk[2 * i] = pack_bf16x2(__uint_as_float(r[0]) + bv.x, __uint_as_float(r[1]) + bv.y);
                        pk[2 * i + 1] = pack_bf16x2(__uint_as_float(r[2]) + bv.z, __uint_as_float(r[3]) + bv.w);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(
                                     stg + (uint32_t)(row * 64 + ((q ^ ((row >> 1) & 3)) << 4))),
                                 "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3])
                                 : "memory");
                }
                fence_proxy_async();
                group_bar(grp);
                if (quad == 0 && lane == 0) {
                    tma_store_3d(&tm_out, stg, n0 + col + c * 32, row0, 0);
                    tma_store_commit();
                }
            }
        };
        if (CO == 256 || chain < R) {
            int u = 0;
            for (int t = 0; t < mine && ok; ++t) {
                const int row0 = ((int)blockIdx.x + t * (int)gridDim.x) * BM * R;
                if (CO == 128) {
                    for (int j = 0; j < nch && ok; ++j, ++u) hidden_chunk(j, u);
                    if (ok) output_tile(chain, row0 + chain * BM, 0, t);
                } else {
                    // chunk c of the whole run belongs to chain c & 1
                    for (int j = 0; j < nch && ok; ++j)
                        if (((t * nch + j) & 1) == chain) hidden_chunk(j, u++);
                    if (ok) output_tile(0, row0, chain * 128, t);
                }
            }
            if (quad == 0 && lane == 0) tma_store_wait<0>();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int CO>
bool launch_co(cudaStream_t stream, const CUtensorMap &tx, const CUtensorMap &t1, const CUtensorMap &t2, const CUtensorMap &to,
               const MlpParams &p)
{
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(transition_kernel<CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
    const int rows = BM * (CO == 128 ? p.tiles : 1), steps = (p.M + rows - 1) / rows;
    const unsigned grid = (unsigned)std::min(steps, std::max(1, sm_count() - runtime().sm_margin));
    KernelTimer timer__("transition", stream);
    launch_chained(transition_kernel<CO>, grid, THREADS, SMEM_BYTES, stream, tx, t1, t2, to, p);
    count_launch();
    return true;
}

// Whether two products through the workspace are faster. While every SM has at most one row tile the one kernel takes as long as
// a tile's chain of hidden chunks, whatever the number of rows; two kernels spread few rows over the chip in both directions.
// Microseconds for h hidden channels (thousands) and m rows (thousands), fitted to 128 to 18944 rows x 256 to 2048 hidden:
//   256 channels: chain 4.6 + 17.2 h, two kernels 9.7 + 5.2 h + 0.76 h m   (2048 x 1024: 23.0 against 17.0, 12288: 23.8 / 25.0,
//                 2048 x 2048: 40.6 / 22.8, 12288: 42.1 / 41.2)
//   128 channels: chain 4.4 +  9.4 h, two kernels 10.5 + 4.6 h + 0.6 h m   (2048 x 2048: 24.0 against 22.2, 4096: 24.1 / 23.9)
// With more row tiles than SMs one kernel is the faster one (40000 x 1024: 59.9 / 70.2) or as fast within a few us (20000: 41.3 /
// 36.3). One row tile of up to 1024 hidden channels stays in one launch without a workspace (22 against 15 us).
bool two_kernels_faster(int64_t M, int c_o, int c_i)
{
    if ((M + BM - 1) / BM > sm_count() || (M <= BM && c_i <= 1024)) return false;
    const double h = c_i * 1e-3, m = (double)M * 1e-3;
    return c_o == 256 ? 4.6 + 17.2 * h > 9.7 + 5.2 * h + 0.76 * h * m : 4.4 + 9.4 * h > 10.5 + 4.6 * h + 0.6 * h * m;
}

}  // namespace

bool tcgen05_transition_bf16(cudaStream_t stream, const void *x, const void *w1, const float *b1, const void *w2, const float *b2,
                             void *out, int64_t M, int c_o, int c_i, bool or_two)
{
    if ((c_o != 128 && c_o != 256) || c_i % BH != 0 || c_i > MAX_HIDDEN || M > INT32_MAX / 2 ||
        ((((uintptr_t)x | (uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)out) & 15u) != 0))
        return false;
    // (the two products want aligned biases, this kernel does not)
    if (or_two && (((uintptr_t)b1 | (uintptr_t)b2) & 15u) == 0 && two_kernels_faster(M, c_o, c_i)) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    CUtensorMap tx, t1, t2, to;
    if (!make_tensor_map_bf16_3d(&tx, x, c_o, M, 1, c_o, (uint64_t)M * c_o, BK, BM, 128) ||
        !make_tensor_map_bf16_3d(&t1, w1, c_o, c_i, 1, c_o, (uint64_t)c_i * c_o, BK, BH, 128) ||
        !make_tensor_map_bf16_3d(&t2, w2, c_i, c_o, 1, c_i, (uint64_t)c_o * c_i, BK, 128, 128) ||
        !make_tensor_map_bf16_3d(&to, out, c_o, M, 1, c_o, (uint64_t)M * c_o, 32, BM, 64))
        return false;
    MlpParams p;
    p.b1 = b1;
    p.b2 = b2;
    p.M = (int)M;
    p.hidden = c_i;
    // two row tiles per CTA once every SM has work that way
    p.tiles = (M + 2 * BM - 1) / (2 * BM) >= sm_count() ? 2 : 1;
    p.err = ew.device;
    return c_o == 128 ? launch_co<128>(stream, tx, t1, t2, to, p) : launch_co<256>(stream, tx, t1, t2, to, p);
}

}  // namespace dev
}  // namespace kutacc
