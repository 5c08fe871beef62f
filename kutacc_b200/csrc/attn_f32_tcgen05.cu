// fp32 gated-attention core on the fifth-generation tensor cores (head size 32).
//
// The operator of src/attention/gating_attention.cpp:73-151 without any bf16 rounding, to fp32 accuracy: both products run
// as tcgen05.mma kind::tf32 on operands split into a tf32 head and a tail (x = hi + lo), lo.hi + hi.lo + hi.hi accumulated
// in fp32 in tensor memory; the softmax is an online softmax in fp32.
//
// A work item is (two batch rows, head h, 128 queries); persistent CTAs, one per SM, take items from an atomic counter.
//   warps 0-7   softmax: warp group w (four warps, 128 tensor-memory lanes) owns batch row w of the item; one thread per
//               query row. The warp's rows of Q and of the gate come by TMA into tiles of its own, from the latter of
//               which the result leaves; the thread splits its row of Q and keeps it in tensor memory, where the first product reads
//               it; per 32-key tile it reads 32 logits, adds mask and pair bias, forms P = exp(x - max), and writes the head
//               of P over the logits and the tail beside them: the A operand of the second product. The logits are
//               double-buffered, so the products of one tile run under the softmax of the other.
//   warp 8      producer: item numbers; TMA loads of K (head and tail, [32 keys x 32]), V^T (head and tail, [32 x 32 keys])
//               and ONE 128 x 32 pair-bias tile, shared by the two batch rows, into a ring of three stages
//   warp 9      mask bias of the tile's keys
//   warps 10-11 MMA issuers, one per warp group. Row 32 of V^T's head is all ones: column 32 of O is the row sum.
// What bounds it: 24 MMA instructions per 32-key tile and warp group, about 55 clocks each at these widths (N = 32 and 48),
// beside a softmax of two warps per scheduler (tensor memory holds no third warp group). The version on mma.sync split K
// and V anew in every CTA and was bound by its shared-memory fragment loads: 269 -> 103 us at 128 x 256 rows, 8 heads.
// Between two items the clocks of a CTA showed 11000, as many as its eight tiles took: rows of Q, gate and result read and written
// by the threads they belong to, 32 lines an instruction. With TMA tiles, the next item's number and first operands early: -> 82 us.
//
// mbarrier conventions as in attn_tcgen05.cu: every barrier is awaited by each of its waiters once per completion, in order;
// all waits are bounded and fall through to the common tail.
#include "common.h"
#include "kernels.h"
#include "launch.cuh"
#include "ptx_utils.cuh"
#include "tcgen05_utils.cuh"
#include "tma_utils.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>

namespace kutacc {
namespace dev {

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int D = 32, BM = 128, BN = 32;        // head size, queries per item, keys per tile
constexpr int MAXG = 2, NST = 3;
constexpr int VT_ROWS = 48;                     // channels, the ones row, zero rows
constexpr int K_BYTES = BN * 128, NB_BYTES = BM * 128;       // one head or tail tile of K
constexpr int VT_HEAD = VT_ROWS * 128, VT_BYTES = VT_HEAD + D * 128;      // V^T: head tile, tail tile (channels only)
constexpr int SOFTMAX_WARPS = 4 * MAXG, PRODUCER_WARP = SOFTMAX_WARPS, MASK_WARP = PRODUCER_WARP + 1, MMA_WARP = PRODUCER_WARP + 2;
constexpr int THREADS = (SOFTMAX_WARPS + 4) * 32;
constexpr int WG_COLS = 256, Q_COL = 0, S_COL = 64, O_COL = 192;     // tensor memory of a warp group; S of buffer b at + 64 b
constexpr int ROWS_BYTES = 32 * 128;            // a warp's 32 rows of one head: Q, the gate, the result
constexpr float kRescaleThreshold = 5.5f;       // P stays below 2^8

struct F32Params {
    const float *bias;                // [B, S] (row stride bias_stride0)
    int avg_split;                    // the result is [B, S, 2*H*D], tf32 heads | tails, instead of [B, S, H*D]
    int64_t bias_stride0;
    int *err;
    int S, H, B, G, n_qt, n_items;
    int *counter;                     // as in attn_tcgen05.cu
    float scale;
};

// D[tmem] (+)= A[tmem] * B[smem], tf32
__device__ __forceinline__ void tc_mma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <bool HAS_NB>
__global__ void __launch_bounds__(THREADS, 1)
attn_f32_tc_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_vt,
                   const __grid_constant__ CUtensorMap tm_nb, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_gate, const __grid_constant__ CUtensorMap tm_avg, const F32Params p)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem_gen = smem_raw + (smem - smem_u32(smem_raw));
    const int G = p.G;
    // stage: K heads x G, K tails x G, then per batch row V^T head and tail, pair bias, mask bias
    const uint32_t off_vt = (uint32_t)(2 * G * K_BYTES), off_nb = off_vt + (uint32_t)(G * VT_BYTES),
                   off_mb = off_nb + (HAS_NB ? NB_BYTES : 0), stage_bytes = off_mb + 1024;
    // before it the warps' tiles of Q and, later, of the gate and the result
    const uint32_t off_stage = 1024u + (uint32_t)(2 * 4 * G * ROWS_BYTES);
    auto stage_base = [&](int s) { return smem + off_stage + (uint32_t)s * stage_bytes; };
    const uint32_t bar = smem;
    auto kv_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto kv_empty = [&](int s) { return bar + 8u * (uint32_t)(NST + s); };
    auto s_full = [&](int w, int b) { return bar + 8u * (uint32_t)(2 * NST + 2 * w + b); };
    auto p_full = [&](int w, int b) { return bar + 8u * (uint32_t)(2 * NST + 2 * MAXG + 2 * w + b); };
    auto o_full = [&](int w) { return bar + 8u * (uint32_t)(2 * NST + 4 * MAXG + w); };
    auto q_full = [&](int w) { return bar + 8u * (uint32_t)(2 * NST + 5 * MAXG + w); };
    auto rows_full = [&](int which, int softmax_warp) { return bar + 8u * (uint32_t)(2 * NST + 6 * MAXG + which * SOFTMAX_WARPS + softmax_warp); };
    const uint32_t it_base = bar + 8u * (2 * NST + 6 * MAXG + 2 * SOFTMAX_WARPS);
    auto it_full = [&](int i) { return it_base + 8u * (uint32_t)(i & 3); };
    const uint32_t item_ring = it_base + 32u, tmem_slot = it_base + 48u;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int S = p.S, nkt = (S + BN - 1) / BN, C = p.H * D;
    auto decode = [&](int w, int &q0, int &h, int &b0) {
        const int qt = w % p.n_qt, hb = w / p.n_qt;
        q0 = qt * BM;
        h = hb % p.H;
        b0 = hb / p.H * G;
    };
    auto item_of = [&](int i, int code) -> int {
        if (!mbar_wait_warp(it_full(i), (uint32_t)((i >> 2) & 1), p.err, code)) return -2;
        int w;
        asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w) : "r"(item_ring + 4u * (uint32_t)(i & 3)));
        return w;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(kv_full(s), 2);
            mbar_init(kv_empty(s), (uint32_t)G);
        }
        for (int w = 0; w < MAXG; ++w) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(s_full(w, b), 2);         // the products' commit, the issuer's own arrival
                mbar_init(p_full(w, b), 4);
            }
            mbar_init(o_full(w), 1);
            mbar_init(q_full(w), 4);
        }
        for (int i = 0; i < 2 * SOFTMAX_WARPS; ++i) mbar_init(rows_full(0, i), 1);       // Q, gate
        for (int i = 0; i < 4; ++i) mbar_init(it_full(i), 1);
        fence_barrier_init();
    }
    // static rows 32..47 of every head tile of V^T: row 32 = 1.0, the others = 0
    for (int i = threadIdx.x; i < NST * G * 128; i += THREADS) {
        const int t = i / 128, rem = i % 128, row = 32 + rem / 8, ch = rem % 8;
        const float v = row == 32 ? 1.0f : 0.0f;
        *reinterpret_cast<float4 *>(smem_gen + off_stage + (t / G) * stage_bytes + off_vt + (t % G) * VT_BYTES + row * 128 + ch * 16) =
            make_float4(v, v, v, v);
    }
    fence_proxy_async();
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, 512);
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

    if (warp == PRODUCER_WARP) {
        // ================= producer =================
        const uint32_t tx = (uint32_t)(2 * G * (K_BYTES + D * 128) + (HAS_NB ? NB_BYTES : 0));
        static_assert(NST <= 3, "item numbers in the ring: as in attn_tcgen05.cu, item i - 3 has been consumed when that of i + 1 is written");
        auto take = [&](int i) -> int {
            int w = 0;
            if (lane == 0) {
                w = atomicAdd(p.counter, 1);
                w = w < p.n_items ? w : -1;
                asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(item_ring + 4u * (uint32_t)(i & 3)), "r"(w) : "memory");
                mbar_arrive(it_full(i));
            }
            return __shfl_sync(0xffffffffu, w, 0);
        };
        auto prefetch_tile = [&](int kt, int q0, int h, int b0) {      // into L2, by the elected lane
            const int k0 = kt * BN;
            for (int t = 0; t < 2; ++t) tma_prefetch_4d(&tm_k, t * D, k0, h, b0);
            for (int r = 0; r < G; ++r)
                for (int t = 0; t < 2; ++t) tma_prefetch_4d(&tm_vt, k0, t * D, h, b0 + r);
            if (HAS_NB) tma_prefetch_3d(&tm_nb, k0, q0, h);
        };
        int g = 0;
        bool ok = true;
        int w = take(0);
        for (int i = 0; ok && w >= 0; ++i) {
            int q0, h, b0, next = -1;
            decode(w, q0, h, b0);
            for (int kt = 0; kt < nkt; ++kt, ++g) {
                const int s = g % NST;
                if (g >= NST && !mbar_wait_warp(kv_empty(s), (uint32_t)((g / NST - 1) & 1), p.err, 71)) {
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t st = stage_base(s);
                    const int k0 = kt * BN;
                    mbar_arrive_expect_tx(kv_full(s), tx);
                    tma_load_4d(st, &tm_k, kv_full(s), 0, k0, h, b0);
                    tma_load_4d(st + G * K_BYTES, &tm_k, kv_full(s), D, k0, h, b0);
                    for (int r = 0; r < G; ++r) {
                        tma_load_4d(st + off_vt + r * VT_BYTES, &tm_vt, kv_full(s), k0, 0, h, b0 + r);
                        tma_load_4d(st + off_vt + r * VT_BYTES + VT_HEAD, &tm_vt, kv_full(s), k0, D, h, b0 + r);
                    }
                    if (HAS_NB) tma_load_3d(st + off_nb, &tm_nb, kv_full(s), k0, q0, h);
                }
                __syncwarp();
                // the next item's number early, and its first operands on their way to L2
                if (kt == max(nkt - 2, 0)) {
                    next = take(i + 1);
                    if (next >= 0) {
                        int q1, h1, b1;
                        decode(next, q1, h1, b1);
                        if (elect_one())
                            for (int t = 0; t < min(nkt, 2); ++t) prefetch_tile(t, q1, h1, b1);
                        __syncwarp();
                    }
                }
            }
            w = next;
        }
    } else if (warp == MASK_WARP) {
        // ================= mask bias =================
        int g = 0;
        bool ok = true;
        for (int i = 0; ok; ++i) {
            const int w = item_of(i, 72);
            if (w < 0) break;
            int q0, h, b0;
            decode(w, q0, h, b0);
            for (int kt = 0; kt < nkt; ++kt, ++g) {
                const int s = g % NST, key = kt * BN + lane;
                float mv[MAXG];
#pragma unroll
                for (int r = 0; r < MAXG; ++r)
                    mv[r] = r < G && key < S ? p.bias[(int64_t)min(b0 + r, p.B - 1) * p.bias_stride0 + key] : -INFINITY;
                if (g >= NST && !mbar_wait_warp(kv_empty(s), (uint32_t)((g / NST - 1) & 1), p.err, 73)) {
                    ok = false;
                    break;
                }
                float *mb = reinterpret_cast<float *>(smem_gen + (stage_base(s) - smem) + off_mb);
#pragma unroll
                for (int r = 0; r < MAXG; ++r)
                    if (r < G) mb[r * BN + lane] = mv[r];
                __syncwarp();
                if (lane == 0) mbar_arrive(kv_full(s));
            }
        }
    } else if (warp >= MMA_WARP) {
        // ================= MMA issuer of warp group w =================
        const int w = warp - MMA_WARP;
        constexpr uint32_t idesc_s = make_instr_desc_tf32(BM, BN), idesc_o = make_instr_desc_tf32(BM, VT_ROWS);
        const uint32_t t0 = tmem_base + (uint32_t)(w * WG_COLS);
        const uint64_t kd0 = make_smem_desc_kmajor(stage_base(0) + w * K_BYTES, 128),
                       vd0 = make_smem_desc_kmajor(stage_base(0) + off_vt + w * VT_BYTES, 128);
        const uint32_t k_tail = (uint32_t)(G * K_BYTES) >> 4, v_tail = VT_HEAD >> 4;
        // S = Q . K^T of global tile g: tail.head + head.tail + head.head (k steps of 8 elements = 32 bytes, 8 columns)
        auto issue_qk = [&](int g) {
            const uint64_t kd = kd0 + (uint32_t)((g % NST) * (int)(stage_bytes >> 4));
            const uint32_t d = t0 + S_COL + (uint32_t)(g & 1) * 64;
#pragma unroll
            for (int pr = 0; pr < 3; ++pr)
#pragma unroll
                for (int k = 0; k < D / 8; ++k)
                    tc_mma_tf32_ts(d, t0 + Q_COL + (pr == 0 ? D : 0) + k * 8, kd + (pr == 1 ? k_tail : 0u) + 2 * k, idesc_s,
                                   (pr > 0 || k > 0) ? 1u : 0u);
            tc_commit(s_full(w, g & 1));
            mbar_arrive(s_full(w, g & 1));          // passes on that the bias tiles have landed, as in attn_tcgen05.cu
        };
        int g = 0;
        bool ok = w < G;
        for (int i = 0; ok; ++i) {
            if (item_of(i, 74) < 0) break;
            if (!mbar_wait_warp(q_full(w), (uint32_t)(i & 1), p.err, 75)) break;
            const int end = g + nkt;
            for (int n = g; n < g + 2 && n < end && ok; ++n) {
                ok = mbar_wait_warp(kv_full(n % NST), (uint32_t)((n / NST) & 1), p.err, 76);
                tc_fence_after();
                if (ok && elect_one()) issue_qk(n);
                __syncwarp();
            }
            for (int kt = 0; kt < nkt && ok; ++kt, ++g) {
                const int b = g & 1;
                ok = mbar_wait_warp(p_full(w, b), (uint32_t)((g >> 1) & 1), p.err, 77);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t vd = vd0 + (uint32_t)((g % NST) * (int)(stage_bytes >> 4));
                    const uint32_t a = t0 + S_COL + (uint32_t)b * 64;
#pragma unroll
                    for (int pr = 0; pr < 3; ++pr)
#pragma unroll
                        for (int k = 0; k < BN / 8; ++k)
                            tc_mma_tf32_ts(t0 + O_COL, a + (pr == 0 ? BN : 0) + k * 8, vd + (pr == 1 ? v_tail : 0u) + 2 * k, pr == 1 ? idesc_s : idesc_o,
                                           (kt > 0 || pr > 0 || k > 0) ? 1u : 0u);
                    tc_commit(kv_empty(g % NST));
                    if (kt == nkt - 1) tc_commit(o_full(w));
                }
                __syncwarp();
                if (g + 2 < end) {
                    ok = mbar_wait_warp(kv_full((g + 2) % NST), (uint32_t)(((g + 2) / NST) & 1), p.err, 78);
                    if (ok && elect_one()) issue_qk(g + 2);       // over P of this tile: in the order of issue
                    __syncwarp();
                }
            }
        }
    } else if (warp < 4 * G) {
        // ================= softmax / epilogue =================
        const int wg = warp >> 2, quad = warp & 3, row = quad * 32 + lane;
        const uint32_t t_w = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(wg * WG_COLS);
        const uint32_t t_o = t_w + O_COL;
        const uint64_t scale2 = pack_f32x2(p.scale, p.scale), log2e2 = pack_f32x2(kLog2e, kLog2e);
        const uint32_t nb_row = off_nb + (uint32_t)row * 128 + (uint32_t)((row & 7) << 4);   // chunk c lies at ^ (c << 4)
        float m = 0.f;                                   // running (possibly stale) max of x
        bool ok = true;

        // a warp whose 32 rows all lie past the item's end only passes on the barriers
        auto do_tile = [&](const int g, const int kt, const bool idle) -> bool {
            const uint32_t st = stage_base(g % NST);
            const uint32_t t_s = t_w + S_COL + (uint32_t)(g & 1) * 64;
            if (!mbar_wait_warp(s_full(wg, g & 1), (uint32_t)((g >> 1) & 1), p.err, 79)) return false;
            if (idle) {
                if (lane == 0) mbar_arrive(p_full(wg, g & 1));
                return true;
            }
            tc_fence_after();
            float pv[32];
            float tmax;
            for (int pass = 0; pass < 2; ++pass) {
                uint32_t r[32];
                tmem_ld_32x32(t_s, r);
                tmem_ld_wait();
                // x = logit * scale + bias (+ pair bias)
                tmax = -INFINITY;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 mb = lds128_f32(st + off_mb + wg * (BN * 4) + c * 16);
                    uint64_t x0 = fma_f32x2(pack_f32x2(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1])), scale2,
                                            pack_f32x2(mb.x, mb.y));
                    uint64_t x1 = fma_f32x2(pack_f32x2(__uint_as_float(r[4 * c + 2]), __uint_as_float(r[4 * c + 3])), scale2,
                                            pack_f32x2(mb.z, mb.w));
                    if (HAS_NB) {
                        const float4 nb = lds128_f32((st + nb_row) ^ (uint32_t)(c << 4));
                        x0 = add_f32x2(x0, pack_f32x2(nb.x, nb.y));
                        x1 = add_f32x2(x1, pack_f32x2(nb.z, nb.w));
                    }
                    unpack_f32x2(x0, pv[4 * c], pv[4 * c + 1]);
                    unpack_f32x2(x1, pv[4 * c + 2], pv[4 * c + 3]);
                    tmax = fmax3(tmax, pv[4 * c], pv[4 * c + 1]);
                    tmax = fmax3(tmax, pv[4 * c + 2], pv[4 * c + 3]);
                }
                // the first tile of an item sets the max, at least the lowest finite number: keys masked with -inf weigh nothing,
                // and a row whose first keys are all of that kind is raised by its first finite one
                if (kt == 0 && pass == 0) m = fmaxf(tmax, -FLT_MAX);
                const bool grow = tmax > m + kRescaleThreshold;
                if (!__any_sync(0xffffffffu, grow)) break;
                // rare: the max of some row grew past the threshold. Rescale those rows of O (and their row sums); the product
                // of the tile before this one must have retired (its stage has been freed).
                const float f = grow ? ex2_approx((m - tmax) * kLog2e) : 1.0f;
                if (grow) m = tmax;
                if (!mbar_wait_warp(kv_empty((g - 1) % NST), (uint32_t)(((g - 1) / NST) & 1), p.err, 80)) return false;
                tc_fence_after();
                uint32_t o[32];
                tmem_ld_32x32(t_o, o);
                uint32_t osum = tmem_ld_32x1(t_o + D);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                tmem_st_32x32(t_o, o);
                tmem_st_32x1(t_o + D, __float_as_uint(__uint_as_float(osum) * f));
                tmem_st_wait();
            }
            // x - m first: with m * log2e folded into one multiply-add its rounding would differ from that of the factor that
            // rescales O, and leave the range of the exponential for masks far below -1e9
            const uint64_t mneg2 = pack_f32x2(-m, -m);
            uint32_t hi[32], lo[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float e0, e1;
                unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(pv[2 * j], pv[2 * j + 1]), mneg2), log2e2), e0, e1);
                const float p0 = ex2_approx(e0), p1 = ex2_approx(e1);
                const float h0 = tf32_head(p0), h1 = tf32_head(p1);
                hi[2 * j] = __float_as_uint(h0);
                hi[2 * j + 1] = __float_as_uint(h1);
                lo[2 * j] = __float_as_uint(p0 - h0);
                lo[2 * j + 1] = __float_as_uint(p1 - h1);
            }
            tmem_st_32x32(t_s, hi);
            tmem_st_32x32(t_s + BN, lo);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(wg, g & 1));
            return true;
        };

        // This warp's rows of Q and of the gate come by TMA into its two tiles; the result leaves from the gate's. (Read row by row
        // by the threads they came to, with 32 lines an instruction, they were half of the kernel's time at 256 keys.)
        const uint32_t q_rows = smem + 1024u + (uint32_t)(warp * 2 * ROWS_BYTES), g_rows = q_rows + ROWS_BYTES;
        auto load_rows = [&](const CUtensorMap *map, int which, int w) {
            int q0, h, b0;
            decode(w, q0, h, b0);
            if (lane == 0) {
                if (which == 1) tma_store_wait_read<0>();
                mbar_arrive_expect_tx(rows_full(which, warp), ROWS_BYTES);
                tma_load_3d(which == 0 ? q_rows : g_rows, map, rows_full(which, warp), h * D, q0 + quad * 32, b0 + wg);
            }
            __syncwarp();
        };
        uint32_t loads[2] = {0, 0}, waits[2] = {0, 0};                // tiles of Q and of the gate
        auto row_chunk = [&](uint32_t rows, int c) { return rows + (uint32_t)(lane * 128 + ((c ^ (lane & 7)) << 4)); };
        auto idle_in = [&](int w) {
            int q0, h, b0;
            decode(w, q0, h, b0);
            return q0 + quad * 32 >= S || b0 + wg >= p.B;
        };
        auto fetch_q = [&](int w) {
            if (idle_in(w)) return;
            load_rows(&tm_q, 0, w);
            ++loads[0];
        };
        // split into tensor memory, once the products with the previous Q have all been formed
        auto publish_q = [&](const bool idle) {
            if (!idle) {
                if (!mbar_wait_warp(rows_full(0, warp), waits[0]++ & 1u, p.err, 84)) {
                    ok = false;
                    return;
                }
                uint32_t hi[32], lo[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 v = lds128_f32(row_chunk(q_rows, c));
                    const float q4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float h = tf32_head(q4[e]);
                        hi[4 * c + e] = __float_as_uint(h);
                        lo[4 * c + e] = __float_as_uint(q4[e] - h);
                    }
                }
                tmem_st_32x32(t_w + Q_COL, hi);
                tmem_st_32x32(t_w + Q_COL + D, lo);
                tmem_st_wait();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full(wg));
        };

        int g = 0;
        int w = item_of(0, 81);
        if (w >= 0) {
            fetch_q(w);
            publish_q(idle_in(w));
        }
        for (int i = 0; w >= 0; ++i) {
            int q0, h, b0, nxt = -1;
            decode(w, q0, h, b0);
            const bool idle = idle_in(w);
            if (!idle) {
                load_rows(&tm_gate, 1, w);
                ++loads[1];
            }
            for (int kt = 0; kt < nkt && ok; ++kt, ++g) {
                if (kt == max(nkt - 2, 0)) {
                    nxt = item_of(i + 1, 82);
                    ok = nxt != -2;
                    if (nxt >= 0) fetch_q(nxt);
                }
                ok = ok && do_tile(g, kt, idle);
            }
            if (!ok) break;
            // every product with this Q has been formed (the logits of its last tile have been read)
            if (nxt >= 0) publish_q(idle_in(nxt));
            if (!ok) break;

            // ---- item epilogue: one row of 32 channels per thread ----
            if (!mbar_wait_warp(o_full(wg), (uint32_t)(i & 1), p.err, 83)) break;
            w = nxt;
            if (idle) continue;
            tc_fence_after();
            uint32_t o[32];
            tmem_ld_32x32(t_o, o);
            const uint32_t osum = tmem_ld_32x1(t_o + D);
            tmem_ld_wait();
            const float inv = 1.0f / __uint_as_float(osum);
            ok = mbar_wait_warp(rows_full(1, warp), waits[1]++ & 1u, p.err, 85);
            if (!ok) break;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 gv = lds128_f32(row_chunk(g_rows, c));
                const float gate[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)      // sigmoid with the hardware reciprocal (2 ulp)
                    o[4 * c + e] = __float_as_uint(__uint_as_float(o[4 * c + e]) * inv * __fdividef(1.0f, 1.0f + __expf(-gate[e])));
            }
            // the result, or its tf32 heads and then, with the same tile, its tails
            for (int t = 0; t < (p.avg_split ? 2 : 1); ++t) {
                if (t == 1) {
                    if (lane == 0) tma_store_wait_read<0>();
                    __syncwarp();
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float4 v = make_float4(__uint_as_float(o[4 * c]), __uint_as_float(o[4 * c + 1]), __uint_as_float(o[4 * c + 2]),
                                           __uint_as_float(o[4 * c + 3]));
                    if (p.avg_split) {
                        const float4 hv = make_float4(tf32_head(v.x), tf32_head(v.y), tf32_head(v.z), tf32_head(v.w));
                        v = t == 0 ? hv : make_float4(v.x - hv.x, v.y - hv.y, v.z - hv.z, v.w - hv.w);
                    }
                    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(row_chunk(g_rows, c)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {                 // rows past S are clipped
                    tma_store_3d(&tm_avg, g_rows, h * D + t * C, q0 + quad * 32, b0 + wg);
                    tma_store_commit();
                }
            }
        }
        // after a wait that ran out: no copy may still be on its way when the CTA exits
        for (int t = 0; t < 2; ++t)
            if (loads[t] != waits[t]) mbar_wait_warp(rows_full(t, warp), waits[t] & 1u, p.err, 86);
        if (lane == 0) tma_store_wait<0>();
    }

    // ================= common tail =================
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(p.counter + 1, 1) == (int)gridDim.x - 1) {
            __threadfence();
            p.counter[0] = 0;
            p.counter[1] = 0;
            __threadfence();
        }
    }
}

int smem_bytes(int G, bool has_nb)
{
    return 1024 + 1024 + 2 * 4 * G * ROWS_BYTES + NST * (G * (2 * K_BYTES + VT_BYTES) + (has_nb ? NB_BYTES : 0) + 1024);
}

}  // namespace

bool tcgen05_attn_f32(cudaStream_t stream, const void *q, const void *k_split, const void *vt_split, int64_t vt_pitch,
                      const void *gate, const void *bias, int64_t bias_stride0, const void *nb, int64_t nb_stride_h,
                      int64_t nb_stride_q, void *avg, bool avg_split, int B, int S, int H, int Dh, float scale)
{
    if (Dh != D || vt_pitch % 4 != 0 || vt_pitch < S) return false;
    if (nb && ((nb_stride_h % 4) || (nb_stride_q % 4) || ((uintptr_t)nb % 16) || nb_stride_h < nb_stride_q)) return false;
    if ((((uintptr_t)q | (uintptr_t)gate | (uintptr_t)avg) & 15u) != 0) return false;
    const int64_t n_qt = (S + BM - 1) / BM, hq = n_qt * H;
    if (hq * B > INT32_MAX / 64) return false;
    KernelErrorWord &ew = kernel_error_word();
    int *counter = work_counter(stream);
    if (ew.device == nullptr || counter == nullptr) return false;
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    F32Params p;
    p.bias = (const float *)bias;
    p.avg_split = avg_split;
    p.bias_stride0 = bias_stride0;
    p.err = ew.device;
    p.S = S;
    p.H = H;
    p.B = B;
    p.G = B * hq <= sms ? 1 : 2;                 // one batch row per CTA while that fits one wave
    p.n_qt = (int)n_qt;
    p.n_items = (int)((B + p.G - 1) / p.G * hq);
    p.counter = counter;
    p.scale = scale;
    const uint64_t Su = (uint64_t)S, Hu = (uint64_t)H, vp = (uint64_t)vt_pitch;
    CUtensorMap tk, tvt, tnb, tq, tg, ta;
    const uint64_t Cu = Hu * D, ca = avg_split ? 2 * Cu : Cu;
    if (!make_tensor_map_f32_3d(&tq, q, Cu, Su, (uint64_t)B, Cu, Su * Cu, D, 32, 128) ||
        !make_tensor_map_f32_3d(&tg, gate, Cu, Su, (uint64_t)B, Cu, Su * Cu, D, 32, 128) ||
        !make_tensor_map_f32_3d(&ta, avg, ca, Su, (uint64_t)B, ca, Su * ca, D, 32, 128))
        return false;
    if (!make_tensor_map_f32_4d(&tk, k_split, 2 * D, Su, Hu, (uint64_t)B, 2 * D * Hu, 2 * D, Su * 2 * D * Hu, D, BN,
                                (uint32_t)p.G, 128) ||
        !make_tensor_map_f32_4d(&tvt, vt_split, Su, 2 * D, Hu, (uint64_t)B, vp, 2 * D * vp, 2 * D * vp * Hu, BN, D, 1, 128))
        return false;
    tnb = tk;
    if (nb && !make_tensor_map_f32_3d(&tnb, nb, Su, Su, Hu, (uint64_t)nb_stride_q, (uint64_t)nb_stride_h, BN, BM, 128)) return false;
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(attn_f32_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MAXG, true)));
        KUTACC_CUDA(cudaFuncSetAttribute(attn_f32_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MAXG, false)));
        configured = true;
    }
    const unsigned grid = (unsigned)std::min(p.n_items, sms);
    KernelTimer timer__("attn_f32_tc", stream);
    if (nb)
        launch_chained(attn_f32_tc_kernel<true>, grid, THREADS, smem_bytes(p.G, true), stream, tk, tvt, tnb, tq, tg, ta, p);
    else
        launch_chained(attn_f32_tc_kernel<false>, grid, THREADS, smem_bytes(p.G, false), stream, tk, tvt, tnb, tq, tg, ta, p);
    count_launch();
    return true;
}

}  // namespace dev
}  // namespace kutacc
