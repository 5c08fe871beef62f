// Fused gated-attention core on the fifth-generation tensor cores (head sizes 8, 16 and 32).
//
// A work item is (up to four batch rows b, head h, 128 queries). The kernel is persistent, one CTA per SM: it takes
// items from an atomic counter until the list is exhausted (a CTA whose SM was busy at launch takes fewer items instead
// of finishing late), and every pipeline below keeps running across item boundaries. Both matrix products run on
// tcgen05.mma with accumulators in tensor memory, issued by one elected lane; the softmax runs on the logits read back
// with tcgen05.ld. The S x S logits never leave the SM.
//
//   warps 0-15  softmax: warp group w (four warps, 128 tensor-memory lanes) owns batch row w of the item and 128 columns
//               of tensor memory; one thread per query row. Per 64-key tile a thread reads its 64 logits in
//               16-column pieces (the next piece is in flight while one is worked on), rounds each raw logit to bf16
//               as the reference's logits scratch does (src/attention/gating_attention.cpp:97-101), adds the mask and
//               pair bias in fp32 (:112-117) and keeps P = exp2((x - max) * log2 e) as packed bf16 in 32
//               registers (narrow heads and 64-channel layers: a bf16 head and a bf16 tail, SPLIT below). P goes back over the logits in tensor memory, where the second product reads it as its A
//               operand: no shared-memory round trip. The running max is the thread's own; it is first taken from the
//               item's first 16 keys and raised only when a tile exceeds it by 2^8 (a stale max cancels in the final
//               division): then the row of O is rescaled and the tile formed again.
//   warp 16     producer: takes the next item number and publishes it to the other roles; TMA tile loads (hardware
//               swizzle) of the four Q tiles and, per 64-key tile, of the four K [64 x D] and V^T [D x 64] tiles and of
//               ONE 128 x 64 pair-bias tile, which the four batch rows share, into a 3-stage ring
//   warp 17     converts the tile's mask-bias values to fp32 (apart from the producer: the two together took longer per
//               tile than the softmax)
//   warps 18-19 MMA issuers, warp group by warp group (two each): O_w (+)= P_w . V_w^T of tile g, then S_w = Q_w . K_w^T of tile
//               g + 1. The row of V^T after the last channel is all ones, so the column of O after the last channel
//               accumulates the row sum of the rounded probabilities for free
//
// What bounds it, and why this split: per logit the softmax issues about six instructions (two conversions per pair for
// the bf16 logit, two packed FMAs, an add, a max3, two unpacks of the pair bias, two exponentials, one pack), so the
// limits are the issue slots (128 lanes per clock and SM) and the MUFU pipe (16 exponentials per clock and SM); what
// keeps a kernel away from them is the latency of the barrier -> tcgen05.ld -> softmax -> tcgen05.st -> barrier ->
// MMA chain of a tile. Four independent chains per SM hide it: while one warp group waits for its products, the warps
// of the other three fill the issue slots of the same schedulers. Measured: triangle attention at 1024 residues (4.3 G
// logits) 2.16 -> 1.57 ms, column attention 384 x 512 x 8 heads 0.41 -> 0.31 ms against two CTAs per SM with one (batch row,
// head, 128 queries) each, P through shared memory and two threads per query row. (Now 1.49 and 0.27 ms, see STAGED.) A share of the
// exponentials on the FMA units, 1 to 4 of 8 pairs, made the call 5 to 22 % longer: instructions are what is short. The single-thread cost of the MMA
// and TMA instructions mattered as much as the split: behind `lane == 0` an instruction took about 70 clocks to
// issue, behind elect_one() about 33.
//
// Fully masked rows stay uniform as in the reference (fp32 absorption of the logit by the -1e9 bias, or by any finite one).
//
// mbarrier phases. A parity wait names "the current or the preceding phase", so every barrier here is awaited by each of
// its waiters once per completion, in order. All waits are bounded; on a timeout the roles fall through to the common
// tail, tensor memory is released, and the host-visible error word carries the site.
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
constexpr int BM = 128;               // queries per item
constexpr int BN = 64;                // keys per tile
constexpr int NST = 3;                // ring depth
constexpr int MAXG = 4;               // batch rows (softmax warp groups) per item
constexpr int NB_BYTES = BM * BN * 2;         // 16 KB, 128-byte rows, 128-byte swizzle
constexpr int MB_BYTES = MAXG * BN * 4;       // mask bias of the tile's keys, fp32
constexpr int SOFTMAX_WARPS = 4 * MAXG;
constexpr int MMA_WARPS = 2;          // warp group w is served by MMA warp w % 2
constexpr int PRODUCER_WARP = SOFTMAX_WARPS, MASK_WARP = SOFTMAX_WARPS + 1, MMA_WARP = SOFTMAX_WARPS + 2;
constexpr int THREADS = (SOFTMAX_WARPS + 2 + MMA_WARPS) * 32;
constexpr int BAR_BYTES = 512;
constexpr int WG_COLS = 128;          // tensor-memory columns of a warp group: S (then P) 0..63, O from 64
constexpr int S_COL = 0, O_COL = 64;
constexpr float kRescaleThreshold = 5.5f;     // P stays below 2^8
constexpr float kFar = 2147483648.f;          // 2^31: mneg below it is within 64 of -m * log2e

// STAGED: a warp's rows of the gate come by TMA into a tile of its own, where the result takes their place; the next item's number and
// first operands are asked for early. The clocks of a CTA showed 6000 between two items of eight tiles of 2700: Q and the first
// tile from memory (3400), rows of gate and result read and written by the threads they belong to, 32 lines an instruction. 384 x 512
// rows x 8 heads: 300 -> 267 us; with a pair bias 512 x 512 x 4 338 -> 317 us (the whole call), 1024 residues 2030 -> 1988. Beside the
// pair bias of heads of 32 there is room for two of its tiles, a ring of their own, and they come one tile after K and V, which a CTA with
// a single short item feels: 4 x 192 rows 20.5 against 22.2 us, 64 residues 28.7 against 30.7. So there, and for narrow heads with a
// pair bias, everything stays in one ring of three. Narrow heads without one have short rows, of which a TMA tile is slow. Heads of 8:
// 256 x 64 rows x 8 25.7 us without the tiles and 27.6 with them, 256 x 128 34.5 and 36.5, but 100 x 256 42.5 and 41.3, 256 x 256 79.5 and 75.8,
// 384 x 512 365 and 336. Heads of 16: 64 x 64 rows x 4 16.0 and 16.5, 256 x 256 x 4 54.0 and 54.6, 300 x 320 x 4 92.8 and 93.9, but with eight items
// or more a CTA 256 x 384 x 8 174.0 and 170.3, 384 x 512 x 8 388 and 381.
template <int D, bool STAGED>
struct Geo {
    static constexpr int ROWS_BYTES = STAGED ? 32 * D * 2 : 0;
    static constexpr int KD = D < 16 ? 16 : D;                // K extent of Q.K^T; TMA zero-fills past D
    static constexpr int ROWB = KD * 2;                       // bytes of a q/k row = swizzle width
    static constexpr int VT_ROWS = (D + 16) / 16 * 16;        // channels, the ones row, zero rows
    static constexpr int Q_BYTES = BM * ROWB, K_BYTES = BN * ROWB, VT_BYTES = VT_ROWS * BN * 2;
    static constexpr int VT_TX = D * BN * 2;                  // bytes TMA writes of a V^T tile
};

template <bool STAGED>
struct RowMaps {                      // [B][S][C], box [D, 32]
    CUtensorMap gate, avg;
};
template <>
struct RowMaps<false> {};

struct AttnParams {
    const __nv_bfloat16 *gate;        // [B, S, H*D]: SPLIT bf16(x.Wg + bg), otherwise bf16(sigmoid(bf16(x.Wg + bg)))
    const __nv_bfloat16 *bias;        // [B, S] (row stride bias_stride0)
    __nv_bfloat16 *avg;               // [B, S, H*D]
    int64_t bias_stride0;
    int *err;
    int S, H, B;
    int G;                            // batch rows per item: 1, 2 or 4
    int n_qt;                         // query tiles per (b, h)
    int n_whole, parts;               // narrow heads: items of G batch rows; each one after them is cut into this many items
    int n_items;
    int nb_head_inner;                // pair-bias tensor map has the dimensions (key, head, query): the heads of a
                                      // query row lie closer together than the rows (a [S, H, S] storage)
    int *counter;                     // [0] next work item of this launch, [1] CTAs that have finished (both zero at
                                      // launch; the last CTA to finish zeroes them again)
    float scale;
};

// SPLIT: 16 bits of P, a bf16 head and a bf16 tail, both multiplied by V^T, for narrow heads and 64-channel layers: heads of 8
// had unrounded probabilities on the CUDA cores, and bf16 ones are less exact against a stale maximum than against the true
// one, where the largest is exactly 1 (error of the layer against 64 bits 1 to 5 % larger; this way 1 % smaller). It costs
// 129 -> 150 us for 256 x 384 rows of 8 heads of 8, 41 -> 49 us for 256 x 256 rows of 4 heads of 16.
// Tails of 16 keys from column tail_col(c, D) on: beside O, and for heads of 32 half of them over logits already read.
__device__ __forceinline__ constexpr int tail_col(int c, int D) { return D < 32 ? 96 + 8 * c : c < 2 ? 112 + 8 * c : 16 + 8 * c; }

template <int D, bool SPLIT, bool HAS_NB, bool STAGED, bool CUT>
__global__ void __launch_bounds__(THREADS, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_vt, const __grid_constant__ CUtensorMap tm_nb,
               const __grid_constant__ RowMaps<STAGED> tm_rows, const AttnParams p)
{
    using T = Geo<D, STAGED>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem_gen = smem_raw + (smem - smem_u32(smem_raw));
    const int G = p.G;
    // shared memory: barriers, Q tiles, rows of the gate, ring of [K x G | V^T x G | pair bias | mask bias]
    const uint32_t off_q = 1024;
    const uint32_t off_rows = off_q + (uint32_t)(G * T::Q_BYTES), off_stage = off_rows + (uint32_t)(G * 4 * T::ROWS_BYTES);
    const uint32_t off_vt = (uint32_t)(G * T::K_BYTES), off_nb = off_vt + (uint32_t)(G * T::VT_BYTES),
                   off_mb = off_nb + (HAS_NB && !STAGED ? NB_BYTES : 0), stage_bytes = off_mb + MB_BYTES;
    auto stage_base = [&](int s) { return smem + off_stage + (uint32_t)s * stage_bytes; };
    auto nb_ring = [&](int g) { return smem + off_stage + NST * stage_bytes + (uint32_t)((g & 1) * NB_BYTES); };     // STAGED
    const uint32_t bar = smem;
    auto kv_full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto kv_empty = [&](int s) { return bar + 8u * (uint32_t)(NST + s); };
    auto s_full = [&](int w) { return bar + 8u * (uint32_t)(2 * NST + w); };
    auto p_full = [&](int w) { return bar + 8u * (uint32_t)(2 * NST + MAXG + w); };
    auto o_full = [&](int w) { return bar + 8u * (uint32_t)(2 * NST + 2 * MAXG + w); };
    const uint32_t q_full = bar + 8u * (2 * NST + 3 * MAXG), q_empty = q_full + 8;
    auto it_full = [&](int i) { return q_full + 16u + 8u * (uint32_t)(i & 3); };      // item number i has been written
    const uint32_t item_ring = q_full + 48u;                                         // four ints
    const uint32_t tmem_slot = q_full + 64u;
    auto g_full = [&](int softmax_warp) { return q_full + 72u + 8u * (uint32_t)softmax_warp; };
    static_assert(8 * (2 * NST + 3 * MAXG) + 72 + 8 * SOFTMAX_WARPS <= BAR_BYTES, "barriers fit their block");

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int S = p.S;
    const int nkt = (S + BN - 1) / BN;
    const int n_mma = min(G, MMA_WARPS);
    // Work items are handed out through an atomic counter in global memory: the producer warp takes the next
    // item number, publishes it to the other roles through a ring of four shared-memory words (one mbarrier each),
    // and publishes -1 when the list is exhausted. Ring depth: the number of item i + 1 is written at the earliest during the loads of
    // item i, once the stage of a tile of that item is free, that is, NST = 3 tiles before it have been consumed. Even where every item has one
    // tile, that was item i - 3, whose number, the last in that slot, every role had read to consume it. There is nothing to spare: an
    // earlier number or a fourth stage needs a longer ring.
    static_assert(NST <= 3, "item numbers in the ring");
    auto rows_of = [&](int w) { return CUT && w >= p.n_whole ? G / p.parts : G; };
    auto decode = [&](int w, int &q0, int &h, int &b0) {
        int sub = 0;
        if (CUT && w >= p.n_whole) {
            const int v = w - p.n_whole;
            sub = v % p.parts * (G / p.parts);
            w = p.n_whole + v / p.parts;
        }
        const int qt = w % p.n_qt, hb = w / p.n_qt;
        q0 = qt * BM;
        h = hb % p.H;
        b0 = hb / p.H * G + sub;
    };
    // item number of this CTA's i-th item, or -1 (bounded wait; -2 on a timeout)
    auto item_of = [&](int i, int code) -> int {
        if (!mbar_wait_warp(it_full(i), (uint32_t)((i >> 2) & 1), p.err, code)) return -2;
        int w;
        asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w) : "r"(item_ring + 4u * (uint32_t)(i & 3)));
        return w;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(kv_full(s), 2);       // the expect_tx arrival of the TMA loads, the mask warp
            mbar_init(kv_empty(s), n_mma);  // each MMA warp's commit after its last P.V^T of the tile
        }
        for (int w = 0; w < MAXG; ++w) {
            mbar_init(s_full(w), 2);        // the products' commit, the issuer's own arrival
            mbar_init(p_full(w), 4);
            mbar_init(o_full(w), 1);
        }
        mbar_init(q_full, 1);
        mbar_init(q_empty, n_mma);
        for (int i = 0; i < 4; ++i) mbar_init(it_full(i), 1);
        for (int i = 0; i < SOFTMAX_WARPS && STAGED; ++i) mbar_init(g_full(i), 1);
        fence_barrier_init();
    }
    // static rows of every V^T tile: row D = 1.0 (row-sum column of O), the rows after it = 0
    constexpr int STATIC_CHUNKS = (T::VT_ROWS - D) * (BN * 2 / 16);
    for (int i = threadIdx.x; i < NST * G * STATIC_CHUNKS; i += THREADS) {
        const int t = i / STATIC_CHUNKS, rem = i % STATIC_CHUNKS, row = D + rem / 8, ch = rem % 8;
        const uint32_t v = row == D ? 0x3F803F80u : 0u;
        uint4 *dst = reinterpret_cast<uint4 *>(smem_gen + off_stage + (t / G) * stage_bytes + off_vt + (t % G) * T::VT_BYTES +
                                               row * 128 + ch * 16);
        *dst = make_uint4(v, v, v, v);
    }
    fence_proxy_async();
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, (uint32_t)(G * WG_COLS));
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0 && elect_one()) {                  // kernel parameters: may be fetched before the predecessor ends
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_vt);
        if (HAS_NB) tma_prefetch_desc(&tm_nb);
        if constexpr (STAGED) {
            tma_prefetch_desc(&tm_rows.gate);
            tma_prefetch_desc(&tm_rows.avg);
        }
    }
    release_successor();
    wait_for_predecessor();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);          // warp-uniform

    if (warp == PRODUCER_WARP) {
        // ================= producer =================
        const uint32_t tx = (uint32_t)(G * (T::K_BYTES + T::VT_TX) + (HAS_NB ? NB_BYTES : 0));
        // number of this CTA's i-th item, published to the other roles
        auto take = [&](int i) -> int {
            int w = 0;
            if (lane == 0) {
                w = atomicAdd(p.counter, 1);
                w = w < p.n_items ? w : -1;
                asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(item_ring + 4u * (uint32_t)(i & 3)), "r"(w) : "memory");
                mbar_arrive(it_full(i));                               // releases the store above
            }
            return __shfl_sync(0xffffffffu, w, 0);
        };
        auto load_q = [&](int i, int q0, int h, int b0) -> bool {
            if (i >= 1 && !mbar_wait_warp(q_empty, (uint32_t)((i - 1) & 1), p.err, 20)) return false;
            if (elect_one()) {
                mbar_arrive_expect_tx(q_full, (uint32_t)(G * T::Q_BYTES));
                tma_load_4d(smem + off_q, &tm_q, q_full, 0, q0, h, b0);
            }
            __syncwarp();
            return true;
        };
        int g = 0;                                      // tiles issued so far (all items)
        bool ok = true;
        int w = take(0);
        int nb_g = -1, nb_k0 = 0, nb_q0 = 0, nb_h = 0;  // the tile whose pair bias has not been asked for
        auto load_nb = [&]() {                          // by the elected lane
            tma_load_3d(nb_ring(nb_g), &tm_nb, kv_full(nb_g % NST), nb_k0, p.nb_head_inner ? nb_h : nb_q0, p.nb_head_inner ? nb_q0 : nb_h);
        };
        for (int i = 0; w >= 0; ++i) {
            int q0, h, b0, next = -1;
            decode(w, q0, h, b0);
            if (!STAGED) ok = load_q(i, q0, h, b0);
            for (int kt = 0; kt < nkt && ok; ++kt, ++g) {
                const int s = g % NST;
                ok = g < NST || mbar_wait_warp(kv_empty(s), (uint32_t)((g / NST - 1) & 1), p.err, 21);
                if (!ok) break;
                const int k0 = kt * BN;
                auto this_nb = [&]() {
                    nb_g = g;
                    nb_k0 = k0;
                    nb_q0 = q0;
                    nb_h = h;
                };
                if (elect_one()) {
                    const uint32_t st = stage_base(s);
                    mbar_arrive_expect_tx(kv_full(s), tx);
                    // K, V^T and Q of batch rows past B are filled with zeros
                    tma_load_4d(st, &tm_k, kv_full(s), 0, k0, h, b0);
                    for (int r = 0; r < G; ++r) tma_load_4d(st + off_vt + r * T::VT_BYTES, &tm_vt, kv_full(s), k0, 0, h, b0 + r);
                    if (HAS_NB && !STAGED) tma_load_3d(st + off_nb, &tm_nb, kv_full(s), k0, p.nb_head_inner ? h : q0, p.nb_head_inner ? q0 : h);
                    // (the stage waited for above belonged to tile g - 3, whose pair bias lay where that of tile g - 1 goes)
                    if (HAS_NB && STAGED && nb_g >= 0) load_nb();
                }
                __syncwarp();
                if (HAS_NB && STAGED) this_nb();
                if (!STAGED) continue;
                // Q after the item's first tile, whose stage is free earlier than the tile of the Q before it
                if (kt == 0) ok = load_q(i, q0, h, b0);
                // The next item's number two tiles before this one's loads end (this tile's stage was free, see above), its Q and first tile on
                // their way to L2.
                if (kt == max(nkt - 2, 0)) {
                    next = take(i + 1);
                    if (next >= 0) {
                        int q1, h1, b1;
                        decode(next, q1, h1, b1);
                        if (elect_one()) {
                            tma_prefetch_4d(&tm_q, 0, q1, h1, b1);
                            tma_prefetch_4d(&tm_k, 0, 0, h1, b1);
                            for (int r = 0; r < G; ++r) tma_prefetch_4d(&tm_vt, 0, 0, h1, b1 + r);
                            if (HAS_NB) tma_prefetch_3d(&tm_nb, 0, p.nb_head_inner ? h1 : q1, p.nb_head_inner ? q1 : h1);
                        }
                        __syncwarp();
                    }
                }
            }
            if (!ok) break;
            w = STAGED ? next : take(i + 1);
        }
        if (HAS_NB && STAGED && ok && nb_g >= 0 &&
            (nb_g < 2 || mbar_wait_warp(kv_empty((nb_g - 2) % NST), (uint32_t)(((nb_g - 2) / NST) & 1), p.err, 19))) {
            if (elect_one()) load_nb();
            __syncwarp();
        }
    } else if (warp == MASK_WARP) {
        // ================= mask bias: fp32 copies of the keys' bias values beside the tile =================
        int g = 0;
        bool ok = true;
        for (int i = 0; ok; ++i) {
            const int w = item_of(i, 35);
            if (w < 0) break;
            int q0, h, b0;
            decode(w, q0, h, b0);
            for (int kt = 0; kt < nkt; ++kt, ++g) {
                const int s = g % NST;
                float mv[2 * MAXG];                    // in flight while the stage drains
#pragma unroll
                for (int r = 0; r < MAXG; ++r)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int key = kt * BN + lane + 32 * j;
                        mv[2 * r + j] = r < G && key < S
                                            ? __bfloat162float(p.bias[(int64_t)min(b0 + r, p.B - 1) * p.bias_stride0 + key])
                                            : -INFINITY;
                    }
                if (g >= NST && !mbar_wait_warp(kv_empty(s), (uint32_t)((g / NST - 1) & 1), p.err, 36)) {
                    ok = false;
                    break;
                }
                float *mb = reinterpret_cast<float *>(smem_gen + (stage_base(s) - smem) + off_mb);
#pragma unroll
                for (int r = 0; r < MAXG; ++r)
                    if (r < G) {
                        mb[r * BN + lane] = mv[2 * r];
                        mb[r * BN + lane + 32] = mv[2 * r + 1];
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive(kv_full(s));
            }
        }
    } else if (warp >= MMA_WARP) {
        // ================= MMA issuer =================
        const int w0 = warp - MMA_WARP;                  // this warp's groups: w0, w0 + 2
        constexpr uint32_t idesc_s = make_instr_desc_bf16(BM, BN);
        constexpr uint32_t idesc_o = make_instr_desc_bf16(BM, T::VT_ROWS);
        auto issue_qk = [&](int s, int w) {
            if (elect_one()) {
                const uint32_t kb = stage_base(s) + w * T::K_BYTES, qb = smem + off_q + w * T::Q_BYTES;
#pragma unroll
                for (int k = 0; k < T::KD / 16; ++k)
                    tc_mma_bf16(tmem_base + w * WG_COLS + S_COL, make_smem_desc_kmajor(qb + k * 32, T::ROWB),
                                make_smem_desc_kmajor(kb + k * 32, T::ROWB), idesc_s, k > 0 ? 1u : 0u);
                tc_commit(s_full(w));
                // The softmax warps read the tile's pair bias and mask bias, which this thread has seen arrive (kv_full): an
                // arrival of its own passes that on, a commit answers only for the tensor core. (A second wait in the
                // softmax warps would cost 1.5 %.)
                mbar_arrive(s_full(w));
            }
            __syncwarp();
        };
        // stage of tile g has landed (and, for the first tile of item i, Q)
        auto wait_loads = [&](int g, int i, bool first) -> bool {
            if (first && !mbar_wait_warp(q_full, (uint32_t)(i & 1), p.err, 22)) return false;
            if (!mbar_wait_warp(kv_full(g % NST), (uint32_t)((g / NST) & 1), p.err, 23)) return false;
            tc_fence_after();
            return true;
        };
        bool more = w0 < G && item_of(0, 32) >= 0;                 // this role needs only to know whether an item exists
        bool ok = true;
        if (more) {
            ok = wait_loads(0, 0, true);
            for (int w = w0; w < G; w += MMA_WARPS)
                if (ok) issue_qk(0, w);
            if (ok && nkt == 1 && elect_one()) tc_commit(q_empty);
        }
        int g = 0;
        for (int i = 0; more && ok; ++i) {
            for (int kt = 0; kt < nkt && ok; ++kt, ++g) {
                const int s = g % NST;
                const bool last = kt == nkt - 1;
                bool next = true;                         // is there a tile g + 1 (possibly of the next item)?
                if (last) {
                    const int nxt = item_of(i + 1, 33);
                    ok = nxt != -2;
                    next = more = nxt >= 0;
                }
                for (int w = w0; w < G; w += MMA_WARPS) {
                    const bool last_w = w + MMA_WARPS >= G;
                    if (!mbar_wait_warp(p_full(w), (uint32_t)(g & 1), p.err, 25)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t vb = stage_base(s) + off_vt + w * T::VT_BYTES, t0 = tmem_base + w * WG_COLS;
#pragma unroll
                        for (int part = SPLIT ? 0 : 1; part < 2; ++part)            // tails, heads
#pragma unroll
                            for (int k = 0; k < BN / 16; ++k)
                                tc_mma_bf16_ts(t0 + O_COL, t0 + (part == 0 ? tail_col(k, D) : S_COL + k * 8),
                                               make_smem_desc_kmajor(vb + k * 32, 128), idesc_o,
                                               (kt > 0 || k > 0 || (SPLIT && part > 0)) ? 1u : 0u);
                        if (last) tc_commit(o_full(w));
                        if (last_w) tc_commit(kv_empty(s));
                    }
                    __syncwarp();
                    // the next logits overwrite P: the tensor core runs the products in the order they are issued
                    if (next) {
                        if (w == w0 && !wait_loads(g + 1, i + 1, last)) {
                            ok = false;
                            break;
                        }
                        issue_qk((g + 1) % NST, w);
                        // the last Q.K^T of an item frees Q
                        if (last_w && (last ? nkt == 1 : kt + 1 == nkt - 1) && elect_one()) tc_commit(q_empty);
                    }
                }
            }
        }
    } else if ((warp >> 2) < G) {
        // ================= softmax / epilogue =================
        const int wg = warp >> 2, quad = warp & 3;       // TMEM lanes 32*quad .. 32*quad+31
        const int row = quad * 32 + lane;                // query row inside the tile
        const uint32_t t_s = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(wg * WG_COLS + S_COL);
        const uint32_t t_o = t_s - S_COL + O_COL;
        const uint64_t scale2 = pack_f32x2(p.scale, p.scale), log2e2 = pack_f32x2(kLog2e, kLog2e);
        const uint32_t nb_row = (STAGED ? 0u : off_nb) + (uint32_t)row * 128 + (uint32_t)((row & 7) << 4);   // chunk c lies at ^ (c << 4)
        const uint32_t mb_row = off_mb + (uint32_t)wg * BN * 4;
        // Running (possibly stale) max of x, at least the lowest finite number: keys masked with -inf then weigh nothing, and
        // a row whose first keys are all of that kind is raised by its first finite one. P = 2^(x * log2e + mneg); the
        // rounding of mneg is the same for all of a row's keys and cancels in the division, and O is rescaled by the
        // difference of the very mneg that P was formed with. Past kFar that rounding would leave the range of the
        // exponential: such rows (masked with the type's lowest value, or masked twice) take x - m first.
        float m = 0.f, mneg = 0.f;
        float limit = 0.f;                               // x above it needs a new max; NaN (always) for a far row
        bool ok = true;
        auto far_row = [&]() { return !(fabsf(mneg) < kFar); };
        auto set_max = [&](float v) {
            m = fmaxf(v, -FLT_MAX);
            mneg = -__fmul_rn(m, kLog2e);
            limit = far_row() ? __int_as_float(0x7fffffff) : m + kRescaleThreshold;
        };

        // one tile of the softmax: global tile g, tile kt of its item
        auto do_tile = [&](const int g, const int kt) -> bool {
            const uint32_t st = stage_base(g % NST);
            if (!mbar_wait_warp(s_full(wg), (uint32_t)(g & 1), p.err, 26)) return false;
            tc_fence_after();
            uint32_t pk[32], late[2][8];              // late: tails of keys 32..63 for heads of 32
            float tmax;
            bool stored = false;                      // P is already in tensor memory
            // x = bf16(logit) * scale + bias (+ pair bias) of the pair of keys 2j, 2j + 1 of a 16-key piece
            struct Piece {
                float mb[16];
                uint32_t nb[8];
            };
            auto fetch = [&](Piece &f, const int c) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v = lds128_f32(st + mb_row + c * 64 + i * 16);
                    f.mb[4 * i] = v.x;
                    f.mb[4 * i + 1] = v.y;
                    f.mb[4 * i + 2] = v.z;
                    f.mb[4 * i + 3] = v.w;
                }
                if (HAS_NB) {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(f.nb[4 * i]), "=r"(f.nb[4 * i + 1]), "=r"(f.nb[4 * i + 2]), "=r"(f.nb[4 * i + 3])
                                     : "r"(((STAGED ? nb_ring(g) : st) + nb_row) ^ (uint32_t)((2 * c + i) << 4)));
                }
            };
            auto x_pair = [&](const uint32_t (&r)[16], const Piece &f, const int j) -> uint64_t {
                uint64_t x2 = fma_f32x2(pack_f32x2(round_to_bf16_f32(__uint_as_float(r[2 * j])),
                                                   round_to_bf16_f32(__uint_as_float(r[2 * j + 1]))),
                                        scale2, pack_f32x2(f.mb[2 * j], f.mb[2 * j + 1]));
                if (HAS_NB) x2 = add_f32x2(x2, pack_f32x2(bf16lo_to_f32(f.nb[j]), bf16hi_to_f32(f.nb[j])));
                return x2;
            };
            auto prob = [&](const float e0, const float e1, uint32_t &hi, uint32_t &lo) {
                const float p0 = ex2_approx(e0), p1 = ex2_approx(e1);
                hi = pack_bf16x2(p0, p1);
                if (SPLIT) lo = pack_bf16x2(p0 - bf16lo_to_f32(hi), p1 - bf16hi_to_f32(hi));
            };
            auto piece = [&](const uint32_t (&r)[16], const int c) {
                Piece f;
                uint32_t lo[8];
                fetch(f, c);
                const uint64_t mneg2 = pack_f32x2(mneg, mneg);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint64_t x2 = x_pair(r, f, j);
                    float x0, x1, e0, e1;
                    unpack_f32x2(x2, x0, x1);
                    tmax = fmax3(tmax, x0, x1);
                    unpack_f32x2(fma_f32x2(x2, log2e2, mneg2), e0, e1);
                    prob(e0, e1, pk[c * 8 + j], lo[j]);
                }
                if (SPLIT && (D < 32 || c < 2)) tmem_st_32x8(t_s - S_COL + tail_col(c, D), lo);
                if (SPLIT && D == 32 && c >= 2) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) late[c & 1][j] = lo[j];
                }
            };
            for (int pass = 0; pass < 2; ++pass) {
                uint32_t a[16], b[16];
                tmax = -INFINITY;
                tmem_ld_32x16(t_s, a);
                tmem_ld_wait16(a);
                if (kt == 0 && pass == 0) {
                    // first tile of an item: the max of its first 16 keys (key 0 always exists)
                    Piece f;
                    fetch(f, 0);
                    float mx = -INFINITY;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float x0, x1;
                        unpack_f32x2(x_pair(a, f, j), x0, x1);
                        mx = fmax3(mx, x0, x1);
                    }
                    set_max(mx);
                }
                tmem_ld_32x16(t_s + 16, b);
                piece(a, 0);
                tmem_ld_wait16(b);
                tmem_ld_32x16(t_s + 32, a);
                piece(b, 1);
                tmem_ld_wait16(a);
                tmem_ld_32x16(t_s + 48, b);
                piece(a, 2);
                tmem_ld_wait16(b);
                piece(b, 3);
                if (!__any_sync(0xffffffffu, !(tmax <= limit))) break;
                // rare: the max of some row grew past the threshold. Rescale those rows of O (and their row sums) and form
                // the tile again against the new max. The product of the previous tile has retired: it was issued
                // before the logits of this one.
                if (SPLIT) tmem_st_wait();
                const bool grow = tmax > m + kRescaleThreshold;
                float f = 1.0f;
                if (grow) {
                    const bool was_far = far_row();
                    const float m_old = m, mneg_old = mneg;
                    set_max(tmax);
                    f = ex2_approx(was_far || far_row() ? (m_old - m) * kLog2e : mneg - mneg_old);
                }
                if (kt > 0 && __any_sync(0xffffffffu, grow)) {
                    constexpr int OC = D < 16 ? 16 : D;
#pragma unroll
                    for (int c = 0; c <= OC; c += 16) {
                        uint32_t o[16];
                        if (c < OC) {
                            tmem_ld_32x16(t_o + c, o);
                            tmem_ld_wait16(o);
#pragma unroll
                            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                            tmem_st_32x16(t_o + c, o);
                        } else if (D >= 16) {
                            const uint32_t osum = tmem_ld_32x1(t_o + D);
                            tmem_ld_wait();
                            tmem_st_32x1(t_o + D, __float_as_uint(__uint_as_float(osum) * f));
                        }
                    }
                    tmem_st_wait();
                }
                if (__any_sync(0xffffffffu, far_row())) {
                    // piece by piece, P over logits already read (a loop, so that the usual path stays short)
                    const float sub = far_row() ? -m : 0.f, add = far_row() ? 0.f : mneg;
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        Piece pc;
                        uint32_t hi[8], lo[8];
                        fetch(pc, c);
                        tmem_ld_32x16(t_s + c * 16, a);
                        tmem_ld_wait16(a);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float e0, e1;
                            unpack_f32x2(fma_f32x2(add_f32x2(x_pair(a, pc, j), pack_f32x2(sub, sub)), log2e2, pack_f32x2(add, add)), e0, e1);
                            prob(e0, e1, hi[j], lo[j]);
                        }
                        tmem_st_32x8(t_s + c * 8, hi);
                        if (SPLIT) tmem_st_32x8(t_s - S_COL + tail_col(c, D), lo);
                    }
                    stored = true;
                    break;
                }
            }
            if (!stored) {
                tmem_st_32x32(t_s, pk);
                if (SPLIT && D == 32) {
                    tmem_st_32x8(t_s - S_COL + tail_col(2, D), late[0]);
                    tmem_st_32x8(t_s - S_COL + tail_col(3, D), late[1]);
                }
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(wg));
            return true;
        };

        const uint32_t rows = smem + off_rows + (uint32_t)(warp * T::ROWS_BYTES);
        uint32_t gates = 0, gate_loads = 0;              // tiles of gate rows waited for, and asked for
        int g = 0;
        for (int i = 0; ok; ++i) {
            const int w = item_of(i, 34);
            if (w < 0) break;
            int q0, h, b0;
            decode(w, q0, h, b0);
            if constexpr (STAGED) {
                const bool any = q0 + quad * 32 < S && b0 + wg < p.B && (!CUT || wg < rows_of(w));
                gate_loads += any ? 1u : 0u;
                if (any && lane == 0) {
                    tma_store_wait_read<0>();
                    mbar_arrive_expect_tx(g_full(warp), (uint32_t)T::ROWS_BYTES);
                    tma_load_3d(rows, &tm_rows.gate, g_full(warp), h * D, q0 + quad * 32, b0 + wg);
                }
                __syncwarp();
            }
            const bool mine = !CUT || wg < rows_of(w);
            if (mine) {
                for (int kt = 0; kt < nkt && ok; ++kt, ++g) ok = do_tile(g, kt);
            } else {                                     // a cut item has no row for this group, which only passes on the barriers
                for (int kt = 0; kt < nkt && ok; ++kt, ++g) {
                    ok = mbar_wait_warp(s_full(wg), (uint32_t)(g & 1), p.err, 26);
                    tc_fence_before();
                    if (ok && lane == 0) mbar_arrive(p_full(wg));
                }
            }
            if (!ok) break;

            // ---- item epilogue: one row of D channels per thread ----
            const int qi = q0 + row, bb = b0 + wg;
            const bool live = mine && bb < p.B && (STAGED ? q0 + quad * 32 < S : qi < S);      // (STAGED: the warp has a row)
            const int64_t base = live && !STAGED ? ((int64_t)bb * S + qi) * (p.H * D) + h * D : 0;
            uint4 gv[D / 8];
#pragma unroll
            for (int c = 0; c < D / 8 && !STAGED; ++c) gv[c] = __ldg(reinterpret_cast<const uint4 *>(p.gate + base) + c);   // in flight
            if (!mbar_wait_warp(o_full(wg), (uint32_t)(i & 1), p.err, 29)) break;
            tc_fence_after();
            uint32_t o[D < 16 ? 16 : D], osum;
            if constexpr (D == 32) {
                tmem_ld_32x32(t_o, o);
                osum = tmem_ld_32x1(t_o + D);
            } else {
                tmem_ld_32x16(t_o, o);
                osum = D == 16 ? tmem_ld_32x1(t_o + D) : 0;
            }
            tmem_ld_wait();
            if (D < 16) osum = o[D];
            const float inv = 1.0f / __uint_as_float(osum);
            if (live) {
                if (STAGED && !mbar_wait_warp(g_full(warp), gates++ & 1u, p.err, 30)) break;
#pragma unroll
                for (int c = 0; c < D / 8; ++c) {
                    // chunk c of this thread's row, in the swizzle of the tensor map
                    const uint32_t at = rows + (uint32_t)(lane * (D * 2) + ((c ^ (D == 32 ? (lane >> 1) & 3 : D == 16 ? (lane >> 2) & 1 : 0)) << 4));
                    if (STAGED)
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(gv[c].x), "=r"(gv[c].y), "=r"(gv[c].z), "=r"(gv[c].w)
                                     : "r"(at));
                    const uint32_t gw[4] = {gv[c].x, gv[c].y, gv[c].z, gv[c].w};
                    uint32_t ow[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        // the weighted average is stored as bf16 before gating in the reference (:128-133)
                        const int e = c * 8 + 2 * j;
                        const uint32_t wa = pack_bf16x2(__uint_as_float(o[e]) * inv, __uint_as_float(o[e + 1]) * inv);
                        float s0 = bf16lo_to_f32(gw[j]), s1 = bf16hi_to_f32(gw[j]);
                        if (SPLIT) {
                            s0 = __fdividef(1.0f, 1.0f + ex2_approx(-s0 * kLog2e));
                            s1 = __fdividef(1.0f, 1.0f + ex2_approx(-s1 * kLog2e));
                        }
                        ow[j] = pack_bf16x2(bf16lo_to_f32(wa) * s0, bf16hi_to_f32(wa) * s1);
                    }
                    if (STAGED)
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(at), "r"(ow[0]), "r"(ow[1]), "r"(ow[2]), "r"(ow[3]) : "memory");
                    else
                        *(reinterpret_cast<uint4 *>(p.avg + base) + c) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                }
                if constexpr (STAGED) {
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {                     // rows past S are clipped
                        tma_store_3d(&tm_rows.avg, rows, h * D, q0 + quad * 32, bb);
                        tma_store_commit();
                    }
                }
            }
        }
        if (STAGED) {
            // after a wait that ran out: no copy may still be on its way when the CTA exits
            if (gates != gate_loads) mbar_wait_warp(g_full(warp), gates & 1u, p.err, 31);
            if (lane == 0) tma_store_wait<0>();
        }
    }

    // ================= common tail =================
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)(G * WG_COLS));
    }
    // The last CTA to get here puts the work counter back to zero for the launch that uses it next (every CTA has
    // taken its last item number by now: the producer's atomics precede the barrier above).
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

template <int D, bool HAS_NB, bool STAGED>
int smem_bytes(int G)
{
    using T = Geo<D, STAGED>;
    return 1024 + 1024 + G * (T::Q_BYTES + 4 * T::ROWS_BYTES) + NST * (G * (T::K_BYTES + T::VT_BYTES) + MB_BYTES) +
           (!HAS_NB ? 0 : STAGED ? 2 : NST) * NB_BYTES;
}

template <int D, bool SPLIT, bool HAS_NB, bool STAGED, bool CUT = false>
bool launch_one(cudaStream_t stream, const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tvt,
                const CUtensorMap &tnb, const RowMaps<STAGED> &rows, const AttnParams &p)
{
    if constexpr (D < 32 && !CUT)
        if (p.parts > 1) return launch_one<D, SPLIT, HAS_NB, STAGED, true>(stream, tq, tk, tvt, tnb, rows, p);
    static bool configured = false;
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(attn_tc_kernel<D, SPLIT, HAS_NB, STAGED, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes<D, HAS_NB, STAGED>(MAXG)));
        configured = true;
    }
    const unsigned grid = (unsigned)std::min<int64_t>(p.n_items, std::max(1, sm_count() - runtime().sm_margin));
    AttnParams q = p;
    q.counter = work_counter(stream);
    if (q.counter == nullptr) return false;
    KernelTimer timer__("attn_core", stream);
    launch_chained(attn_tc_kernel<D, SPLIT, HAS_NB, STAGED, CUT>, grid, THREADS, smem_bytes<D, HAS_NB, STAGED>(p.G), stream, tq, tk, tvt, tnb, rows, q);
    count_launch();
    return true;
}

// How the work is cut into items. More batch rows per CTA overlap more chains and share the pair-bias tile, fewer rows spread a
// small problem over more SMs: the choice minimises waves x (relative time of an item with that many rows). Measured per full wave
// against one row, at 128, 256, 384 and 1024 positions: four rows 2.4 (with pair bias 3.2), 2.3, 2.1, 1.8 with heads of 32, 1.4 to
// 2.1 with narrower ones; two rows 1.3 to 1.6 and 1.0 to 1.5. Narrow heads: what is left for the last wave is cut into items of two
// or one batch rows where that ends sooner: 256 x 256 rows of 4 heads of 16, the whole call, 63.7 -> 62.5 us (with heads of 32 the
// kernel that can do this lost 1 to 3 % and gained nothing; narrow ones whose items stay whole run without it, 85 x 85 rows of 4
// heads of 16 24.4 against 24.1 us; without a full wave before them fewer rows for all items do the same for less, 64 x 64 rows 19.6
// against 18.9 us, 16 x 48 rows of 8 heads of 8 18.9 against 18.4).
void plan_items(AttnParams &p, int64_t sms, bool cut)
{
    const int groups[3] = {4, 2, 1};
    const double t[3] = {2.03, 1.36, 1.0};
    double best = 1e30;
    for (int i = 0; i < 3; ++i) {
        const int64_t items = (int64_t)(p.B + groups[i] - 1) / groups[i] * p.H * p.n_qt, whole = items / sms * sms, last = items - whole;
        for (int j = i; j < (cut && whole > 0 ? 3 : i + 1); ++j) {
            const int parts = groups[i] / groups[j];
            const double cost = (double)(whole / sms) * t[i] + (double)((last * parts + sms - 1) / sms) * t[j];
            if (cost < (j > i ? best * 0.99 : best)) {
                best = cost;
                p.G = groups[i];
                p.parts = parts;
                p.n_whole = (int)(parts == 1 ? items : whole);
                p.n_items = (int)(parts == 1 ? items : whole + last * parts);
            }
        }
    }
}

template <int D, bool SPLIT>
bool launch_d(cudaStream_t stream, const void *q, const void *k, const void *vt, int64_t vt_pitch, const void *nb,
              int64_t nb_stride_h, int64_t nb_stride_q, AttnParams &p)
{
    using T = Geo<D, true>;
    const uint64_t Su = (uint64_t)p.S;
    CUtensorMap tq, tk, tvt, tnb;
    const uint64_t H = (uint64_t)p.H, B = (uint64_t)p.B, vp = (uint64_t)vt_pitch;
    const uint32_t G = (uint32_t)p.G;
    if (!make_tensor_map_bf16_4d(&tq, q, D, Su, H, B, D, Su * D, Su * D * H, T::KD, BM, G, T::ROWB)) return false;
    if (!make_tensor_map_bf16_4d(&tk, k, D, Su, H, B, D, Su * D, Su * D * H, T::KD, BN, G, T::ROWB)) return false;
    if (!make_tensor_map_bf16_4d(&tvt, vt, Su, D, H, B, vp, D * vp, D * vp * H, BN, D, 1, 128)) return false;
    // where the items are long, or many (see Geo)
    const int64_t sms = std::max(1, sm_count() - runtime().sm_margin);
    const bool staged = D == 32 ? !nb || p.n_items > sms : !nb && p.S > 3 * BN && (D == 8 || p.n_items >= 8 * sms);
    RowMaps<true> rows;
    if (staged) {
        const int swizzle = D == 8 ? 0 : D * 2;
        if (!make_tensor_map_bf16_3d(&rows.gate, p.gate, H * D, Su, B, H * D, Su * H * D, D, 32, swizzle) ||
            !make_tensor_map_bf16_3d(&rows.avg, p.avg, H * D, Su, B, H * D, Su * H * D, D, 32, swizzle))
            return false;
    }
    p.nb_head_inner = 0;
    if (nb) {
        if (nb_stride_h < nb_stride_q) {
            // heads closer together than query rows: dimensions in the order of their strides (key, head, query); the
            // box takes one head, so the tile in shared memory is the same 128 rows x 64 keys
            p.nb_head_inner = 1;
            if (!make_tensor_map_bf16_3d(&tnb, nb, Su, (uint64_t)p.H, Su, (uint64_t)nb_stride_h, (uint64_t)nb_stride_q, BN, 1,
                                         128, BM))
                return false;
        } else if (!make_tensor_map_bf16_3d(&tnb, nb, Su, Su, (uint64_t)p.H, (uint64_t)nb_stride_q, (uint64_t)nb_stride_h, BN,
                                            BM, 128)) {
            return false;
        }
        if constexpr (D == 32) {
            if (staged) return launch_one<D, SPLIT, true, true>(stream, tq, tk, tvt, tnb, rows, p);
        }
        return launch_one<D, SPLIT, true, false>(stream, tq, tk, tvt, tnb, RowMaps<false>{}, p);
    }
    tnb = tk;
    if constexpr (D < 32) {
        if (!staged) return launch_one<D, SPLIT, false, false>(stream, tq, tk, tvt, tnb, RowMaps<false>{}, p);
    }
    return launch_one<D, SPLIT, false, true>(stream, tq, tk, tvt, tnb, rows, p);
}

}  // namespace

bool tcgen05_attn_core_bf16(cudaStream_t stream, const void *q, const void *k, const void *vt, int64_t vt_pitch,
                            const void *gate, const void *bias, int64_t bias_stride0, const void *nb,
                            int64_t nb_stride_h, int64_t nb_stride_q, void *avg, int B, int S, int H, int D,
                            float scale, bool gate_is_sigmoid)
{
    if ((D != 8 && D != 16 && D != 32) || (gate_is_sigmoid && D != 32) || vt_pitch % 8 != 0) return false;
    if (nb && ((nb_stride_h % 8) || (nb_stride_q % 8) || ((uintptr_t)nb % 16))) return false;
    if ((((uintptr_t)gate | (uintptr_t)avg) & 15u) != 0) return false;
    const int64_t n_qt = (S + BM - 1) / BM;
    if (n_qt * H * B > INT32_MAX / 2) return false;          // work items are counted in 32 bits
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    AttnParams p;
    p.gate = (const __nv_bfloat16 *)gate;
    p.bias = (const __nv_bfloat16 *)bias;
    p.avg = (__nv_bfloat16 *)avg;
    p.bias_stride0 = bias_stride0;
    p.err = ew.device;
    p.S = S;
    p.H = H;
    p.B = B;
    p.n_qt = (int)n_qt;
    plan_items(p, std::max(1, sm_count() - runtime().sm_margin), D < 32);
    p.scale = scale;
    p.counter = nullptr;
    switch (D) {
        case 8: return launch_d<8, true>(stream, q, k, vt, vt_pitch, nb, nb_stride_h, nb_stride_q, p);
        case 16: return launch_d<16, true>(stream, q, k, vt, vt_pitch, nb, nb_stride_h, nb_stride_q, p);
        default:
            return gate_is_sigmoid ? launch_d<32, false>(stream, q, k, vt, vt_pitch, nb, nb_stride_h, nb_stride_q, p)
                                   : launch_d<32, true>(stream, q, k, vt, vt_pitch, nb, nb_stride_h, nb_stride_q, p);
    }
}

}  // namespace dev
}  // namespace kutacc
