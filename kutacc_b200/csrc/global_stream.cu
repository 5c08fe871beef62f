// Extra-MSA global column attention as three streaming kernels (64 channels, 8 heads x 8).
//
// Reference path: src/attention/global_attention.cpp:30-164. A column's query needs the masked mean of all its rows, its
// output needs the softmax over all its rows: two passes over x that nothing can join. A single kernel that holds each
// column in the shared memory of a thread-block cluster reads x once, but its stages (pool, exchange, softmax, exchange,
// output) run one after another with two columns per SM, and it is bound by that chain: 235 us at 384 x 5120 rows where
// its bytes take 77 (163 us here). Here every stage is a stream with enough independent work in flight:
//   kv    x once: masked partial sums of every 32 or 64 rows, k = x.Wk^T and v = x.Wv^T (bf16, 32 bytes per row)        (:44-89)
//   core  one CTA per column: q from the partial sums, logits, softmax, weighted v from k and v                      (:76-133)
//   out   x again, last rows first (what the kv kernel read last is still in L2): gate, gated average, output     (:90-94, :134-163)
// Rows of a column are split by S alone, so a column's result does not depend on the batch it is in.
//
// bf16 rounding points of the reference that are kept: q_avg, q, k, v, logits, wa, gate, gated gate, out. Probabilities are
// rounded to bf16 un-normalised (they feed the tensor cores); the reference rounds them after normalising.
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

constexpr int C = 64, H = 8, D = 8;
constexpr int REC_BYTES = 512 + 512 + 64;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int POOL_PITCH = C + 4;            // floats per partial sum: 64 channels, the mask sum, padding

__device__ __forceinline__ float rbf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float bits_to_f32(unsigned short b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint4 lds128_u32(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void mma_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}

struct StreamArgs {
    const __nv_bfloat16 *x;                  // [B, S, 64]
    const unsigned short *mask;              // [B, S] bf16 bits
    const __nv_bfloat16 *wq, *wk, *wv;
    // k, v and mask of every 32 rows (8 j + r) as one record, in the order in which the softmax kernel's lanes take them:
    //   k    [row r = g][channels 2t, 2t+1][j]   512 bytes
    //   v    [channel g][rows r = 2t, 2t+1][j]   512 bytes
    //   mask [t][j][rows r = 2t, 2t+1]            64 bytes; -inf past the last row
    unsigned char *rec;                      // [B, nrec][REC_BYTES]
    float *pool;                             // [B, chunks, POOL_PITCH]
    float *hwa;                              // [B, 64]: weighted average / 2
    int B, S, nrec;                          // nrec: records per column
    int chunk_rows, chunks;                  // rows per partial sum (32 or 64) and their number per column
    int keep_from;                           // units from here on should stay in L2 for the out kernel
    int *err;
};

// ---- kv: a warp streams one chunk after another, 16 rows per step -----------------------------------------------------
// 16 rows are 2 KB of consecutive memory: one bulk copy into the warp's own ring of shared-memory slots, issued NS steps ahead
// (192 KB of ring per SM without a register held for it; with the rows in registers, one step ahead, 76 us at 384 x 5120
// rows). Lane (g, t) takes channels 8t..8t+7 and 32+8t..32+8t+7 of rows g and g + 8. The products sum over the channels in
// whatever order both operands agree on: k step ks takes channels 32 (ks / 2) + 8 t + 4 (ks % 2) .. + 3 of lane t, and the
// weights are held in that order. Bound by HBM: 251 MB in, 71 MB out at that shape, 57 us.
constexpr int KV_WARPS = 8, NS = 6, STEP_BYTES = 16 * C * 2;
constexpr int KV_SMEM = KV_WARPS * NS * (STEP_BYTES + 8);

__global__ void __launch_bounds__(KV_WARPS * 32, 2) global_kv_kernel(const StreamArgs a)
{
    extern __shared__ __align__(128) unsigned char kv_smem[];
    release_successor();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nwarps = gridDim.x * KV_WARPS, units = a.B * a.chunks;
    const uint32_t slots = smem_u32(kv_smem) + (uint32_t)(warp * NS * STEP_BYTES);
    const uint32_t bars = smem_u32(kv_smem) + (uint32_t)(KV_WARPS * NS * STEP_BYTES + warp * NS * 8);
    if (lane == 0) {
        for (int i = 0; i < NS; ++i) mbar_init(bars + 8 * i, 1);
        fence_barrier_init();
    }
    __syncwarp();
    wait_for_predecessor();
    uint32_t wk[4][2], wv[4][2];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const int ch = (ks >> 1) * 32 + 8 * t + (ks & 1) * 4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            wk[ks][i] = *reinterpret_cast<const uint32_t *>(a.wk + g * C + ch + 2 * i);
            wv[ks][i] = *reinterpret_cast<const uint32_t *>(a.wv + g * C + ch + 2 * i);
        }
    }
    const int u0 = blockIdx.x * KV_WARPS + warp;
    auto rows_of = [&](int c) { return min(a.chunk_rows, a.S - c * a.chunk_rows); };

    // the copies run ahead of the work: unit, its first row and rows, row within it
    const uint64_t first = l2_evict_first(), normal = l2_evict_normal();
    int iu = u0, ir = 0, irows = 0, issued = 0;
    int64_t irow = 0;
    auto enter_issue = [&]() {
        if (iu < units) {
            const int c = iu % a.chunks;
            irow = (int64_t)(iu / a.chunks) * a.S + c * a.chunk_rows;
            irows = rows_of(c);
            ir = 0;
        }
    };
    auto issue = [&]() {                     // the next step's copy (whole warp, lane 0 acts)
        if (iu >= units) return;
        if (lane == 0) {
            const uint32_t slot = (uint32_t)(issued % NS), bytes = (uint32_t)min(16, irows - ir) * (C * 2);
            mbar_arrive_expect_tx(bars + 8 * slot, bytes);
            bulk_load(slots + slot * STEP_BYTES, a.x + (irow + ir) * C, bytes, bars + 8 * slot, iu < a.keep_from ? first : normal);
        }
        ++issued;
        ir += 16;
        if (ir >= irows) {
            iu += nwarps;
            enter_issue();
        }
    };
    enter_issue();
    for (int i = 0; i < NS; ++i) issue();

    // a chunk's mask: row lane + 32 i of the chunk, the next chunk's on its way
    unsigned short mk[2], mk_next[2];
    auto load_mask = [&](int u) {
        if (u >= units) return;
        const int c = u % a.chunks, rows = rows_of(c);
        const unsigned short *mp = a.mask + (int64_t)(u / a.chunks) * a.S + c * a.chunk_rows;
#pragma unroll
        for (int i = 0; i < 2; ++i) mk_next[i] = lane + 32 * i < rows ? __ldg(mp + lane + 32 * i) : (unsigned short)0;
    };
    load_mask(u0);
    bool ok = true;
    int step = 0;
    for (int u = u0; u < units && ok; u += nwarps) {
        const int b = u / a.chunks, c = u % a.chunks, rows = rows_of(c);
        unsigned char *rec = a.rec + ((int64_t)b * a.nrec + c * (a.chunk_rows / 32)) * REC_BYTES;    // the chunk's first record
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mk[i] = mk_next[i];
            if (32 * i < rows)
                reinterpret_cast<unsigned short *>(rec + i * REC_BYTES + 1024)[(((lane & 7) >> 1) * 4 + (lane >> 3)) * 2 + (lane & 1)] =
                    lane + 32 * i < rows ? mk[i] : (unsigned short)0xFF80;
        }
        load_mask(u + nwarps);
        float acc[16], msum = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        uint32_t kw[2] = {0, 0}, vw[2] = {0, 0};                         // of the record's first 16 rows
        for (int r = 0; r < (rows + 31) / 32 * 32; r += 16) {
            uint4 x[2][2] = {};
            if (r < rows) {
                const uint32_t slot = (uint32_t)(step % NS);
                ok = mbar_wait_warp(bars + 8 * slot, (uint32_t)((step / NS) & 1), a.err, 97);
                if (!ok) break;
                ++step;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf)
                        x[i][hf] = lds128_u32(slots + slot * STEP_BYTES + (uint32_t)((g + 8 * i) * 128 + hf * 64 + t * 16));
                if (r + 16 > rows) {         // rows past the end hold what was in the slot before
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        if (r + g + 8 * i >= rows) x[i][0] = x[i][1] = make_uint4(0, 0, 0, 0);
                }
                __syncwarp();
                issue();                     // refills this slot
            }
            const unsigned mw = r < 32 ? mk[0] : mk[1];
            const float m0 = bits_to_f32((unsigned short)__shfl_sync(0xffffffffu, mw, (r & 31) + g));
            const float m1 = bits_to_f32((unsigned short)__shfl_sync(0xffffffffu, mw, (r & 31) + g + 8));
            float kacc[4] = {0.f, 0.f, 0.f, 0.f}, v0[4] = {0.f, 0.f, 0.f, 0.f}, v1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const uint32_t w0[4] = {x[0][hf].x, x[0][hf].y, x[0][hf].z, x[0][hf].w};
                const uint32_t w1[4] = {x[1][hf].x, x[1][hf].y, x[1][hf].z, x[1][hf].w};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int ks = hf * 2 + q;
                    const uint32_t af[4] = {w0[2 * q], w1[2 * q], w0[2 * q + 1], w1[2 * q + 1]};
                    const uint32_t wvf[4] = {wv[ks][0], 0u, wv[ks][1], 0u};
                    mma_bf16_16816(kacc, af, wk[ks][0], wk[ks][1]);
                    mma_bf16_16816(v0, wvf, af[0], af[2]);               // v^T of rows 0..7
                    mma_bf16_16816(v1, wvf, af[1], af[3]);               // rows 8..15
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[hf * 8 + 2 * e] = fmaf(bf16lo_to_f32(w1[e]), m1, fmaf(bf16lo_to_f32(w0[e]), m0, acc[hf * 8 + 2 * e]));
                    acc[hf * 8 + 2 * e + 1] = fmaf(bf16hi_to_f32(w1[e]), m1, fmaf(bf16hi_to_f32(w0[e]), m0, acc[hf * 8 + 2 * e + 1]));
                }
            }
            msum += m0 + m1;
            const uint32_t k0 = pack_bf16x2(kacc[0], kacc[1]), k1 = pack_bf16x2(kacc[2], kacc[3]);
            const uint32_t y0 = pack_bf16x2(v0[0], v0[1]), y1 = pack_bf16x2(v1[0], v1[1]);
            if ((r & 16) == 0) {
                kw[0] = k0;
                kw[1] = k1;
                vw[0] = y0;
                vw[1] = y1;
            } else {                         // 32 rows are complete: 512 contiguous bytes per store
                uint4 *dst = reinterpret_cast<uint4 *>(rec + (r / 32) * REC_BYTES) + lane;
                dst[0] = make_uint4(kw[0], kw[1], k0, k1);
                dst[32] = make_uint4(vw[0], vw[1], y0, y1);
            }
        }
        // sum over the eight row lanes by halves: lane (g, t) ends with two of its quad's 16 channels after 14 shuffles
        float *pp = a.pool + (int64_t)u * POOL_PITCH;
#pragma unroll
        for (int n = 8; n >= 2; n >>= 1) {
            const bool up = (lane & (2 * n)) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
            }
            msum += __shfl_xor_sync(0xffffffffu, msum, 2 * n);
        }
        *reinterpret_cast<float2 *>(pp + (g >> 2) * 32 + 8 * t + (g & 3) * 2) = make_float2(acc[0], acc[1]);
        if (lane == 0) pp[C] = msum;
    }
    // after a wait that ran out: no copy may still be on its way when the CTA exits
    if (!ok)
        for (int i = step; i < issued; ++i) mbar_wait_warp(bars + 8 * (uint32_t)(i % NS), (uint32_t)((i / NS) & 1), a.err, 98);
}

// ---- core: one CTA per column, whose pairs of records are dealt to SLICES slices -----------------------------------------------
// A pair is one bulk copy of 2176 bytes into the warp's ring, QN pairs ahead of the arithmetic. (As three copies per record
// the copies themselves were the bound, 26 us for 61440 records.) Sixteen slices per column whatever the number of columns: a
// column's sums are split the same way in every batch. More columns than SMs run two CTAs per SM on a shorter ring (250
// columns x 1500 rows: 41.6 us for the three kernels, with one CTA per SM 44.7); fewer have the longer ring (64 x 5120: 41 us,
// with the shorter 46). Where those come in two waves and the columns are short, up to 2048 rows, three CTAs per SM (shared memory holds
// no fourth) of eight warps, each with two slices one after the other: one wave of the chain from the partial sums to the query instead
// of two (297 x 128: 17.2 -> 15.7 us, 384 x 512: 31.3 -> 29.7, 384 x 2000: 77.4 -> 77.2; but 384 x 5120: 162.9 -> 163.4). From 445
// columns on (148 SMs) they come in two waves either way and sixteen warps are faster: 445 x 512 32.6 -> 31.7 us, 592 x 512 37.4 -> 35.6, 500 x 1000 61.3 -> 57.2.
// Half of a long column's time is issue slots (two rows a packed operation and a flushed exponential: 141 instructions a record
// of 32 rows; 384 x 5120, the three kernels 164.7 -> 162.9 us).
constexpr int SLICES = 16, Q_BYTES = 2 * REC_BYTES;
constexpr int core_smem(int warps, int qn) { return warps * qn * (Q_BYTES + 8); }

template <int WARPS, int QN>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 3 : QN == 3 ? 2 : 1) global_softmax_kernel(const StreamArgs a)
{
    constexpr int NR = 7;                        // row groups of the pooled sums: a thread for each and channel in sixteen warps
    static_assert(NR * (C + 1) <= SLICES * 32 && SLICES % WARPS == 0, "");
    extern __shared__ __align__(128) unsigned char core_dyn[];
    __shared__ float red[NR][C + 1], qa[C];
    __shared__ __align__(16) float q_s[C];
    __shared__ float s_m[SLICES][H], s_part[SLICES][H][1 + D];
    release_successor();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int b = blockIdx.x, nrec = a.nrec;
    const uint32_t slots = smem_u32(core_dyn) + (uint32_t)(warp * QN * Q_BYTES);
    const uint32_t bars = smem_u32(core_dyn) + (uint32_t)(WARPS * QN * Q_BYTES + warp * QN * 8);
    if (lane == 0) {
        for (int i = 0; i < QN; ++i) mbar_init(bars + 8 * i, 1);
        fence_barrier_init();
    }
    __syncwarp();
    wait_for_predecessor();
    const uint64_t policy = l2_evict_first();    // read once, and x should stay
    const int n_first = max(0, ((nrec + 1) / 2 - warp + SLICES - 1) / SLICES);         // pairs of slice `warp`; slice warp + WARPS follows
    static_assert(SLICES <= 2 * WARPS, "at most two slices a warp");
    auto first_record = [&](int i) {             // of this warp's i-th pair; from nrec on there is none
        return 2 * (WARPS == SLICES || i < n_first ? warp + i * SLICES : warp + WARPS + (i - n_first) * SLICES);
    };
    auto issue = [&](int i) {
        const int r0 = first_record(i);
        if (lane == 0 && r0 < nrec) {
            const uint32_t slot = (uint32_t)(i % QN), bytes = (uint32_t)min(2, nrec - r0) * REC_BYTES;
            mbar_arrive_expect_tx(bars + 8 * slot, bytes);
            bulk_load(slots + slot * Q_BYTES, a.rec + ((int64_t)b * nrec + r0) * REC_BYTES, bytes, bars + 8 * slot, policy);
        }
    };
    for (int i = 0; i < QN; ++i) issue(i);
    const float scale = 1.0f / sqrtf((float)D);
    for (int i = tid; i < NR * (C + 1); i += WARPS * 32) {
        const int grp = i / (C + 1), ch = i % (C + 1);
        const float *pp = a.pool + (int64_t)b * a.chunks * POOL_PITCH + ch;
        float s = 0.f;
#pragma unroll 8
        for (int c = grp; c < a.chunks; c += NR) s += pp[(int64_t)c * POOL_PITCH];
        red[grp][ch] = s;
    }
    __syncthreads();
    if (tid < C) {
        float s = 0.f, ms = 0.f;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            s += red[i][tid];
            ms += red[i][C];
        }
        qa[tid] = rbf(s * (1.0f / (ms + 1e-10f)));
    }
    __syncthreads();
#pragma unroll
    for (int o = tid >> 3; o < C; o += WARPS * 4) {
        const int part = tid & 7;
        const uint4 raw = __ldg(reinterpret_cast<const uint4 *>(a.wq + o * C) + part);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s = fmaf(qa[part * 8 + 2 * e], bf16lo_to_f32(w[e]), s);
            s = fmaf(qa[part * 8 + 2 * e + 1], bf16hi_to_f32(w[e]), s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if (part == 0) q_s[o] = rbf(s);
    }
    __syncthreads();

    // thread (g, t) owns head g: logits^T [8 heads x 16] = q.k^T, wa [8 x 8] += P.v
    const uint32_t aq = pack_bf16x2(q_s[g * D + 2 * t], q_s[g * D + 2 * t + 1]);
    float m_run, wa[4];
    uint64_t l2;                                 // sums of the even and of the odd rows' probabilities
    const uint64_t scale2 = pack_f32x2(scale, scale), big2 = pack_f32x2(1e9f, 1e9f), nbig2 = pack_f32x2(-1e9f, -1e9f);
    const uint64_t log2e2 = pack_f32x2(kLog2e, kLog2e);
    // logits of the record at `src`, two rows at a time; its v stays in registers
    auto logits = [&](uint32_t src, uint64_t (&xv)[4], uint4 &vq) -> float {
        const uint4 kq = lds128_u32(src + lane * 16), mq = lds128_u32(src + 1024 + t * 16);
        vq = lds128_u32(src + 512 + lane * 16);
        const uint32_t kk[4] = {kq.x, kq.y, kq.z, kq.w}, mm[4] = {mq.x, mq.y, mq.z, mq.w};
        float tmax = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float l[4] = {0.f, 0.f, 0.f, 0.f}, x0, x1;
            mma_1688(l, aq, 0u, kk[j]);
            xv[j] = fma_f32x2(pack_f32x2(round_to_bf16_f32(l[0]), round_to_bf16_f32(l[1])), scale2,
                              fma_f32x2(pack_f32x2(bf16lo_to_f32(mm[j]), bf16hi_to_f32(mm[j])), big2, nbig2));
            unpack_f32x2(xv[j], x0, x1);
            tmax = fmax3(tmax, x0, x1);
        }
        return tmax;
    };
    auto accumulate = [&](const uint64_t (&xv)[4], const uint4 &vq) {
        const uint64_t neg2 = pack_f32x2(-m_run, -m_run);
        uint32_t pk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float e0, e1;
            unpack_f32x2(mul_f32x2(add_f32x2(xv[j], neg2), log2e2), e0, e1);
            e0 = ex2_approx(e0);
            e1 = ex2_approx(e1);
            l2 = add_f32x2(l2, pack_f32x2(e0, e1));
            pk[j] = pack_bf16x2(e0, e1);
        }
        const uint32_t pa[4] = {pk[0], 0u, pk[1], 0u}, pb[4] = {pk[2], 0u, pk[3], 0u};
        mma_bf16_16816(wa, pa, vq.x, vq.y);
        mma_bf16_16816(wa, pb, vq.z, vq.w);
    };
    bool ok = true;
    int n = 0;
#pragma unroll 1
    for (int slice = warp; slice < SLICES && ok; slice += WARPS) {
        m_run = -INFINITY;
        l2 = 0;
        wa[0] = wa[1] = wa[2] = wa[3] = 0.f;
        // The running max may be stale by up to 5.5 (P below 2^8; it cancels in the division): a step needs a vote and no
        // exchange of maxima unless some row exceeds it by more.
        for (int r0 = 2 * slice; r0 < nrec; r0 += 2 * SLICES, ++n) {
            uint64_t x0[4], x1[4];
            uint4 v0, v1;
            const uint32_t slot = (uint32_t)(n % QN), src = slots + slot * Q_BYTES;
            ok = mbar_wait_warp(bars + 8 * slot, (uint32_t)((n / QN) & 1), a.err, 99);
            if (!ok) break;
            const bool two = r0 + 1 < nrec;
            float tmax = logits(src, x0, v0);
            if (two) tmax = fmaxf(tmax, logits(src + REC_BYTES, x1, v1));
            __syncwarp();
            issue(n + QN);                       // refills the slot
            if (__any_sync(0xffffffffu, tmax > m_run + 5.5f)) {
                tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
                tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
                const float m_new = fmaxf(m_run, tmax);              // finite: every record holds a row
                const float corr = __expf(m_run - m_new);            // first step: exp(-inf) = 0
                m_run = m_new;
                l2 = mul_f32x2(l2, pack_f32x2(corr, corr));
                wa[0] *= corr;
                wa[1] *= corr;
            }
            accumulate(x0, v0);
            if (two) accumulate(x1, v1);
        }
        float l_run, l_odd;
        unpack_f32x2(l2, l_run, l_odd);
        l_run += l_odd;
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
        if (t == 0) {
            s_m[slice][g] = m_run;
            s_part[slice][g][0] = l_run;
        }
        s_part[slice][g][1 + 2 * t] = wa[0];
        s_part[slice][g][2 + 2 * t] = wa[1];
    }
    // after a wait that ran out: no copy may still be on its way when the CTA exits
    if (!ok)
        for (int i = n; i < n + QN; ++i)
            if (first_record(i) < nrec) mbar_wait_warp(bars + 8 * (uint32_t)(i % QN), (uint32_t)((i / QN) & 1), a.err, 100);
    __syncthreads();
    if (tid < C) {
        const int h = tid >> 3, d = tid & 7;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < SLICES; ++w) mx = fmaxf(mx, s_m[w][h]);
        float l = 0.f, av = 0.f;
#pragma unroll
        for (int w = 0; w < SLICES; ++w) {
            const float f = s_m[w][h] == -INFINITY ? 0.f : __expf(s_m[w][h] - mx);
            l += s_part[w][h][0] * f;
            av += s_part[w][h][1 + d] * f;
        }
        a.hwa[(int64_t)b * C + tid] = 0.5f * rbf(av / l);
    }
}

// ---- out: gate = x.Wg^T + bg; out = (sigmoid(gate) * wa).Wo^T + bo -----------------------------------------------
//   warp 0      data: TMA loads of 128-row tiles into a ring of slots, TMA stores of the finished rows out of the same slots
//   warp 1      MMA issuer
//   warps 4-19  four groups of four warps, one row per thread; group e finishes tiles e, e + 4, ...: gated rows as bf16 over
//               the gate's accumulator in tensor memory, which the second product reads as its A operand; out rows over the
//               x tile in shared memory
// Four chains hide the products and the tensor-memory round trips behind each other's arithmetic; the ring holds ten
// tiles, of which four are being worked on. Bound by HBM and L2 (x in, out written): 75 us at 384 x 5120 rows, 502 MB.
constexpr int BM = 128, NSLOT = 10, NGRP = 4;
constexpr int SLOT_BYTES = BM * C * 2;
constexpr int OUT_THREADS = 20 * 32;
constexpr int OFF_WG = NSLOT * SLOT_BYTES, OFF_WO = OFF_WG + C * C * 2, OFF_VEC = OFF_WO + C * C * 2;
constexpr int VEC_FLOATS = 2 * C + NGRP * 2 * C;             // bg, bo, two buffers of hwa per group
constexpr int OFF_BAR = OFF_VEC + VEC_FLOATS * 4;
constexpr int OUT_SMEM = OFF_BAR + 8 * (2 * NSLOT + 3 * NGRP) + 16 + 1024;
constexpr int CHAIN_COLS = 128, G_COL = 0, O_COL = 64;
static_assert(OUT_SMEM <= 232448, "shared memory of one CTA");

struct OutArgs {
    const float *bg, *bo, *hwa;
    const __nv_bfloat16 *wg, *wo;
    int chunks, tiles;                       // 128-row tiles per column, and in all
    bool pass_l2;                            // x and the result leave L2 first
    int *err;
};

__global__ void __launch_bounds__(OUT_THREADS, 1)
global_stream_out_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap omap, const OutArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *gen = smem_raw + (smem - smem_u32(smem_raw));
    const uint32_t bar = smem + OFF_BAR;
    auto full = [&](int s) { return bar + 8u * (uint32_t)s; };
    auto done = [&](int s) { return bar + 8u * (uint32_t)(NSLOT + s); };
    auto g_done = [&](int e) { return bar + 8u * (uint32_t)(2 * NSLOT + e); };
    auto p_ready = [&](int e) { return bar + 8u * (uint32_t)(2 * NSLOT + NGRP + e); };
    auto o_done = [&](int e) { return bar + 8u * (uint32_t)(2 * NSLOT + 2 * NGRP + e); };
    const uint32_t tmem_slot = bar + 8u * (2 * NSLOT + 3 * NGRP);
    float *vec = reinterpret_cast<float *>(gen + OFF_VEC);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int mine = (int)blockIdx.x < a.tiles ? (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    // this CTA's t-th tile, last rows first
    auto tile_of = [&](int t, int &b, int &row0) {
        const int T = a.tiles - 1 - ((int)blockIdx.x + t * (int)gridDim.x);
        b = T / a.chunks;
        row0 = T % a.chunks * BM;
    };

    if (tid == 0) {
        for (int s = 0; s < NSLOT; ++s) {
            mbar_init(full(s), 1);
            mbar_init(done(s), 4);
        }
        for (int e = 0; e < NGRP; ++e) {
            mbar_init(g_done(e), 1);
            mbar_init(p_ready(e), 4);
            mbar_init(o_done(e), 1);
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
    release_successor();
    wait_for_predecessor();
    // weights: 16-byte chunks in the K-major 128-byte-swizzle operand layout
    for (int i = tid; i < C * 8; i += OUT_THREADS) {
        const int r = i >> 3, c = i & 7, dst = r * 128 + ((c ^ (r & 7)) << 4);
        *reinterpret_cast<uint4 *>(gen + OFF_WG + dst) = __ldg(reinterpret_cast<const uint4 *>(a.wg + r * C) + c);
        *reinterpret_cast<uint4 *>(gen + OFF_WO + dst) = __ldg(reinterpret_cast<const uint4 *>(a.wo + r * C) + c);
    }
    if (tid < C) {
        vec[tid] = a.bg[tid];
        vec[C + tid] = a.bo[tid];
    }
    fence_proxy_async();
    __syncthreads();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_desc(&xmap);
            tma_prefetch_desc(&omap);
            int issued = 0, freed = 0, b, row0;
            const uint64_t policy = a.pass_l2 ? l2_evict_first() : l2_evict_normal();
            bool ok = true;
            auto issue_loads = [&]() {
                while (issued < mine && issued - NSLOT < freed) {
                    tile_of(issued, b, row0);
                    const int s = issued % NSLOT;
                    mbar_arrive_expect_tx(full(s), SLOT_BYTES);
                    tma_load_3d(smem + s * SLOT_BYTES, &xmap, full(s), 0, row0, b, policy);
                    ++issued;
                }
            };
            issue_loads();
            for (int t = 0; t < mine; ++t) {
                const int s = t % NSLOT;
                if (!mbar_wait(done(s), (uint32_t)((t / NSLOT) & 1), a.err, 91)) {
                    ok = false;
                    break;
                }
                tile_of(t, b, row0);
                tma_store_3d(&omap, smem + s * SLOT_BYTES, 0, row0, b, policy);
                tma_store_commit();
                tma_store_wait_read<1>();                        // all but the newest store have left their slots
                freed = t;
                issue_loads();
            }
            // unwinding: no load may still be in flight into this CTA's shared memory when it exits
            if (!ok)
                for (int t = max(0, issued - NSLOT); t < issued; ++t) mbar_wait(full(t % NSLOT), (uint32_t)((t / NSLOT) & 1), a.err, 92);
            tma_store_wait<0>();
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_instr_desc_bf16(BM, C);
        const uint64_t xd = make_smem_desc_kmajor(smem, 128), gd = make_smem_desc_kmajor(smem + OFF_WG, 128),
                       od = make_smem_desc_kmajor(smem + OFF_WO, 128);
        bool ok = true;
        auto gate = [&](int t) {
            const int s = t % NSLOT, e = t % NGRP;
            ok = mbar_wait_warp(full(s), (uint32_t)((t / NSLOT) & 1), a.err, 93);
            if (!ok) return;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < C / 16; ++k)
                    tc_mma_bf16(tmem_base + e * CHAIN_COLS + G_COL, xd + (uint32_t)(s * (SLOT_BYTES >> 4)) + 2 * k, gd + 2 * k, idesc,
                                k > 0 ? 1u : 0u);
                tc_commit(g_done(e));
            }
            __syncwarp();
        };
        for (int t = 0; t < NGRP && t < mine && ok; ++t) gate(t);
        for (int t = 0; t < mine && ok; ++t) {
            const int e = t % NGRP;
            ok = mbar_wait_warp(p_ready(e), (uint32_t)((t / NGRP) & 1), a.err, 94);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t c0 = tmem_base + e * CHAIN_COLS;
#pragma unroll
                for (int k = 0; k < C / 16; ++k)
                    tc_mma_bf16_ts(c0 + O_COL, c0 + G_COL + k * 8, od + 2 * k, idesc, k > 0 ? 1u : 0u);
                tc_commit(o_done(e));
            }
            __syncwarp();
            // overwrites the gated rows: the tensor core runs the products in the order they are issued
            if (t + NGRP < mine) gate(t + NGRP);
        }
    } else if (warp >= 4) {
        const int e = (warp - 4) >> 2, quad = warp & 3, row = quad * 32 + lane, gtid = tid - 128 - e * 128;
        const uint32_t tc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(e * CHAIN_COLS);
        const uint32_t bg_a = smem + OFF_VEC, bo_a = bg_a + C * 4;
        float *hw = vec + 2 * C + e * 2 * C;
        int b, row0;
        float next = 0.f;
        if (e < mine && gtid < C) {
            tile_of(e, b, row0);
            next = __ldg(a.hwa + (int64_t)b * C + gtid);
        }
        int n = 0;
        for (int t = e; t < mine; t += NGRP, ++n) {
            // the tile's column: wa / 2 into this group's buffer n & 1, the one after it on its way
            if (gtid < C) {
                hw[(n & 1) * C + gtid] = next;
                if (t + NGRP < mine) {
                    tile_of(t + NGRP, b, row0);
                    next = __ldg(a.hwa + (int64_t)b * C + gtid);
                }
            }
            asm volatile("bar.sync %0, 128;\n" ::"r"(e + 1) : "memory");
            const uint32_t hw_a = smem + OFF_VEC + (uint32_t)((2 * C + e * 2 * C + (n & 1) * C) * 4);
            const int s = t % NSLOT;
            const uint32_t par = (uint32_t)(n & 1);
            if (!mbar_wait_warp(g_done(e), par, a.err, 95)) break;
            tc_fence_after();
            uint32_t pk[32];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t v[32];
                tmem_ld_32x32(tc + G_COL + hf * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 bg = lds128_f32(bg_a + (uint32_t)((hf * 32 + 4 * j) * 4)), hv = lds128_f32(hw_a + (uint32_t)((hf * 32 + 4 * j) * 4));
                    const float bgs[4] = {bg.x, bg.y, bg.z, bg.w}, hws[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int i0 = 4 * j + 2 * i;
                        float g0, g1, t0, t1, p0, p1;
                        unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(v[i0]), __uint_as_float(v[i0 + 1])),
                                               pack_f32x2(bgs[2 * i], bgs[2 * i + 1])), g0, g1);
                        // gate is a bf16 tensor in the reference; sigmoid(g) = 0.5 tanh(g / 2) + 0.5
                        unpack_f32x2(mul_f32x2(pack_f32x2(round_to_bf16_f32(g0), round_to_bf16_f32(g1)), pack_f32x2(0.5f, 0.5f)), t0, t1);
                        const uint64_t hw2 = pack_f32x2(hws[2 * i], hws[2 * i + 1]);         // wa / 2
                        unpack_f32x2(fma_f32x2(pack_f32x2(tanh_approx(t0), tanh_approx(t1)), hw2, hw2), p0, p1);
                        pk[hf * 16 + 2 * j + i] = pack_bf16x2(p0, p1);
                    }
                }
            }
            tmem_st_32x32(tc + G_COL, pk);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready(e));
            if (!mbar_wait_warp(o_done(e), par, a.err, 96)) break;
            tc_fence_after();
            const uint32_t rowaddr = smem + s * SLOT_BYTES + row * 128;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t v[32];
                tmem_ld_32x32(tc + O_COL + hf * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int i0 = q * 8 + 4 * i;
                        const float4 bo = lds128_f32(bo_a + (uint32_t)((hf * 32 + i0) * 4));
                        float o0, o1, o2, o3;
                        unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(v[i0]), __uint_as_float(v[i0 + 1])), pack_f32x2(bo.x, bo.y)), o0, o1);
                        unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(v[i0 + 2]), __uint_as_float(v[i0 + 3])), pack_f32x2(bo.z, bo.w)), o2, o3);
                        w[2 * i] = pack_bf16x2(o0, o1);
                        w[2 * i + 1] = pack_bf16x2(o2, o3);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(rowaddr + (((hf * 4 + q) ^ (row & 7)) << 4)),
                                 "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                                 : "memory");
                }
            }
            fence_proxy_async();                                 // the TMA store reads what these threads wrote
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(done(s));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

struct StreamPlan {
    int nrec, chunk_rows, chunks;
    size_t off_pool, off_hwa, bytes;
};
StreamPlan make_plan(int64_t B, int64_t S)
{
    StreamPlan p;
    p.nrec = (int)((S + 31) / 32);
    // A chunk is a warp's unit of work: small ones spread few columns over the chip (16 x 5120 rows: 25 us in chunks of 128, 22
    // in 64), large ones write fewer partial sums. It depends on S alone, like everything that a sum's order depends on.
    p.chunk_rows = S <= 1024 ? 32 : 64;
    p.chunks = (int)((S + p.chunk_rows - 1) / p.chunk_rows);
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    p.off_pool = up((size_t)B * p.nrec * REC_BYTES);
    p.off_hwa = p.off_pool + up((size_t)B * p.chunks * POOL_PITCH * 4);
    p.bytes = p.off_hwa + up((size_t)B * C * 4);
    return p;
}

// x is read twice. What the kv kernel reads last should still be in L2 when the out kernel starts from there, beside the records that
// the softmax kernel reads in between: the units before go first when room is made, like the records once they have been read. Of the L2
// 90 MB are counted on. 384 x 5120 rows: 179.5 -> 173.7 us; all of x first 176, nothing first 178.
constexpr int64_t kL2Bytes = (int64_t)126 << 20;

int keep_from(int64_t B, int64_t S, const StreamPlan &p)
{
    const int64_t x_bytes = B * S * C * 2, keep = std::max<int64_t>(0, kL2Bytes * 5 / 7 - (int64_t)p.bytes), units = B * p.chunks;
    return keep >= x_bytes ? 0 : (int)(units - units * keep / x_bytes);
}

// Whether x, read for the last time, and the result leave L2 first. The next operator reads the result and, for the residual, x. Where it
// would find a good part of both, they stay: with the sum of x and the result in the place of x after the call, 384 x 1000 rows 65.6 -> 63.9 us,
// 128 x 5120 99.3 -> 98.0, 384 x 2000 119.4 -> 116.8. Where x, the result and another tensor fit beside the records nothing has to go, and the
// call itself is shorter with the hint: 300 x 1000 rows 40.4 -> 38.5 us, with the sum 53.1 -> 52.0. And where not even x fits there is little to be
// found: 384 x 5120 rows, new inputs each time, 169.4 -> 167.0 us; with the sum 270.5 -> 273.0.
bool passes_l2(int64_t B, int64_t S, const StreamPlan &p)
{
    const int64_t x_bytes = B * S * C * 2, records = (int64_t)p.bytes;
    return 3 * x_bytes + records <= kL2Bytes || x_bytes + records > kL2Bytes;
}

}  // namespace

bool global_stream_covers(int heads, int head_size, int64_t out_row_stride)
{
    return heads == H && head_size == D && (out_row_stride % 8) == 0 && out_row_stride >= C;
}

size_t global_stream_scratch_bytes(int64_t B, int64_t S) { return make_plan(B, S).bytes; }

bool launch_global_stream_bf16(cudaStream_t stream, const void *x, const void *mask, const void *wq, const void *wk,
                               const void *wv, const void *wg, const float *bg, const void *wo, const float *bo,
                               void *out, int64_t out_row_stride, void *scratch, int B, int S)
{
    if (B < 1 || S < 1 || !global_stream_covers(H, D, out_row_stride)) return false;
    if ((((uintptr_t)x | (uintptr_t)out | (uintptr_t)wq | (uintptr_t)wg | (uintptr_t)wo | (uintptr_t)scratch) & 15u) != 0) return false;
    if ((((uintptr_t)wk | (uintptr_t)wv) & 3u) != 0) return false;
    KernelErrorWord &ew = kernel_error_word();
    if (ew.device == nullptr) return false;
    const StreamPlan pl = make_plan(B, S);
    char *ws = (char *)scratch;
    StreamArgs a;
    a.x = (const __nv_bfloat16 *)x;
    a.mask = (const unsigned short *)mask;
    a.wq = (const __nv_bfloat16 *)wq;
    a.wk = (const __nv_bfloat16 *)wk;
    a.wv = (const __nv_bfloat16 *)wv;
    a.rec = (unsigned char *)ws;
    a.pool = (float *)(ws + pl.off_pool);
    a.hwa = (float *)(ws + pl.off_hwa);
    a.B = B;
    a.S = S;
    a.nrec = pl.nrec;
    a.chunk_rows = pl.chunk_rows;
    a.chunks = pl.chunks;
    a.keep_from = keep_from(B, S, pl);
    a.err = ew.device;
    OutArgs o;
    o.bg = bg;
    o.bo = bo;
    o.hwa = a.hwa;
    o.wg = (const __nv_bfloat16 *)wg;
    o.wo = (const __nv_bfloat16 *)wo;
    o.chunks = (S + BM - 1) / BM;
    if ((int64_t)pl.chunks * B > INT32_MAX / 4) return false;
    o.tiles = o.chunks * B;
    o.pass_l2 = passes_l2(B, S, pl);
    o.err = ew.device;
    CUtensorMap xmap, omap;
    if (!make_tensor_map_bf16_3d(&xmap, x, C, (uint64_t)S, (uint64_t)B, C, (uint64_t)S * C, C, BM, 128) ||
        !make_tensor_map_bf16_3d(&omap, out, C, (uint64_t)S, (uint64_t)B, (uint64_t)out_row_stride,
                                 (uint64_t)S * (uint64_t)out_row_stride, C, BM, 128))
        return false;
    static bool configured = false;
    static int fit16 = 0, fit8 = 0;              // CTAs of the softmax kernel's two forms per SM
    if (!configured) {
        KUTACC_CUDA(cudaFuncSetAttribute(global_kv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM));
        KUTACC_CUDA(cudaFuncSetAttribute(global_softmax_kernel<8, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, core_smem(8, 3)));
        KUTACC_CUDA(cudaFuncSetAttribute(global_softmax_kernel<16, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, core_smem(16, 3)));
        KUTACC_CUDA(cudaFuncSetAttribute(global_softmax_kernel<16, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, core_smem(16, 4)));
        KUTACC_CUDA(cudaFuncSetAttribute(global_stream_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM));
        KUTACC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit16, global_softmax_kernel<16, 3>, 16 * 32, core_smem(16, 3)));
        KUTACC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit8, global_softmax_kernel<8, 3>, 8 * 32, core_smem(8, 3)));
        configured = true;
    }
    const int sms = std::max(1, sm_count() - runtime().sm_margin);
    {
        KernelTimer timer__("global_kv", stream);
        const int64_t units = (int64_t)B * pl.chunks;
        launch_chained(global_kv_kernel, (unsigned)std::min<int64_t>((units + KV_WARPS - 1) / KV_WARPS, (int64_t)sms * 2), KV_WARPS * 32,
                       KV_SMEM, stream, a);
    }
    {
        KernelTimer timer__("global_softmax", stream);
        const int at16 = std::max(1, fit16) * sms, at8 = std::max(1, fit8) * sms, w16 = (B + at16 - 1) / at16, w8 = (B + at8 - 1) / at8;       // waves
        if (2 * w8 <= w16 && pl.nrec <= 64)
            launch_chained(global_softmax_kernel<8, 3>, (unsigned)B, 8 * 32, core_smem(8, 3), stream, a);
        else if (B > sms)
            launch_chained(global_softmax_kernel<16, 3>, (unsigned)B, 16 * 32, core_smem(16, 3), stream, a);
        else
            launch_chained(global_softmax_kernel<16, 4>, (unsigned)B, 16 * 32, core_smem(16, 4), stream, a);
    }
    {
        KernelTimer timer__("global_stream_out", stream);
        launch_chained(global_stream_out_kernel, (unsigned)std::min(o.tiles, sms), OUT_THREADS, OUT_SMEM, stream, xmap, omap, o);
    }
    count_launch(3);
    return true;
}

}  // namespace dev
}  // namespace kutacc
