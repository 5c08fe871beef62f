// LayerNorm of rows that lie in shared memory, in place: statistics and arithmetic of layernorm.cu, one bf16 rounding.
#pragma once
#include "ptx_utils.cuh"

namespace kutacc {
namespace dev {

// U rows per group of LPR lanes; addr[i] is this lane's 16-byte chunk (8 channels) of row i. The first lane of a group has the
// row's first channels; gs and bs are gamma and beta of this lane's channels. The whole warp calls it.
template <int LPR, int U>
__device__ __forceinline__ void layernorm_smem_rows(const uint32_t (&addr)[U], const float (&gs)[8], const float (&bs)[8], float eps)
{
    constexpr float inv_n = 1.0f / (float)(8 * LPR);
    const int first = (threadIdx.x & 31) / LPR * LPR;
    uint32_t w[U][4];
    float delta[U], sum[U], sum2[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(w[i][0]), "=r"(w[i][1]), "=r"(w[i][2]), "=r"(w[i][3]) : "r"(addr[i]) : "memory");
#pragma unroll
    for (int i = 0; i < U; ++i) {
        delta[i] = bf16lo_to_f32(__shfl_sync(0xffffffffu, w[i][0], first));      // the row's first channel
        sum[i] = sum2[i] = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float a = bf16lo_to_f32(w[i][e]) - delta[i], b = bf16hi_to_f32(w[i][e]) - delta[i];
            sum[i] += a;
            sum2[i] = fmaf(a, a, sum2[i]);
            sum[i] += b;
            sum2[i] = fmaf(b, b, sum2[i]);
        }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < U; ++i) {
            sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
            sum2[i] += __shfl_xor_sync(0xffffffffu, sum2[i], o);
        }
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const float mean = fmaf(sum[i], inv_n, delta[i]);
        const float var = fmaxf((sum2[i] - sum[i] * sum[i] * inv_n) * inv_n, 0.f);
        const float rstd = rsqrtf(var + eps), shift = -rstd * mean;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            w[i][e] = pack_bf16x2(fmaf(fmaf(bf16lo_to_f32(w[i][e]), rstd, shift), gs[2 * e], bs[2 * e]),
                                  fmaf(fmaf(bf16hi_to_f32(w[i][e]), rstd, shift), gs[2 * e + 1], bs[2 * e + 1]));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr[i]), "r"(w[i][0]), "r"(w[i][1]), "r"(w[i][2]), "r"(w[i][3])
                     : "memory");
    }
}

}  // namespace dev
}  // namespace kutacc
