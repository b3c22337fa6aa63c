// Attention of one query row by one warp on the CUDA cores: the general path, and what the tensor-core f32 kernel falls back to
// for rows whose result is not finite. Scores are folded in ascending order with one fma per step, softmax is online over
// blocks of 32 keys.
#pragma once

#include <math_constants.h>

#include "common.cuh"

namespace mimk {
namespace attn_row {

__device__ __forceinline__ float ld(const float* p, int64_t i) { return __ldg(p + i); }
__device__ __forceinline__ float ld(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st(float* p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void st(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }

// Row i of head h, by the calling warp; qs: its own MAX_D floats of shared memory.
template <class T, int MAX_D>
__device__ __forceinline__ void row(float* qs, const T* __restrict__ Q, const T* __restrict__ K, const T* __restrict__ V,
                                    T* __restrict__ O, float* __restrict__ lse, int64_t h, int64_t i, int64_t Sq, int64_t Sk,
                                    int D, float scale, int causal) {
    const int lane = threadIdx.x & 31;
    const T* q = Q + (h * Sq + i) * D;
    const T* k = K + h * Sk * D;
    const T* v = V + h * Sk * D;
    for (int d = lane; d < D; d += 32) qs[d] = ld(q, d);
    __syncwarp();
    int64_t limit = causal ? i + 1 + (Sk - Sq) : Sk;
    if (limit > Sk) limit = Sk;
    float o_acc[MAX_D / 32];
#pragma unroll
    for (int t = 0; t < MAX_D / 32; ++t) o_acc[t] = 0.f;
    float m = -CUDART_INF_F, l = 0.f;
    for (int64_t j0 = 0; j0 < limit; j0 += 32) {
        const int64_t j = j0 + lane;
        float s         = -CUDART_INF_F;
        if (j < limit) {
            float acc      = 0.f;
            const T* kj    = k + j * D;
            for (int d = 0; d < D; ++d) acc = fmaf(qs[d], ld(kj, d), acc);
            s = acc * scale;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float alpha = (m == -CUDART_INF_F) ? 0.f : expf(m - m_new);
        // (keys that score minus infinity, and none better so far, weigh nothing)
        const float p     = (j < limit) ? expf(s - (m_new == -CUDART_INF_F ? 0.f : m_new)) : 0.f;
        l                 = l * alpha + warp_sum(p);
#pragma unroll
        for (int t = 0; t < MAX_D / 32; ++t) o_acc[t] *= alpha;
        const int n = int(limit - j0 < 32 ? limit - j0 : 32);
        for (int jj = 0; jj < n; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const T* vj    = v + (j0 + jj) * D;
#pragma unroll
            for (int t = 0; t < MAX_D / 32; ++t) {
                const int d = lane + 32 * t;
                if (d < D) o_acc[t] = fmaf(pj, ld(vj, d), o_acc[t]);
            }
        }
        m = m_new;
    }
    T* o            = O + (h * Sq + i) * D;
    // no weight at all: zeros for a row that sees no key, else every score is minus infinity and the softmax has no value
    const float inv = l > 0.f ? 1.f / l : l == 0.f && limit > 0 ? CUDART_NAN_F : 0.f;
#pragma unroll
    for (int t = 0; t < MAX_D / 32; ++t) {
        const int d = lane + 32 * t;
        if (d < D) st(o, d, o_acc[t] * inv);
    }
    if (lse && lane == 0) lse[h * Sq + i] = l > 0.f ? m + logf(l) : -CUDART_INF_F;
}

}  // namespace attn_row
}  // namespace mimk
