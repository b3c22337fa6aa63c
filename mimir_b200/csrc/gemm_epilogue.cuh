// What the epilogues of the bf16 contraction kernels share: the `post` slot on a run of columns, and plain stores of a staged piece.
#pragma once

#include "common.cuh"

namespace mimk {

// `post` on 32 consecutive columns of one row, from column `col0` on: one dispatch and 16-byte loads for the whole run (an
// operator dispatched per element, each with its own loads and bounds, takes as long as the contraction of its tile).
// row / full: the row operand, and the full operand's row; either may be null. Columns from n on are left as they are.
template <class TOut>
__device__ __forceinline__ void apply_post_32(int post, float (&v)[32], const float* row, const TOut* full, int64_t col0, int64_t n) {
    float b[32];
    if (row && col0 + 32 <= n && (reinterpret_cast<uintptr_t>(row + col0) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(row + col0) + i);
            b[4 * i] = q.x, b[4 * i + 1] = q.y, b[4 * i + 2] = q.z, b[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) b[i] = row && col0 + i < n ? __ldg(row + col0 + i) : 0.f;
    }
#define MIMK_CASE(POST)                                                       \
    case POST:                                                                \
        _Pragma("unroll") for (int i = 0; i < 32; ++i) v[i] = apply_post(POST, v[i], b[i], 0.f); \
        break;
    switch (post) {
        MIMK_CASE(MIMK_POST_BIAS) MIMK_CASE(MIMK_POST_BIAS_RELU) MIMK_CASE(MIMK_POST_BIAS_TANH) MIMK_CASE(MIMK_POST_RELU) MIMK_CASE(MIMK_POST_SILU)
        case MIMK_POST_ADD_FULL:
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (full && col0 + i < n) v[i] += float(full[col0 + i]);
            break;
        default: break;
    }
#undef MIMK_CASE
}

// One 32-row piece of a staged result (128-byte-swizzled rows at `buf`) to a matrix that bulk stores cannot write (a row pitch
// that is no multiple of 16 bytes, or a base that is not aligned): the warp stores each row with neighbouring lanes on
// neighbouring elements, two bf16 per lane where the pair is aligned.
__device__ __forceinline__ void store_piece(const uint8_t* buf, __nv_bfloat16* c, int64_t ldc, int64_t rows, int64_t cols, int lane) {
    const int n = int(rows < 32 ? rows : 32), m = int(cols < 64 ? cols : 64);
    uint16_t* dst = reinterpret_cast<uint16_t*>(c);
    const int odd0 = int(reinterpret_cast<uintptr_t>(dst) >> 1) & 1, step = int(ldc) & 1;
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
        if (r >= n) break;
        // this lane's pair of the row, elements 2 lane and 2 lane + 1, and (shifted by one) the pair that straddles two words
        const uint32_t w    = *reinterpret_cast<const uint32_t*>(buf + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
        const uint32_t next = __shfl_down_sync(0xffffffffu, w, 1);
        if (!((odd0 + r * step) & 1)) {  // the row starts on a word
            if (2 * lane + 1 < m) reinterpret_cast<uint32_t*>(dst)[lane] = w;
            else if (2 * lane < m) dst[2 * lane] = uint16_t(w);
        } else {
            if (2 * lane + 2 < m) *reinterpret_cast<uint32_t*>(dst + 2 * lane + 1) = __funnelshift_r(w, next, 16);
            else if (2 * lane + 1 < m) dst[2 * lane + 1] = uint16_t(w >> 16);
            if (lane == 0 && m > 0) dst[0] = uint16_t(w);
        }
        dst += ldc;
    }
}

}  // namespace mimk
