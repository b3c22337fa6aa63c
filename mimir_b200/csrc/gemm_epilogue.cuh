// What the epilogues of the bf16 contraction kernels share: the `post` slot on a run of columns, and plain stores of a staged piece.
#pragma once

#include "common.cuh"

namespace mimk {

// The row operand's values for a tile's columns [n0, n0 + 256): eight per lane, requested before the tile is waited for, zeros where there
// are none.
__device__ __forceinline__ void load_row_256(float (&mine)[8], const float* row, int64_t n0, int64_t n, int lane) {
#pragma unroll
    for (int i = 0; i < 8; ++i) mine[i] = row && n0 + lane * 8 + i < n ? __ldg(row + n0 + lane * 8 + i) : 0.f;
}
// `post` on 32 consecutive columns of one row, from column `c` of the tile on, by a whole warp: one dispatch for the whole run (an
// operator dispatched per element, each with its own loads and bounds, takes as long as the contraction of its tile), the row operand
// from the lanes that hold it (loaded here, 16 bytes at a time, it held up every run: 2048 x 2304 x 2048 with bias and relu 29.5 us, 26.6 now).
// full: the full operand at these columns of this lane's row, `left` of which exist, or null.
template <class TOut>
__device__ __forceinline__ void apply_post_32(int post, float (&v)[32], const float (&mine)[8], int c, const TOut* full, int64_t left) {
    float b[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) b[i] = __shfl_sync(0xffffffffu, mine[i & 7], (c >> 3) + (i >> 3));
#define MIMK_CASE(POST)                                                       \
    case POST:                                                                \
        _Pragma("unroll") for (int i = 0; i < 32; ++i) v[i] = apply_post(POST, v[i], b[i], 0.f); \
        break;
    switch (post) {
        MIMK_CASE(MIMK_POST_BIAS) MIMK_CASE(MIMK_POST_BIAS_RELU) MIMK_CASE(MIMK_POST_BIAS_TANH) MIMK_CASE(MIMK_POST_RELU) MIMK_CASE(MIMK_POST_SILU)
        case MIMK_POST_ADD_FULL:
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (full && i < left) v[i] += float(full[i]);
            break;
        default: break;
    }
#undef MIMK_CASE
}

// One 32-row piece of a tile's result (128-byte-swizzled rows at `buf`, the piece before it at `before`) to a bf16 matrix that bulk stores
// cannot write (a row pitch that is no multiple of 16 bytes, or a base that is not aligned): the warp stores each row with neighbouring lanes
// on neighbouring words. Where a row starts in the middle of a word, its last element waits for the next piece, so that single elements are
// stored at the ends of the tile only. Eight rows' words are read before the first is stored. What bounds it: the instructions per row (2000 x
// 5003 x 2048, at first row by row with tests of its own for each: 60 us; 47 now; 39 by bulk stores, for a width of 5008; storing
// whole sectors only, carried from piece to piece, gains nothing).
__device__ __forceinline__ void store_piece(const uint8_t* buf, const uint8_t* before, bool first, bool last, __nv_bfloat16* c, int64_t ldc, int64_t rows,
                                            int64_t cols, int lane) {
    const int n = int(rows < 32 ? rows : 32), m = int(cols < 64 ? cols : 64);
    uint16_t* dst = reinterpret_cast<uint16_t*>(c);
    const int odd0 = int(reinterpret_cast<uintptr_t>(dst) >> 1) & 1, step = int(ldc) & 1;
    const uint8_t* prev_at = lane ? buf : before;
    const int prev = (lane + 31) & 31;
    const bool has_prev = lane > 0 || !first;
    // what this lane stores of every row, settled before the rows (tested row by row the tests take longer than the stores). Even: the row
    // starts on a word, elements 2 lane and 2 lane + 1; odd: elements 2 lane - 1 and 2 lane; and single elements where the pair is not whole:
    // the last one (even: w's first; odd: p's second, or w's second at the tile's end), the tile's first (odd: w's first).
    const bool pair_even = 2 * lane + 1 < m, one_even = 2 * lane == m - 1;
    const bool pair_odd = 2 * lane < m && has_prev, start = first && lane == 0 && m > 0, rest = 2 * lane == m && has_prev;
    const bool one_odd = start || rest || (last && m == 64 && lane == 31);
    const int one_at   = start ? 0 : rest ? m - 1 : 63;
#pragma unroll 1
    for (int r0 = 0; r0 < n; r0 += 8) {
        uint32_t w[8], p[8];  // this lane's pair of elements of each row, and the pair before it
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            w[j] = *reinterpret_cast<const uint32_t*>(buf + (r0 + j) * 128 + (((lane >> 2) ^ j) << 4) + (lane & 3) * 4);
            p[j] = *reinterpret_cast<const uint32_t*>(prev_at + (r0 + j) * 128 + (((prev >> 2) ^ j) << 4) + (prev & 3) * 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j, dst += ldc) {
            const bool odd = (odd0 + (r0 + j) * step) & 1, there = r0 + j < n;
            const uint32_t both = odd ? __funnelshift_r(p[j], w[j], 16) : w[j];
            const uint32_t one  = odd ? (rest ? p[j] : w[j]) >> (start ? 0 : 16) : w[j];
            if (there && (odd ? pair_odd : pair_even)) *reinterpret_cast<uint32_t*>(dst + 2 * lane - int(odd)) = both;
            if (there && (odd ? one_odd : one_even)) dst[odd ? one_at : 2 * lane] = uint16_t(one);
        }
    }
}

}  // namespace mimk
