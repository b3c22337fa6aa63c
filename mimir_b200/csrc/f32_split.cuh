// f32 operands for the bf16 tensor cores: every value as the exact sum of three bf16 pieces, and the shared-memory tiles that
// hold the pieces.
//
// An f32 significand has 24 bits and a bf16 one 8, so cutting x after its first 8 bits, and what is left after its next 8,
// gives x = h + m + l exactly, unless bits of l lie below 2^-133, where bf16 ends: from values below 2^-109 on. The cutting
// says so (lost_bits), and what such values may have spoiled is computed again by the scalar fold. Of the nine products of two such sums the six with at least 2^-16 of the value are taken,
//     h h,  h m + m h,  h l + m m + l h,
// the three left out are below 2^-22 of it. An infinite or NaN operand leaves NaN in a piece, so every cell it reaches
// comes out non-finite and is computed again by the scalar fold.
//
// Tiles: [rows x 32] bf16, K contiguous, 64-byte rows, 64-byte swizzle (16-byte unit u of row r lies at u ^ ((r >> 1) & 3)).
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace mimk {
namespace f32split {

constexpr int BK = 32;  // k per tile row

__device__ __forceinline__ uint32_t upper_halves(float a, float b) {
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float lower_part(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xffff0000u); }

__device__ __forceinline__ void st_shared16(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// What the cutting returns has bits set here if a value was not the sum of its pieces (an infinite or NaN one included).
constexpr uint32_t lost_bits = 0xffff;
// A sum of |a b| over k terms is off by less than k (max |a| + max |b|) times this where values have lost bits.
constexpr float LOST_ABS = 0x1p-133f;

// Eight consecutive k of one row, cut into pieces and stored at `addr` of the three piece tiles (`piece_bytes` apart). Values
// that are bf16 already are their own first piece (PIECES = 1).
template <int PIECES = 3>
__device__ __forceinline__ uint32_t split_store8(uint32_t addr, uint32_t piece_bytes, const float (&x)[8]) {
    uint32_t lost = 0;
    st_shared16(addr, upper_halves(x[0], x[1]), upper_halves(x[2], x[3]), upper_halves(x[4], x[5]), upper_halves(x[6], x[7]));
    if constexpr (PIECES == 3) {
        float r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = lower_part(x[i]);
        st_shared16(addr + piece_bytes, upper_halves(r[0], r[1]), upper_halves(r[2], r[3]), upper_halves(r[4], r[5]),
                    upper_halves(r[6], r[7]));
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = lower_part(r[i]), lost |= __float_as_uint(r[i]);
        st_shared16(addr + 2 * piece_bytes, upper_halves(r[0], r[1]), upper_halves(r[2], r[3]), upper_halves(r[4], r[5]),
                    upper_halves(r[6], r[7]));
    }
    return lost;
}
// Four consecutive k of a row, half a 16-byte unit.
template <int PIECES = 3>
__device__ __forceinline__ uint32_t split_store4(uint32_t addr, uint32_t piece_bytes, const float* x) {
    float r[4]    = {x[0], x[1], x[2], x[3]};
    uint32_t lost = 0;
#pragma unroll
    for (int t = 0; t < PIECES; ++t) {
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr + t * piece_bytes), "r"(upper_halves(r[0], r[1])), "r"(upper_halves(r[2], r[3]))
                     : "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (t == 2) lost |= __float_as_uint(r[i]);
            r[i] = lower_part(r[i]);
        }
    }
    return lost;
}
__device__ __forceinline__ uint32_t half_unit_offset(int row, int half) {
    return uint32_t(row * 64 + (((half >> 1) ^ ((row >> 1) & 3)) << 4) + (half & 1) * 8);
}
__device__ __forceinline__ uint32_t unit_offset(int row, int unit) { return uint32_t(row * 64 + ((unit ^ ((row >> 1) & 3)) << 4)); }

// Shared-memory matrix descriptor of such a tile: K-major, 64-byte swizzle (layout 4), 512 bytes between groups of eight rows.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr & 0x3FFFFu) >> 4);
    d |= uint64_t(1) << 16;
    d |= uint64_t(512 >> 4) << 32;
    d |= uint64_t(1) << 46;
    d |= uint64_t(4) << 61;
    return d;
}

// D = A B^T over `blocks` 32-wide k-blocks, the products smallest first over all of them: the tensor core cuts off what its
// accumulator update cannot hold, which costs least while the accumulator is small (and so only 2 x blocks updates by full-size
// terms count). stage[b]: descriptor of block b's A tiles, its B tiles behind them; the h piece first. PIECES = 1: the product of the h pieces
// alone.
// Called by the lane that issues, from descriptors that the whole warp has made: made by lane 0 in a branch of its own they are not known to be
// uniform, and moving them costs about 50 clocks per MMA.
template <int PIECES, int A_PIECE, int B_PIECE>
__device__ __forceinline__ void mma_six(uint32_t d, const uint64_t (&stage)[2], int blocks, uint32_t idesc) {
    constexpr int B_OFF = PIECES * A_PIECE;
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0}, FIRST = PIECES == 1 ? 5 : 0;
#pragma unroll
    for (int t = FIRST; t < 6; ++t)
#pragma unroll
        for (int b = 0; b < 2; ++b)
            if (b < blocks)
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    sm100::mma_f16_ss(d, stage[b] + ((PA[t] * A_PIECE + k * 32) >> 4), stage[b] + ((B_OFF + PB[t] * B_PIECE + k * 32) >> 4), idesc,
                                      (t > FIRST || b > 0 || k > 0) ? 1u : 0u);
}

__device__ __forceinline__ float load1(const float* p) { return __ldg(p); }
__device__ __forceinline__ float load1(const __nv_bfloat16* p) {
    return __uint_as_float(uint32_t(__ldg(reinterpret_cast<const unsigned short*>(p))) << 16);
}
// Four consecutive elements from `at`, as f32, under the rules of load8 (vec: one aligned load).
__device__ __forceinline__ void load4(float* x, const float* at, bool there, int left, bool vec) {
    if (there && vec && left >= 4) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(at));
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = there && i < left ? load1(at + i) : 0.f;
    }
}
__device__ __forceinline__ void load4(float* x, const __nv_bfloat16* at, bool there, int left, bool vec) {
    if (there && vec && left >= 4) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(at));
        x[0] = __uint_as_float(v.x << 16), x[1] = __uint_as_float(v.x & 0xffff0000u);
        x[2] = __uint_as_float(v.y << 16), x[3] = __uint_as_float(v.y & 0xffff0000u);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = there && i < left ? load1(at + i) : 0.f;
    }
}
// Eight consecutive elements from `at`, as f32: `left` of them exist (zeros for the rest), none where the row is not there. vec:
// `at` is 16-byte aligned.
__device__ __forceinline__ void load8(float (&x)[8], const __nv_bfloat16* at, bool there, int left, bool vec) {
    if (there && vec && left >= 8) {
        const uint4 v       = __ldg(reinterpret_cast<const uint4*>(at));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) x[2 * i] = __uint_as_float(w[i] << 16), x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = there && i < left ? load1(at + i) : 0.f;
    }
}
__device__ __forceinline__ void load8(float (&x)[8], const float* at, bool there, int left, bool vec) {
    if (there && vec && left >= 8) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(at)), b = __ldg(reinterpret_cast<const float4*>(at + 4));
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = there && i < left ? load1(at + i) : 0.f;
    }
}

}  // namespace f32split
}  // namespace mimk
