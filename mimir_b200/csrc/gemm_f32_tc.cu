// f32 contraction on the tensor cores with f32-grade accuracy, in one launch.
//
// Every tensor program the reference can lower today is f32 (its Ring has one element type and the LLVM emitter knows
// half / float / double only, MimIR src/mim/plug/ll/ll.cpp:139-145), so the f32 `product_2d` is the path existing
// programs take. Each operand value is cut into three bf16 pieces that sum to it exactly, and the six products that matter
// are accumulated by tcgen05.mma (f32_split.cuh).
//
//   warps 0..15   read the operands and write their pieces into shared-memory tiles (each eight-k unit of the next k-block is
//                 requested as soon as the present one's has left its registers), add finished accumulators to sums in registers
//   warp 16       one thread issues the MMAs, 128 x BN x 32 per k-block; every two k-blocks go into a fresh accumulator
// The tensor core does not round its accumulator updates to nearest; with four updates by full-size terms per accumulator (all
// small terms first) and ordinary f32 adds between accumulators, the error stays below that of an f32 fold for any K.
// Accumulators are added in pairs. Few tiles: the pairs of one tile are dealt out to a cluster of two, four or eight CTAs, which exchange
// them through distributed shared memory (about 14 bytes a clock per SM, what bounds such products: by single accumulators 128 x 1024 x
// 784 took 17 us), or one accumulator to a CTA where there are as many, their pairs added at the end. They are added in order whatever the grid as long as each CTA can hold its own to the end and they are at most nine:
// K <= 1152, with 128 columns K <= 256 * split. Up to there a small product has the bits of the same cells of a large one, which programs rely on
// (and the tests hold, to K = 1028). Beyond that a CTA adds its own first, fewer tiles change hands, the sums round less, and the bits follow the split.
// That bits agree is what nine is for: 128 x 2048 x 1152, nine pairs held 24.3 us and 1.247e-7, as sums 20.5 and 1.203e-7; 128 x 1024 x 1536,
// twelve: 24.4 and 1.280e-7, 20.5 and 1.227e-7; 300 x 300 x 3000, 24: 31.6 and 27 us.
//
// The operands are read as the caller has them: any extents, strides and alignment, no copies, no scratch. What bounds it:
// shared-memory bandwidth (a k-block of 128 x 128 moves 96 KB into the MMA and 48 KB from the loaders; measured 100 clocks per
// instruction of 64 clocks' arithmetic) next to the loaders' instructions. Many tiles: the operands
// are cut beforehand instead (gemm_tf32.cu). Measured: 1000^3 29 us (30 as three TF32 products, 2e-6 off; here 1.3e-7), 4096 x 128 x
// 4096 45 (112), 64 of 512^3 220 (830 on the CUDA cores), 24 of 503 x 2052 x 407 342 (1062).
#include <type_traits>

#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;
using namespace f32split;

namespace {

constexpr int BM = 128;
constexpr int CHUNK = 2;        // k-blocks per accumulator
constexpr int LOADERS = 512, NUM_THREADS = LOADERS + 32, MMA_WARP = LOADERS / 32;
constexpr int STAGES = 4, GROUP_M = 16, HELD_PAIRS = 9;
constexpr int A_PIECE = BM * BK * 2;

template <int BN, class TIn> struct Cfg {
    static constexpr int PIECES  = sizeof(TIn) == 4 ? 3 : 1;
    static constexpr int B_PIECE = BN * BK * 2;
    static constexpr int STAGE_BYTES = PIECES * (A_PIECE + B_PIECE);
    static constexpr int PITCH = BN + 4, PART_BYTES = BM * PITCH * 4;  // a partial tile; they lie over the stages
    static constexpr int NACC  = 512 / BN;                             // accumulators in tensor memory
    static constexpr int SLOTS = BN == 128 ? 2 : 4;                    // pairs of them that a CTA of a cluster may hold to the end
    static constexpr int TILE_BYTES = STAGES * STAGE_BYTES > SLOTS * PART_BYTES ? STAGES * STAGE_BYTES : SLOTS * PART_BYTES;
    static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 256;
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
};

struct Bars {
    uint64_t full[STAGES], empty[STAGES], acc_full[8];
    uint32_t tmem_base;
    int abort_flag;
    // not zero: a value of this CTA's k-blocks was not the sum of its pieces; then whether some values are below all their pieces, and
    // what sums have to reach for all that not to matter (0: nothing lost)
    uint32_t lost, deep, max_a, max_b;
    float bound;
};

// A convolution as a contraction: row = output pixel (image, oh, ow), k = (input channel, kh, kw), column = filter. Rows of the
// patch matrix are gathered from the image as the loaders read them.
// tap_major (channels a multiple of 8): k = (kh, kw, input channel) instead, in the filters too, so that the eight k of a unit
// share one tap: one test whether it lies inside, and addresses a plane apart. With k in the order of the filters, every element has its own tap and
// test: 16 x 128 x 56 x 56, 128 filters of 3 x 3: 207 us.
struct ConvShape {
    int cin, h, w, kh, kw, oh, ow, stride_h, stride_w, dil_h, dil_w, pad_h, pad_w, tap_major;
};

struct Params {
    const void* A;
    const void* B;
    void* C;
    ConvShape conv;
    int64_t M, N, K, sa, sb, sc;
    const float* post_row;
    const void* post_full;
    int post, b_nk, vec_a, vec_b, vec_c, split;
    int64_t tiles_m, tiles_n;
    int* status;
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t saddr, uint32_t rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_cluster1(uint32_t saddr, uint32_t rank) {
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// A wait of a whole warp, with one outcome for all its lanes.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

__device__ __forceinline__ void tile_coords(int64_t tile, int64_t tiles_m, int64_t tiles_n, int64_t& tm, int64_t& tn) {
    const int64_t per_group = GROUP_M * tiles_n;
    const int64_t group     = tile / per_group;
    const int64_t first_m   = group * GROUP_M;
    const int64_t gsize     = (tiles_m - first_m) < GROUP_M ? (tiles_m - first_m) : GROUP_M;
    const int64_t in_group  = tile % per_group;
    tm                      = first_m + in_group % gsize;
    tn                      = in_group / gsize;
}

__device__ __forceinline__ int cv_pixels(const Params& p) { return p.conv.oh * p.conv.ow; }

// four neighbouring results of one row; vec: they are one aligned store, and n is a multiple of 4
template <class TOut>
__device__ __forceinline__ void store4(TOut* row, int64_t col, int64_t n, float4 q, bool vec) {
    if (col >= n) return;
    if (vec) {
        if (sizeof(TOut) == 4) *reinterpret_cast<float4*>(row + col) = q;
        else *reinterpret_cast<uint2*>(row + col) = make_uint2(pack_bf16x2(q.x, q.y), pack_bf16x2(q.z, q.w));
    } else {
        row[col] = TOut(q.x);
        if (col + 1 < n) row[col + 1] = TOut(q.y);
        if (col + 2 < n) row[col + 2] = TOut(q.z);
        if (col + 3 < n) row[col + 3] = TOut(q.w);
    }
}

// The scalar fold of one cell -- ascending k, one fma per step, what the CUDA-core kernel computes -- for cells the pieces make
// non-finite (an operand of the fold was inf / NaN, or the sum overflowed), and for cells as small as the bits lost in cutting.
template <class TIn, bool CONV>
__device__ __noinline__ float scalar_fold(const Params& p, int64_t bz, int64_t row, int64_t col) {
    const TIn* A = static_cast<const TIn*>(p.A) + bz * p.sa;
    const TIn* B = static_cast<const TIn*>(p.B) + bz * p.sb;
    float v = 0.f;
    if (CONV) {  // padding read as zeros
        const ConvShape& cv = p.conv;
        const int pixels  = cv.oh * cv.ow;
        const int64_t img = row / pixels;
        const int y = int(row - img * pixels) / cv.ow, x = int(row - img * pixels) - y * cv.ow;
        const TIn* im = A + img * (int64_t(cv.cin) * cv.h * cv.w);
        const int taps = cv.kh * cv.kw;
        for (int ci = 0; ci < cv.cin; ++ci)
            for (int kr = 0; kr < cv.kh; ++kr)
                for (int kq = 0; kq < cv.kw; ++kq) {
                    const int iy = y * cv.stride_h - cv.pad_h + kr * cv.dil_h, ix = x * cv.stride_w - cv.pad_w + kq * cv.dil_w;
                    const bool in = unsigned(iy) < unsigned(cv.h) && unsigned(ix) < unsigned(cv.w);
                    const int tap = kr * cv.kw + kq;
                    const TIn* wt = B + col * p.K + (cv.tap_major ? tap * cv.cin + ci : ci * taps + tap);
                    v = fmaf(in ? load1(im + (int64_t(ci) * cv.h + iy) * cv.w + ix) : 0.f, load1(wt), v);
                }
    } else {
        const TIn* ar = A + row * p.K;
        const TIn* br = p.b_nk ? B + col * p.K : B + col;
        const int64_t step = p.b_nk ? 1 : p.N;
        for (int64_t k = 0; k < p.K; ++k) v = fmaf(load1(ar + k), load1(br + k * step), v);
    }
    return v;
}

// How many of a tile's accumulators go to each CTA of a cluster: whole pairs, so that half as many partial tiles change hands; one each where
// there are CTAs enough, and the pairs are added when the tile is stored; one by one in convolutions, and beyond HELD_PAIRS, where
// each CTA adds up its own in any case. (Always whole pairs, us: 1710 x 104 x 233 9.9 -> 12.0, 23 x 719 x 472 10.2 -> 11.0, 62 x 36 x 2364 18.4 -> 19.3.)
__host__ __device__ inline int share_of(int chunks, int split, bool conv) {
    if (conv || chunks > 2 * HELD_PAIRS || chunks <= split) return (chunks + split - 1) / split;
    return ((chunks + 1) / 2 + split - 1) / split * 2;
}

// What a CTA works on: a tile of a batch entry, and of its k-blocks the accumulators [ch0, ch1).
template <int BN> struct Place {
    int rank, ch0, ch1, kb0, kb1, per, chunks;
    int64_t bz, m0, n0;
    __device__ __forceinline__ explicit Place(const Params& p) {
        const int64_t tiles = p.tiles_m * p.tiles_n;
        rank                = int(blockIdx.x % unsigned(p.split));  // a cluster is `split` consecutive CTAs
        const int64_t item  = blockIdx.x / unsigned(p.split);
        bz                  = item / tiles;
        int64_t tm, tn;
        tile_coords(item - bz * tiles, p.tiles_m, p.tiles_n, tm, tn);
        m0 = tm * BM, n0 = tn * BN;
        const int all_kb = int((p.K + BK - 1) / BK);
        chunks = (all_kb + CHUNK - 1) / CHUNK, per = share_of(chunks, p.split, p.conv.cin > 0);
        ch0 = rank * per < chunks ? rank * per : chunks, ch1 = ch0 + per < chunks ? ch0 + per : chunks;
        kb0 = ch0 * CHUNK, kb1 = ch1 * CHUNK < all_kb ? ch1 * CHUNK : all_kb;
    }
};

// Four neighbouring sums of one row: non-finite ones and those below `bound` (zeros, if so said) folded again, `post`, stored.
template <class TIn, class TOut>
__device__ __forceinline__ void finish4(const Params& p, TOut* out, const TOut* post_full, int64_t bz, int64_t row, int64_t col, float4 q, float bound,
                                        bool zeros) {
    if (row >= p.M || col >= p.N) return;
    float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (col + e >= p.N) break;
        if (!isfinite(v[e]) || (fabsf(v[e]) < bound && (v[e] != 0.f || zeros))) v[e] = scalar_fold<TIn, false>(p, bz, row, col + e);
        const float rowv = p.post_row ? __ldg(p.post_row + col + e) : 0.f;
        const float full = post_full ? float(post_full[row * p.N + col + e]) : 0.f;
        v[e]             = apply_post(p.post, v[e], rowv, full);
    }
    store4(out + row * p.N, col, p.N, make_float4(v[0], v[1], v[2], v[3]), p.vec_c);
}

// The accumulators of a tile in order, each CTA of the cluster a share of the rows. hold: every pair of them has a partial tile of its
// own, or each of them, where each is a CTA's only one; else each CTA has one.
template <int BN, class TIn, class TOut, bool CONV>
__device__ __forceinline__ void store_tile(const Params& p, const Place<BN>& at, uint32_t base, bool hold, float bound, bool zeros) {
    using C = Cfg<BN, TIn>;
    const bool pairs = hold && at.per > 1, singles = hold && at.per == 1;
    const int rows = BM / p.split, held = pairs ? at.per / 2 : 1, used = pairs ? (at.chunks + 1) / 2 : (at.chunks + at.per - 1) / at.per;
    TOut* out             = static_cast<TOut*>(p.C) + at.bz * p.sc;
    const TOut* post_full = p.post_full ? static_cast<const TOut*>(p.post_full) + at.bz * p.sc : nullptr;
    for (int i = threadIdx.x; i < rows * (BN / 4); i += NUM_THREADS) {
        // CONV: neighbouring threads take neighbouring pixels, else neighbouring columns
        const int r = at.rank * rows + (CONV ? i % rows : i / (BN / 4)), col = (CONV ? i / rows : i % (BN / 4)) * 4;
        const int64_t row = at.m0 + r, gcol = at.n0 + col;
        if (row >= p.M || gcol >= p.N) continue;
        const uint32_t a = base + uint32_t(r * C::PITCH + col) * 4;
        float4 q         = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int t0 = 0; t0 < used; t0 += 4) {  // four on their way at a time, added in order
            float4 w[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
                w[t] = t0 + t < used ? ld_cluster4(a + ((t0 + t) % held) * C::PART_BYTES, uint32_t((t0 + t) / held)) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (singles)  // (the same adds as where a pair is one CTA's)
#pragma unroll
                for (int t = 0; t < 4; t += 2) {
                    w[t].x += w[t + 1].x, w[t].y += w[t + 1].y, w[t].z += w[t + 1].z, w[t].w += w[t + 1].w;
                    w[t + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
            for (int t = 0; t < 4; ++t) q.x += w[t].x, q.y += w[t].y, q.z += w[t].z, q.w += w[t].w;
        }
        if (CONV) {
            const int pixels  = cv_pixels(p);
            const int64_t img = row / pixels;
            TOut* plane       = out + (img * p.N + gcol) * pixels + (row - img * pixels);
            const float v[4]  = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (gcol + e < p.N) {
                    const bool again = !isfinite(v[e]) || (fabsf(v[e]) < bound && (v[e] != 0.f || zeros));
                    plane[int64_t(e) * pixels] = TOut(again ? scalar_fold<TIn, CONV>(p, at.bz, row, gcol + e) : v[e]);
                }
        } else {
            finish4<TIn, TOut>(p, out, post_full, at.bz, row, gcol, q, bound, zeros);
        }
    }
}

template <int BN, class TIn> __device__ __forceinline__ bool holds(const Params& p, const Place<BN>& at) { return p.split > 1 && p.conv.cin == 0 && at.chunks <= 2 * HELD_PAIRS && at.per <= 2 * Cfg<BN, TIn>::SLOTS; }

// Bits were lost in cutting this CTA's part of the operands: what a sum has to reach for that not to matter, 22 bits above the loss,
// from the largest finite magnitudes among the CTA's rows, columns and k; a sum of exactly zero can be short of something only if there
// are values below 2^-133. (It finds its place again, and loads four rows at a time: kept for it, or with eight, registers are spilled
// by the loaders' loop, 1000^3 31 -> 35 us.) By all warps: 16 of 1000 x 1000 x 64 with softmax weights of 1e-38 67 us, 264 by one.
// CONV: the largest of the image rows that the tile's windows reach, all channels.
template <class TIn, int BN, bool CONV>
__device__ __noinline__ void find_bound(const Params& p, Bars* bars) {
    const Place<BN> at(p);
    const TIn* A = static_cast<const TIn*>(p.A) + at.bz * p.sa;
    const TIn* B = static_cast<const TIn*>(p.B) + at.bz * p.sb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t k0 = int64_t(at.kb0) * BK, k1 = int64_t(at.kb1) * BK < p.K ? int64_t(at.kb1) * BK : p.K;
    const int64_t rows = p.M - at.m0 < BM ? p.M - at.m0 : BM, cols = p.N - at.n0 < BN ? p.N - at.n0 : BN;
    uint32_t deep = 0;
    // the largest of `n` rows of `len` elements, `pitch` apart; four rows of 128 elements on their way at a time
    auto largest = [&](const TIn* first, int64_t n, int64_t pitch, int64_t len, bool vec) {
        uint32_t most = 0;
        for (int64_t r = warp * 4; r < n; r += NUM_THREADS / 32 * 4)
            for (int64_t c = lane * 4; c < len; c += 128) {
                float x[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) load4(x[j], first + (r + j) * pitch + c, r + j < n, int(len - c < 4 ? len - c : 4), vec);
#pragma unroll
                for (int j = 0; j < 4 * 4; ++j) {
                    const uint32_t u = __float_as_uint(x[j >> 2][j & 3]) & 0x7fffffffu;
                    if (u < 0x7f800000u) most = max(most, u), deep |= u > 0u && u < __float_as_uint(LOST_ABS);
                }
            }
        return __reduce_max_sync(0xffffffffu, most);
    };
    uint32_t a = 0;
    if (CONV) {
        const ConvShape& cv  = p.conv;
        const int64_t pixels = int64_t(cv.oh) * cv.ow, plane = int64_t(cv.h) * cv.w, last = at.m0 + rows - 1;
        for (int64_t img = at.m0 / pixels; img * pixels <= last; ++img) {
            const int y0 = img * pixels < at.m0 ? int(at.m0 - img * pixels) / cv.ow : 0;
            const int y1 = last - img * pixels < pixels ? int(last - img * pixels) / cv.ow : cv.oh - 1;
            const int top = max(y0 * cv.stride_h - cv.pad_h, 0), bottom = min(y1 * cv.stride_h - cv.pad_h + (cv.kh - 1) * cv.dil_h, cv.h - 1);
            if (top <= bottom) a = max(a, largest(A + img * cv.cin * plane + int64_t(top) * cv.w, cv.cin, plane, int64_t(bottom - top + 1) * cv.w, false));
        }
    } else {
        a = largest(A + at.m0 * p.K + k0, rows, p.K, k1 - k0, p.vec_a);
    }
    const TIn* b0    = p.b_nk ? B + at.n0 * p.K + k0 : B + k0 * p.N + at.n0;
    const uint32_t b = p.b_nk ? largest(b0, cols, p.K, k1 - k0, p.vec_b)
                              : largest(b0, k1 - k0, p.N, cols, p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(b0) & 15) == 0);
    deep             = __reduce_or_sync(0xffffffffu, deep);
    if (lane == 0) atomicMax(&bars->max_a, a), atomicMax(&bars->max_b, b), atomicOr(&bars->deep, deep);
    __syncthreads();
    if (threadIdx.x == 0) bars->bound = float(k1 - k0) * (0x1p22f * LOST_ABS) * (__uint_as_float(bars->max_a) + __uint_as_float(bars->max_b));
    __syncthreads();
}

template <int BN, class TIn, class TOut, bool CONV>
__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ Params p) {
    using C = Cfg<BN, TIn>;
    constexpr int PIECES = C::PIECES;
    constexpr bool LOSES = PIECES == 3;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;
    Bars* bars              = reinterpret_cast<Bars*>(smem_raw + (base - raw_addr) + C::TILE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const Place<BN> place(p);
    const int rank = place.rank, ch0 = place.ch0, ch1 = place.ch1, kb0 = place.kb0, kb1 = place.kb1, per = place.per, chunks = place.chunks;
    const int64_t bz = place.bz, m0 = place.m0, n0 = place.n0;
    const TIn* A = static_cast<const TIn*>(p.A) + bz * p.sa;
    const TIn* B = static_cast<const TIn*>(p.B) + bz * p.sb;
    // this CTA's accumulators stay in tensor memory to the end and leave one by one, or are added up as they are finished
    const bool hold = holds<BN, TIn>(p, place);

    // A thread's part of a k-block. Where memory runs along k: four k of one or two rows 64 apart, eight lanes to a row's 128
    // bytes. Where it runs along the rows (B stored [K, N], the pixels of an image): eight k of one row, a warp's lanes on
    // neighbouring rows.
    const int across = (warp >> 2) * 32 + lane, unit = warp & 3, along = tid >> 3, half = tid & 7;
    constexpr int NB = BN / 64;
    const bool has_b = BN == 128 || p.b_nk || tid < BN * 4;
    float fa[8], fb[8];
    const TIn* a_at;                // CONV: the first tap of the pixel's window; else the thread's first row of A
    const TIn* b_at = p.b_nk ? B + (n0 + along) * p.K + half * 4 : B + int64_t(unit * 8) * p.N + n0 + across;
    int rows_in = 0, cols_in = 0;   // CONV: bit i: tap row / column i of this pixel lies inside the image
    const ConvShape& cv = p.conv;
    if (CONV) {
        const int64_t row = m0 + across;
        const int pixels  = cv.oh * cv.ow;
        const int64_t img = row / pixels;
        const int pix = int(row - img * pixels), y = pix / cv.ow;
        const int ih0 = y * cv.stride_h - cv.pad_h, iw0 = (pix - y * cv.ow) * cv.stride_w - cv.pad_w;
        a_at = A + img * (int64_t(cv.cin) * cv.h * cv.w) + (int64_t(ih0) * cv.w + iw0);  // only taps inside are read
        if (row < p.M) {
            for (int r = 0; r < cv.kh; ++r) rows_in |= int(unsigned(ih0 + r * cv.dil_h) < unsigned(cv.h)) << r;
            for (int q = 0; q < cv.kw; ++q) cols_in |= int(unsigned(iw0 + q * cv.dil_w) < unsigned(cv.w)) << q;
        }
    } else {
        a_at = A + (m0 + along) * p.K + half * 4;
    }
    auto fetch_a = [&](int kb) {
        const int64_t k0 = int64_t(kb) * BK;
        if (CONV && cv.tap_major) {
            const int k = int(k0) + unit * 8, tap = k / cv.cin, r = tap / cv.kw, q = tap - r * cv.kw, plane = cv.h * cv.w;
            const bool in = k < int(p.K) && ((rows_in >> r) & (cols_in >> q) & 1);
            const TIn* at = a_at + (k - tap * cv.cin) * int64_t(plane) + (r * cv.dil_h * cv.w + q * cv.dil_w);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                fa[j] = in ? load1(at) : 0.f;
                at += plane;
            }
        } else if (CONV) {
            const int k = int(k0) + unit * 8, taps = cv.kh * cv.kw;
            const int ci = k / taps;
            int r = (k - ci * taps) / cv.kw, q = k - ci * taps - r * cv.kw;
            // offsets of taps that are read fit 31 bits (mimk_conv sees to it); the others wrap
            const unsigned w = cv.w, plane = cv.h * w, down = cv.dil_h * w;
            unsigned off = ci * plane + r * down + q * cv.dil_w;
            const unsigned next_row = down - cv.kw * cv.dil_w, next_plane = plane - cv.kh * down;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool in = (rows_in >> r) & (cols_in >> q) & int(k + j < int(p.K));
                fa[j]         = in ? load1(a_at + int(off)) : 0.f;
                off += cv.dil_w;
                if (++q == cv.kw) {
                    q = 0, off += next_row;
                    if (++r == cv.kh) r = 0, off += next_plane;
                }
            }
        } else {
            const int left = int(p.K - k0) - half * 4;
            load4(fa, a_at + k0, m0 + along < p.M, left, p.vec_a);
            load4(fa + 4, a_at + k0 + 64 * p.K, m0 + along + 64 < p.M, left, p.vec_a);
        }
    };
    auto fetch_b = [&](int kb) {
        if (!has_b) return;
        const int64_t k0 = int64_t(kb) * BK;
        if (p.b_nk) {
            const int left = int(p.K - k0) - half * 4;
            load4(fb, b_at + k0, n0 + along < p.N, left, p.vec_b);
            if (NB == 2) load4(fb + 4, b_at + k0 + 64 * p.K, n0 + along + 64 < p.N, left, p.vec_b);
        } else {
            const TIn* at  = b_at + k0 * p.N;
            const int left = int(p.K - k0) - unit * 8;
            const bool in  = n0 + across < p.N;
#pragma unroll
            for (int j = 0; j < 8; ++j) fb[j] = in && j < left ? load1(at + j * p.N) : 0.f;
        }
    };
    uint32_t lost = 0;
    // (CONV: at once, for a register that its loaders have not got)
    auto note = [&](uint32_t bits) {
        if (!CONV) lost |= bits;
        else if (LOSES && (bits & lost_bits)) bars->lost = 1;
    };
    auto store_a = [&](uint32_t at) {
        if (CONV) {
            note(split_store8<PIECES>(at + unit_offset(across, unit), A_PIECE, fa));
        } else {
            note(split_store4<PIECES>(at + half_unit_offset(along, half), A_PIECE, fa));
            note(split_store4<PIECES>(at + half_unit_offset(along + 64, half), A_PIECE, fa + 4));
        }
    };
    auto store_b = [&](uint32_t at) {
        if (p.b_nk) {
            note(split_store4<PIECES>(at + half_unit_offset(along, half), C::B_PIECE, fb));
            if (NB == 2) note(split_store4<PIECES>(at + half_unit_offset(along + 64, half), C::B_PIECE, fb + 4));
        } else if (has_b) {
            note(split_store8<PIECES>(at + unit_offset(across, unit), C::B_PIECE, fb));
        }
    };
    if (warp < MMA_WARP && kb0 < kb1) {  // on their way while the barriers and the tensor memory are set up
        fetch_a(kb0);
        fetch_b(kb0);
    }

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), LOADERS / 32);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (int b = 0; b < C::NACC; ++b) mbar_init(smem_u32(&bars->acc_full[b]), 1);
        bars->abort_flag = 0;
        bars->lost = bars->deep = bars->max_a = bars->max_b = 0, bars->bound = 0.f;
        fence_barrier_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&bars->tmem_base), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

    if (warp == MMA_WARP) {
        {
            const bool leader    = elect_one();
            const uint64_t desc0 = smem_desc_sw64(base);
            const uint32_t idesc = idesc_bf16_f32(BM, BN, 0, 0);
            uint32_t stage = 0, phase = 0;
            for (int kb = kb0, c = 0; kb < kb1; kb += CHUNK, ++c) {
                // A full stage also says that every warp has added up the chunk four before this one, so an accumulator is free
                // when its turn comes again.
                uint64_t at[CHUNK];
                uint32_t empty[CHUNK];
                const int n = kb1 - kb < CHUNK ? kb1 - kb : CHUNK;
                bool ok = true;
#pragma unroll
                for (int b = 0; b < CHUNK; ++b) {
                    if (b < n && ok) ok = warp_wait(smem_u32(&bars->full[stage]), phase, abort_flag);
                    at[b] = desc0 + stage * (C::STAGE_BYTES >> 4), empty[b] = smem_u32(&bars->empty[stage]);
                    if (b < n && ++stage == STAGES) stage = 0, phase ^= 1u;
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = uint32_t(c) % C::NACC;
                if (leader) {
                    mma_six<PIECES, A_PIECE, C::B_PIECE>(tmem_base + acc * BN, at, n, idesc);
#pragma unroll
                    for (int b = 0; b < CHUNK; ++b)
                        if (b < n) mma_commit(empty[b]);
                    mma_commit(smem_u32(&bars->acc_full[acc]));
                }
            }
        }
        __syncwarp();
    } else {
        static_assert(CHUNK == 2 && STAGES == 2 * CHUNK && C::NACC >= 4, "see the waits of the MMA warp");
        constexpr int COLS = BN / 4;  // accumulator columns per warp
        const uint32_t quarter = uint32_t(warp & 3), col0 = uint32_t(warp >> 2) * COLS, lanes = (quarter * 32u) << 16;
        float sum[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
        // sixteen columns, from `h` on, of this CTA's chunk c; the registers are valid after tmem_ld_wait
        auto ready   = [&](int c) {
            const bool ok = warp_wait(smem_u32(&bars->acc_full[uint32_t(c) % C::NACC]), uint32_t(c / C::NACC) & 1u, abort_flag);
            tc_fence_after();
            return ok;
        };
        auto request = [&](int c, int h, uint32_t (&r)[16]) { tmem_ld_32x16(tmem_base + uint32_t(c) % C::NACC * BN + col0 + lanes + h, r); };
        auto add     = [&](auto h, const uint32_t (&r)[16]) {
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[decltype(h)::value + i] += __uint_as_float(r[i]);
            tc_fence_before();
        };
        // chunks c and c + 1 (or c alone) added up and to the sums
        auto pair = [&](int c) {
#pragma unroll
            for (int h = 0; h < COLS; h += 16) {
                uint32_t r[16], second[16];
                request(c, h, r);
                if (c + 1 < ch1 - ch0) {
                    request(c + 1, h, second);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) second[i] = 0;
                }
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[h + i] += __uint_as_float(r[i]) + __uint_as_float(second[i]);
            }
            tc_fence_before();
        };
        using First  = std::integral_constant<int, 0>;
        using Second = std::integral_constant<int, COLS == 32 ? 16 : 0>;
        uint32_t stage = 0, phase = 0;
        auto load_block = [&](int kb) {
            if (!warp_wait(smem_u32(&bars->empty[stage]), phase ^ 1u, abort_flag)) return false;
            const uint32_t s0 = base + stage * C::STAGE_BYTES;
            store_a(s0);
            if (kb + 1 < kb1) fetch_a(kb + 1);
            store_b(s0 + PIECES * A_PIECE);
            if (kb + 1 < kb1) fetch_b(kb + 1);
            else if (LOSES && (lost & lost_bits)) bars->lost = 1;
            fence_proxy_async_smem();  // the MMA reads shared memory through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->full[stage]));
            if (++stage == STAGES) stage = 0, phase ^= 1u;
            return true;
        };
        bool ok   = true;
        int added = 0;
        for (int c = 0; c < ch1 - ch0; ++c) {
            // A read of tensor memory waits behind the MMAs in the queue (about 1200 clocks). Where the loaders wait for memory too
            // (an image's patches), it is requested before a block is loaded and added after it (16 x 128 x 56 x 56, 128 filters of
            // 3 x 3: 241 -> 201 us; bf16 248 -> 279, 2048^3 163 -> 170, so not there). The chunk read is complete: its stages are in use again.
            constexpr bool EARLY = CONV && PIECES == 3;
            const int kb = kb0 + c * CHUNK;
            const bool second = kb + 1 < kb1;
            if constexpr (EARLY) {
                const bool due = !hold && c >= 3;
                uint32_t r[16];
                if (!(ok = !due || ready(added))) break;
                if (due) request(added, 0, r);
                if (!(ok = load_block(kb))) break;
                if (due) add(First{}, r);
                if (COLS == 32 && due) request(added, 16, r);
                if (second && !(ok = load_block(kb + 1))) break;
                if (COLS == 32 && due) add(Second{}, r);
                added += due;
            } else {
                if (!(ok = load_block(kb) && (!second || load_block(kb + 1)))) break;
                if (!hold && c >= 3 && (c & 1)) {
                    if (!(ok = ready(added) && ready(added + 1))) break;
                    pair(added);
                    added += 2;
                }
            }
        }
        auto part = [&](int slot, const float (&x)[COLS]) {
            const uint32_t a = base + slot * C::PART_BYTES + (uint32_t(quarter * 32 + lane) * C::PITCH + col0) * 4;
#pragma unroll
            for (int i = 0; i < COLS; i += 4)
                st_shared16(a + i * 4, __float_as_uint(x[i]), __float_as_uint(x[i + 1]), __float_as_uint(x[i + 2]), __float_as_uint(x[i + 3]));
        };
        // Once the last chunk is finished every MMA of this CTA is complete, and the stages become its partial tiles.
        if (hold) {
            if (ok && ch1 > ch0) ok = ready(ch1 - ch0 - 1);
            for (int c = 0; c < ch1 - ch0 && ok; c += 2) {  // (the last being ready, all are)
#pragma unroll
                for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
                pair(c);
                part(c / 2, sum);
            }
        } else {
            if (ok && added < ch1 - ch0) ok = ready(ch1 - ch0 - 1);
            if constexpr (CONV && PIECES == 3) {
                for (; added < ch1 - ch0 && ok; ++added) {
                    uint32_t r[16];
                    request(added, 0, r);
                    add(First{}, r);
                    if (COLS == 32) {
                        request(added, 16, r);
                        add(Second{}, r);
                    }
                }
            } else {
                for (; added < ch1 - ch0 && ok; added += 2) pair(added);
            }
            part(0, sum);
        }
    }
    __syncthreads();
    if (LOSES && bars->lost) find_bound<TIn, BN, CONV>(p, bars);
    // (an abandoned wait leaves MMAs that read the stages; their results are marked invalid by the status word)
    if (p.split > 1) cluster_sync();
    float bound   = 0.f;
    uint32_t deep = 0;
    if (LOSES) {  // (a lane asks a CTA each: one after the other the answers take 2000 clocks)
        if (lane < p.split) bound = __uint_as_float(ld_cluster1(smem_u32(&bars->bound), uint32_t(lane))), deep = ld_cluster1(smem_u32(&bars->deep), uint32_t(lane));
        bound = warp_sum(bound), deep = __reduce_or_sync(0xffffffffu, deep);
    }
    store_tile<BN, TIn, TOut, CONV>(p, place, base, hold, bound, deep != 0);
    if (p.split > 1) cluster_sync();  // no CTA of the cluster exits while another may read its partial tiles

    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(&bars->tmem_base), 512);
    }
    if (tid == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

template <int BN, class TIn, class TOut, bool CONV>
int launch(const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = gemm_f32_tc_kernel<BN, TIn, TOut, CONV>;
    constexpr int SMEM = Cfg<BN, TIn>::SMEM_BYTES;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[dev & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas)), cfg.blockDim = dim3(NUM_THREADS), cfg.dynamicSmemBytes = SMEM, cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(p.split), attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    return note_cuda_error(cudaLaunchKernelEx(&cfg, kern, p));
}

// Tile width and split: the pair with the least estimated time, rounds * (fixed + k-blocks per CTA * per k-block), a round being
// the tiles that are on the chip at once: one CTA per SM; clusters leave SMs of a partly filled group idle (15 of eight were on
// the chip at once, 16 took two rounds; of four 32). Measured per k-block: 1.15 us (128 wide), 0.95 (64); fixed 8 us, 9 with the
// exchange. 1000^3: 128 wide split 2, 29 us (128 / 1: 48, 64 / 1: 40); 300 x 300 x 3000: 64 wide split 8, 20 (64 / 1: 99).
struct Plan {
    int bn, split;
    double us;
};
// singly: accumulators are dealt out one by one.
Plan make_plan(int64_t m, int64_t n, int64_t k, int64_t batch, int sm_count, bool singly) {
    const int64_t tiles_m = (m + BM - 1) / BM;
    const int kb = int((k + BK - 1) / BK), chunks = (kb + CHUNK - 1) / CHUNK;
    Plan best{64, 1, 1e300};
    for (int wide = 0; wide < 2; ++wide)
        for (int split = 1; split <= 8; split *= 2) {
            if (split > 1 && share_of(chunks, split, singly) == share_of(chunks, split / 2, singly)) break;  // no fewer for a CTA than with half the CTAs
            const int64_t items = tiles_m * ((n + (wide ? 127 : 63)) / (wide ? 128 : 64)) * batch;
            int64_t room        = split == 1 ? sm_count : split == 2 ? sm_count / 2 - 4 : split == 4 ? sm_count / 4 - 5 : sm_count / 8 - 3;
            if (room < 1) room = 1;  // (a slice of a GPU)
            const double rounds = double((items + room - 1) / room);
            const int per       = share_of(chunks, split, singly) * CHUNK;
            const bool singles  = !singly && split > 1 && per == CHUNK;  // of 128 columns: twice the bytes to exchange (172 x 740 x 340 10.2 -> 11.1 us)
            const double time   = rounds * ((split > 1 ? 9.0 : 8.0) + (per < kb ? per : kb) * (wide ? 1.15 : 0.95) + (singles && wide ? 1.6 : 0.0));
            if (time < best.us) best = Plan{wide ? 128 : 64, split, time};
        }
    return best;
}

template <class TIn, class TOut, bool CONV>
int plan_and_launch(Params& p, int64_t batch, int sm_count, cudaStream_t s) {
    const Plan plan = make_plan(p.M, p.N, p.K, batch, sm_count, CONV);
    p.split = plan.split, p.tiles_m = (p.M + BM - 1) / BM, p.tiles_n = (p.N + plan.bn - 1) / plan.bn;
    const int64_t ctas = p.tiles_m * p.tiles_n * batch * p.split;
    return plan.bn == 128 ? launch<128, TIn, TOut, CONV>(p, ctas, s) : launch<64, TIn, TOut, CONV>(p, ctas, s);
}

}  // namespace

static int extents_fit(const mimk_gemm_desc& d) {
    if (d.k <= 0) return 0;
    if (d.m >= (int64_t(1) << 31) || d.n >= (int64_t(1) << 31) || d.k >= (int64_t(1) << 31)) return 0;
    const int64_t tiles = ((d.m + BM - 1) / BM) * ((d.n + 63) / 64);
    return tiles < (int64_t(1) << 28) && d.batch < (int64_t(1) << 28) && tiles * d.batch < (int64_t(1) << 28);  // one grid
}
// (by single accumulators: the choice against three TF32 products, which are less accurate, is not to move with how pairs fall to CTAs)
double gemm_f32_tc_us(int64_t m, int64_t n, int64_t k, int64_t batch, int sm_count) { return make_plan(m, n, k, batch, sm_count, true).us; }
int gemm_f32_tc_supported(const mimk_gemm_desc& d) { return d.in_dtype == MIMK_F32 && extents_fit(d); }

static Params product_params(const mimk_gemm_desc& d, const DeviceInfo& dev) {
    Params p{};
    p.A = d.a, p.B = d.b, p.C = d.c;
    p.M = d.m, p.N = d.n, p.K = d.k;
    p.sa = d.batch > 1 ? d.stride_a : 0, p.sb = d.batch > 1 ? d.stride_b : 0, p.sc = d.batch > 1 ? d.stride_c : 0;
    p.post_row = static_cast<const float*>(d.post_row), p.post_full = d.post_full, p.post = d.post;
    p.b_nk  = d.b_layout == MIMK_B_NK;
    p.vec_a = d.k % 4 == 0 && aligned16(d.a) && p.sa % 4 == 0;
    p.vec_b = d.k % 4 == 0 && aligned16(d.b) && p.sb % 4 == 0;
    p.vec_c = d.n % 4 == 0 && aligned16(d.c) && p.sc % 4 == 0;
    p.status = dev.status_dev;
    return p;
}

int gemm_f32_tc(const mimk_gemm_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    if (gemm_tf32_preferred(d, dev->sm_count, gemm_f32_tc_us(d.m, d.n, d.k, d.batch, dev->sm_count))) {
        const int r = gemm_tf32(d, s);
        if (r != MIMK_E_UNSUPPORTED) return r;
    }
    Params p = product_params(d, *dev);
    return d.out_dtype == MIMK_BF16 ? plan_and_launch<float, __nv_bfloat16, false>(p, d.batch, dev->sm_count, s)
                                    : plan_and_launch<float, float, false>(p, d.batch, dev->sm_count, s);
}

// bf16 operands, an f32 result, extents or alignment that TMA cannot take. One piece per value, accumulators of 64 k and f32 adds
// between them: an accumulator kept over all of K (gemm_tc.cu) loses up to 2e-6 of a result that the CUDA-core fold gives to 4e-7,
// which a result in f32 shows (2000 x 5003 x 2048).
int gemm_bf16_chunked(const mimk_gemm_desc& d, cudaStream_t s) {
    if (d.in_dtype != MIMK_BF16 || d.out_dtype != MIMK_F32 || !extents_fit(d)) return MIMK_E_UNSUPPORTED;
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p = product_params(d, *dev);
    return plan_and_launch<__nv_bfloat16, float, false>(p, d.batch, dev->sm_count, s);
}

static int64_t conv_oh(const mimk_conv_desc& d) { return (d.h + 2 * d.pad_h - d.dil_h * (d.kh - 1) - 1) / d.stride_h + 1; }
static int64_t conv_ow(const mimk_conv_desc& d) { return (d.w + 2 * d.pad_w - d.dil_w * (d.kw - 1) - 1) / d.stride_w + 1; }

// Gathering costs more than the plan's k-blocks: rounds * (14 + 1.75 us per k-block), 7 + 1.25 up to 64 filters, within 15 % of the
// measured 214 us (16 x 128 x 56 x 56, 128 filters of 3 x 3), 69 (of 1 x 1), 79 (6 images), 380 (32 x 256 x 28 x 28, 256 of 3 x 3),
// 161 (64 filters). f32 over a cluster stays here: each CTA adds its own accumulators first, which leaves less rounding than one long
// sum (4 x 256 x 28 x 28, 256 filters of 3 x 3, 77 us and 1.50e-7 against 73 and 1.65e-7).
int conv_tc_preferred(const mimk_conv_desc& d, int sm_count) {
    const int64_t pixels = d.n * conv_oh(d) * conv_ow(d), k = d.cin * d.kh * d.kw;
    const Plan plan = make_plan(pixels, d.cout, k, 1, sm_count, true);
    if (d.dtype == MIMK_F32 && plan.split > 1) return 1;
    const int64_t tiles = ((pixels + BM - 1) / BM) * ((d.cout + plan.bn - 1) / plan.bn);
    const double kb = double((k + BK - 1) / BK), round = plan.bn == 128 ? 14.0 + 1.75 * kb : 7.0 + 1.25 * kb;
    return !conv_pieces_preferred(d, sm_count, plan.split > 1 ? plan.us : double((tiles + sm_count - 1) / sm_count) * round);
}

int conv_tc(const mimk_conv_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p{};
    const int64_t oh = conv_oh(d), ow = conv_ow(d);
    p.A = d.x, p.B = d.filters, p.C = d.out;
    p.M = d.n * oh * ow, p.N = d.cout, p.K = d.cin * d.kh * d.kw;
    p.conv = ConvShape{int(d.cin), int(d.h), int(d.w), int(d.kh), int(d.kw), int(oh), int(ow), int(d.stride_h), int(d.stride_w),
                       int(d.dil_h), int(d.dil_w), int(d.pad_h), int(d.pad_w), d.by_tap};
    p.b_nk   = 1;
    p.vec_b  = p.K % (d.dtype == MIMK_F32 ? 4 : 8) == 0 && aligned16(d.filters);
    p.status = dev->status_dev;
    return d.dtype == MIMK_F32 ? plan_and_launch<float, float, true>(p, 1, dev->sm_count, s)
                               : plan_and_launch<__nv_bfloat16, __nv_bfloat16, true>(p, 1, dev->sm_count, s);
}

}  // namespace mimk
