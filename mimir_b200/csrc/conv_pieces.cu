// Convolution as shifted products over an image that is laid out for the tensor cores once.
//
//   cut kernel    one pass over image and filters: channels last, the padding written as zeros, f32 values cut into three bf16 pieces
//                 (f32_split.cuh). With strides the pixels are dealt out to one grid per remainder of their coordinates, so that
//                 whatever the stride, window and dilation, the pixels that one tap reads for consecutive output positions are
//                 consecutive rows: tap (r, q) of output row v is row v + shift(r, q).
//   conv kernel   D[filter, position] over (tap, channel block of 32): both operands come by TMA (box of 32 channels x rows x pieces),
//                 no address arithmetic, tests or cutting in the loop. Positions run over the padded width (a window that crosses
//                 the edge of an image gives a column that is not stored: 7 % at 56 x 56 with a 3 x 3 window).
//     warps 0..7  add finished accumulators to sums in registers, store the tile by pixels (NCHW)
//     warp 8      TMA, warp 9 one thread issues the MMAs, 128 x BN x 16
//     warps 10, 11  read the cut kernel's records (f32) while the first tile is multiplied
// Every block of 64 channels goes into a fresh accumulator, and accumulators are added with ordinary f32 adds (the tensor core does not
// round its updates to nearest: over all of K in one accumulator a bf16 convolution was off by up to 2e-5 before its result was rounded).
// f32: the products of small pieces first. Cells that are not finite, or so small that bits lost in
// cutting tiny values (below 2^-109, f32_split.cuh) could show, are folded again by the scalar code: each block of the cut kernel says
// whether it lost any, and where one did, the storing warps look for the largest magnitudes that their cells come from.
//
// Against gathering the image by the contraction's own loaders (gemm_f32_tc.cu), where every value is fetched, tested and cut again
// for each tap that reads it: 16 x 128 x 56 x 56, 128 filters of 3 x 3, f32 214 -> 82 us (cut 16, conv 61), bf16 247 -> 40;
// 32 x 256 x 28 x 28, 256 of 3 x 3: f32 380 -> 195, bf16 462 -> 67. What bounds the f32 form: shared memory, 116 clocks per MMA of 96 (its
// operands 10 KB and 5 KB of TMA writes). Also measured: blocks of 32 channels in 64-byte rows, 105 us (TMA takes as long for a row of 64
// bytes as for one of 128); four accumulators of 128 columns, 114; MMAs issued by lane 0 in a branch of its own, 95.
#include <math_constants.h>

#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;
using namespace f32split;

namespace {

constexpr int BM = 128, BKC = 64, NUM_THREADS = 384, TMA_WARP = 8, MMA_WARP = 9, RECORDS_WARP = 10;
constexpr int STORE_REGS = 224, ISSUE_REGS = 56;  // two warpgroups and one, of 168 a thread at launch
static_assert(2 * STORE_REGS + ISSUE_REGS <= 3 * 168, "setmaxnreg waits for ever for more than the launch was given");
constexpr int A_BYTES = BM * BKC * 2;
constexpr int PITCH = 33, STAGING = 8 * 32 * PITCH * 4;  // a 32 x 32 block per storing warp

// A slot holds one piece of both operands, 64 channels. The pieces l, h of a block go through one ring and m through another, in the
// order the products need them, and leave as soon as their last product is done: l after two of six, m after five, h at the end.
template <int BN, int PIECES> struct Cfg {
    static constexpr int SLOT_BYTES = A_BYTES + BN * BKC * 2;
    static constexpr int ROOM  = (232448 - STAGING - 1024 - 512) / SLOT_BYTES;
    static constexpr int M_SLOTS = PIECES == 3 ? (ROOM >= 6 ? 2 : 1) : 0, X_SLOTS = ROOM - M_SLOTS;
    static constexpr int SMEM_BYTES = ROOM * SLOT_BYTES + STAGING + 1024 + 512;
    static constexpr int NACC = 512 / BN;  // accumulators in tensor memory
    static_assert(X_SLOTS >= 3 && X_SLOTS <= 6, "a block's l and h, and the next block's l on its way");
};

struct Bars {
    uint64_t full[6], empty[6], m_full[2], m_empty[2], acc_full[4], acc_empty[4];
    uint32_t tmem_base;
    int abort_flag;
    uint64_t records;                       // the cut kernel's records have been read
    uint32_t flags[2];                      // what two warps found there
};
struct Ring {  // a place in a ring of N slots
    uint32_t slot = 0, phase = 0;
    template <int N> __device__ __forceinline__ void step() {
        if (++slot == N) slot = 0, phase ^= 1u;
    }
};

// the image laid out: grids of [n, hq, wq] rows of `pitch` channels, one per remainder of the padded coordinates by the strides
// (one in all where the window is one pixel high / wide)
struct Shape {
    int n, cin, h, w, cout, kh, kw, oh, ow, stride_h, stride_w, dil_h, dil_w, pad_h, pad_w, by_tap;
    int hp, wp, hq, wq, grids_h, grids_w, pitch;
};
// What a block of the cut kernel says (f32): bits of a value were lost; a value was below all its pieces.
constexpr uint32_t LOST = 1, DEEP = 2;

struct Params {
    Shape c;
    const void* x;
    const void* filters;
    void* out;
    int64_t tiles_m, tiles_n;
    int* status;
    uint32_t* records;             // LOST and DEEP, a word per block of the cut kernel
    int64_t image_blocks, blocks;  // the image's, then the filters'
    const __nv_bfloat16 *image_h, *filters_h;  // the first pieces
};

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

template <class TIn>
__device__ __forceinline__ const TIn* filter_at(const Shape& c, const void* filters, int co, int ci, int tap) {
    const int taps = c.kh * c.kw;
    return static_cast<const TIn*>(filters) + int64_t(co) * c.cin * taps + (c.by_tap ? tap * c.cin + ci : ci * taps + tap);
}

// N neighbouring channels cut and stored, the pieces `piece` elements apart; flags: LOST and DEEP.
template <int PIECES, int N>
__device__ __forceinline__ void store_pieces(__nv_bfloat16* dst, int64_t piece, const float (&x)[N], uint32_t& flags) {
    float v[N];
    uint32_t lost = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = x[i];
#pragma unroll
    for (int t = 0; t < PIECES; ++t) {
        if constexpr (N == 4) *reinterpret_cast<uint2*>(dst + t * piece) = make_uint2(upper_halves(v[0], v[1]), upper_halves(v[2], v[3]));
        else *reinterpret_cast<uint32_t*>(dst + t * piece) = upper_halves(v[0], v[1]);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (t == 2) lost |= __float_as_uint(v[i]);
            v[i] = lower_part(v[i]);
        }
    }
    if (PIECES == 3 && (lost & lost_bits)) {
        flags |= LOST;
#pragma unroll
        for (int i = 0; i < N; ++i) flags |= x[i] != 0.f && fabsf(x[i]) < LOST_ABS ? DEEP : 0u;
    }
}

// Blocks [0, image_blocks): one padded image row that some tap reads and 64 channels, turned in shared memory; the others: 2048 filter elements
// each.
template <class TIn, int PIECES>
__global__ void __launch_bounds__(256) conv_cut_kernel(const Params p, __nv_bfloat16* __restrict__ image, __nv_bfloat16* __restrict__ filters,
                                                       int64_t image_piece, int64_t filter_piece) {
    __shared__ float tile[64][65];
    const Shape& c   = p.c;
    const int groups = (c.pitch + 63) / 64, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    uint32_t flags = 0;
    auto leave = [&]() {  // the block's record
        if constexpr (PIECES == 3) {
            uint32_t all = 0;
            if (__syncthreads_or(flags)) all = LOST | (__syncthreads_or(flags & DEEP) ? DEEP : 0u);
            if (threadIdx.x == 0) p.records[blockIdx.x] = all;
        }
    };
    const int64_t rows = p.image_blocks;
    if (blockIdx.x >= rows) {
        const int taps = c.kh * c.kw;
        int64_t i      = ((blockIdx.x - rows) * 256 + threadIdx.x) * 2;
        const int64_t n = int64_t(c.cout) * taps * c.pitch, step = (gridDim.x - rows) * 512;
        for (; i < n; i += step) {
            const int64_t t = i / c.pitch;
            const int ci = int(i - t * c.pitch), co = int(t / taps), tap = int(t - int64_t(co) * taps);
            const float v[2] = {ci < c.cin ? load1(filter_at<TIn>(c, p.filters, co, ci, tap)) : 0.f,
                                ci + 1 < c.cin ? load1(filter_at<TIn>(c, p.filters, co, ci + 1, tap)) : 0.f};
            store_pieces<PIECES>(filters + i, filter_piece, v, flags);
        }
        return leave();
    }
    const int64_t line = blockIdx.x / groups;
    // (rows and columns behind the padded image, which the grids have where it is no multiple of the strides, are written as zeros too)
    const int lines = c.hq * c.grids_h, width = c.wq * c.stride_w;
    const int c0 = int(blockIdx.x - line * groups) * 64, img = int(line / lines), in_image = int(line - int64_t(img) * lines);
    const int yq = in_image / c.grids_h, yg = in_image - yq * c.grids_h, yi = yq * c.stride_h + yg - c.pad_h;
    const bool inside = unsigned(yi) < unsigned(c.h);
    const int64_t plane = int64_t(c.h) * c.w, grid_rows = int64_t(c.n) * c.hq * c.wq;
    __nv_bfloat16* line_out = image + (int64_t(yg) * c.grids_w * grid_rows + (int64_t(img) * c.hq + yq) * c.wq) * c.pitch + c0;
    const TIn* src = static_cast<const TIn*>(p.x) + (int64_t(img) * c.cin + c0) * plane + int64_t(inside ? yi : 0) * c.w;
    for (int x0 = 0; x0 < width; x0 += 64) {
        const int xi  = x0 + tx - c.pad_w;
        const bool in0 = inside && unsigned(xi) < unsigned(c.w), in1 = inside && unsigned(xi + 32) < unsigned(c.w);
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int ch = ty + 8 * (j >> 1);
            v[j]         = ((j & 1) ? in1 : in0) && c0 + ch < c.cin ? load1(src + ch * plane + xi + (j & 1) * 32) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) tile[tx + (j & 1) * 32][ty + 8 * (j >> 1)] = v[j];
        __syncthreads();
        const int ch = (tx & 15) * 4;  // four channels of every sixteenth pixel: half a warp writes 128 bytes of each piece
        if (c0 + ch < c.pitch) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int px = j * 16 + ty * 2 + (tx >> 4), x = x0 + px;
                const int xg = c.stride_w == 1 ? 0 : x % c.stride_w, xq = c.stride_w == 1 ? x : x / c.stride_w;
                if (x >= width || xg >= c.grids_w) continue;
                const float w[4] = {tile[px][ch], tile[px][ch + 1], tile[px][ch + 2], tile[px][ch + 3]};
                store_pieces<PIECES>(line_out + (xg * grid_rows + xq) * c.pitch + ch, image_piece, w, flags);
            }
        }
        if (x0 + 64 < width) __syncthreads();
    }
    leave();
}

// The scalar fold of one cell, ascending (channel, kh, kw), one fma per step, padding read as zeros: for cells the pieces make
// non-finite (an operand was inf / NaN, or the sum overflowed), and for cells as small as the bits lost in cutting.
template <class TIn>
__device__ __noinline__ float scalar_fold(const Params& p, int img, int co, int y, int x) {
    const Shape& c = p.c;
    const TIn* im  = static_cast<const TIn*>(p.x) + int64_t(img) * c.cin * c.h * c.w;
    float v        = 0.f;
    for (int ci = 0; ci < c.cin; ++ci)
        for (int r = 0; r < c.kh; ++r)
            for (int q = 0; q < c.kw; ++q) {
                const int iy = y * c.stride_h - c.pad_h + r * c.dil_h, ix = x * c.stride_w - c.pad_w + q * c.dil_w;
                const bool in = unsigned(iy) < unsigned(c.h) && unsigned(ix) < unsigned(c.w);
                v = fmaf(in ? load1(im + (int64_t(ci) * c.h + iy) * c.w + ix) : 0.f, load1(filter_at<TIn>(c, p.filters, co, ci, r * c.kw + q)), v);
            }
    return v;
}

// Bits were lost in cutting: what the sums of 32 filters from m0 on at `width` positions from n0 on have to reach for that not to matter, 22
// bits above the loss, from the largest finite magnitudes among those filters and the rows of the grids that their taps read. (A sum of exactly
// zero can be short of something only if values lie below all their pieces.) By a whole warp, from the first pieces, which are short of
// a value by less than 2^-7 of it.
__device__ __noinline__ float lost_bound(const Params& p, int m0, int n0, int width) {
    const Shape& c = p.c;
    const int lane = threadIdx.x & 31;
    auto largest = [&](const __nv_bfloat16* from, int64_t elements) {  // a multiple of eight, 16-byte aligned
        uint32_t most = 0;
#pragma unroll 8
        for (int64_t i = lane * 8; i < elements; i += 256) {
            const uint4 q       = __ldg(reinterpret_cast<const uint4*>(from + i));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t lo = w[j] << 16 & 0x7fffffffu, hi = w[j] & 0x7fff0000u;
                most = max(most, max(lo < 0x7f800000u ? lo : 0u, hi < 0x7f800000u ? hi : 0u));
            }
        }
        return __uint_as_float(__reduce_max_sync(0xffffffffu, most));
    };
    const int64_t grid_rows = int64_t(c.n) * c.hq * c.wq, grids = int64_t(c.grids_h) * c.grids_w;
    const int64_t reach = int64_t((c.kh - 1) * c.dil_h / c.stride_h) * c.wq + (c.kw - 1) * c.dil_w / c.stride_w;
    float x = 0.f;
    for (int64_t g = 0; g < grids; ++g) {
        const int64_t first = g * grid_rows + n0, end = first + width + reach < grids * grid_rows ? first + width + reach : grids * grid_rows;
        if (first < end) x = fmaxf(x, largest(p.image_h + first * c.pitch, (end - first) * c.pitch));
    }
    const int64_t row = int64_t(c.kh) * c.kw * c.pitch;
    const float w = m0 < c.cout ? largest(p.filters_h + m0 * row, (c.cout - m0 < 32 ? c.cout - m0 : 32) * row) : 0.f;
    return float(c.cin * c.kh * c.kw) * (0x1p22f * 1.01f * LOST_ABS) * (x + w);
}

// The cells of 32 filters and `width` positions that a warp has just stored, those so small that lost bits could show folded again. (A pass of
// its own: in the store loop, where it is hardly ever needed, it made a layer of 113 us 1 to 2 us longer.) The look for the largest magnitudes
// is most of its time where few cells are that small: 16 x 128 x 56 x 56, 128 filters of 3 x 3, with one value of 1e-40 190 us, 86 without; where
// the rest of that image is zero, 1.4 ms (18 with each position's cells folded by one lane).
__device__ __noinline__ void fold_small_again(const Params& p, int m0, int n0, int width, bool zeros) {
    const Shape& c    = p.c;
    const float bound = lost_bound(p, m0, n0, width);
    const int per_image = c.hq * c.wq, rows = c.cout - m0 < 32 ? c.cout - m0 : 32;
    const int64_t pixels = int64_t(c.oh) * c.ow;
    const int lane = threadIdx.x & 31;
    for (int v0 = n0; v0 < n0 + width; v0 += 32) {
        auto cell = [&](int v, auto&& use) {  // use(the first filter's cell at the position, if there is one; its image, row and column)
            const int img = v / per_image, in = v - img * per_image, y = in / c.wq, x = in - y * c.wq;
            if (img < c.n && y < c.oh && x < c.ow)
                use(static_cast<float*>(p.out) + (int64_t(img) * c.cout + m0) * pixels + (int64_t(y) * c.ow + x), img, y, x);
        };
        uint32_t again = 0;  // filters, at this lane's position
        cell(v0 + lane, [&](const float* at, int, int, int) {
            for (int r = 0; r < rows; ++r) {
                const float value = at[r * pixels];
                again |= uint32_t(fabsf(value) < bound && (value != 0.f || zeros)) << r;
            }
        });
        // a lane folds its position's cells, or each lane its filter's at the positions concerned (often few, of all filters)
        uint32_t positions = __ballot_sync(0xffffffffu, again != 0);
        if (__reduce_max_sync(0xffffffffu, uint32_t(__popc(again))) <= uint32_t(__popc(positions))) {
            cell(v0 + lane, [&](float* at, int img, int y, int x) {
                for (; again; again &= again - 1) {
                    const int r    = __ffs(again) - 1;
                    at[r * pixels] = scalar_fold<float>(p, img, m0 + r, y, x);
                }
            });
        } else {
            for (; positions; positions &= positions - 1) {
                const int from = __ffs(positions) - 1;
                if (__shfl_sync(0xffffffffu, again, from) >> lane & 1)
                    cell(v0 + from, [&](float* at, int img, int y, int x) { at[lane * pixels] = scalar_fold<float>(p, img, m0 + lane, y, x); });
            }
        }
        __syncwarp();
    }
}

template <int BN, int PIECES, class T>
__global__ void __launch_bounds__(NUM_THREADS, 1)
conv_pieces_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ Params p) {
    using C = Cfg<BN, PIECES>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw), base = (raw_addr + 1023u) & ~1023u;
    uint8_t* after           = smem_raw + (base - raw_addr) + C::ROOM * C::SLOT_BYTES;
    Bars* bars               = reinterpret_cast<Bars*>(after + STAGING);
    volatile int* abort_flag = &bars->abort_flag;
    const Shape& c           = p.c;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t num_tiles = p.tiles_m * p.tiles_n;
    const int taps = c.kh * c.kw, cblocks = (c.cin + BKC - 1) / BKC, num_kb = taps * cblocks;

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::X_SLOTS; ++i) {
            mbar_init(smem_u32(&bars->full[i]), 1);
            mbar_init(smem_u32(&bars->empty[i]), 1);
        }
        for (int i = 0; i < C::M_SLOTS; ++i) {
            mbar_init(smem_u32(&bars->m_full[i]), 1);
            mbar_init(smem_u32(&bars->m_empty[i]), 1);
        }
        for (int b = 0; b < C::NACC; ++b) {
            mbar_init(smem_u32(&bars->acc_full[b]), 1);
            mbar_init(smem_u32(&bars->acc_empty[b]), 8);
        }
        mbar_init(smem_u32(&bars->records), 2);
        bars->abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&bars->tmem_base), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

    const uint32_t m_base = base + C::X_SLOTS * C::SLOT_BYTES;

    if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGS));
    if (warp == TMA_WARP) {
        if (lane == 0) {
            Ring x, m;
            bool ok = true;
            const int grid_rows = c.n * c.hq * c.wq;
            auto load = [&](uint32_t full, uint32_t empty, uint32_t phase, uint32_t at, int ax, int bx, int m0, int row, int piece) {
                if (!(ok = mbar_wait(empty, phase ^ 1u, abort_flag))) return;
                mbar_expect_tx(full, C::SLOT_BYTES);
                tma_load_3d(at, &tmA, ax, m0, piece, full);
                tma_load_3d(at + A_BYTES, &tmB, bx, row, piece, full);
            };
            for (int64_t tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                const int m0 = int(tile % p.tiles_m) * BM, n0 = int(tile / p.tiles_m) * BN;
                for (int r = 0, tap = 0; r < c.kh && ok; ++r)
                    for (int q = 0; q < c.kw && ok; ++q, ++tap) {
                        const int dy = r * c.dil_h, dx = q * c.dil_w;
                        const int grid = (dy % c.stride_h) * c.grids_w + dx % c.stride_w;
                        const int row  = n0 + grid * grid_rows + dy / c.stride_h * c.wq + dx / c.stride_w;
                        for (int cb = 0; cb < cblocks && ok; ++cb) {
                            const int ax = tap * c.pitch + cb * BKC, bx = cb * BKC;
                            for (int t = PIECES == 3 ? 2 : 0; t >= 0 && ok; t -= 2) {  // l, h
                                load(smem_u32(&bars->full[x.slot]), smem_u32(&bars->empty[x.slot]), x.phase, base + x.slot * C::SLOT_BYTES, ax, bx, m0, row, t);
                                x.step<C::X_SLOTS>();
                            }
                            if constexpr (PIECES == 3) {
                                if (!ok) break;
                                load(smem_u32(&bars->m_full[m.slot]), smem_u32(&bars->m_empty[m.slot]), m.phase, m_base + m.slot * C::SLOT_BYTES, ax, bx, m0, row, 1);
                                m.step<C::M_SLOTS>();
                            }
                        }
                    }
            }
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        {
            // (the whole warp runs, one lane issues: with lane 0 alone in the branch the descriptors are not known to be uniform, and moving them
            // costs about 50 clocks per MMA)
            const bool leader = elect_one();
            const uint32_t idesc = idesc_bf16_f32(BM, BN, 0, 0);
            Ring x, m;
            Ring acc;
            bool ok = true;
            const uint64_t desc0 = smem_desc_sw128(base, 16, 1024);
            // the product of the pieces in two places over `steps` times 16 channels; first: into a fresh accumulator
            auto product = [&](uint32_t d, uint32_t a, uint32_t b, int steps, bool first) {
                const uint64_t da = desc0 + a * (C::SLOT_BYTES >> 4), db = desc0 + b * (C::SLOT_BYTES >> 4) + (A_BYTES >> 4);
                if (leader)
#pragma unroll
                    for (int k = 0; k < BKC / 16; ++k)
                        if (k < steps) mma_f16_ss(d, da + k * 2, db + k * 2, idesc, (!first || k > 0) ? 1u : 0u);
            };
            auto commit = [&](uint32_t bar) { if (leader) mma_commit(bar); };
            auto wait = [&](uint64_t& bar, uint32_t phase) { return ok = warp_wait(smem_u32(&bar), phase, abort_flag); };
            for (int64_t tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                for (int kb = 0, cb = 0; kb < num_kb; ++kb) {
                    const int left = c.cin - cb * BKC, steps = left >= BKC ? BKC / 16 : (left + 15) / 16;
                    if (++cb == cblocks) cb = 0;
                    if (!wait(bars->acc_empty[acc.slot], acc.phase ^ 1u)) break;
                    const uint32_t d = tmem_base + acc.slot * BN;
                    if constexpr (PIECES == 3) {
                        const uint32_t lo = x.slot;
                        const uint32_t lo_empty = smem_u32(&bars->empty[x.slot]);
                        if (!wait(bars->full[x.slot], x.phase)) break;
                        x.step<C::X_SLOTS>();
                        const uint32_t hi = x.slot;
                        const uint32_t hi_empty = smem_u32(&bars->empty[x.slot]);
                        if (!wait(bars->full[x.slot], x.phase)) break;
                        x.step<C::X_SLOTS>();
                        tc_fence_after();
                        product(d, lo, hi, steps, true);
                        product(d, hi, lo, steps, false);
                        commit(lo_empty);
                        const uint32_t mid = C::X_SLOTS + m.slot;
                        if (!wait(bars->m_full[m.slot], m.phase)) break;
                        tc_fence_after();
                        product(d, mid, mid, steps, false);
                        product(d, mid, hi, steps, false);
                        product(d, hi, mid, steps, false);
                        commit(smem_u32(&bars->m_empty[m.slot]));
                        m.step<C::M_SLOTS>();
                        product(d, hi, hi, steps, false);
                        commit(hi_empty);
                    } else {
                        if (!wait(bars->full[x.slot], x.phase)) break;
                        tc_fence_after();
                        product(d, x.slot, x.slot, steps, true);
                        commit(smem_u32(&bars->empty[x.slot]));
                        x.step<C::X_SLOTS>();
                    }
                    commit(smem_u32(&bars->acc_full[acc.slot]));
                    acc.step<C::NACC>();
                }
            }
        }
        __syncwarp();
    } else if (PIECES == 3) {
        uint32_t flags = 0;
#pragma unroll 8
        for (int64_t i = (threadIdx.x - RECORDS_WARP * 32) * 4; i < p.blocks; i += 256) {
            const uint4 r = __ldg(reinterpret_cast<const uint4*>(p.records + i));
            flags |= r.x | (i + 1 < p.blocks ? r.y : 0u) | (i + 2 < p.blocks ? r.z : 0u) | (i + 3 < p.blocks ? r.w : 0u);
        }
        flags = __reduce_or_sync(0xffffffffu, flags);
        if (lane == 0) {
            bars->flags[warp - RECORDS_WARP] = flags;
            mbar_arrive(smem_u32(&bars->records));
        }
        __syncwarp();
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(STORE_REGS));
        constexpr int HALF = BN / 2;
        static_assert(HALF % 32 == 0, "blocks of 32 columns");
        const uint32_t quarter = uint32_t(warp & 3), col0 = uint32_t(warp >> 2) * HALF;
        float* block = reinterpret_cast<float*>(after) + warp * (32 * PITCH);
        Ring acc;
        bool ok      = true;
        const int per_image  = c.hq * c.wq;
        const int64_t pixels = int64_t(c.oh) * c.ow;
        for (int64_t tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
            const int m0 = int(tile % p.tiles_m) * BM, n0 = int(tile / p.tiles_m) * BN;
            float sum[HALF];
#pragma unroll
            for (int i = 0; i < HALF; ++i) sum[i] = 0.f;
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!(ok = warp_wait(smem_u32(&bars->acc_full[acc.slot]), acc.phase, abort_flag))) break;
                tc_fence_after();
                // as many columns requested as registers allow, then one wait: a read of tensor memory stands in line behind the MMAs that are
                // queued
                const uint32_t t0  = tmem_base + acc.slot * BN + col0 + ((quarter * 32u) << 16);
                constexpr int WIDE = HALF <= 96 ? HALF : 64;
#pragma unroll
                for (int i0 = 0; i0 < HALF; i0 += WIDE) {
                    uint32_t r[WIDE / 32][32];
#pragma unroll
                    for (int i = 0; i < WIDE / 32; ++i) tmem_ld_32x32(t0 + i0 + i * 32, r[i]);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < WIDE; ++i) sum[i0 + i] += __uint_as_float(r[i / 32][i % 32]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[acc.slot]));
                acc.step<C::NACC>();
            }
            if (PIECES == 3) ok = ok && warp_wait(smem_u32(&bars->records), 0, abort_flag);  // (complete from the first tile on)
            if (!ok) break;
            const int rows = c.cout - (m0 + int(quarter) * 32);
#pragma unroll
            for (int i = 0; i < HALF; i += 32) {
#pragma unroll
                for (int j = 0; j < 32; ++j) block[lane * PITCH + j] = sum[i + j];
                __syncwarp();
                const int v = n0 + int(col0) + i + lane, img = v / per_image, in = v - img * per_image, y = in / c.wq, x = in - y * c.wq;
                const bool there = img < c.n && y < c.oh && x < c.ow;
                const int co     = m0 + int(quarter) * 32;
                T* dst           = static_cast<T*>(p.out) + (int64_t(img) * c.cout + co) * pixels + (int64_t(y) * c.ow + x);
                float value[32], probe = 0.f;  // (a sum of v * 0 is zero where all are finite)
#pragma unroll
                for (int r = 0; r < 32; ++r) value[r] = block[r * PITCH + lane], probe = fmaf(value[r], 0.f, probe);
                if (there) {
#pragma unroll
                    for (int r = 0; r < 32; ++r)
                        if (r < rows) dst[r * pixels] = T(value[r]);
                    if (probe != 0.f)
                        for (int r = 0; r < 32 && r < rows; ++r)
                            if (!isfinite(block[r * PITCH + lane])) dst[r * pixels] = T(scalar_fold<T>(p, img, co + r, y, x));
                }
                __syncwarp();
            }
            if constexpr (PIECES == 3) {
                const uint32_t flags = bars->flags[0] | bars->flags[1];
                if (flags) fold_small_again(p, m0 + int(quarter) * 32, n0 + int(col0), HALF, flags & DEEP);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

Shape make_shape(const mimk_conv_desc& d) {
    Shape c{};
    c.n = int(d.n), c.cin = int(d.cin), c.h = int(d.h), c.w = int(d.w), c.cout = int(d.cout), c.kh = int(d.kh), c.kw = int(d.kw);
    c.stride_h = int(d.stride_h), c.stride_w = int(d.stride_w), c.dil_h = int(d.dil_h), c.dil_w = int(d.dil_w);
    c.pad_h = int(d.pad_h), c.pad_w = int(d.pad_w), c.by_tap = d.by_tap;
    c.hp = c.h + 2 * c.pad_h, c.wp = c.w + 2 * c.pad_w;
    c.oh = (c.hp - c.dil_h * (c.kh - 1) - 1) / c.stride_h + 1, c.ow = (c.wp - c.dil_w * (c.kw - 1) - 1) / c.stride_w + 1;
    c.hq = (c.hp + c.stride_h - 1) / c.stride_h, c.wq = (c.wp + c.stride_w - 1) / c.stride_w;
    c.grids_h = c.kh == 1 ? 1 : c.stride_h, c.grids_w = c.kw == 1 ? 1 : c.stride_w;
    c.pitch = (c.cin + 15) & ~15;  // (whole sectors: 24 channels in rows of 48 bytes 78 us, 45 now; 16 x 24 x 56 x 56, 128 filters of 3 x 3, f32)
    return c;
}

struct Sizes {
    int64_t image, filters;  // elements of one piece
    size_t bytes(int pieces) const { return size_t(pieces) * size_t(image + filters) * 2 + 512; }
};
Sizes make_sizes(const Shape& c) {
    return Sizes{int64_t(c.grids_h) * c.grids_w * c.n * c.hq * c.wq * c.pitch, int64_t(c.cout) * c.kh * c.kw * c.pitch};
}

// Tile width: the one with the least estimated time: launches, a pass over the image at 4.1 TB/s, and rounds of a tile per SM. Measured
// per block of 64 channels, f32: 1.52 us (128 wide) and 1.85 (192), what the tile's shared-memory traffic takes at 106 bytes a clock
// (of 288 and 360 KB, a third of it written by TMA); bf16 0.5, 0.63 and 0.82 (256), the loads and what reading the accumulators
// leaves uncovered (one accumulator over all of K: 0.45, 0.55, 0.7; one per 128 channels saves a third of that, and rounds more).
struct Plan {
    int bn;
    double us;
};
Plan make_plan(const Shape& c, int pieces, int sm_count) {
    const int64_t positions = int64_t(c.n) * c.hq * c.wq, tiles_m = (c.cout + BM - 1) / BM;
    const double kb = double(c.kh) * c.kw * ((c.cin + BKC - 1) / BKC);
    const Sizes s   = make_sizes(c);
    const double bytes = double(c.n) * c.cin * c.h * c.w * (pieces == 3 ? 4 : 2) + double(s.bytes(pieces));
    const double part  = double((c.cin < BKC ? c.cin : BKC) + 15) / 16 / 4;  // of a block's MMAs that are issued
    Plan best{128, 1e300};
    for (int bn : {128, 192, 256}) {
        if (pieces == 3 && bn == 256) continue;
        const double rounds = double((tiles_m * ((positions + bn - 1) / bn) + sm_count - 1) / sm_count);
        const double loads = pieces == 3 ? (bn == 128 ? 0.95 : 1.2) : (bn == 128 ? 0.5 : bn == 192 ? 0.63 : 0.82);
        const double mmas  = (pieces == 3 ? (bn == 128 ? 1.52 : 1.85) : 0.0) * part;
        const double us    = 11.0 + bytes / 4.1e6 + rounds * (4.0 + kb * (mmas > loads ? mmas : loads));
        if (us < best.us) best = Plan{bn, us};
    }
    return best;
}

int make_tmap(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t pieces, uint64_t piece_elems, uint32_t box_rows) {
    cuuint64_t dims[3]    = {inner, rows, pieces};
    cuuint64_t strides[2] = {inner * 2, piece_elems * 2};
    cuuint32_t box[3]     = {BKC, box_rows, 1};
    return encode_tmap_bf16(out, base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int BN, int PIECES, class T>
int launch(Params& p, __nv_bfloat16* image, __nv_bfloat16* filters, const Sizes& sizes, int sm_count, cudaStream_t s) {
    const Shape& c = p.c;
    auto kern      = conv_pieces_kernel<BN, PIECES, T>;
    constexpr int SMEM = Cfg<BN, PIECES>::SMEM_BYTES;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[dev & 63] = true;
    }
    const int64_t positions = int64_t(c.n) * c.hq * c.wq;
    CUtensorMap tmA, tmB;
    MIMK_TRY(make_tmap(&tmA, filters, uint64_t(c.kh) * c.kw * c.pitch, uint64_t(c.cout), PIECES, uint64_t(sizes.filters), BM));
    MIMK_TRY(make_tmap(&tmB, image, uint64_t(c.pitch), uint64_t(positions) * c.grids_h * c.grids_w, PIECES, uint64_t(sizes.image), BN));
    p.tiles_m = (c.cout + BM - 1) / BM, p.tiles_n = (positions + BN - 1) / BN;
    const int64_t tiles = p.tiles_m * p.tiles_n;
    kern<<<unsigned(tiles < sm_count ? tiles : sm_count), NUM_THREADS, SMEM, s>>>(tmA, tmB, p);
    return launch_status();
}

}  // namespace

// Whether this route takes the convolution: 16 channels and more (a row of fewer takes TMA as long: 25 x 3 x 56 x 61, 128 filters of 3 x 3, 161 us
// against 106), 31-bit rows, a buffer of at most 1 GiB, an estimate below `other_us`, and f32 only where the error is no larger than the
// gathering kernel's. That one's accumulators hold 64 k whatever the channels; here it is one per tap and 64 channels, and the more of them are
// added the larger the error. Measured, here / gathered, 1e-7: up to nine accumulators 1.15 / 1.26 (16 channels), 1.35 / 1.35 (56); whole blocks of
// 64 channels the same at any window; 32 channels 1.41 / 1.41 in 25 taps, 1.65 / 1.54 in 49; 24 channels 1.40 / 1.38, 1.65 / 1.48, and 2.20 / 1.74 in
// 121; 56 in 25 taps 1.53 / 1.51; 72 in 9 taps (18 accumulators) 1.46 / 1.40.
int conv_pieces_preferred(const mimk_conv_desc& d, int sm_count, double other_us) {
    if (d.cin < 16 || d.n < 1 || d.cout < 1 || d.n >= (1 << 30) || d.cout >= (1 << 30)) return 0;
    const double rows = double(d.n) * (double(d.h) + 2.0 * double(d.pad_h) + double(d.stride_h)) * (double(d.w) + 2.0 * double(d.pad_w) + double(d.stride_w));
    if (rows >= double(1 << 30) || double(d.cin + 16) * double(d.kh) * double(d.kw) >= double(1 << 30)) return 0;
    const Shape c    = make_shape(d);
    const int pieces = d.dtype == MIMK_F32 ? 3 : 1;
    const int accumulators = c.kh * c.kw * ((c.cin + BKC - 1) / BKC);
    if (pieces == 3 && c.cin % BKC != 0 && accumulators > (c.cin == 32 ? 25 : 10)) return 0;
    if (make_sizes(c).bytes(pieces) > (size_t(1) << 30)) return 0;
    return make_plan(c, pieces, sm_count).us < other_us;
}

// MIMK_E_UNSUPPORTED, with nothing launched, where the buffer cannot be had: under stream capture (a graph must not hold on to the
// cached buffer) and when there is no memory for it.
int conv_pieces(const mimk_conv_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    MIMK_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) return MIMK_E_UNSUPPORTED;
    Params p{};
    p.c = make_shape(d);
    const int pieces  = d.dtype == MIMK_F32 ? 3 : 1;
    const Sizes sizes = make_sizes(p.c);
    void* scratch     = nullptr;
    const Shape& c    = p.c;
    const int64_t extra = (sizes.filters + 2047) / 2048;
    p.image_blocks      = int64_t(c.n) * c.hq * c.grids_h * ((c.pitch + 63) / 64);
    p.blocks            = p.image_blocks + (extra < 1024 ? extra : 1024);
    ScratchLease lease;  // of both launches
    if (lease.take(sizes.bytes(pieces) + size_t(p.blocks) * 4 + 512, &scratch, s) != MIMK_OK) {
        cudaGetLastError();
        return MIMK_E_UNSUPPORTED;
    }
    auto* image   = static_cast<__nv_bfloat16*>(scratch);
    auto* filters = reinterpret_cast<__nv_bfloat16*>((reinterpret_cast<uintptr_t>(image + pieces * sizes.image) + 255) & ~uintptr_t(255));
    p.x = d.x, p.filters = d.filters, p.out = d.out, p.status = dev->status_dev;
    p.image_h = image, p.filters_h = filters;
    p.records = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(filters + pieces * sizes.filters) + 255) & ~uintptr_t(255));
    const unsigned blocks = unsigned(p.blocks);
    if (pieces == 3) conv_cut_kernel<float, 3><<<blocks, 256, 0, s>>>(p, image, filters, sizes.image, sizes.filters);
    else conv_cut_kernel<__nv_bfloat16, 1><<<blocks, 256, 0, s>>>(p, image, filters, sizes.image, sizes.filters);
    MIMK_TRY(launch_status());
    const int bn = make_plan(c, pieces, dev->sm_count).bn;
    if (pieces == 3)
        return bn == 128 ? launch<128, 3, float>(p, image, filters, sizes, dev->sm_count, s) : launch<192, 3, float>(p, image, filters, sizes, dev->sm_count, s);
    return bn == 128   ? launch<128, 1, __nv_bfloat16>(p, image, filters, sizes, dev->sm_count, s)
           : bn == 192 ? launch<192, 1, __nv_bfloat16>(p, image, filters, sizes, dev->sm_count, s)
                       : launch<256, 1, __nv_bfloat16>(p, image, filters, sizes, dev->sm_count, s);
}

}  // namespace mimk
