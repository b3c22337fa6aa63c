// f32 contraction on the tensor cores with f32-grade accuracy, in one launch.
//
// Every tensor program the reference can lower today is f32 (its Ring has one element type and the LLVM emitter knows
// half / float / double only, MimIR src/mim/plug/ll/ll.cpp:139-145), so the f32 `product_2d` is the path existing
// programs take. Each operand value is cut into three bf16 pieces that sum to it exactly, and the six products that matter
// are accumulated by tcgen05.mma (f32_split.cuh).
//
//   loaders      8 or 16 warps: read the operands (next k-block into registers while the present one is cut and stored), write
//                the pieces into shared-memory tiles, and add each finished k-block's accumulator to sums in registers
//   last warp    one thread issues the MMAs: 128 x BN x 32 per k-block, every k-block into a fresh one of four accumulators
// The tensor core does not round its accumulator updates to nearest; with one k-block (2 x 6 updates, the small terms first)
// per accumulator and ordinary f32 adds between k-blocks, the error stays that of an f32 fold for any K (2-norm 1.1e-7 to
// 1.3e-7 for K from 64 to 4096; the scalar fold has 1.5e-7 to 1.2e-6).
//
// The operands are read as the caller has them: any extents, strides and alignment, no copies, no scratch. What bounds it:
// the loaders' instructions and shared-memory bandwidth (a k-block of 128 x 128 moves 96 KB into the MMA and 48 KB from the
// loaders, 1150 clocks, against 770 of arithmetic). Too few tiles for the chip: the k-blocks of one tile are dealt out to a
// cluster of up to eight CTAs, which add their partial tiles through distributed shared memory in a fixed order.
#include <cstdlib>

#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;
using namespace f32split;

namespace {

constexpr int BM = 128;
constexpr int NBUF = 4;         // accumulators in tensor memory
constexpr int LAG = 2;          // k-blocks between storing one and adding its accumulator
constexpr int GROUP_M = 16;
constexpr int A_PIECE = BM * BK * 2;

template <int BN, class TIn> struct Cfg {
    static constexpr int PIECES  = sizeof(TIn) == 4 ? 3 : 1;
    static constexpr int STAGES  = BN == 128 || PIECES == 1 ? 4 : 3;  // BN 64: two CTAs can share an SM
    static constexpr int B_PIECE = BN * BK * 2;
    static constexpr int STAGE_BYTES = PIECES * (A_PIECE + B_PIECE);
    static constexpr int PITCH = BN + 4;  // floats per row of the partial tile, which lies over the stages
    static constexpr int TILE_BYTES = STAGES * STAGE_BYTES > BM * PITCH * 4 ? STAGES * STAGE_BYTES : BM * PITCH * 4;
    static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 256;
};

struct Bars {
    uint64_t full[4], empty[4], acc_full[NBUF];
    uint32_t tmem_base;
    int abort_flag;
};

// A convolution as a contraction: row = output pixel (image, oh, ow), k = (input channel, kh, kw), column = filter. Rows of the
// patch matrix are gathered from the image as the loaders read them.
struct ConvShape {
    int cin, h, w, kh, kw, oh, ow, stride_h, stride_w, dil_h, dil_w, pad_h, pad_w;
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
__device__ __forceinline__ float ld_cluster1(uint32_t saddr, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld_32x16(taddr, r); }

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

// LOADERS: 512 threads, and the SM for one CTA alone; or 256, and two CTAs (BN 64) that hide each other's waits.
template <int BN, int LOADERS, class TIn, class TOut, bool CONV>
__global__ void __launch_bounds__(LOADERS + 32, LOADERS == 512 ? 1 : 2) gemm_f32_tc_kernel(const Params p) {
    using C = Cfg<BN, TIn>;
    constexpr int PIECES = C::PIECES, MMA_WARP = LOADERS / 32;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;
    Bars* bars              = reinterpret_cast<Bars*>(smem_raw + (base - raw_addr) + C::TILE_BYTES);
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int64_t tiles = p.tiles_m * p.tiles_n;
    const int rank      = int(blockIdx.x % unsigned(p.split));  // a cluster is `split` consecutive CTAs
    const int64_t item  = blockIdx.x / unsigned(p.split), bz = item / tiles;
    int64_t tm, tn;
    tile_coords(item - bz * tiles, p.tiles_m, p.tiles_n, tm, tn);
    const int64_t m0 = tm * BM, n0 = tn * BN;
    const TIn* A = static_cast<const TIn*>(p.A) + bz * p.sa;
    const TIn* B = static_cast<const TIn*>(p.B) + bz * p.sb;
    const int64_t all_kb = (p.K + BK - 1) / BK, per = (all_kb + p.split - 1) / p.split;
    const int64_t kb0    = rank * per < all_kb ? rank * per : all_kb;
    const int num_kb     = int(kb0 + per < all_kb ? per : all_kb - kb0);

    // What a loader thread holds of one k-block: one or two eight-k units of A and at most one of B. Where memory runs along k a
    // unit's row is u / 4; where it runs along the rows (B stored [K, N], the pixels of an image) a warp takes one unit of 32
    // neighbouring rows. The first loads are on their way while the barriers and the tensor memory are set up.
    constexpr int UA = BM * 4 / LOADERS;
    static_assert(BN * 4 <= LOADERS, "one unit of B per thread");
    const int across = (warp >> 2) * 32 + lane, unit = warp & 3;
    const bool has_b = BN * 4 == LOADERS || tid < BN * 4;
    const int b_row = p.b_nk ? tid >> 2 : across, b_unit = p.b_nk ? tid & 3 : unit;
    float fa[UA][8], fb[8];
    const TIn* a_at[UA];           // CONV: the first tap of the pixel's window; else the thread's row of A, at its unit
    int rows_in[UA], cols_in[UA];  // CONV: bit i: tap row / column i of this pixel lies inside the image
    const ConvShape& cv = p.conv;
#pragma unroll
    for (int i = 0; i < UA; ++i) {
        rows_in[i] = cols_in[i] = 0;
        if (CONV) {
            const int64_t row = m0 + across + i * (LOADERS / 4);
            const int pixels  = cv.oh * cv.ow;
            const int64_t img = row / pixels;
            const int pix = int(row - img * pixels), y = pix / cv.ow;
            const int ih0 = y * cv.stride_h - cv.pad_h, iw0 = (pix - y * cv.ow) * cv.stride_w - cv.pad_w;
            a_at[i] = A + img * (int64_t(cv.cin) * cv.h * cv.w) + (int64_t(ih0) * cv.w + iw0);  // only taps inside are read
            if (row < p.M) {
                for (int r = 0; r < cv.kh; ++r) rows_in[i] |= int(unsigned(ih0 + r * cv.dil_h) < unsigned(cv.h)) << r;
                for (int q = 0; q < cv.kw; ++q) cols_in[i] |= int(unsigned(iw0 + q * cv.dil_w) < unsigned(cv.w)) << q;
            }
        } else {
            const int u = tid + i * LOADERS;
            a_at[i] = A + (m0 + (u >> 2)) * p.K + (u & 3) * 8;
        }
    }
    const TIn* b_at = p.b_nk ? B + (n0 + b_row) * p.K + b_unit * 8 : B + int64_t(b_unit * 8) * p.N + n0 + b_row;
    auto fetch = [&](int kb) {
        const int64_t k0 = (kb0 + kb) * BK;
        if (CONV) {
            const int k = int(k0) + unit * 8, taps = cv.kh * cv.kw;
            const int ci = k / taps;
            int r = (k - ci * taps) / cv.kw, q = k - ci * taps - r * cv.kw;
            int off = ci * (cv.h * cv.w) + r * cv.dil_h * cv.w + q * cv.dil_w;
            const int next_row = cv.dil_h * cv.w - cv.kw * cv.dil_w, next_plane = cv.h * cv.w - cv.kh * cv.dil_h * cv.w;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
#pragma unroll
                for (int i = 0; i < UA; ++i) {
                    const bool in = (rows_in[i] >> r) & (cols_in[i] >> q) & int(k + j < int(p.K));
                    fa[i][j]      = in ? load1(a_at[i] + off) : 0.f;
                }
                off += cv.dil_w;
                if (++q == cv.kw) {
                    q = 0, off += next_row;
                    if (++r == cv.kh) r = 0, off += next_plane;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < UA; ++i) {
                const int u = tid + i * LOADERS;
                load8(fa[i], a_at[i] + k0, m0 + (u >> 2) < p.M, int(p.K - k0) - (u & 3) * 8, p.vec_a);
            }
        }
        if (has_b) {
            const bool there = n0 + b_row < p.N;
            const int left   = int(p.K - k0) - b_unit * 8;
            if (p.b_nk) {
                load8(fb, b_at + k0, there, left, p.vec_b);
            } else {
                const TIn* at = b_at + k0 * p.N;
#pragma unroll
                for (int j = 0; j < 8; ++j) fb[j] = there && j < left ? load1(at + j * p.N) : 0.f;
            }
        }
    };
    auto store = [&](uint32_t s0) {
#pragma unroll
        for (int i = 0; i < UA; ++i) {
            const int u = tid + i * LOADERS;
            split_store8<PIECES>(s0 + (CONV ? unit_offset(across + i * (LOADERS / 4), unit) : unit_offset(u >> 2, u & 3)), A_PIECE, fa[i]);
        }
        if (has_b) split_store8<PIECES>(s0 + PIECES * A_PIECE + unit_offset(b_row, b_unit), C::B_PIECE, fb);
    };
    if (warp < MMA_WARP && num_kb > 0) fetch(0);

    if (tid == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), LOADERS / 32);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (int b = 0; b < NBUF; ++b) mbar_init(smem_u32(&bars->acc_full[b]), 1);
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&bars->tmem_base), NBUF * BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

    if (warp == MMA_WARP) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16_f32(BM, BN, 0, 0);
            uint32_t stage = 0, phase = 0;
            for (int kb = 0; kb < num_kb; ++kb) {
                // A full stage also says that every loader warp has read the accumulator of k-block kb - 1 - LAG, so the buffer
                // of kb - NBUF is free.
                if (!mbar_wait(smem_u32(&bars->full[stage]), phase, abort_flag)) break;
                tc_fence_after();
                const uint32_t s0 = base + stage * C::STAGE_BYTES;
                mma_six<PIECES>(tmem_base + (kb & (NBUF - 1)) * BN, s0, A_PIECE, s0 + PIECES * A_PIECE, C::B_PIECE, idesc);
                mma_commit(smem_u32(&bars->empty[stage]));
                mma_commit(smem_u32(&bars->acc_full[kb & (NBUF - 1)]));
                if (++stage == C::STAGES) stage = 0, phase ^= 1u;
            }
        }
        __syncwarp();
    } else {
        static_assert(NBUF > LAG + 1, "an accumulator is read before its buffer comes round again");
        constexpr int COLS = BN / (LOADERS / 128);  // accumulator columns per warp
        float sum[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
        const uint32_t quarter = uint32_t(warp & 3), col0 = uint32_t(warp >> 2) * COLS;
        auto drain = [&](int kb) {
            const int b = kb & (NBUF - 1);
            if (!warp_wait(smem_u32(&bars->acc_full[b]), uint32_t(kb / NBUF) & 1u, abort_flag)) return false;
            tc_fence_after();
            uint32_t r[COLS];
            tmem_ld_cols(tmem_base + b * BN + col0 + ((quarter * 32u) << 16), r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < COLS; ++i) sum[i] += __uint_as_float(r[i]);
            tc_fence_before();
            return true;
        };
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (int kb = 0; kb < num_kb; ++kb) {
            if (!(ok = warp_wait(smem_u32(&bars->empty[stage]), phase ^ 1u, abort_flag))) break;
            store(base + stage * C::STAGE_BYTES);
            fence_proxy_async_smem();  // the MMA reads shared memory through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->full[stage]));
            if (++stage == C::STAGES) stage = 0, phase ^= 1u;
            if (kb + 1 < num_kb) fetch(kb + 1);
            if (kb >= LAG && !(ok = drain(kb - LAG))) break;
        }
        for (int kb = num_kb > LAG ? num_kb - LAG : 0; kb < num_kb && ok; ++kb) ok = drain(kb);
        // every MMA of this CTA is complete: the stages become the partial tile
#pragma unroll
        for (int i = 0; i < COLS; i += 4) {
            const uint32_t a = base + (uint32_t(quarter * 32 + lane) * C::PITCH + col0 + i) * 4;
            st_shared16(a, __float_as_uint(sum[i]), __float_as_uint(sum[i + 1]), __float_as_uint(sum[i + 2]), __float_as_uint(sum[i + 3]));
        }
    }
    __syncthreads();
    // (an abandoned wait leaves MMAs that read the stages; their results are marked invalid by the status word)
    if (p.split > 1) cluster_sync();

    if (CONV && warp < MMA_WARP) {
        // the filters' planes: neighbouring lanes take neighbouring pixels (a thread keeps one pixel: the rows divide the threads)
        const int rows = BM / p.split, r = rank * rows + tid % rows, pixels = cv.oh * cv.ow;
        const int64_t row = m0 + r;
        if (row < p.M) {
            const int64_t img = row / pixels;
            TOut* out         = static_cast<TOut*>(p.C) + img * p.N * pixels + (row - img * pixels);
            for (int col = tid / rows; col < BN && n0 + col < p.N; col += LOADERS / rows) {
                const uint32_t a = base + uint32_t(r * C::PITCH + col) * 4;
                float v          = 0.f;
                for (int s = 0; s < p.split; ++s)
                    v += p.split > 1 ? ld_cluster1(a, uint32_t(s)) : *reinterpret_cast<const float*>(smem_raw + (a - raw_addr));
                if (!isfinite(v)) {  // the scalar fold, ascending k, padding read as zeros
                    const int y = int(row - img * pixels) / cv.ow, x = int(row - img * pixels) - y * cv.ow;
                    const TIn* im = A + img * (int64_t(cv.cin) * cv.h * cv.w);
                    const TIn* wt = B + (n0 + col) * p.K;
                    v = 0.f;
                    for (int ci = 0; ci < cv.cin; ++ci)
                        for (int kr = 0; kr < cv.kh; ++kr)
                            for (int kq = 0; kq < cv.kw; ++kq, ++wt) {
                                const int iy = y * cv.stride_h - cv.pad_h + kr * cv.dil_h, ix = x * cv.stride_w - cv.pad_w + kq * cv.dil_w;
                                const bool in = unsigned(iy) < unsigned(cv.h) && unsigned(ix) < unsigned(cv.w);
                                v = fmaf(in ? load1(im + (int64_t(ci) * cv.h + iy) * cv.w + ix) : 0.f, load1(wt), v);
                            }
                }
                out[(n0 + col) * pixels] = TOut(v);
            }
        }
    } else if (warp < MMA_WARP) {
        constexpr int LPR = BN / 4, RPW = 32 / LPR;  // lanes per row, rows per warp and step
        const int rows = BM / p.split, col = (lane % LPR) * 4;
        const int64_t gcol = n0 + col;
        TOut* out             = static_cast<TOut*>(p.C) + bz * p.sc;
        const TOut* post_full = p.post_full ? static_cast<const TOut*>(p.post_full) + bz * p.sc : nullptr;
        for (int r = rank * rows + warp * RPW + lane / LPR; r < (rank + 1) * rows; r += MMA_WARP * RPW) {
            const int64_t row = m0 + r;
            if (row >= p.M || gcol >= p.N) continue;
            const uint32_t a = base + uint32_t(r * C::PITCH + col) * 4;
            float v[4]       = {0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s < p.split; ++s) {
                const float4 q = p.split > 1 ? ld_cluster4(a, uint32_t(s)) : *reinterpret_cast<const float4*>(smem_raw + (a - raw_addr));
                v[0] += q.x, v[1] += q.y, v[2] += q.z, v[3] += q.w;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t n = gcol + i;
                if (n >= p.N) break;
                // A non-finite cell: an operand of its fold was inf / NaN, or the sum overflowed. Such cells take the scalar
                // fold of the CUDA-core kernel -- ascending k, one fma per step -- from the caller's operands.
                if (!isfinite(v[i])) {
                    const TIn* ar = A + row * p.K;
                    const TIn* br = p.b_nk ? B + n * p.K : B + n;
                    const int64_t step = p.b_nk ? 1 : p.N;
                    float acc = 0.f;
                    for (int64_t k = 0; k < p.K; ++k) acc = fmaf(load1(ar + k), load1(br + k * step), acc);
                    v[i] = acc;
                }
                const float rowv = p.post_row ? __ldg(p.post_row + n) : 0.f;
                const float full = post_full ? float(post_full[row * p.N + n]) : 0.f;
                v[i]             = apply_post(p.post, v[i], rowv, full);
            }
            TOut* dst = out + row * p.N + gcol;
            if (p.vec_c) {  // four results are one aligned store, and N is a multiple of 4
                if (sizeof(TOut) == 4)
                    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                else
                    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (gcol + i < p.N) dst[i] = TOut(v[i]);
            }
        }
    }
    if (p.split > 1) cluster_sync();  // no CTA of the cluster exits while another may read its partial tile

    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, NBUF * BN);
    }
    if (tid == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

template <int BN, int LOADERS, class TIn, class TOut, bool CONV>
int launch(const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = gemm_f32_tc_kernel<BN, LOADERS, TIn, TOut, CONV>;
    constexpr int SMEM = Cfg<BN, TIn>::SMEM_BYTES;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[dev & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas)), cfg.blockDim = dim3(LOADERS + 32), cfg.dynamicSmemBytes = SMEM, cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(p.split), attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    return note_cuda_error(cudaLaunchKernelEx(&cfg, kern, p));
}

// Tile width and split. Tiles of 128 x 128 read a third less shared memory per flop; 128 x 64 puts two CTAs on an SM, which
// hides the start and end of a tile, and leaves a smaller last wave.
template <class TIn, class TOut, bool CONV>
int plan_and_launch(Params& p, int64_t batch, int sm_count, cudaStream_t s) {
    p.tiles_m = (p.M + BM - 1) / BM;
    const int64_t kb = (p.K + BK - 1) / BK, wide = p.tiles_m * ((p.N + 127) / 128) * batch;
    int bn = p.N > 64 && wide >= sm_count && kb >= 8 ? 128 : 64;
    if (getenv("SW_BN")) bn = atoi(getenv("SW_BN"));
    p.tiles_n = (p.N + bn - 1) / bn;
    const int64_t items = p.tiles_m * p.tiles_n * batch;
    p.split = 1;
    while (p.split < 8 && items * p.split * 2 <= sm_count && kb >= p.split * 2) p.split *= 2;
    if (getenv("SW_SPLIT")) p.split = atoi(getenv("SW_SPLIT"));
    const int64_t ctas = items * p.split;
    if (bn == 128) return launch<128, 512, TIn, TOut, CONV>(p, ctas, s);
    if (getenv("SW_LD") ? atoi(getenv("SW_LD")) == 512 : ctas <= sm_count) return launch<64, 512, TIn, TOut, CONV>(p, ctas, s);
    return launch<64, 256, TIn, TOut, CONV>(p, ctas, s);
}

}  // namespace

int gemm_f32_tc_supported(const mimk_gemm_desc& d) {
    if (d.in_dtype != MIMK_F32 || d.k <= 0) return 0;
    if (d.m >= (int64_t(1) << 31) || d.n >= (int64_t(1) << 31) || d.k >= (int64_t(1) << 31)) return 0;
    const int64_t tiles = ((d.m + BM - 1) / BM) * ((d.n + 63) / 64);
    return tiles < (int64_t(1) << 28) && d.batch < (int64_t(1) << 28) && tiles * d.batch < (int64_t(1) << 28);  // one grid
}

int gemm_f32_tc(const mimk_gemm_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p{};
    p.A = d.a, p.B = d.b, p.C = d.c;
    p.M = d.m, p.N = d.n, p.K = d.k;
    p.sa = d.batch > 1 ? d.stride_a : 0, p.sb = d.batch > 1 ? d.stride_b : 0, p.sc = d.batch > 1 ? d.stride_c : 0;
    p.post_row = static_cast<const float*>(d.post_row), p.post_full = d.post_full, p.post = d.post;
    p.b_nk  = d.b_layout == MIMK_B_NK;
    p.vec_a = d.k % 4 == 0 && aligned16(d.a) && p.sa % 4 == 0;
    p.vec_b = d.k % 4 == 0 && aligned16(d.b) && p.sb % 4 == 0;
    p.vec_c = d.n % 4 == 0 && aligned16(d.c) && p.sc % 4 == 0;
    p.status = dev->status_dev;
    return d.out_dtype == MIMK_BF16 ? plan_and_launch<float, __nv_bfloat16, false>(p, d.batch, dev->sm_count, s)
                                    : plan_and_launch<float, float, false>(p, d.batch, dev->sm_count, s);
}

int conv_tc(const mimk_conv_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p{};
    const int64_t oh = (d.h + 2 * d.pad_h - d.dil_h * (d.kh - 1) - 1) / d.stride_h + 1, ow = (d.w + 2 * d.pad_w - d.dil_w * (d.kw - 1) - 1) / d.stride_w + 1;
    p.A = d.x, p.B = d.filters, p.C = d.out;
    p.M = d.n * oh * ow, p.N = d.cout, p.K = d.cin * d.kh * d.kw;
    p.conv = ConvShape{int(d.cin), int(d.h), int(d.w), int(d.kh), int(d.kw), int(oh), int(ow), int(d.stride_h), int(d.stride_w),
                       int(d.dil_h), int(d.dil_w), int(d.pad_h), int(d.pad_w)};
    p.b_nk   = 1;
    p.vec_b  = p.K % (d.dtype == MIMK_F32 ? 4 : 8) == 0 && aligned16(d.filters);
    p.status = dev->status_dev;
    return d.dtype == MIMK_F32 ? plan_and_launch<float, float, true>(p, 1, dev->sm_count, s)
                               : plan_and_launch<__nv_bfloat16, __nv_bfloat16, true>(p, 1, dev->sm_count, s);
}

}  // namespace mimk
