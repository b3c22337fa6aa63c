// CUDA-core contraction: the f32 path of the dot family and the landing place for bf16 shapes the tensor-core
// kernel does not take (extents that break TMA's 16-byte rules).
//
// Each output cell is folded in ascending k with one fused multiply-add per step -- the per-cell order every
// CPU nest of the reference keeps (MimIR src/mim/plug/btensor/btensor.mim:348) under its `fast` math mode,
// which permits contraction (src/mim/plug/ll/ll.cpp:55-68). Shapes are arbitrary (the reference tests
// 5x33 . (7x33)^T, lit/tensor/fc_exec.mim:36); out-of-range tile cells are predicated off.
#include "common.cuh"

namespace mimk {
namespace {

constexpr int TM = 64, TN = 64, TK = 16;

__device__ __forceinline__ float ld(const float* p, int64_t i) { return __ldg(p + i); }
__device__ __forceinline__ float ld(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st(float* p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void st(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }

template <class TIn, class TOut>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const TIn* __restrict__ A, const TIn* __restrict__ B,
                                                       TOut* __restrict__ C, int64_t M, int64_t N, int64_t K,
                                                       int64_t sa, int64_t sb, int64_t sc, int b_nk, int post,
                                                       const float* __restrict__ post_row,
                                                       const TOut* __restrict__ post_full) {
    __shared__ float As[TK][TM + 4];
    __shared__ float Bs[TK][TN + 4];
    const int64_t batch = blockIdx.z;
    A += batch * sa;
    B += batch * sb;
    C += batch * sc;
    if (post_full) post_full += batch * sc;
    const int64_t m0 = int64_t(blockIdx.y) * TM, n0 = int64_t(blockIdx.x) * TN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4] = {};
    // Each thread moves four A and four B elements per k-tile. The next tile's elements are fetched into registers before
    // the current tile is multiplied, so their global-memory latency overlaps the arithmetic (small problems have too few
    // CTAs to hide it by occupancy). The per-cell order of the fold is untouched: ascending k, one fma per step.
    float ra[4], rb[4];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i  = threadIdx.x + r * 256;
            const int kk = i % TK, mm = i / TK;
            const int64_t m = m0 + mm, k = k0 + kk;
            ra[r] = (m < M && k < K) ? ld(A, m * K + k) : 0.f;
            if (b_nk) {
                const int64_t n = n0 + mm;
                rb[r] = (n < N && k < K) ? ld(B, n * K + k) : 0.f;
            } else {
                const int nn = i % TN, kb = i / TN;
                const int64_t n = n0 + nn, kr = k0 + kb;
                rb[r] = (n < N && kr < K) ? ld(B, kr * N + n) : 0.f;
            }
        }
    };
    if (K > 0) fetch(0);
    for (int64_t k0 = 0; k0 < K; k0 += TK) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = threadIdx.x + r * 256;
            As[i % TK][i / TK] = ra[r];  // A tile: TM x TK, read with k fastest (unit stride in memory)
            if (b_nk) Bs[i % TK][i / TK] = rb[r];
            else Bs[i / TN][i % TN] = rb[r];
        }
        __syncthreads();
        if (k0 + TK < K) fetch(k0 + TK);
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t n = n0 + tx * 4 + j;
            if (n >= N) continue;
            const float row  = post_row ? post_row[n] : 0.f;
            const float full = post_full ? float(post_full[m * N + n]) : 0.f;
            st(C, m * N + n, apply_post(post, acc[i][j], row, full));
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Small f32 products: 32 x 32 tiles, or 16 x 32 where those leave most SMs without one, the K extent staged in 128-wide chunks by
// asynchronous copies.
//
// A product like 256^3 has 16 tiles of 64 x 64: sixteen CTAs on 148 SMs, each walking K in sixteen steps that every one
// pay a global-memory latency. Here the same product is 128 CTAs, and both chunks of a K <= 256 are in flight from the
// first instruction (two stages; longer K streams through them), so a CTA waits for memory once. The fold per cell is
// the one above -- ascending k, one fma per step -- so the two kernels agree bit for bit.
// Copies of 16 bytes where an operand's rows allow them, of 4 else (1024 x 10 x 128: 10.8 us on the kernel above, 3.7 here; 1000 x 61 x 250 stored [N, K] 17 and 5).
// Thread (tx, ty) of the 16 x 16 block owns rows ty (and ty + 16) and, for B stored [N, K], columns tx, tx + 16 (both operands
// K-major in shared memory, read four k at a time: a quarter-warp reads one A address and eight B rows whose pitch of
// KC + 4 floats spreads them over all banks); for B stored [K, N], columns 2 tx, 2 tx + 1 (one 8-byte read per k).
// What bounds it: the launch, one trip to memory and the issue of 13 instructions per 4 k and cell pair. 256^3: 5.7 us (6.4 with
// 32-row tiles on 64 CTAs).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int SN = 32, KC = 128, KP = KC + 4, NP = SN + 4;

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
    const int sz     = valid ? 16 : 0;  // 0: nothing is read, the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
    const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
    const int sz     = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}

// A [rows x width] part of a row-major matrix, `pitch` elements a row in memory and `to_pitch` in shared memory; zeros outside.
template <int ROWS, int WIDTH>
__device__ __forceinline__ void stage_part(float* to, int to_pitch, const float* from, int64_t pitch, int64_t rows, int64_t cols, bool vec) {
    if (vec) {
        constexpr int PER_ROW = WIDTH / 4;
#pragma unroll
        for (int r = 0; r < ROWS * PER_ROW / 256; ++r) {
            const int g = threadIdx.x + r * 256, row = g / PER_ROW, col = g % PER_ROW * 4;
            const bool ok = row < rows && col < cols;
            cp_async16(to + row * to_pitch + col, ok ? from + row * pitch + col : from, ok);
        }
    } else {
#pragma unroll 4
        for (int r = 0; r < ROWS * WIDTH / 256; ++r) {
            const int g = threadIdx.x + r * 256, row = g / WIDTH, col = g % WIDTH;
            const bool ok = row < rows && col < cols;
            cp_async4(to + row * to_pitch + col, ok ? from + row * pitch + col : from, ok);
        }
    }
}

// RT: rows of a thread. VEC: both operands by 16 bytes, which K is a multiple of then. (B stored [N, K]: tested at run time, with a loop for the
// rest of K, 733 x 634 x 16 4.9 -> 5.1 us, 4 of 107 x 204 x 188 5.7 -> 6.3. Stored [K, N] such an instance is slower: 41 x 168 x 252 5.2 -> 5.6.)
template <bool B_NK, int RT, bool VEC>
__global__ void __launch_bounds__(256) gemm_simt_small_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                             float* __restrict__ C, int64_t M, int64_t N, int64_t K,
                                                             int64_t sa, int64_t sb, int64_t sc, int post, int vec_a, int vec_b,
                                                             const float* __restrict__ post_row,
                                                             const float* __restrict__ post_full) {
    extern __shared__ __align__(16) float smem[];
    constexpr int SM = 16 * RT, A_FLOATS = SM * KP, B_FLOATS = B_NK ? SN * KP : KC * NP;
    const int64_t batch = blockIdx.z;
    A += batch * sa;
    B += batch * sb;
    C += batch * sc;
    if (post_full) post_full += batch * sc;
    const int64_t m0 = int64_t(blockIdx.y) * SM, n0 = int64_t(blockIdx.x) * SN;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;

    auto stage = [&](int buf, int64_t k0) {
        float* As = smem + buf * (A_FLOATS + B_FLOATS);
        float* Bs = As + A_FLOATS;
        stage_part<SM, KC>(As, KP, A + m0 * K + k0, K, M - m0, K - k0, VEC || vec_a);
        if (B_NK) stage_part<SN, KC>(Bs, KP, B + n0 * K + k0, K, N - n0, K - k0, VEC || vec_b);
        else stage_part<KC, SN>(Bs, NP, B + k0 * N + n0, N, K - k0, N - n0, VEC || vec_b);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[RT][2] = {};
    const int64_t chunks = (K + KC - 1) / KC;
    if (chunks > 0) stage(0, 0);
    if (chunks > 1) stage(1, KC);
    for (int64_t c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float* As = smem + int(c & 1) * (A_FLOATS + B_FLOATS);
        const float* Bs = As + A_FLOATS;
        const int kn    = int(K - c * KC < KC ? K - c * KC : KC);
        int k           = 0;
#pragma unroll 4
        for (; VEC ? k < kn : k + 4 <= kn; k += 4) {
            float av[RT][4];
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(As + (ty + 16 * i) * KP + k);
                av[i][0] = a.x, av[i][1] = a.y, av[i][2] = a.z, av[i][3] = a.w;
            }
            if (B_NK) {
                const float4 b0 = *reinterpret_cast<const float4*>(Bs + tx * KP + k);
                const float4 b1 = *reinterpret_cast<const float4*>(Bs + (tx + 16) * KP + k);
                const float bv0[4] = {b0.x, b0.y, b0.z, b0.w}, bv1[4] = {b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < RT; ++i) acc[i][0] = fmaf(av[i][q], bv0[q], acc[i][0]), acc[i][1] = fmaf(av[i][q], bv1[q], acc[i][1]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 b = *reinterpret_cast<const float2*>(Bs + (k + q) * NP + tx * 2);
#pragma unroll
                    for (int i = 0; i < RT; ++i) acc[i][0] = fmaf(av[i][q], b.x, acc[i][0]), acc[i][1] = fmaf(av[i][q], b.y, acc[i][1]);
                }
            }
        }
        for (; !VEC && k < kn; ++k) {
            const float b0 = B_NK ? Bs[tx * KP + k] : Bs[k * NP + tx * 2], b1 = B_NK ? Bs[(tx + 16) * KP + k] : Bs[k * NP + tx * 2 + 1];
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const float a = As[(ty + 16 * i) * KP + k];
                acc[i][0] = fmaf(a, b0, acc[i][0]), acc[i][1] = fmaf(a, b1, acc[i][1]);
            }
        }
        __syncthreads();
        if (c + 2 < chunks) stage(int(c & 1), (c + 2) * KC);
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int64_t m = m0 + ty + 16 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int64_t n = n0 + (B_NK ? tx + 16 * j : tx * 2 + j);
            if (n >= N) continue;
            const float row  = post_row ? post_row[n] : 0.f;
            const float full = post_full ? post_full[m * N + n] : 0.f;
            C[m * N + n]     = apply_post(post, acc[i][j], row, full);
        }
    }
}

bool vec_a(const mimk_gemm_desc& d) { return d.k % 4 == 0 && aligned16(d.a) && d.stride_a % 4 == 0; }
bool vec_b(const mimk_gemm_desc& d) { return (d.b_layout == MIMK_B_NK ? d.k : d.n) % 4 == 0 && aligned16(d.b) && d.stride_b % 4 == 0; }

// Worth it while the 64 x 64 tiling leaves most SMs without a tile. With copies of 4 bytes, which take as long as a short K, not with many tiles
// either. This kernel / the one above, us: 217 x 1298 x 17 (287 tiles of 32 x 32) 4.6 / 6.7, 303 x 1139 x 21 (360) 6.2 / 6.8, 2070 x 194 x 20 (455) 5.9 / 6.8, 2152 x 197 x 13
// (476) 7.3 / 5.8, 693 x 731 x 15 (506) 7.2 / 5.7; 1978 x 347 x 109 (682) 13.9 / 17.0, 697 x 1101 x 83 (770) 13.3 / 14.8, 808 x 1267 x 195 (1040)
// 33.7 / 27.8.
bool small_tiles_apply(const mimk_gemm_desc& d) {
    if (d.in_dtype != MIMK_F32 || d.out_dtype != MIMK_F32 || d.k < 1) return false;
    const int64_t big = ((d.m + TM - 1) / TM) * ((d.n + TN - 1) / TN) * d.batch;
    if (big >= 2 * 148 || (d.m + 31) / 32 > 65535 || d.batch > 65535) return false;
    const int64_t tiles = ((d.m + 31) / 32) * ((d.n + SN - 1) / SN) * d.batch;
    return (vec_a(d) && vec_b(d)) || tiles * 10 <= 31 * 148 || (tiles <= 6 * 148 && d.k >= 48);
}

template <bool B_NK, int RT, bool VEC>
int launch_small(const mimk_gemm_desc& d, cudaStream_t s) {
    constexpr int SMEM = 2 * (16 * RT * KP + (B_NK ? SN * KP : KC * NP)) * int(sizeof(float));
    auto kern          = gemm_simt_small_kernel<B_NK, RT, VEC>;
    static bool configured[64] = {};  // per instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[dev & 63] = true;
    }
    dim3 grid((unsigned)((d.n + SN - 1) / SN), (unsigned)((d.m + 16 * RT - 1) / (16 * RT)), (unsigned)d.batch);
    kern<<<grid, 256, SMEM, s>>>(static_cast<const float*>(d.a), static_cast<const float*>(d.b), static_cast<float*>(d.c),
                                 d.m, d.n, d.k, d.stride_a, d.stride_b, d.stride_c, d.post, vec_a(d), vec_b(d),
                                 static_cast<const float*>(d.post_row), static_cast<const float*>(d.post_full));
    return launch_status();
}
template <bool B_NK, int RT>
int launch_small(const mimk_gemm_desc& d, bool vec, cudaStream_t s) {
    if constexpr (B_NK)
        if (vec) return launch_small<true, RT, true>(d, s);
    return launch_small<B_NK, RT, false>(d, s);
}
int launch_small(const mimk_gemm_desc& d, cudaStream_t s) {
    // 16 rows while the device has an SM for each such tile
    int st                = MIMK_OK;
    const DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    const bool narrow = ((d.m + 15) / 16) * ((d.n + SN - 1) / SN) * d.batch <= dev->sm_count;
    const bool vec = vec_a(d) && vec_b(d);
    if (d.b_layout == MIMK_B_NK) return narrow ? launch_small<true, 1>(d, vec, s) : launch_small<true, 2>(d, vec, s);
    return narrow ? launch_small<false, 1>(d, vec, s) : launch_small<false, 2>(d, vec, s);
}

template <class TIn, class TOut>
int launch(const mimk_gemm_desc& d, cudaStream_t s) {
    dim3 grid((unsigned)((d.n + TN - 1) / TN), (unsigned)((d.m + TM - 1) / TM), (unsigned)d.batch);
    if (grid.y > 65535 || grid.z > 65535) return MIMK_E_UNSUPPORTED;
    gemm_simt_kernel<TIn, TOut><<<grid, 256, 0, s>>>(
        static_cast<const TIn*>(d.a), static_cast<const TIn*>(d.b), static_cast<TOut*>(d.c), d.m, d.n, d.k, d.stride_a,
        d.stride_b, d.stride_c, d.b_layout == MIMK_B_NK, d.post, static_cast<const float*>(d.post_row),
        static_cast<const TOut*>(d.post_full));
    return launch_status();
}

}  // namespace

// Where f32 products stay on the CUDA cores (times: CUDA-graph replays, warm, CUDA cores against tensor cores).
//   batches below 2^25 multiply-adds      64 of 64^3: 4.5 / 8.4 us; above: 10 of 76 x 704 x 448, 33.6 / 19.1
//   K <= 256: below 5 * 2^24 where the small-tile kernel applies and copies 16 bytes at a time (256^3: 5.7 / 7.8 us; 815 x 524 x 168: 13 / 15;
//             784 x 1024 x 128: 13.9 / 10.7), else 2^24 (245 x 674 x 146: 15.3 / 10.0).
//             Rows that are no multiple of four below 20 * 2^24: any part of such a product has the bits of the small product of the
//             same rows and columns, which is worth more there than the time (1280 x 961 x 256: 60 / 25; x 128: 34 / 20; 4096 x 250 x
//             17: 8.5 / 10.5). Above, K <= 32 only (4096 x 4001 x 17: 97 / 101; x 64: 144 / 112; x 256: 408 / 171)
//   longer K: only what is hardly any work (the CUDA cores walk all of K in one CTA: 32 x 1024 x 1024, 19.0 / 11.2)
int gemm_simt_preferred(const mimk_gemm_desc& d) {
    const double work = double(d.m) * double(d.n) * double(d.k);
    if (d.batch > 1) return work * double(d.batch) < double(1 << 25);
    if (d.k > 256) return d.k < 1024 && work < double(1 << 20);
    if (d.n % 4 != 0 && (d.k <= 32 || work < double(20 << 24))) return 1;
    return work < (small_tiles_apply(d) && vec_a(d) && vec_b(d) ? double(5 << 24) : double(1 << 24));
}

int gemm_simt(const mimk_gemm_desc& d, cudaStream_t s) {
    if (small_tiles_apply(d)) return launch_small(d, s);
    if (d.in_dtype == MIMK_F32 && d.out_dtype == MIMK_F32) return launch<float, float>(d, s);
    if (d.in_dtype == MIMK_F32 && d.out_dtype == MIMK_BF16) return launch<float, __nv_bfloat16>(d, s);
    if (d.in_dtype == MIMK_BF16 && d.out_dtype == MIMK_F32) return launch<__nv_bfloat16, float>(d, s);
    if (d.in_dtype == MIMK_BF16 && d.out_dtype == MIMK_BF16) return launch<__nv_bfloat16, __nv_bfloat16>(d, s);
    return MIMK_E_DTYPE;
}

}  // namespace mimk
