// Attention of a few query rows (1 to 16 per head, one step of generation) against a long key / value sequence: bf16 in and out,
// f32 scores, statistics and accumulation, head_dim 64 or 128 (MimIR lit/tensor/attn_exec.mim:20-22).
//
// What bounds it is reading K and V once: with r query rows a loaded byte carries 2 r flops, far below the chip's ridge. The
// tcgen05 kernel has 128-row tiles, so it would do 8 to 128 times the exponentials and could give each head to one SM only.
// Here the keys of a head are dealt out to a cluster of up to eight CTAs of four warps, and every warp streams its own run of
// keys, 16 at a time, through a ring of its own that one elected lane has filled by TMA (a copy for K's tile, one for V's; no barrier of the CTA in the
// loop). The first product has the query rows as its M, the second has the head's elements as its M and the rows as its N, eight at
// a time: its right operand is then the first one's result as it lies in the registers, and up to eight rows cost half of sixteen. The fragments
// come by ldmatrix from the swizzled tiles, V's transposed.
// Next to the bytes it is instructions that count, with one or two warps to a scheduler: 16 copies of 16 bytes by every lane, and V's keys interleaved
// by byte permutes, made 450 instructions a step and 4.4 TB/s. Before / after, inputs not in L2: 128 heads x 1 x 4096 x 128 62 -> 47 us (5.7 TB/s),
// 256 x 1 x 8192 x 128 214 -> 161, 8 x 1 x 8192 x 128 24 -> 16, 32 x 11 x 5000 x 128 39 -> 28, 256 x 1 x 8192 x 64 137 -> 87. The copies
// issued by lane 0 in a branch of its own, not by a lane elected from a converged warp: 65536 keys of one head 77 us, 54 so. Twice the stages
// change nothing; the next step's scores beside this step's softmax take a stage from the copies in flight (67 us).
// Each warp keeps its own running maximum, sum and output; they are merged through (distributed) shared memory in a fixed order.
#include <math_constants.h>

#include <type_traits>

#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {
namespace {

constexpr int ROWS = 16, WARPS = 4, THREADS = WARPS * 32, STEP = 16;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

template <int D> struct Ring {
    static constexpr int STAGES = D == 128 ? 3 : 4, CTAS = D == 128 ? 2 : 3;
    static constexpr int HALVES = D / 64, TILE = STEP * 128;  // a tile: the step's keys x 64 elements, 128-byte swizzle
    static constexpr int STAGE_BYTES = 2 * HALVES * TILE;     // K's tiles, V's tiles
    static constexpr int WARP_BYTES = STAGES * STAGE_BYTES;
    static_assert(WARP_BYTES >= ROWS * D * 4, "a warp's part of the output lies over its ring");
};

struct Params {
    const __nv_bfloat16 *q, *v;
    __nv_bfloat16* o;
    float* lse;
    int64_t sq, sk;
    float scale;
    int causal, split;
    int* status;
};

// Four 8 x 8 matrices, of which lane l gives the address of row l % 8 of matrix l / 8: lane l gets elements 2 (l % 4) and the next of row l / 4
// (TRANS: of column l / 4).
template <bool TRANS>
__device__ __forceinline__ void ld_matrix(uint32_t (&r)[4], uint32_t a) {
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float quad_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(const float* p, int rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(uint32_t(__cvta_generic_to_shared(p))), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ bool has_nonfinite(uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; }
// Scores are kept in powers of two, or in powers of e where the weights are kept in f32.
template <bool F32W> __device__ __forceinline__ float power(float x) { return F32W ? expf(x) : exp2f(x); }
// weight of a part whose running maximum is m, in a whole of maximum M; a part without keys has none
template <bool F32W> __device__ __forceinline__ float part_weight(float m, float M) { return m == -CUDART_INF_F ? 0.f : power<F32W>(m - M); }

// F32W: the weights enter the second product as three bf16 pieces that sum to the f32 value, not rounded to bf16.
// NT: tiles of eight query rows.
template <int D, bool F32W, int NT>
__global__ void __launch_bounds__(THREADS, Ring<D>::CTAS) attn_few_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Params p) {
    constexpr int MT = D / 16;  // k-steps of the first product, tiles of 16 rows (elements of the head) of the second
    using R = Ring<D>;
    extern __shared__ __align__(1024) uint8_t ring[];
    constexpr int stages = R::STAGES, warp_bytes = R::WARP_BYTES;
    auto part_o = [&](int w) { return reinterpret_cast<float*>(ring + w * warp_bytes); };  // [ROWS][D], once the loop is over
    __shared__ __align__(8) uint64_t full[WARPS][stages];
    __shared__ int abort_flag;
    __shared__ float part_m[WARPS][ROWS], part_l[WARPS][ROWS];
    __shared__ float cta_m[ROWS], cta_l[ROWS];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int rank  = int(blockIdx.x % unsigned(p.split));  // a cluster is `split` consecutive CTAs
    const int64_t h = blockIdx.x / unsigned(p.split);
    const __nv_bfloat16* Q = p.q + h * p.sq * D;
    const __nv_bfloat16* V = p.v + h * p.sk * D;
    const int64_t steps = (p.sk + STEP - 1) / STEP, per = (steps + p.split * WARPS - 1) / (p.split * WARPS);
    const int64_t s0 = (rank * WARPS + warp) * per, s1 = s0 + per < steps ? s0 + per : steps;
    const float scale = F32W ? p.scale : p.scale * LOG2E;

    const uint32_t mine = sm100::smem_u32(ring) + warp * warp_bytes;
    auto bar   = [&](int stage) { return sm100::smem_u32(&full[warp][stage]); };
    auto fetch = [&](int64_t step, int stage) {
        sm100::mbar_expect_tx(bar(stage), R::STAGE_BYTES);
        sm100::tma_load_4d(mine + stage * R::STAGE_BYTES, &tmK, 0, int(step * STEP), 0, int(h), bar(stage));
        sm100::tma_load_4d(mine + stage * R::STAGE_BYTES + R::HALVES * R::TILE, &tmV, 0, int(step * STEP), 0, int(h), bar(stage));
    };
    int64_t issued = s0 + stages < s1 ? s0 + stages : s1;  // steps whose copies have been requested
    if (tid == 0) abort_flag = 0;
    if (lane == 0) {
        for (int i = 0; i < stages; ++i) sm100::mbar_init(bar(i), 1);
        sm100::fence_barrier_init();
        sm100::fence_proxy_async_smem();
        for (int64_t step = s0; step < issued; ++step) fetch(step, int(step - s0));
    }
    __syncthreads();

    uint32_t q[MT][4];  // rows g and g + 8, elements 2 c and 2 c + 8 of each 16
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = g + 8 * (e & 1);
            q[i][e] = (e & 1) < NT && row < p.sq ? __ldg(reinterpret_cast<const uint32_t*>(Q + row * D + i * 16 + (e >> 1) * 8 + 2 * c)) : 0u;
        }
    // o[i][n]: elements i * 16 + g and 8 further of the head, of rows n * 8 + 2 c and the next
    float o[MT][NT][4], m[NT], l[NT];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[i][n][e] = 0.f;
#pragma unroll
    for (int n = 0; n < NT; ++n) m[n] = -CUDART_INF_F, l[n] = 0.f;
    // a row sees keys [0, limit)
    auto limit_of = [&](int row) {
        const int64_t n = p.causal ? row + 1 + p.sk - p.sq : p.sk;
        return n < p.sk ? n : p.sk;
    };
    int64_t limit[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) limit[n] = limit_of(g + 8 * n);
    const int64_t seen_by_all = limit_of(0);

    // addresses within a tile: K's rows of keys, V's of keys with the elements as the result's rows
    const int krow = lane & 7, vrow = (lane >> 4) * 8 + (lane & 7);
    uint32_t ku[2], vu[4];
#pragma unroll
    for (int j = 0; j < 2; ++j) ku[j] = krow * 128 + (((4 * j + (lane >> 3)) ^ krow) << 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) vu[j] = vrow * 128 + (((2 * j + ((lane >> 3) & 1)) ^ krow) << 4);

    bool alive = true;
    int stage  = 0;
    uint32_t phase = 0;
    for (int64_t step = s0; step < s1; ++step) {
        if (step < issued) alive &= bool(__all_sync(0xffffffffu, sm100::mbar_wait(bar(stage), phase, &abort_flag)));  // (one outcome for the warp)
        const uint32_t kt = mine + stage * R::STAGE_BYTES, vt = kt + R::HALVES * R::TILE;
        float s[2][4] = {}, s2[2][4] = {};  // two chains of dependent products for each eight keys
#pragma unroll
        for (int i = 0; i < MT / 2; ++i)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                uint32_t b[4];
                ld_matrix<false>(b, kt + (i >> 1) * R::TILE + t * 1024 + ku[i & 1]);
                mma16816(s[t], q[2 * i][0], q[2 * i][1], q[2 * i][2], q[2 * i][3], b[0], b[1]);
                mma16816(s2[t], q[2 * i + 1][0], q[2 * i + 1][1], q[2 * i + 1][2], q[2 * i + 1][3], b[2], b[3]);
            }
        uint32_t vr[MT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i) ld_matrix<true>(vr[i], vt + (i >> 2) * R::TILE + vu[i & 3]);
        // scores of this lane: key step * 16 + t * 8 + 2c + (e & 1), row g + 8 (e >> 1); `left`: how many of the step's keys the row sees
        const bool whole = step * STEP + STEP <= seen_by_all;
        int left[NT];
        float mx[NT], from[NT];
        bool grown = false;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int64_t there = limit[n] - step * STEP;
            left[n] = there < 0 ? 0 : there > STEP ? STEP : int(there);
            mx[n]   = -CUDART_INF_F;
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 2 * n; e < 2 * n + 2; ++e) {
                    s[t][e] = (s[t][e] + s2[t][e]) * scale;
                    if (whole || t * 8 + 2 * c + (e & 1) < left[n]) mx[n] = fmaxf(mx[n], s[t][e]);
                }
            grown |= mx[n] > m[n];
        }
        if (__any_sync(0xffffffffu, grown)) {  // a maximum has grown (rare after the first steps)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float m_new = fmaxf(m[n], quad_max(mx[n])), alpha = part_weight<F32W>(m[n], m_new);
                m[n] = m_new;
                l[n] *= alpha;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float a = __shfl_sync(0xffffffffu, alpha, (2 * c + e) * 4);
#pragma unroll
                    for (int i = 0; i < MT; ++i) o[i][n][e] *= a, o[i][n][e + 2] *= a;
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            from[n] = m[n] == -CUDART_INF_F ? 0.f : m[n];  // keys that score minus infinity so far weigh nothing
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 2 * n; e < 2 * n + 2; ++e) {
                    s[t][e] = whole || t * 8 + 2 * c + (e & 1) < left[n] ? power<F32W>(s[t][e] - from[n]) : 0.f;
                    l[n] += s[t][e];
                }
        }
        __syncwarp();  // every lane has the step's fragments
        if (alive && step + stages < s1 && sm100::elect_one()) fetch(step + stages, stage);
        if (alive && issued < s1) ++issued;
        if (++stage == stages) stage = 0, phase ^= 1;
        // A key that a row does not see must not reach it even as 0 times an infinity: such a block, where it holds one, is
        // added cell by cell over the keys each row sees.
        bool odd_block = false;
        if (!whole) {
            bool bad = false;
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) bad = bad || has_nonfinite(vr[i][e]);
            odd_block = __any_sync(0xffffffffu, bad);
        }
        if (!odd_block) {
#pragma unroll
            for (int piece = 0; piece < (F32W ? 3 : 1); ++piece)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    uint32_t b[2];
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        float &lo = s[t][2 * n], &hi = s[t][2 * n + 1];
                        b[t] = F32W ? f32split::upper_halves(lo, hi) : pack_bf16x2(lo, hi);
                        if (F32W) lo = f32split::lower_part(lo), hi = f32split::lower_part(hi);
                    }
#pragma unroll
                    for (int i = 0; i < MT; ++i) mma16816(o[i][n], vr[i][0], vr[i][1], vr[i][2], vr[i][3], b[0], b[1]);
                }
        } else {
            for (int kk = 0; kk < STEP; ++kk) {
                const int64_t key = step * STEP + kk;
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float lo = kk < 8 ? s[0][2 * n] : s[1][2 * n], hi = kk < 8 ? s[0][2 * n + 1] : s[1][2 * n + 1];
                        float pr = __shfl_sync(0xffffffffu, (kk & 1) ? hi : lo, (2 * c + e) * 4 + ((kk & 7) >> 1));
                        if (!F32W) pr = __bfloat162float(__float2bfloat16_rn(pr));
                        if (key < limit_of(n * 8 + 2 * c + e))
#pragma unroll
                            for (int i = 0; i < MT; ++i)
#pragma unroll
                                for (int half = 0; half < 2; ++half)
                                    o[i][n][e + 2 * half] = fmaf(pr, __bfloat162float(V[key * D + i * 16 + half * 8 + g]), o[i][n][e + 2 * half]);
                    }
            }
        }
    }
    __syncwarp();  // every lane is done with the warp's ring

    // the warps' parts -> this CTA's part (in the first warp's place) -> the rows of the head, each CTA of the cluster some
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        l[n] = quad_sum(l[n]);
        if (c == 0) part_m[warp][g + 8 * n] = m[n], part_l[warp][g + 8 * n] = l[n];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) part_o(warp)[(n * 8 + 2 * c + (e & 1)) * D + i * 16 + (e >> 1) * 8 + g] = o[i][n][e];
    }
    __syncthreads();
    const int cells = int(p.sq) * D;
    for (int i = tid; i < cells; i += THREADS) {
        const int row = i / D, col = i % D;
        float M = part_m[0][row];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) M = fmaxf(M, part_m[w][row]);
        float sum = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float wt = part_weight<F32W>(part_m[w][row], M);
            sum += wt * part_o(w)[i];
            den += wt * part_l[w][row];
        }
        part_o(0)[i] = sum;
        if (col == 0) cta_m[row] = M, cta_l[row] = den;
    }
    __syncthreads();
    if (p.split > 1) cluster_sync();
    for (int i = rank * THREADS + tid; i < cells; i += p.split * THREADS) {
        const int row = i / D, col = i % D;
        float M = -CUDART_INF_F, sum = 0.f, den = 0.f;
        if (p.split > 1) {
            for (int r = 0; r < p.split; ++r) M = fmaxf(M, ld_cluster(&cta_m[row], r));
            for (int r = 0; r < p.split; ++r) {
                const float wt = part_weight<F32W>(ld_cluster(&cta_m[row], r), M);
                sum += wt * ld_cluster(part_o(0) + i, r);
                den += wt * ld_cluster(&cta_l[row], r);
            }
        } else {
            M = cta_m[row], sum = part_o(0)[i], den = cta_l[row];
        }
        // no weight at all: zeros for a row that sees no key, else every score is minus infinity and the softmax has no value
        const bool none = den == 0.f && (!p.causal || row + 1 + p.sk - p.sq > 0);
        const float inv = none ? CUDART_NAN_F : den > 0.f ? 1.f / den : 0.f;
        p.o[(h * p.sq + row) * D + col] = __float2bfloat16_rn(sum * inv);
        if (p.lse && col == 0) p.lse[h * p.sq + row] = den > 0.f ? (F32W ? M : M * LN2) + logf(den) : -CUDART_INF_F;
    }
    if (tid == 0 && abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
    if (p.split > 1) cluster_sync();  // no CTA of the cluster exits while another may read its part
}

template <int D, bool F32W, int NT>
int launch(const CUtensorMap& tmK, const CUtensorMap& tmV, const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = attn_few_kernel<D, F32W, NT>;
    constexpr int SMEM = WARPS * Ring<D>::WARP_BYTES;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[dev & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas)), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = SMEM, cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(p.split), attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    return note_cuda_error(cudaLaunchKernelEx(&cfg, kern, tmK, tmV, p));
}

}  // namespace

int attn_few_supported(const mimk_attn_desc& d) {
    if (d.dtype != MIMK_BF16 || (d.head_dim != 64 && d.head_dim != 128)) return 0;
    if (d.seq_q < 1 || d.seq_q > ROWS || d.seq_k < 1 || d.seq_k >= (int64_t(1) << 31)) return 0;
    if (d.batch_heads >= (int64_t(1) << 27)) return 0;
    return aligned16(d.q) && aligned16(d.k) && aligned16(d.v);
}

// With more than eight rows the second tile of rows makes this kernel's steps twice as long, while the 128-row kernel (attn_tc_p.cu) gives a
// head to each SM whatever its rows: it is ahead where one round of heads leaves few SMs idle, the longer the fewer the keys. Its time / this
// kernel's, us, 128 heads x 128: 16 rows, 100 keys 7.9 / 10.3, 400 12.6 / 16.3, 1000 18.7 / 19.7, 2500 no more; 11 rows, 400 12.5 / 13.8, 1000
// 18.7 / 17.1; 10 rows, 400 12.5 / 13.1, 1000 18.7 / 16.5. With a head on every SM there are no idle SMs whose share of the memory's rate the others take: 148
// heads, 4096 keys, 16 rows 56.0 / 60.4, 12 rows 56.1 / 58.4, 5500 keys no more. At head_dim 64, with more or with fewer heads it is behind (200 heads x 16 x 1000 36.9 / 24.4).
int attn_heads_fill(const mimk_attn_desc& d, int sm_count) {
    if (d.head_dim != 128 || d.seq_q <= 10 || d.batch_heads > sm_count || d.batch_heads * 5 < sm_count * 4) return 0;
    return d.seq_k <= 75 * d.seq_q || (d.batch_heads * 20 >= sm_count * 19 && d.seq_k >= 2000 && d.seq_k <= 5000);
}

int attn_few(const mimk_attn_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p;
    p.q = static_cast<const __nv_bfloat16*>(d.q), p.v = static_cast<const __nv_bfloat16*>(d.v);
    p.status = dev->status_dev;
    p.o = static_cast<__nv_bfloat16*>(d.o), p.lse = d.lse;
    p.sq = d.seq_q, p.sk = d.seq_k, p.scale = d.scale, p.causal = d.causal;
    // As many CTAs per head as the SMs hold at once (two each): a second round of CTAs would pay the start of its stream and the
    // merge, together several steps, again (128 heads x 4096 keys: split 1 / 2 / 4 / 8: 46 / 46 / 50 / 56 us; 8 x 8192: 52 / 32 /
    // 22 / 17). Every warp has at least three steps.
    p.split = 1;
    while (p.split < 8 && d.batch_heads * p.split * 2 <= 2 * int64_t(dev->sm_count) && d.seq_k >= int64_t(p.split) * 2 * WARPS * 3 * STEP) p.split *= 2;
    // The calls that the 128-row kernel takes too (attn_tc_p.cu) have weights rounded to bf16, as there; the others, whose general
    // path keeps them in f32 (attn_row.cuh), keep them here.
    const int64_t ctas = d.batch_heads * p.split;
    CUtensorMap tK, tV;
    // [heads][keys][head_dim / 64][64]: a step's tiles of K, or of V, in one copy
    const uint64_t row = uint64_t(d.head_dim) * 2;
    const cuuint64_t dims[4] = {64, cuuint64_t(d.seq_k), cuuint64_t(d.head_dim / 64), cuuint64_t(d.batch_heads)}, strides[3] = {row, 128, cuuint64_t(d.seq_k) * row};
    const cuuint32_t box[4] = {64, STEP, cuuint32_t(d.head_dim / 64), 1};
    MIMK_TRY(encode_tmap_bf16(&tK, d.k, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B));
    MIMK_TRY(encode_tmap_bf16(&tV, d.v, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B));
    auto run = [&](auto w, auto n) {
        constexpr bool F32W = decltype(w)::value;
        constexpr int NT    = decltype(n)::value;
        return d.head_dim == 128 ? launch<128, F32W, NT>(tK, tV, p, ctas, s) : launch<64, F32W, NT>(tK, tV, p, ctas, s);
    };
    auto run_rows = [&](auto w) {
        return d.seq_q <= 8 ? run(w, std::integral_constant<int, 1>{}) : run(w, std::integral_constant<int, 2>{});
    };
    return attn_tc_persistent_supported(d) ? run_rows(std::false_type{}) : run_rows(std::true_type{});
}

}  // namespace mimk
