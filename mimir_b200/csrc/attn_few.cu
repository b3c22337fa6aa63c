// Attention of a few query rows (1 to 16 per head, one step of generation) against a long key / value sequence: bf16 in and out,
// f32 scores, statistics and accumulation, head_dim 64 or 128 (MimIR lit/tensor/attn_exec.mim:20-22).
//
// What bounds it is reading K and V once: with r query rows a loaded byte carries 2 r flops, far below the chip's ridge. The
// tcgen05 kernel has 128-row tiles, so it would do 8 to 128 times the exponentials and could give each head to one SM only.
// Here the keys of a head are dealt out to a cluster of up to eight CTAs of four warps, and every warp streams its own run of
// keys, 16 at a time, into mma.sync fragments (16 rows are exactly its M). The copies are asynchronous, each lane reads from
// shared memory only what it fetched itself, and so there is no barrier in the loop. Both products may take their contracted
// index in any order as long as both operands use the same one, so
//   K   a lane takes 16 consecutive bytes of a key (head_dim 8c .. 8c+7 of each 32), which are the fragments of two k-steps
//   V   a lane takes 16 consecutive bytes of four keys; pairs of keys are interleaved by byte permutes, and the eight elements
//       belong to eight different column tiles of the result
// Measured: 128 heads x 1 x 4096 x 128, 61 us (4.4 TB/s, as the 128-row kernel); 8 x 1 x 8192 x 128, 22 us; causal, with f32 weights,
// 32 x 11 x 5000 x 128, 32 us (26 with weights rounded to bf16: the products of two more pieces are no longer hidden). One bulk copy per
// key instead of 16 lanes' copies was slower (69 and 32 us for the first two), registers instead of the ring too.
// Each warp keeps its own running maximum, sum and output; they are merged through (distributed) shared memory in a fixed order.
#include <math_constants.h>

#include "common.cuh"
#include "f32_split.cuh"

namespace mimk {
namespace {

constexpr int ROWS = 16, WARPS = 4, THREADS = WARPS * 32, STEP = 16;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

template <int D> struct Ring {
    static constexpr int STAGES = D == 128 ? 3 : 4;
    static constexpr int CHUNKS = D / 8;  // 16-byte pieces per lane and step: half K, half V
    static constexpr int WARP_BYTES = STAGES * CHUNKS * 32 * 16;
    static_assert(WARP_BYTES >= ROWS * D * 4, "a warp's part of the output lies over its ring");
};

struct Params {
    const __nv_bfloat16 *q, *k, *v;
    __nv_bfloat16* o;
    float* lse;
    int64_t sq, sk;
    float scale;
    int causal, split;
};

__device__ __forceinline__ uint4 ld_row(const __nv_bfloat16* p, bool there) {
    return there ? __ldg(reinterpret_cast<const uint4*>(p)) : make_uint4(0, 0, 0, 0);
}
// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void copy16(uint32_t dst, const __nv_bfloat16* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
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
__device__ __forceinline__ bool has_nonfinite(uint4 v) {
    auto bad = [](uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; };
    return bad(v.x) || bad(v.y) || bad(v.z) || bad(v.w);
}
// Scores are kept in powers of two, or in powers of e where the weights are kept in f32.
template <bool F32W> __device__ __forceinline__ float power(float x) { return F32W ? expf(x) : exp2f(x); }
// weight of a part whose running maximum is m, in a whole of maximum M; a part without keys has none
template <bool F32W> __device__ __forceinline__ float part_weight(float m, float M) { return m == -CUDART_INF_F ? 0.f : power<F32W>(m - M); }

// F32W: the weights enter the second product as three bf16 pieces that sum to the f32 value, not rounded to bf16.
template <int D, bool F32W>
__global__ void __launch_bounds__(THREADS, D == 128 ? 2 : 3) attn_few_kernel(const Params p) {
    constexpr int G = D / 32, CH = D / 64;
    using R = Ring<D>;
    extern __shared__ __align__(16) uint8_t ring[];
    auto part_o = [&](int w) { return reinterpret_cast<float*>(ring + w * R::WARP_BYTES); };  // [ROWS][D], once the loop is over
    __shared__ float part_m[WARPS][ROWS], part_l[WARPS][ROWS];
    __shared__ float cta_m[ROWS], cta_l[ROWS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int rank  = int(blockIdx.x % unsigned(p.split));  // a cluster is `split` consecutive CTAs
    const int64_t h = blockIdx.x / unsigned(p.split);
    const __nv_bfloat16* Q = p.q + h * p.sq * D;
    const __nv_bfloat16* K = p.k + h * p.sk * D;
    const __nv_bfloat16* V = p.v + h * p.sk * D;
    const int64_t steps = (p.sk + STEP - 1) / STEP, per = (steps + p.split * WARPS - 1) / (p.split * WARPS);
    const int64_t s0 = (rank * WARPS + warp) * per, s1 = s0 + per < steps ? s0 + per : steps;
    const float scale = F32W ? p.scale : p.scale * LOG2E;

    const uint32_t mine = uint32_t(__cvta_generic_to_shared(ring)) + warp * R::WARP_BYTES + lane * 16;
    auto slot  = [&](int64_t step, int piece) { return mine + (unsigned(step - s0) % R::STAGES * R::CHUNKS + piece) * 512; };
    auto fetch = [&](int64_t step) {  // this lane's pieces of the step's K and V; a step that is not there is an empty group
        if (step < s1) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const int64_t key = step * STEP + t * 8 + g;
                    copy16(slot(step, t * G + i), key < p.sk ? K + key * D + i * 32 + c * 8 : K, key < p.sk);
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    const int64_t key = step * STEP + (j >> 1) * 8 + 2 * c + (j & 1);
                    copy16(slot(step, 2 * G + j * CH + ch), key < p.sk ? V + key * D + ch * 64 + g * 8 : V, key < p.sk);
                }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < R::STAGES - 1; ++i) fetch(s0 + i);

    uint4 q[2][G];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < G; ++i) q[r][i] = ld_row(Q + (g + 8 * r) * D + i * 32 + c * 8, g + 8 * r < p.sq);
    float o[CH][8][4], m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int ch = 0; ch < CH; ++ch)
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[ch][t][e] = 0.f;
    // rows g and g + 8 see keys [0, limit)
    int64_t limit[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        limit[r] = p.causal ? g + 8 * r + 1 + p.sk - p.sq : p.sk;
        if (limit[r] > p.sk) limit[r] = p.sk;
    }
    const int64_t seen_by_all = p.causal && p.sk - p.sq + 1 < p.sk ? p.sk - p.sq + 1 : p.sk;

    for (int64_t step = s0; step < s1; ++step) {
        fetch(step + R::STAGES - 1);  // over the step before this one, whose pieces are in registers or used up
        asm volatile("cp.async.wait_group %0;" ::"n"(R::STAGES - 1) : "memory");
        // all of the step's fragments first: the copies into registers overlap one another and the first product
        uint4 kr[2][G], vr[4][CH];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < G; ++i) kr[t][i] = ld_shared16(slot(step, t * G + i));
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) vr[j][ch] = ld_shared16(slot(step, 2 * G + j * CH + ch));
        float s[2][4] = {}, s2[2][4] = {};  // two chains of dependent products for each eight keys
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                mma16816(s[t], q[0][i].x, q[1][i].x, q[0][i].y, q[1][i].y, kr[t][i].x, kr[t][i].y);
                mma16816(s2[t], q[0][i].z, q[1][i].z, q[0][i].w, q[1][i].w, kr[t][i].z, kr[t][i].w);
            }
        // scores of this lane: key step * 16 + t * 8 + 2c + (e & 1), row g + 8 (e >> 1); `left[r]`: how many of the step's keys
        // the row sees
        const bool whole = step * STEP + STEP <= seen_by_all;
        int left[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t n = limit[r] - step * STEP;
            left[r]         = n < 0 ? 0 : n > STEP ? STEP : int(n);
        }
        float mx[2] = {-CUDART_INF_F, -CUDART_INF_F}, alpha[2], from[2];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[t][e] = (s[t][e] + s2[t][e]) * scale;
                if (whole || t * 8 + 2 * c + (e & 1) < left[e >> 1]) mx[e >> 1] = fmaxf(mx[e >> 1], s[t][e]);
            }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float m_new = fmaxf(m[r], quad_max(mx[r]));
            alpha[r]          = part_weight<F32W>(m[r], m_new);
            m[r]              = m_new;
            from[r]           = m_new == -CUDART_INF_F ? 0.f : m_new;  // keys that score minus infinity so far weigh nothing
            l[r] *= alpha[r];
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[t][e] = whole || t * 8 + 2 * c + (e & 1) < left[e >> 1] ? power<F32W>(s[t][e] - from[e >> 1]) : 0.f;
                l[e >> 1] += s[t][e];
            }
        if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {  // a maximum has grown (rare after the first steps)
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
#pragma unroll
                for (int t = 0; t < 8; ++t)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[ch][t][e] *= alpha[e >> 1];
        }
        // A key that a row does not see must not reach it even as 0 times an infinity: such a block, where it holds one, is
        // added cell by cell over the keys each row sees.
        bool odd_block = false;
        if (!whole) {
            bool bad = false;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) bad = bad || has_nonfinite(vr[j][ch]);
            odd_block = __any_sync(0xffffffffu, bad);
        }
        if (!odd_block) {
#pragma unroll
            for (int piece = 0; piece < (F32W ? 3 : 1); ++piece) {
                uint32_t a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float &lo = s[i >> 1][(i & 1) * 2], &hi = s[i >> 1][(i & 1) * 2 + 1];
                    a[i] = F32W ? f32split::upper_halves(lo, hi) : pack_bf16x2(lo, hi);
                    if (F32W) lo = f32split::lower_part(lo), hi = f32split::lower_part(hi);
                }
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    const uint32_t w0[4] = {vr[0][ch].x, vr[0][ch].y, vr[0][ch].z, vr[0][ch].w}, w1[4] = {vr[1][ch].x, vr[1][ch].y, vr[1][ch].z, vr[1][ch].w};
                    const uint32_t w2[4] = {vr[2][ch].x, vr[2][ch].y, vr[2][ch].z, vr[2][ch].w}, w3[4] = {vr[3][ch].x, vr[3][ch].y, vr[3][ch].z, vr[3][ch].w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        mma16816(o[ch][2 * u], a[0], a[1], a[2], a[3], __byte_perm(w0[u], w1[u], 0x5410), __byte_perm(w2[u], w3[u], 0x5410));
                        mma16816(o[ch][2 * u + 1], a[0], a[1], a[2], a[3], __byte_perm(w0[u], w1[u], 0x7632), __byte_perm(w2[u], w3[u], 0x7632));
                    }
                }
            }
        } else {
            for (int kk = 0; kk < STEP; ++kk) {
                const int at      = (lane & ~3) | ((kk & 7) >> 1);
                const int64_t key = step * STEP + kk;
                float pr[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float lo = kk < 8 ? s[0][2 * r] : s[1][2 * r], hi = kk < 8 ? s[0][2 * r + 1] : s[1][2 * r + 1];
                    pr[r] = __shfl_sync(0xffffffffu, (kk & 1) ? hi : lo, at);
                    if (!F32W) pr[r] = __bfloat162float(__float2bfloat16_rn(pr[r]));
                }
#pragma unroll
                for (int ch = 0; ch < CH; ++ch)
#pragma unroll
                    for (int t = 0; t < 8; ++t)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (key < limit[e >> 1])
                                o[ch][t][e] = fmaf((e >> 1) ? pr[1] : pr[0], __bfloat162float(V[key * D + ch * 64 + (2 * c + (e & 1)) * 8 + t]), o[ch][t][e]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();  // every lane is done with the warp's ring

    // the warps' parts -> this CTA's part (in the first warp's place) -> the rows of the head, each CTA of the cluster some
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] = quad_sum(l[r]);
        if (c == 0) part_m[warp][g + 8 * r] = m[r], part_l[warp][g + 8 * r] = l[r];
#pragma unroll
        for (int ch = 0; ch < CH; ++ch)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int t = 0; t < 8; t += 4)
                    *reinterpret_cast<float4*>(part_o(warp) + (g + 8 * r) * D + ch * 64 + (2 * c + e) * 8 + t) =
                        make_float4(o[ch][t][2 * r + e], o[ch][t + 1][2 * r + e], o[ch][t + 2][2 * r + e], o[ch][t + 3][2 * r + e]);
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
    if (p.split > 1) cluster_sync();  // no CTA of the cluster exits while another may read its part
}

template <int D, bool F32W>
int launch(const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = attn_few_kernel<D, F32W>;
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
    return note_cuda_error(cudaLaunchKernelEx(&cfg, kern, p));
}

}  // namespace

int attn_few_supported(const mimk_attn_desc& d) {
    if (d.dtype != MIMK_BF16 || (d.head_dim != 64 && d.head_dim != 128)) return 0;
    if (d.seq_q < 1 || d.seq_q > ROWS || d.seq_k < 1 || d.seq_k >= (int64_t(1) << 31)) return 0;
    if (d.batch_heads >= (int64_t(1) << 27)) return 0;
    return aligned16(d.q) && aligned16(d.k) && aligned16(d.v);
}

// The 128-row kernel gives each SM a head and at head_dim 128 streams it as fast as eight warps here do, so where its rounds of
// heads leave few SMs idle it is ahead: 128 heads x 4096: 55.5 / 60.8 us; 256 x 8192: 202 / 215. Not so 64 x 1000: 18.1 / 17.3, or
// at head_dim 64 (256 x 8192: 175 / 109).
int attn_heads_fill(const mimk_attn_desc& d) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev || d.head_dim != 128) return 0;
    const int64_t rounds = (d.batch_heads + dev->sm_count - 1) / dev->sm_count;
    return d.batch_heads * 5 >= rounds * dev->sm_count * 4;
}

int attn_few(const mimk_attn_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p;
    p.q = static_cast<const __nv_bfloat16*>(d.q), p.k = static_cast<const __nv_bfloat16*>(d.k), p.v = static_cast<const __nv_bfloat16*>(d.v);
    p.o = static_cast<__nv_bfloat16*>(d.o), p.lse = d.lse;
    p.sq = d.seq_q, p.sk = d.seq_k, p.scale = d.scale, p.causal = d.causal;
    // As many CTAs per head as the SMs hold at once (two each): a second round of CTAs would pay the start of its stream and the
    // merge, together several steps, again (128 heads x 4096 keys: split 1 / 2 / 4 / 8: 64 / 61 / 65 / 74 us; 8 x 8192: 118 / 64 /
    // 36 / 22). Every warp has at least three steps.
    p.split = 1;
    while (p.split < 8 && d.batch_heads * p.split * 2 <= 2 * int64_t(dev->sm_count) && d.seq_k >= int64_t(p.split) * 2 * WARPS * 3 * STEP) p.split *= 2;
    // The calls that the 128-row kernel takes too (attn_tc_p.cu) have weights rounded to bf16, as there; the others, whose general
    // path keeps them in f32 (attn_row.cuh), keep them here.
    const int64_t ctas = d.batch_heads * p.split;
    if (attn_tc_persistent_supported(d)) return d.head_dim == 128 ? launch<128, false>(p, ctas, s) : launch<64, false>(p, ctas, s);
    return d.head_dim == 128 ? launch<128, true>(p, ctas, s) : launch<64, true>(p, ctas, s);
}

}  // namespace mimk
