// f32 attention on the tensor cores in one launch: softmax(scale * Q K^T [+ causal mask]) V (MimIR lit/tensor/attn_exec.mim:20-22)
// with f32-grade accuracy, any lengths and alignment, head_dim up to 128. Scores and probabilities never leave the SM.
//
// A CTA owns 128 query rows of one head and walks the keys in blocks of 64. Q, K, V and the probabilities are cut into three
// bf16 pieces each (f32_split.cuh), both products take the six piece products that matter:
//   warps 0..7   read K and V, store their pieces (V transposed) in shared memory; scores from tensor memory -> online softmax
//                in registers (a row is shared by two threads) -> the pieces of P into tensor memory; add the finished block's
//                P V, rescaled, to the output rows kept in registers, with ordinary f32 adds
//   warp 8       issues S = Q K^T (operands in shared memory) and P V (P read from tensor memory)
// P V of a block runs while K of the next is read and cut, the next scores while V is; only the softmax leaves the tensor
// cores idle, and head_dim <= 64 has a second CTA on the SM for that. What bounds it: the shared-memory reads of S (A 4 KB and
// B 2 KB per instruction, 48 clocks against 32 of arithmetic) and the serial chain score -> softmax -> P V.
// Measured: 32 heads x 1000 x 64, 116 us (71 TFLOP/s; 771 us as three passes over a score matrix); 127 heads x 215 x 64, 36 us, and
// 11 x 1047 x 128, 97 us (1760 and 7710 us with a warp per row). 2-norm error 1.7e-7 to 3.8e-7.
//
// Rows whose result is not finite (an infinite or NaN operand, an overflow), or so small that bits lost in the cutting of tiny
// values (and weights) would show, are computed again by the general path.
#include "attn_row.cuh"
#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;
using namespace f32split;

namespace {

constexpr int BQ = 128, BKEYS = 64, WORKERS = 256, NUM_THREADS = WORKERS + 32;

template <int DP> struct Cfg {
    static constexpr int TILES = DP / 32;  // 32-wide tiles along head_dim
    static constexpr int Q_PIECE = BQ * DP * 2, K_PIECE = BKEYS * DP * 2, V_PIECE = DP * BKEYS * 2;
    static constexpr int K_AT = 3 * Q_PIECE, V_AT = K_AT + 3 * K_PIECE, TILE_BYTES = V_AT + 3 * V_PIECE;
    static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 2048 + 256;
    // tensor memory: scores, P V of one block, the pieces of P (two bf16 per column)
    static constexpr int S_COL = 0, O_COL = BKEYS, P_COL = O_COL + DP, COLS = P_COL + 96 <= 256 ? 256 : 512;
};

struct Bars {
    uint64_t k_full, v_full, p_full, s_full, o_full, pair[4], all;
    uint32_t tmem_base;
    int abort_flag;
    uint32_t max_qk, max_v;  // the largest magnitudes that were cut
    uint32_t zeros, deep;    // a result is exactly zero; then: V has values below all their pieces
};

struct Params {
    const float *q, *k, *v;
    float *o, *lse;
    int64_t sq, sk;
    int d, causal, vec_q, vec_k, vec_o;
    float scale;
    int64_t q_tiles;
    int* status;
};

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
// The warps that share a barrier meet: the two of 32 rows, or all eight (a bounded wait like any other: a named barrier would keep one
// of them for good once another has given up).
__device__ __forceinline__ bool pair_meet(uint64_t* bar, uint32_t& parity, volatile int* abort_flag) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(bar));
    const bool ok = warp_wait(smem_u32(bar), parity, abort_flag);
    parity ^= 1u;
    return ok;
}

template <int DP>
__global__ void __launch_bounds__(NUM_THREADS, DP <= 64 ? 2 : 1) attn_f32_tc_kernel(const Params p) {
    using C = Cfg<DP>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;
    float* pair_max = reinterpret_cast<float*>(smem_raw + (base - raw_addr) + C::TILE_BYTES);  // [2][128], later: row not finite
    float* pair_sum = pair_max + 256;
    Bars* bars      = reinterpret_cast<Bars*>(smem_raw + (base - raw_addr) + C::TILE_BYTES + 2048);
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // late query tiles first: under a causal mask they are the long ones
    const int64_t h  = blockIdx.x / p.q_tiles, q0 = (p.q_tiles - 1 - blockIdx.x % p.q_tiles) * BQ;
    const int64_t last_row = q0 + BQ - 1 < p.sq - 1 ? q0 + BQ - 1 : p.sq - 1;
    int64_t visible = p.causal ? last_row + 1 + p.sk - p.sq : p.sk;  // keys that some row of the tile sees
    visible = visible < 0 ? 0 : (visible > p.sk ? p.sk : visible);
    const int blocks = int((visible + BKEYS - 1) / BKEYS);
    const float* Q = p.q + h * p.sq * p.d;
    const float* K = p.k + h * p.sk * p.d;
    const float* V = p.v + h * p.sk * p.d;

    if (tid == 0) {
        mbar_init(smem_u32(&bars->k_full), WORKERS / 32);
        mbar_init(smem_u32(&bars->v_full), WORKERS / 32);
        mbar_init(smem_u32(&bars->p_full), WORKERS / 32);
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&bars->pair[i]), 2);
        mbar_init(smem_u32(&bars->all), WORKERS / 32);
        bars->max_qk = bars->max_v = bars->zeros = bars->deep = 0;
        mbar_init(smem_u32(&bars->s_full), 1);
        mbar_init(smem_u32(&bars->o_full), 1);
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(&bars->tmem_base), C::COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};

    if (warp == 8) {
        if (lane == 0) {
            const uint32_t idesc_s = idesc_bf16_f32(BQ, BKEYS, 0, 0), idesc_o = idesc_bf16_f32(BQ, DP, 0, 0);
            auto scores = [&](uint32_t parity) {
                if (!mbar_wait(smem_u32(&bars->k_full), parity, abort_flag)) return false;
                tc_fence_after();
#pragma unroll
                for (int t = 0; t < 6; ++t)
                    for (int ks = 0; ks < DP / 16; ++ks)
                        mma_f16_ss(tmem + C::S_COL, smem_desc_sw64(base + PA[t] * C::Q_PIECE + (ks >> 1) * (BQ * 64) + (ks & 1) * 32),
                                   smem_desc_sw64(base + C::K_AT + PB[t] * C::K_PIECE + (ks >> 1) * (BKEYS * 64) + (ks & 1) * 32),
                                   idesc_s, (t > 0 || ks > 0) ? 1u : 0u);
                mma_commit(smem_u32(&bars->s_full));
                return true;
            };
            bool ok = blocks == 0 || scores(0);
            for (int j = 0; j < blocks && ok; ++j) {
                const uint32_t parity = j & 1;
                if (!(ok = mbar_wait(smem_u32(&bars->v_full), parity, abort_flag))) break;
                if (!(ok = mbar_wait(smem_u32(&bars->p_full), parity, abort_flag))) break;
                tc_fence_after();
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int ks = 0; ks < BKEYS / 16; ++ks)
                        mma_f16_ts(tmem + C::O_COL, tmem + C::P_COL + PA[t] * 32 + ks * 8,
                                   smem_desc_sw64(base + C::V_AT + PB[t] * C::V_PIECE + (ks >> 1) * (DP * 64) + (ks & 1) * 32), idesc_o,
                                   (t > 0 || ks > 0) ? 1u : 0u);
                mma_commit(smem_u32(&bars->o_full));
                if (j + 1 < blocks) ok = scores(parity ^ 1u);
            }
        }
        __syncwarp();
    } else {
        constexpr int HALF = DP / 2;  // output columns per thread
        const int quarter = warp & 3, half = warp >> 2;
        const int r       = quarter * 32 + lane;  // this thread's row of the tile: tensor-memory lane r
        const uint32_t lanes = uint32_t(quarter * 32) << 16;
        float o[HALF], m = -CUDART_INF_F, l = 0.f;
        float most_qk = 0.f, most_v = 0.f;
        auto see = [](float& most, const float (&x)[8]) {
#pragma unroll
            for (int i = 0; i < 8; i += 2) most = fmaxf(fmaxf(most, fabsf(x[i])), fabsf(x[i + 1]));
        };
#pragma unroll
        for (int i = 0; i < HALF; ++i) o[i] = 0.f;

        auto fetch_k = [&](float (&x)[C::TILES][8], int j) {
            const int64_t key = int64_t(j) * BKEYS + (tid >> 2);
#pragma unroll
            for (int t = 0; t < C::TILES; ++t)
                load8(x[t], K + key * p.d + t * 32 + (tid & 3) * 8, key < p.sk, p.d - t * 32 - (tid & 3) * 8, p.vec_k);
        };
        auto store_k = [&](const float (&x)[C::TILES][8]) {
#pragma unroll
            for (int t = 0; t < C::TILES; ++t)
                see(most_qk, x[t]), split_store8(base + C::K_AT + t * (BKEYS * 64) + unit_offset(tid >> 2, tid & 3), C::K_PIECE, x[t]);
        };
        auto fetch_v = [&](float (&x)[C::TILES][8], int j) {  // eight keys of one column; neighbouring lanes, neighbouring columns
            const int64_t key = int64_t(j) * BKEYS + warp * 8;
#pragma unroll
            for (int t = 0; t < C::TILES; ++t)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    x[t][i] = t * 32 + lane < p.d && key + i < p.sk ? __ldg(V + (key + i) * p.d + t * 32 + lane) : 0.f;
        };
        auto store_v = [&](const float (&x)[C::TILES][8]) {
#pragma unroll
            for (int t = 0; t < C::TILES; ++t)
                see(most_v, x[t]), split_store8(base + C::V_AT + (warp >> 2) * (DP * 64) + unit_offset(t * 32 + lane, warp & 3), C::V_PIECE, x[t]);
        };
        auto publish = [&](uint64_t* bar) {  // this warp's shared-memory stores are ready for the MMA
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(bar));
        };

        if (blocks > 0) {
            for (int t = 0; t < C::TILES; ++t)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int row = (tid >> 2) + i * 64;
                    float x[8];
                    load8(x, Q + (q0 + row) * p.d + t * 32 + (tid & 3) * 8, q0 + row < p.sq, p.d - t * 32 - (tid & 3) * 8, p.vec_q);
                    see(most_qk, x);
                    split_store8(base + t * (BQ * 64) + unit_offset(row, tid & 3), C::Q_PIECE, x);
                }
            float x[C::TILES][8];
            fetch_k(x, 0);
            store_k(x);
            publish(&bars->k_full);
            fetch_v(x, 0);
            store_v(x);
            publish(&bars->v_full);
        }
        // keys [0, limit) take part in this row
        int64_t limit = p.causal ? q0 + r + 1 + p.sk - p.sq : p.sk;
        limit = limit > p.sk ? p.sk : limit;
        bool ok = true;
        uint32_t meeting = 0;
        for (int j = 0; j < blocks; ++j) {
            const uint32_t parity = j & 1;
            const bool more       = j + 1 < blocks;
            float x[C::TILES][8];
            if (more) fetch_k(x, j + 1);
            if (!(ok = warp_wait(smem_u32(&bars->s_full), parity, abort_flag))) break;
            tc_fence_after();
            uint32_t sr[32];
            tmem_ld_32x32(tmem + C::S_COL + half * 32 + lanes, sr);
            tmem_ld_wait();
            const int64_t left = limit - int64_t(j) * BKEYS - half * 32;  // of this thread's 32 keys, the first `left` count
            float mx = -CUDART_INF_F;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float s = __uint_as_float(sr[i]) * p.scale;
                sr[i] = __float_as_uint(s);
                if (i < left) mx = fmaxf(mx, s);
            }
            pair_max[half * 128 + r] = mx;
            if (!(ok = pair_meet(&bars->pair[quarter], meeting, abort_flag))) break;
            mx = fmaxf(mx, pair_max[(half ^ 1) * 128 + r]);
            const float m_new = fmaxf(m, mx);
            const float alpha = m == -CUDART_INF_F ? 0.f : expf(m - m_new);
            const float from  = m_new == -CUDART_INF_F ? 0.f : m_new;  // keys that score minus infinity so far weigh nothing
            m                 = m_new;
            float part = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float e = i < left ? expf(__uint_as_float(sr[i]) - from) : 0.f;
                part += e;
                sr[i] = __float_as_uint(e);
            }
            l = l * alpha + part;
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) {
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    w[i] = __byte_perm(sr[2 * i], sr[2 * i + 1], 0x7632);
                    if (piece < 2) {
                        sr[2 * i]     = __float_as_uint(lower_part(__uint_as_float(sr[2 * i])));
                        sr[2 * i + 1] = __float_as_uint(lower_part(__uint_as_float(sr[2 * i + 1])));
                    }
                }
                tmem_st_32x32_x16(tmem + C::P_COL + piece * 32 + half * 16 + lanes, w);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->p_full));
            if (more) {  // the scores are read and the MMAs that read K are complete: the next K
                store_k(x);
                publish(&bars->k_full);
                fetch_v(x, j + 1);
            }
            if (!(ok = warp_wait(smem_u32(&bars->o_full), parity, abort_flag))) break;
            tc_fence_after();
            const uint32_t t0 = tmem + C::O_COL + half * HALF + lanes;
#pragma unroll
            for (int c = 0; c < HALF; c += 16) {
                uint32_t w[16];
                tmem_ld_32x16(t0 + c, w);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c + i] = fmaf(o[c + i], alpha, __uint_as_float(w[i]));
            }
            tc_fence_before();
            if (more) {
                store_v(x);
                publish(&bars->v_full);
            }
        }
        pair_sum[half * 128 + r] = l;
        // What the cutting may have lost: a value below 2^-109 the bits under 2^-133. Scores are off by less than d (max |q| + max |k|)
        // 2^-133, a result by 2^-133 for V, whose weights sum to at least one, and by keys * max |v| * 2^-133 for the weights.
        const uint32_t mqk = __reduce_max_sync(0xffffffffu, __float_as_uint(most_qk)), mv = __reduce_max_sync(0xffffffffu, __float_as_uint(most_v));
        if (lane == 0) atomicMax(&bars->max_qk, mqk), atomicMax(&bars->max_v, mv);
        uint32_t together = 0;
        ok = ok && pair_meet(&bars->all, together, abort_flag);
        l += pair_sum[(half ^ 1) * 128 + r];
        auto shared          = [](const uint32_t* word) { return *reinterpret_cast<const volatile uint32_t*>(word); };
        const bool spoiled   = fabsf(p.scale) * p.d * 2.f * LOST_ABS * __uint_as_float(shared(&bars->max_qk)) > 0x1p-24f;
        const float small    = 0x1p22f * LOST_ABS * (1.f + float(visible) * __uint_as_float(shared(&bars->max_v)));  // 22 bits above the loss
        // a row both of whose threads saw only finite results that are large enough is written here, any other one below
        const float inv = l > 0.f ? 1.f / l : 0.f;
        bool finite     = isfinite(l) && (l > 0.f || limit <= 0) && !spoiled, zero = false;  // (keys seen and no weight: the general path)
#pragma unroll
        for (int i = 0; i < HALF; ++i) {
            o[i] *= inv;
            finite = finite && isfinite(o[i]) && (fabsf(o[i]) >= small || o[i] == 0.f);
            zero   = zero || (o[i] == 0.f && half * HALF + i < p.d);
        }
        // A zero is short of something only if V has values below all their pieces.
        zero = zero && q0 + r < p.sq && limit > 0;
        if (__any_sync(0xffffffffu, zero) && lane == 0) bars->zeros = 1;
        ok = ok && pair_meet(&bars->all, together, abort_flag);
        if (__any_sync(0xffffffffu, shared(&bars->zeros) != 0)) {
            bool deep = false;
            for (int64_t i = tid; i < visible * p.d; i += WORKERS) {
                const float v = fabsf(__ldg(V + i));
                deep          = deep || (v > 0.f && v < LOST_ABS);
            }
            if (__any_sync(0xffffffffu, deep) && lane == 0) bars->deep = 1;
            ok     = ok && pair_meet(&bars->all, together, abort_flag);
            finite = finite && !(zero && shared(&bars->deep));
        }
        pair_max[half * 128 + r] = finite ? 0.f : 1.f;  // (its last reads as a maximum lie before the exchange of sums)
        ok = ok && pair_meet(&bars->pair[quarter], meeting, abort_flag);
        const bool there = ok && q0 + r < p.sq;
        const bool redo  = there && (pair_max[r] != 0.f || pair_max[128 + r] != 0.f);
        if (there && !redo) {
            float* dst = p.o + (h * p.sq + q0 + r) * p.d + half * HALF;
#pragma unroll
            for (int i = 0; i < HALF; i += 4) {
                if (p.vec_o && half * HALF + i + 4 <= p.d) {
                    *reinterpret_cast<float4*>(dst + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (half * HALF + i + e < p.d) dst[i + e] = o[i + e];
                }
            }
            if (p.lse && half == 0) p.lse[h * p.sq + q0 + r] = l > 0.f ? m + logf(l) : -CUDART_INF_F;
        }
        // every MMA of the tile is complete, so the Q tiles become each warp's row buffer; the two warps of a quarter take its
        // rows in turn
        unsigned again = __ballot_sync(0xffffffffu, redo);
        if (again) {
            float* qs = reinterpret_cast<float*>(smem_raw + (base - raw_addr)) + warp * 128;
            while (again) {
                const int i = __ffs(again) - 1;
                again &= again - 1;
                if ((i & 1) != half) continue;
                __syncwarp();
                attn_row::row<float, 128>(qs, p.q, p.k, p.v, p.o, p.lse, h, q0 + quarter * 32 + i, p.sq, p.sk, p.d, p.scale, p.causal);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, C::COLS);
    }
    if (tid == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

template <int DP>
int launch(const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = attn_f32_tc_kernel<DP>;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<DP>::SMEM_BYTES));
        configured[dev & 63] = true;
    }
    kern<<<unsigned(ctas), NUM_THREADS, Cfg<DP>::SMEM_BYTES, s>>>(p);
    return launch_status();
}

}  // namespace

int attn_f32_tc_supported(const mimk_attn_desc& d) {
    if (d.dtype != MIMK_F32 || d.head_dim < 1 || d.head_dim > 128 || d.seq_k < 1) return 0;
    const int64_t q_tiles = (d.seq_q + BQ - 1) / BQ;
    return d.seq_q < (int64_t(1) << 31) && d.seq_k < (int64_t(1) << 31) && q_tiles < (int64_t(1) << 30) / d.batch_heads;
}

int attn_f32_tc(const mimk_attn_desc& d, cudaStream_t s) {
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    Params p;
    p.q = static_cast<const float*>(d.q), p.k = static_cast<const float*>(d.k), p.v = static_cast<const float*>(d.v);
    p.o = static_cast<float*>(d.o), p.lse = d.lse;
    p.sq = d.seq_q, p.sk = d.seq_k, p.d = int(d.head_dim), p.causal = d.causal, p.scale = d.scale;
    p.vec_q = p.d % 4 == 0 && aligned16(d.q), p.vec_k = p.d % 4 == 0 && aligned16(d.k), p.vec_o = p.d % 4 == 0 && aligned16(d.o);
    p.q_tiles = (d.seq_q + BQ - 1) / BQ;
    p.status  = dev->status_dev;
    const int64_t ctas = p.q_tiles * d.batch_heads;
    if (p.d <= 32) return launch<32>(p, ctas, s);
    if (p.d <= 64) return launch<64>(p, ctas, s);
    if (p.d <= 96) return launch<96>(p, ctas, s);
    return launch<128>(p, ctas, s);
}

}  // namespace mimk
