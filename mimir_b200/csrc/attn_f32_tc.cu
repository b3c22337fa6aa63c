// f32 attention on the tensor cores in one launch: softmax(scale * Q K^T [+ causal mask]) V (MimIR lit/tensor/attn_exec.mim:20-22)
// with f32-grade accuracy, any lengths and alignment, head_dim up to 128. Scores and probabilities never leave the SM.
//
// A tile of 128 query rows of one head walks the keys in blocks of 64. Q, K, V and the probabilities are cut into three bf16
// pieces each (f32_split.cuh), both products take the six piece products that matter:
//   workers      scores from tensor memory -> online softmax in registers -> the pieces of P into tensor memory; add the finished
//                block's P V, rescaled, to the output rows kept in registers, with ordinary f32 adds
//   MMA warp     issues S = Q K^T (operands in shared memory) and P V (P read from tensor memory); the next block's S as soon as
//                this one's has been read, so it runs beside the softmax
// Many keys and several tiles a head (LAID): K and V are cut once, by a launch of their own, and come by TMA, piece by piece in the
// order of the products. head_dim <= 64: two tiles share them on an SM (a row is one thread's, 8 warps of workers, two MMA warps);
// beyond, one tile (a row is shared by two threads). Otherwise the workers also read and cut K and V (V transposed) for each tile,
// and head_dim <= 64 has two CTAs per SM.
// What bounds it: LAID with two tiles the MMAs (N = 64: 46 clocks each with P in tensor memory, 57 with Q in shared memory, against 32
// of arithmetic; 4600 clocks a block for both tiles), else the chain score -> softmax -> P V (3400 a block).
// Measured (K and V cut by the workers before): 32 heads x 1000 x 64 65 us (119); 128 x 1024 x 64 241 (410); 128 x 2000 x 32 causal 329 (651);
// 8 x 2048 x 128 110 (175); 11 x 1047 x 128 71 (99). 2-norm error 1.7e-7 to 4e-7.
//
// Rows whose result is not finite (an infinite or NaN operand, an overflow), or so small that bits lost in the cutting of tiny
// values (and weights) would show, are computed again by the general path.
#include <type_traits>

#include "attn_common.cuh"
#include "attn_row.cuh"
#include "common.cuh"
#include "f32_split.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;
using namespace f32split;
using namespace attn;

namespace {

constexpr float LOG2E = 1.4426950408889634f;

constexpr int BQ = 128, BKEYS = 64;

// What a group of workers and its MMA warp share.
struct Group {
    uint64_t q_full, p_full, s_full, o_full, s_free, pair[4], all;
    uint32_t max_qk, max_v;  // the largest magnitudes that were cut
    uint32_t zeros, deep;    // a result is exactly zero; then: V has values below all their pieces
};
struct Bars {
    Group group[2];
    uint64_t k_full, v_full;  // the workers' K and V
    uint64_t k_there[2][3], k_free[2][3], v_there[2][3], v_free[2][3];  // LAID: stages of pieces
    uint32_t tmem_base;
    int abort_flag;
};

template <int DP, bool LAID> struct Cfg {
    static constexpr int GROUPS = LAID && DP <= 64 ? 2 : 1;  // query tiles per CTA
    static constexpr int STAGES = GROUPS;                    // of K and V
    static constexpr int SPLIT  = 3 - GROUPS;                // threads of a row
    static constexpr int WORKERS = BQ * SPLIT, WORKER_WARPS = WORKERS / 32;  // of one query tile
    static constexpr int MMA_WARP = GROUPS * WORKER_WARPS, K_WARP = MMA_WARP + GROUPS, V_WARP = K_WARP + 1;
    static constexpr int NUM_THREADS = 32 * (LAID ? V_WARP + 1 : K_WARP);
    static constexpr int CTAS  = DP <= 64 && !LAID ? 2 : 1;  // per SM
    static constexpr int TILES = DP / 32;  // 32-wide tiles along head_dim
    static constexpr int ATOMS = (DP + 63) / 64, ATOM_BYTES = BKEYS * 128;  // LAID: K and V lie in 64-wide boxes of 64 keys, 128-byte rows
    static constexpr int Q_PIECE = BQ * DP * 2, K_PIECE = LAID ? ATOMS * ATOM_BYTES : BKEYS * DP * 2, V_PIECE = K_PIECE;
    static constexpr int K_AT = GROUPS * 3 * Q_PIECE, V_AT = K_AT + STAGES * 3 * K_PIECE, TILE_BYTES = V_AT + STAGES * 3 * V_PIECE;
    static constexpr int ROWS_AT = TILE_BYTES, ROWS_BYTES = SPLIT == 2 ? 3 * 256 * 4 : 0;  // what the two threads of a row exchange
    static constexpr int BARS_AT = ROWS_AT + GROUPS * ROWS_BYTES;
    static constexpr int SMEM_BYTES = BARS_AT + 1024 + int(sizeof(Bars));
    // tensor memory of a group: scores, P V of one block, the pieces of P (two bf16 per column)
    static constexpr int S_COL = 0, O_COL = BKEYS, P_COL = O_COL + DP, COLS = P_COL + 96 <= 256 ? 256 : 512;
    static_assert(CTAS * (SMEM_BYTES + 1024) <= 233472 && GROUPS * CTAS * COLS <= 512, "an SM's shared and tensor memory");
    // two tiles: registers move from the warpgroup that loads and issues to the two of workers (168 a thread at launch)
    static constexpr int WORKER_REGS = 224, ISSUE_REGS = 56;
    static_assert(GROUPS == 1 || (NUM_THREADS == 384 && 2 * WORKER_REGS + ISSUE_REGS <= 3 * 168), "setmaxnreg waits for ever for more than the launch was given");
    static_assert(ATOM_BYTES % 1024 == 0 && (3 * Q_PIECE) % 1024 == 0, "128-byte swizzle");
};

struct Params {
    const float *q, *k, *v;
    float *o, *lse;
    int64_t sq, sk;
    int d, causal, vec_q, vec_k, vec_o;
    float scale;
    int64_t q_tiles, items;  // query tiles of a head, and CTAs that share them
    int per_cta;             // query tiles of a CTA
    int* status;
    const float* most;  // LAID: the largest magnitudes of K and of V in each block of 64 keys of each head
    int64_t kv_blocks;
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

// A block of 64 keys of one head cut into pieces, K and V ([piece][head][key][dp], zeros behind d), and its largest magnitudes.
__global__ void __launch_bounds__(256) attn_cut_kernel(const float* __restrict__ k, const float* __restrict__ v, __nv_bfloat16* __restrict__ pieces,
                                                       float* __restrict__ most, int64_t sk, int64_t kv_blocks, int d, int dp, int vec, int64_t piece) {
    __shared__ float warp_most[8];
    const int64_t head = blockIdx.x / kv_blocks, block = blockIdx.x - head * kv_blocks;
    const int64_t first = head * sk + block * BKEYS;
    const int keys = int(sk - block * BKEYS < BKEYS ? sk - block * BKEYS : BKEYS), quads = dp / 4;
    for (int which = 0; which < 2; ++which) {
        const float* src   = (which ? v : k) + first * d;
        __nv_bfloat16* dst = pieces + which * 3 * piece + first * dp;
        float largest      = 0.f;
#pragma unroll 4
        for (int i = threadIdx.x; i < keys * quads; i += 256) {
            const int row = i / quads, col = (i - row * quads) * 4;
            float x[4];
            load4(x, src + int64_t(row) * d + col, true, d - col, vec);
#pragma unroll
            for (int e = 0; e < 4; ++e) largest = fmaxf(largest, fabsf(x[e]));
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                *reinterpret_cast<uint2*>(dst + t * piece + int64_t(row) * dp + col) = make_uint2(upper_halves(x[0], x[1]), upper_halves(x[2], x[3]));
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = lower_part(x[e]);
            }
        }
        largest = warp_max(largest);
        if ((threadIdx.x & 31) == 0) warp_most[threadIdx.x >> 5] = largest;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < 8; ++i) largest = fmaxf(largest, warp_most[i]);
            most[int64_t(blockIdx.x) * 2 + which] = largest;
        }
        __syncthreads();
    }
}

// LAID: K and V have been cut by attn_cut_kernel and come by TMA, for up to two query tiles; else the workers read and cut them.
template <int DP, bool LAID>
__global__ void __launch_bounds__(Cfg<DP, LAID>::NUM_THREADS, Cfg<DP, LAID>::CTAS)
attn_f32_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Params p) {
    using C = Cfg<DP, LAID>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;
    uint8_t* smem           = smem_raw + (base - raw_addr);
    Bars* bars              = reinterpret_cast<Bars*>(smem + C::BARS_AT);
    volatile int* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // late query tiles first: under a causal mask they are the long ones
    const int64_t h = blockIdx.x / p.items, item = p.items - 1 - blockIdx.x % p.items;
    // a tile's blocks of keys: those that some of its rows sees
    auto blocks_of = [&](int g) {
        const int64_t q0 = (item * p.per_cta + g) * BQ;
        if (q0 >= p.sq || g >= p.per_cta) return 0;
        const int64_t last_row = q0 + BQ - 1 < p.sq - 1 ? q0 + BQ - 1 : p.sq - 1;
        int64_t visible        = p.causal ? last_row + 1 + p.sk - p.sq : p.sk;
        visible                = visible < 0 ? 0 : (visible > p.sk ? p.sk : visible);
        return int((visible + BKEYS - 1) / BKEYS);
    };
    const int group = warp < C::MMA_WARP ? warp / C::WORKER_WARPS : warp < C::K_WARP ? warp - C::MMA_WARP : 0;
    Group* own      = &bars->group[group];
    // (of a CTA's two tiles the later has no fewer blocks; every block goes through both tiles' MMA warps)
    const int blocks = blocks_of(group), most_blocks = C::GROUPS == 2 ? max(blocks_of(0), blocks_of(1)) : blocks;
    const float* Q = p.q + h * p.sq * p.d;
    const float* K = p.k + h * p.sk * p.d;
    const float* V = p.v + h * p.sk * p.d;

    if (threadIdx.x == 0) {
        for (int g = 0; g < C::GROUPS; ++g) {
            Group& b = bars->group[g];
            mbar_init(smem_u32(&b.q_full), C::WORKER_WARPS), mbar_init(smem_u32(&b.p_full), C::WORKER_WARPS), mbar_init(smem_u32(&b.s_free), C::WORKER_WARPS);
            mbar_init(smem_u32(&b.s_full), 1), mbar_init(smem_u32(&b.o_full), 1), mbar_init(smem_u32(&b.all), C::WORKER_WARPS);
            for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&b.pair[i]), 2);
            b.max_qk = b.max_v = b.zeros = b.deep = 0;
        }
        if (LAID) {
            for (int s = 0; s < C::STAGES; ++s)
                for (int i = 0; i < 3; ++i) {
                    mbar_init(smem_u32(&bars->k_there[s][i]), 1), mbar_init(smem_u32(&bars->k_free[s][i]), C::GROUPS);
                    mbar_init(smem_u32(&bars->v_there[s][i]), 1), mbar_init(smem_u32(&bars->v_free[s][i]), C::GROUPS);
                }
        } else {
            mbar_init(smem_u32(&bars->k_full), C::WORKER_WARPS), mbar_init(smem_u32(&bars->v_full), C::WORKER_WARPS);
        }
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == C::MMA_WARP) {
        tmem_alloc(smem_u32(&bars->tmem_base), C::GROUPS * C::COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base) + group * C::COLS;
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};

    if (warp >= C::MMA_WARP) {
    if constexpr (C::GROUPS == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::ISSUE_REGS));
    if (LAID && warp >= C::K_WARP) {
        if (lane == 0) {
            // the pieces of a block in the order in which the products need them; a piece's place is free once its last product is done
            constexpr int ORDER[3] = {0, 2, 1};
            const bool is_v        = warp == C::V_WARP;
            const CUtensorMap* map = is_v ? &tmV : &tmK;
            bool ok                = true;
            uint32_t stage = 0, phase = 0;
            for (int j = 0; j < most_blocks && ok; ++j) {
                uint64_t *there = is_v ? bars->v_there[stage] : bars->k_there[stage], *free = is_v ? bars->v_free[stage] : bars->k_free[stage];
                const uint32_t at = base + (is_v ? C::V_AT : C::K_AT) + stage * 3 * C::K_PIECE;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int t = ORDER[i];
                    if (ok) ok = mbar_wait(smem_u32(&free[t]), phase ^ 1u, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(smem_u32(&there[t]), C::K_PIECE);
#pragma unroll
                    for (int a = 0; a < C::ATOMS; ++a)
                        tma_load_4d(at + t * C::K_PIECE + a * C::ATOM_BYTES, map, a * 64, j * BKEYS, int(h), t, smem_u32(&there[t]));
                }
                if (++stage == C::STAGES) stage = 0, phase ^= 1u;
            }
        }
        __syncwarp();
    } else if (LAID) {
        {
            // (the whole warp runs, one lane issues: with lane 0 alone in the branch the descriptors are not known to be uniform, and moving them
            // costs about 50 clocks per MMA)
            const bool leader = elect_one();
            const uint32_t idesc_s = idesc_bf16_f32(BQ, BKEYS, 0, 0), idesc_o = idesc_bf16_f32(BQ, DP, 0, 1);
            auto commit = [&](uint32_t bar) { if (leader) mma_commit(bar); };
            const uint64_t q0_desc = smem_desc_sw64(base + group * 3 * C::Q_PIECE), k0_desc = smem_desc_sw128(base + C::K_AT, 16, 1024);
            const uint64_t v0_desc = smem_desc_sw128(base + C::V_AT, C::ATOM_BYTES, 1024);
            bool ok = true;
            // the six products of block j in three steps, each as soon as its pieces are there; a block this tile does not see is passed on
            auto products = [&](uint64_t (*there)[3], uint64_t (*free)[3], int j, auto&& product) {
                const uint32_t stage = C::STAGES == 2 ? j & 1 : 0, parity = (C::STAGES == 2 ? j >> 1 : j) & 1;
                auto wait = [&](int t) { ok = ok && warp_wait(smem_u32(&there[stage][t]), parity, abort_flag); };
                wait(0), wait(2);
                if (!ok) return;
                tc_fence_after();
                product(stage, std::integral_constant<int, 0>{}), product(stage, std::integral_constant<int, 1>{});
                commit(smem_u32(&free[stage][2]));
                wait(1);
                if (!ok) return;
                tc_fence_after();
                product(stage, std::integral_constant<int, 2>{}), product(stage, std::integral_constant<int, 3>{}), product(stage, std::integral_constant<int, 4>{});
                commit(smem_u32(&free[stage][1]));
                product(stage, std::integral_constant<int, 5>{});
                commit(smem_u32(&free[stage][0]));
            };
            auto scores = [&](int j) {
                if (j > 0) ok = ok && warp_wait(smem_u32(&own->s_free), (j - 1) & 1, abort_flag);
                if (ok)
                    products(bars->k_there, bars->k_free, j, [&](uint32_t stage, auto which) {
                        constexpr int t = decltype(which)::value;
                        const uint64_t k = k0_desc + stage * (3 * C::K_PIECE >> 4);
                        if (leader)
#pragma unroll
                            for (int ks = 0; ks < DP / 16; ++ks)
                                mma_f16_ss(tmem + C::S_COL, q0_desc + ((PA[t] * C::Q_PIECE + (ks >> 1) * (BQ * 64) + (ks & 1) * 32) >> 4),
                                           k + ((PB[t] * C::K_PIECE + (ks >> 2) * C::ATOM_BYTES + (ks & 3) * 32) >> 4), idesc_s, (t > 0 || ks > 0) ? 1u : 0u);
                    });
                if (ok) commit(smem_u32(&own->s_full));
            };
            if (blocks > 0) ok = warp_wait(smem_u32(&own->q_full), 0, abort_flag);
            if (blocks > 0 && ok) scores(0);
            for (int j = 0; j < blocks && ok; ++j) {
                if (j + 1 < blocks) scores(j + 1);  // while the softmax of this block runs
                ok = ok && warp_wait(smem_u32(&own->p_full), j & 1, abort_flag);
                if (ok)
                    products(bars->v_there, bars->v_free, j, [&](uint32_t stage, auto which) {
                        constexpr int t = decltype(which)::value;
                        const uint64_t v = v0_desc + stage * (3 * C::V_PIECE >> 4);
                        if (leader)
#pragma unroll
                            for (int ks = 0; ks < BKEYS / 16; ++ks)
                                mma_f16_ts(tmem + C::O_COL, tmem + C::P_COL + PA[t] * 32 + ks * 8, v + ((PB[t] * C::V_PIECE + ks * 2048) >> 4), idesc_o,
                                           (t > 0 || ks > 0) ? 1u : 0u);
                    });
                if (ok) commit(smem_u32(&own->o_full));
            }
            auto pass = [&](uint64_t (*there)[3], uint64_t (*free)[3], int j) {
                const uint32_t stage = C::STAGES == 2 ? j & 1 : 0, parity = (C::STAGES == 2 ? j >> 1 : j) & 1;
                for (int t = 0; t < 3 && ok; ++t)
                    if ((ok = warp_wait(smem_u32(&there[stage][t]), parity, abort_flag)) && leader) mbar_arrive(smem_u32(&free[stage][t]));
            };
            for (int j = blocks; j < most_blocks && ok; ++j) {
                pass(bars->k_there, bars->k_free, j);
                pass(bars->v_there, bars->v_free, j);
            }
        }
        __syncwarp();
    } else {
        {
            const bool leader = elect_one();
            const uint32_t idesc_s = idesc_bf16_f32(BQ, BKEYS, 0, 0), idesc_o = idesc_bf16_f32(BQ, DP, 0, 0);
            const uint64_t q_desc = smem_desc_sw64(base), k_desc = smem_desc_sw64(base + C::K_AT), v_desc = smem_desc_sw64(base + C::V_AT);
            auto scores = [&](uint32_t parity) {
                if (!warp_wait(smem_u32(&bars->k_full), parity, abort_flag)) return false;
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int t = 0; t < 6; ++t)
#pragma unroll
                        for (int ks = 0; ks < DP / 16; ++ks)
                            mma_f16_ss(tmem + C::S_COL, q_desc + ((PA[t] * C::Q_PIECE + (ks >> 1) * (BQ * 64) + (ks & 1) * 32) >> 4),
                                       k_desc + ((PB[t] * C::K_PIECE + (ks >> 1) * (BKEYS * 64) + (ks & 1) * 32) >> 4), idesc_s, (t > 0 || ks > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&own->s_full));
                }
                return true;
            };
            bool ok = blocks == 0 || scores(0);
            for (int j = 0; j < blocks && ok; ++j) {
                const uint32_t parity = j & 1;
                if (!(ok = warp_wait(smem_u32(&bars->v_full), parity, abort_flag))) break;
                if (!(ok = warp_wait(smem_u32(&own->p_full), parity, abort_flag))) break;
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int t = 0; t < 6; ++t)
#pragma unroll
                        for (int ks = 0; ks < BKEYS / 16; ++ks)
                            mma_f16_ts(tmem + C::O_COL, tmem + C::P_COL + PA[t] * 32 + ks * 8,
                                       v_desc + ((PB[t] * C::V_PIECE + (ks >> 1) * (DP * 64) + (ks & 1) * 32) >> 4), idesc_o, (t > 0 || ks > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&own->o_full));
                }
                if (j + 1 < blocks) ok = scores(parity ^ 1u);
            }
        }
        __syncwarp();
    }
    } else if (group < p.per_cta && (item * p.per_cta + group) * BQ < p.sq) {
        if constexpr (C::GROUPS == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::WORKER_REGS));
        constexpr int HALF = DP / C::SPLIT, KEYS = BKEYS / C::SPLIT;  // output columns and keys of a block per thread
        const int tid = threadIdx.x - group * C::WORKERS, quarter = warp & 3, half = C::SPLIT == 2 ? (warp >> 2) & 1 : 0;
        const int64_t q0 = (item * p.per_cta + group) * BQ;
        float* pair_max  = reinterpret_cast<float*>(smem + C::ROWS_AT + group * C::ROWS_BYTES);  // [parity][2][128], later: row not finite
        float* pair_sum  = pair_max + 512;
        const uint32_t q_tile = base + group * 3 * C::Q_PIECE;
        const int r       = quarter * 32 + lane;  // this thread's row of the tile: tensor-memory lane r
        const uint32_t lanes = uint32_t(quarter * 32) << 16;
        float o[HALF], m = -CUDART_INF_F, from = 0.f;
        uint64_t sums[2] = {0, 0};  // of the weights, in four parts (one sum of a long row loses more than the products do)
        bool l_any = false;  // some key scored above minus infinity
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
            constexpr int ROWS = 512 / C::WORKERS;
#pragma unroll
            for (int t = 0; t < C::TILES; ++t) {
                float x[ROWS][8];  // all on their way before the first is stored
#pragma unroll
                for (int i = 0; i < ROWS; ++i) {
                    const int row = (tid >> 2) + i * (C::WORKERS / 4);
                    load8(x[i], Q + (q0 + row) * p.d + t * 32 + (tid & 3) * 8, q0 + row < p.sq, p.d - t * 32 - (tid & 3) * 8, p.vec_q);
                }
#pragma unroll
                for (int i = 0; i < ROWS; ++i)
                    see(most_qk, x[i]), split_store8(q_tile + t * (BQ * 64) + unit_offset((tid >> 2) + i * (C::WORKERS / 4), tid & 3), C::Q_PIECE, x[i]);
            }
            if (LAID) {
                publish(&own->q_full);
            } else {
                float x[C::TILES][8];
                fetch_k(x, 0);
                store_k(x);
                publish(&bars->k_full);
                fetch_v(x, 0);
                store_v(x);
                publish(&bars->v_full);
            }
        }
        // keys [0, limit) take part in this row
        int64_t limit = p.causal ? q0 + r + 1 + p.sk - p.sq : p.sk;
        limit = limit > p.sk ? p.sk : limit;
        bool ok = true;
        uint32_t meeting = 0;
        float alpha = 0.f;
        auto add_block = [&](int j) {  // P V of block j, with the factor that came with its maximum
            if (!(ok = warp_wait(smem_u32(&own->o_full), j & 1, abort_flag))) return;
            tc_fence_after();
            const uint32_t t0     = tmem + C::O_COL + half * HALF + lanes;
            const uint64_t alpha2 = pack2(alpha, alpha);
            constexpr int WIDE    = C::SPLIT == 1 ? HALF : 16;  // (as many as registers allow)
#pragma unroll
            for (int c = 0; c < HALF; c += WIDE) {
                uint32_t w[WIDE / 16][16];
#pragma unroll
                for (int u = 0; u < WIDE / 16; ++u) tmem_ld_32x16(t0 + c + u * 16, w[u]);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < WIDE; i += 2)
                    unpack2(fma2(pack2(o[c + i], o[c + i + 1]), alpha2, pack2(__uint_as_float(w[i / 16][i % 16]), __uint_as_float(w[i / 16][i % 16 + 1]))),
                            o[c + i], o[c + i + 1]);
            }
            tc_fence_before();
        };
        for (int j = 0; j < blocks; ++j) {
            const uint32_t parity = j & 1;
            const bool more       = !LAID && j + 1 < blocks;
            float x[C::TILES][8];
            if (more) fetch_k(x, j + 1);
            if (!(ok = warp_wait(smem_u32(&own->s_full), parity, abort_flag))) break;
            tc_fence_after();
            uint32_t sr[KEYS];
#pragma unroll
            for (int c = 0; c < KEYS; c += 32) tmem_ld_slice(tmem + C::S_COL + half * KEYS + c + lanes, sr + c);
            tmem_ld_wait();
            if (LAID) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&own->s_free));
            }
            const int64_t rest = limit - int64_t(j) * BKEYS - half * KEYS;
            const int left     = rest > KEYS ? KEYS : int(rest < 0 ? 0 : rest);  // of this thread's keys, the first `left` count
            float top[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};  // (chains of their own)
            const uint64_t scale2 = pack2(p.scale, p.scale), none2 = pack2(-0.f, -0.f);
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) {
                float x, y;
                unpack2(fma2(pack2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), scale2, none2), x, y);
                sr[i] = __float_as_uint(x), sr[i + 1] = __float_as_uint(y);
            }
            if (!__all_sync(0xffffffffu, left == KEYS)) {
#pragma unroll
                for (int i = 0; i < KEYS; ++i)
                    if (i >= left) sr[i] = __float_as_uint(-CUDART_INF_F);
            }
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) top[(i >> 1) & 3] = max3(top[(i >> 1) & 3], __uint_as_float(sr[i]), __uint_as_float(sr[i + 1]));
            float mx = max3(fmaxf(top[0], top[1]), top[2], top[3]);
            if constexpr (C::SPLIT == 2) {
            float* shared_max = pair_max + parity * 256;  // (a warp may be one block ahead of the other)
            shared_max[half * 128 + r] = mx;
            if (!(ok = pair_meet(&own->pair[quarter], meeting, abort_flag))) break;
            mx = fmaxf(mx, shared_max[(half ^ 1) * 128 + r]);
            }
            // weights are 2^(s log2 e - from), one rounding for product and difference; `from` is the rounded product of the maximum, the
            // same for every key until a larger score comes
            m                  = fmaxf(m, mx);
            const float before = from;
            from               = m == -CUDART_INF_F ? 0.f : m * LOG2E;  // keys that score minus infinity so far weigh nothing
            const float factor = l_any ? exp2f(before - from) : 0.f;
            l_any              = l_any || m != -CUDART_INF_F;
            // (exp2f, not the instruction alone, which gives no denormal weights; telling the blocks without any apart costs more in code
            // that each launch fetches anew than it saves: 8 of 128 x 128 x 64 22.6 -> 25.3 us)
            const uint64_t log2e2 = pack2(LOG2E, LOG2E), from2 = pack2(-from, -from);
            uint64_t part[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
#pragma unroll
            for (int i = 0; i < KEYS; i += 2) {
                float x, y;
                unpack2(fma2(pack2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), log2e2, from2), x, y);
                x = exp2f(x), y = exp2f(y);
                part[(i >> 1) & 1] = add2(part[(i >> 1) & 1], pack2(x, y));
                sr[i] = __float_as_uint(x), sr[i + 1] = __float_as_uint(y);
            }
            sums[0] = fma2(sums[0], pack2(factor, factor), part[0]), sums[1] = fma2(sums[1], pack2(factor, factor), part[1]);
            if (LAID && j > 0) {  // the block before this one, whose P V ran meanwhile; its P is read
                add_block(j - 1);
                if (!ok) break;
            }
            alpha = factor;
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) {
#pragma unroll
                for (int c = 0; c < KEYS / 2; c += 16) {
                uint32_t w[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int i = c + u;
                    w[u] = __byte_perm(sr[2 * i], sr[2 * i + 1], 0x7632);
                    if (piece < 2) {  // what the upper halves leave
                        float x, y;
                        unpack2(add2(pack2(__uint_as_float(sr[2 * i]), __uint_as_float(sr[2 * i + 1])),
                                     pack2(-__uint_as_float(sr[2 * i] & 0xffff0000u), -__uint_as_float(sr[2 * i + 1] & 0xffff0000u))), x, y);
                        sr[2 * i] = __float_as_uint(x), sr[2 * i + 1] = __float_as_uint(y);
                    }
                }
                tmem_st_32x32_x16(tmem + C::P_COL + piece * 32 + half * (KEYS / 2) + c + lanes, w);
                }
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&own->p_full));
            if (more) {  // the scores are read and the MMAs that read K are complete: the next K
                store_k(x);
                publish(&bars->k_full);
                fetch_v(x, j + 1);
            }
            if (!LAID) {
                add_block(j);
                if (!ok) break;
            }
            if (more) {
                store_v(x);
                publish(&bars->v_full);
            }
        }
        if (LAID && blocks > 0 && ok) add_block(blocks - 1);
        if (LAID)
            for (int t = tid; t < blocks; t += C::WORKERS) {
                const float* most = p.most + (h * p.kv_blocks + t) * 2;
                most_qk = fmaxf(most_qk, __ldg(most)), most_v = fmaxf(most_v, __ldg(most + 1));
            }
        float l, part[3];
        unpack2(sums[0], l, part[0]), unpack2(sums[1], part[1], part[2]);
        l = (l + part[0]) + (part[1] + part[2]);
        if (C::SPLIT == 2) pair_sum[half * 128 + r] = l;
        const int64_t seen = int64_t(blocks) * BKEYS < p.sk ? int64_t(blocks) * BKEYS : p.sk;  // keys that some row of the tile sees, to a block's end
        // What the cutting may have lost: a value below 2^-109 the bits under 2^-133. Scores are off by less than d (max |q| + max |k|)
        // 2^-133, a result by 2^-133 for V, whose weights sum to at least one, and by keys * max |v| * 2^-133 for the weights.
        const uint32_t mqk = __reduce_max_sync(0xffffffffu, __float_as_uint(most_qk)), mv = __reduce_max_sync(0xffffffffu, __float_as_uint(most_v));
        if (lane == 0) atomicMax(&own->max_qk, mqk), atomicMax(&own->max_v, mv);
        uint32_t together = 0;
        ok = ok && pair_meet(&own->all, together, abort_flag);
        if (C::SPLIT == 2) l += pair_sum[(half ^ 1) * 128 + r];
        auto shared          = [](const uint32_t* word) { return *reinterpret_cast<const volatile uint32_t*>(word); };
        const bool spoiled   = fabsf(p.scale) * p.d * 2.f * LOST_ABS * __uint_as_float(shared(&own->max_qk)) > 0x1p-24f;
        const float small    = 0x1p22f * LOST_ABS * (1.f + float(seen) * __uint_as_float(shared(&own->max_v)));  // 22 bits above the loss
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
        if (__any_sync(0xffffffffu, zero) && lane == 0) own->zeros = 1;
        ok = ok && pair_meet(&own->all, together, abort_flag);
        if (__any_sync(0xffffffffu, shared(&own->zeros) != 0)) {
            bool deep = false;
            for (int64_t i = tid; i < seen * p.d; i += C::WORKERS) {
                const float v = fabsf(__ldg(V + i));
                deep          = deep || (v > 0.f && v < LOST_ABS);
            }
            if (__any_sync(0xffffffffu, deep) && lane == 0) own->deep = 1;
            ok     = ok && pair_meet(&own->all, together, abort_flag);
            finite = finite && !(zero && shared(&own->deep));
        }
        if constexpr (C::SPLIT == 2) {
            pair_max[half * 128 + r] = finite ? 0.f : 1.f;  // (its last reads as a maximum lie before the exchange of sums)
            ok = ok && pair_meet(&own->pair[quarter], meeting, abort_flag);
            finite = pair_max[r] == 0.f && pair_max[128 + r] == 0.f;
        }
        const bool there = ok && q0 + r < p.sq;
        const bool redo  = there && !finite;
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
            if (p.lse && half == 0) p.lse[h * p.sq + q0 + r] = l > 0.f ? m + fmaf(fmaf(m, LOG2E, -from), -0.693147180559945f, logf(l)) : -CUDART_INF_F;
        }
        // every MMA of the tile is complete, so the Q tiles become each warp's row buffer; the two warps of a quarter take its
        // rows in turn
        unsigned again = __ballot_sync(0xffffffffu, redo);
        if (again) {
            float* qs = reinterpret_cast<float*>(smem + group * 3 * C::Q_PIECE) + (warp % C::WORKER_WARPS) * 128;
            while (again) {
                const int i = __ffs(again) - 1;
                again &= again - 1;
                if (C::SPLIT == 2 && (i & 1) != half) continue;
                __syncwarp();
                attn_row::row<float, 128>(qs, p.q, p.k, p.v, p.o, p.lse, h, q0 + quarter * 32 + i, p.sq, p.sk, p.d, p.scale, p.causal);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == C::MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, C::GROUPS * C::COLS);
    }
    if (threadIdx.x == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

template <int DP, bool LAID>
int launch(const CUtensorMap& tmK, const CUtensorMap& tmV, Params& p, int64_t heads, int sm_count, cudaStream_t s) {
    using C   = Cfg<DP, LAID>;
    auto kern = attn_f32_tc_kernel<DP, LAID>;
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
        configured[dev & 63] = true;
    }
    // two tiles on an SM share K and V; while there is an SM for each, each has its own
    p.per_cta = C::GROUPS == 2 && p.q_tiles * heads > sm_count ? 2 : 1;
    p.items   = (p.q_tiles + p.per_cta - 1) / p.per_cta;
    kern<<<unsigned(p.items * heads), C::NUM_THREADS, C::SMEM_BYTES, s>>>(tmK, tmV, p);
    return launch_status();
}
template <bool LAID>
int launch_for(const CUtensorMap& tmK, const CUtensorMap& tmV, Params& p, int64_t heads, int sm_count, cudaStream_t s) {
    if (p.d <= 32) return launch<32, LAID>(tmK, tmV, p, heads, sm_count, s);
    if (p.d <= 64) return launch<64, LAID>(tmK, tmV, p, heads, sm_count, s);
    if (p.d <= 96) return launch<96, LAID>(tmK, tmV, p, heads, sm_count, s);
    return launch<128, LAID>(tmK, tmV, p, heads, sm_count, s);
}

int make_tmap(CUtensorMap* out, const void* base, uint64_t dp, uint64_t sk, uint64_t heads, uint64_t piece) {
    const cuuint64_t dims[4] = {dp, sk, heads, 3}, strides[3] = {dp * 2, sk * dp * 2, piece * 2};
    const cuuint32_t box[4]  = {64, BKEYS, 1, 1};
    return encode_tmap_bf16(out, base, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Whether K and V are cut by a launch of their own: several query tiles read each head's, so many keys that it pays for the launch, and the
// pieces take at most 1 GiB. Measured, cut before / by the workers, us: 8 x 300 x 300 x 128 46 / 41, 128 x 256 x 256 x 32 30 / 25, 64 x 512 x 512 x
// 32 38 / 38, 20 x 400 x 400 x 64 38 / 42, 8 x 600 x 600 x 128 58 / 66, 8 x 300 x 2000 x 64 81 / 132.
bool laid_out_pays(const mimk_attn_desc& d, int64_t q_tiles) {
    const double bytes = 12.0 * double(d.batch_heads) * double(d.seq_k) * double((d.head_dim + 7) & ~int64_t(7));
    return q_tiles >= 2 && d.seq_k >= 384 && bytes <= double(1 << 30) && d.batch_heads * ((d.seq_k + BKEYS - 1) / BKEYS) < (int64_t(1) << 31);
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
    CUtensorMap tmK{}, tmV{};
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    MIMK_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
    // (under stream capture a graph must not hold on to the cached buffer; without memory for it the workers cut, too)
    if (cap == cudaStreamCaptureStatusNone && laid_out_pays(d, p.q_tiles)) {
        const int64_t dp = (d.head_dim + 7) & ~int64_t(7), piece = d.batch_heads * d.seq_k * dp, blocks = (d.seq_k + BKEYS - 1) / BKEYS;
        void* scratch    = nullptr;
        ScratchLease lease;  // of both launches
        if (lease.take(size_t(piece) * 12 + size_t(d.batch_heads * blocks) * 8, &scratch, s) == MIMK_OK) {
            auto* pieces = static_cast<__nv_bfloat16*>(scratch);
            auto* most   = reinterpret_cast<float*>(pieces + 6 * piece);
            p.most = most, p.kv_blocks = blocks;
            MIMK_TRY(make_tmap(&tmK, pieces, uint64_t(dp), uint64_t(d.seq_k), uint64_t(d.batch_heads), uint64_t(piece)));
            MIMK_TRY(make_tmap(&tmV, pieces + 3 * piece, uint64_t(dp), uint64_t(d.seq_k), uint64_t(d.batch_heads), uint64_t(piece)));
            attn_cut_kernel<<<unsigned(d.batch_heads * blocks), 256, 0, s>>>(p.k, p.v, pieces, most, d.seq_k, blocks, p.d, int(dp),
                                                                            p.vec_k && aligned16(d.v), piece);
            MIMK_TRY(launch_status());
            return launch_for<true>(tmK, tmV, p, d.batch_heads, dev->sm_count, s);
        }
        cudaGetLastError();
    }
    return launch_for<false>(tmK, tmV, p, d.batch_heads, dev->sm_count, s);
}

}  // namespace mimk
