// bf16 contraction on the tensor cores (tcgen05) for results with too few tiles for the chip: a few rows against a large weight
// matrix (one step of generation), narrow results over a long contracted extent, small layers. Same operator as gemm_tc.cu
// (`dot_product_impl`, MimIR src/mim/plug/tensor/tensor.mim:1367-1411, with the `post` slot of
// src/mim/plug/tensor/phase/fuse.cpp:408-534).
//
// gemm_tc.cu gives each 128 x 256 tile to one SM, so 16 rows x 14336 columns keep 56 of 148 SMs busy. Here the tiles are 128 x 64
// or 128 x 128 (gated: half as many columns of each of the two operands), the k-blocks of a tile are dealt out to a cluster of
// up to eight CTAs, and two CTAs share an SM. What bounds such a product is the bytes of the right operand, so the shared memory
// goes to its stages: of the left operand only the rows that exist are staged (the MMA reads on into the next tiles for the
// others; a row of the result depends on its own row only, and those are not stored).
//   warp 0      TMA producer    warp 1   MMA issuer, one accumulator
//   warps 2..5  accumulator -> f32 partial tile in shared memory, over the stages
//   all         after a cluster barrier: the partial tiles are added in rank order through distributed shared memory, each CTA
//               a share of the cells, `post`, and stored with neighbouring lanes on neighbouring columns (any pitch and alignment,
//               one destination or each of a gather's)
#include "common.cuh"
#include "sm100.cuh"

namespace mimk {

using namespace sm100;

namespace {

constexpr int BM = 128, BK = 64, MAX_STAGES = 8, NUM_THREADS = 192;
constexpr int STAGE_BUDGET = 100 * 1024;  // two CTAs per SM

struct Bars {
    uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Bars) <= 256, "barrier block too large");

struct Params {
    int64_t M, N, K, stride_c, ldc, col_off;
    int64_t tiles_m, tiles_n;
    int a_batched, b_batched, a_rows, stages, split, vec_c;
    int a_panel_kb, a_panel_rows;  // A as panels one below the other: k-blocks of a panel, rows from one to the next
    int n_dst;
    void* dst[MIMK_MAX_GATHER];
    const float* post_row;
    const void* post_full;
    int post;
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

template <int BN, bool B_MN, bool GATED, class TOut>
__global__ void __launch_bounds__(NUM_THREADS, 2)
gemm_tc_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmB2, const Params p) {
    constexpr int BNO = GATED ? BN / 2 : BN;  // result columns per tile
    constexpr int B_BYTES = BN * BK * 2, PITCH = BN + 4;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    Bars* bars              = reinterpret_cast<Bars*>(smem_raw);  // in front of the tiles
    const uint32_t tiles_at = ((raw_addr + 1023u) & ~1023u) + 1024;
    const uint32_t a_bytes = uint32_t(p.a_rows) * BK * 2, b_at = tiles_at + p.stages * a_bytes;
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int rank     = int(blockIdx.x % unsigned(p.split));  // a cluster is `split` consecutive CTAs
    const int64_t item = blockIdx.x / unsigned(p.split), tiles = p.tiles_m * p.tiles_n, bz = item / tiles;
    const int64_t tn = (item - bz * tiles) / p.tiles_m, tm = (item - bz * tiles) % p.tiles_m;  // the tiles of one column of B together
    const int64_t m0 = tm * BM, n0 = tn * BNO;
    const int all_kb = int((p.K + BK - 1) / BK), per = (all_kb + p.split - 1) / p.split;
    const int kb0 = rank * per < all_kb ? rank * per : all_kb, kb1 = kb0 + per < all_kb ? kb0 + per : all_kb;

    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        mbar_init(smem_u32(&bars->acc_full), 1);
        bars->abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (GATED) tma_prefetch_desc(&tmB2);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&bars->tmem_base), BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            const int za = p.a_batched ? int(bz) : 0, zb = p.b_batched ? int(bz) : 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(smem_u32(&bars->empty[stage]), phase ^ 1u, abort_flag)) break;
                const uint32_t full = smem_u32(&bars->full[stage]), sa = tiles_at + stage * a_bytes, sb = b_at + stage * B_BYTES;
                mbar_expect_tx(full, a_bytes + B_BYTES);
                const int panel = kb / p.a_panel_kb;
                tma_load_3d(sa, &tmA, (kb - panel * p.a_panel_kb) * BK, int(m0) + panel * p.a_panel_rows, za, full);
                if (!B_MN) {
                    tma_load_3d(sb, &tmB, kb * BK, int(n0), zb, full);
                    if (GATED) tma_load_3d(sb + B_BYTES / 2, &tmB2, kb * BK, int(n0), zb, full);
                } else {
#pragma unroll
                    for (int j = 0; j < BNO / 64; ++j) {
                        tma_load_3d(sb + j * (BK * 128), &tmB, int(n0) + j * 64, kb * BK, zb, full);
                        if (GATED) tma_load_3d(sb + B_BYTES / 2 + j * (BK * 128), &tmB2, int(n0) + j * 64, kb * BK, zb, full);
                    }
                }
                if (++stage == uint32_t(p.stages)) stage = 0, phase ^= 1u;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16_f32(BM, BN, 0, B_MN ? 1 : 0);
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!(ok = mbar_wait(smem_u32(&bars->full[stage]), phase, abort_flag))) break;
                tc_fence_after();
                const uint32_t sa = tiles_at + stage * a_bytes, sb = b_at + stage * B_BYTES;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    mma_f16_ss(tmem, smem_desc_sw128(sa + k * 32, 16, 1024),
                               smem_desc_sw128(sb + (B_MN ? k * 2048 : k * 32), B_MN ? BK * 128 : 16, 1024), idesc,
                               (kb > kb0 || k > 0) ? 1u : 0u);
                mma_commit(smem_u32(&bars->empty[stage]));
                if (++stage == uint32_t(p.stages)) stage = 0, phase ^= 1u;
            }
            if (ok && kb1 > kb0) mma_commit(smem_u32(&bars->acc_full));
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3;
        const bool any    = kb1 > kb0;  // a rank without k-blocks adds zeros
        const bool ok     = !any || __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->acc_full), 0, abort_flag));
        if (ok && m0 + quarter * 32 < p.M) {
            tc_fence_after();
            const uint32_t row_at = tiles_at + uint32_t(quarter * 32 + lane) * PITCH * 4;
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                uint32_t r[32];
                if (any) {
                    tmem_ld_32x32(tmem + c + (uint32_t(quarter * 32) << 16), r);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = 0;
                }
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_at + (c + i) * 4), "r"(r[i]), "r"(r[i + 1]),
                                 "r"(r[i + 2]), "r"(r[i + 3])
                                 : "memory");
            }
            tc_fence_before();
        }
    }
    __syncthreads();
    if (p.split > 1) cluster_sync();

    const int rows = int(p.M - m0 < BM ? p.M - m0 : BM);
    const TOut* post_full = p.post_full ? static_cast<const TOut*>(p.post_full) + bz * p.stride_c : nullptr;
    for (int i = rank * NUM_THREADS + tid; i < rows * (BNO / 4); i += p.split * NUM_THREADS) {
        const int r = i / (BNO / 4), c = (i % (BNO / 4)) * 4;
        const int64_t row = m0 + r, col = n0 + c;
        if (col >= p.N) continue;
        const uint32_t a = tiles_at + uint32_t(r * PITCH + c) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < p.split; ++s) {
            const float4 q = ld_cluster4(a, uint32_t(s));
            v[0] += q.x, v[1] += q.y, v[2] += q.z, v[3] += q.w;
            if (GATED) {
                const float4 w = ld_cluster4(a + BNO * 4, uint32_t(s));
                u[0] += w.x, u[1] += w.y, u[2] += w.z, u[3] += w.w;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (col + e >= p.N) break;
            if (GATED) v[e] = (v[e] / (1.f + __expf(-v[e]))) * u[e];
            const float rowv = p.post_row ? __ldg(p.post_row + col + e) : 0.f;
            const float full = post_full ? float(post_full[row * p.N + col + e]) : 0.f;
            v[e]             = apply_post(p.post, v[e], rowv, full);
        }
        for (int t = 0; t < p.n_dst; ++t) {
            TOut* dst = static_cast<TOut*>(p.dst[t]) + bz * p.stride_c + row * p.ldc + p.col_off + col;
            if (p.vec_c) {  // four results are one aligned store, and N is a multiple of 4
                if (sizeof(TOut) == 4)
                    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                else
                    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (col + e < p.N) dst[e] = TOut(v[e]);
            }
        }
    }
    if (p.split > 1) cluster_sync();  // no CTA of the cluster exits while another may read its partial tile

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, BN);
    }
    if (tid == 0 && *abort_flag) *p.status = MIMK_E_DEVICE_WAIT;
}

template <int BN, bool B_MN, bool GATED, class TOut>
int launch(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tB2, const Params& p, int64_t ctas, cudaStream_t s) {
    auto kern = gemm_tc_split_kernel<BN, B_MN, GATED, TOut>;
    constexpr int PART_BYTES = BM * (BN + 4) * 4, MOST = 2048 + STAGE_BUDGET;
    static_assert(PART_BYTES <= STAGE_BUDGET, "the partial tile lies over the stages");
    static bool configured[64] = {};  // per template instance and device: the attribute is a per-device setting
    int dev = 0;
    MIMK_CUDA_TRY(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
        MIMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST));
        configured[dev & 63] = true;
    }
    // (the MMA reads 128 rows from the last left tile on, which stays inside the right operand's stages)
    const int stage_bytes = p.stages * (p.a_rows * BK * 2 + BN * BK * 2);
    const int need        = 2048 + (stage_bytes > PART_BYTES ? stage_bytes : PART_BYTES);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ctas)), cfg.blockDim = dim3(NUM_THREADS), cfg.dynamicSmemBytes = size_t(need), cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(p.split), attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    return note_cuda_error(cudaLaunchKernelEx(&cfg, kern, tA, tB, tB2, p));
}

template <bool B_MN, class TOut>
int pick(int bn, bool gated, const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tB2, const Params& p, int64_t ctas, cudaStream_t s) {
    if constexpr (sizeof(TOut) == 2) {
        if (gated) return launch<128, B_MN, true, TOut>(tA, tB, tB2, p, ctas, s);
    }
    if (gated) return MIMK_E_DTYPE;
    return bn == 128 ? launch<128, B_MN, false, TOut>(tA, tB, tB2, p, ctas, s) : launch<64, B_MN, false, TOut>(tA, tB, tB2, p, ctas, s);
}

}  // namespace

// Few tiles of the one-CTA kernel's 128 x 256 (gated 128 x 128), and K long enough to deal out. The one-CTA kernel takes about
// 0.3 us per k-block of its single round; this one starts and merges 4 us slower and works on several k-blocks of a tile at once:
// 16 x 14336 x 4096 (56 tiles): 32.9 -> 24.3 us; 256 x 4096 x 4096 (32): 23.6 -> 17.7; 5000 x 64 x 8192 (40): 40.6 -> 17.7;
// 300 x 200 x 16000 (3): 74.6 -> 16.7. Beyond the rule: 128 x 8192 x 1024: 10.0 against 12.1; 700 x 3008 x 8192 (72): 43.5 / 42.4;
// 2048 x 1024 x 4096 (64): 24.1 / 27.1; 256^3: 6.3 / 7.0. With few rows the bytes of B decide, and more SMs fetch them faster.
// A shorter K pays for the exchange with fewer tiles only: 16 x 14336 x 1024 (56): 10.9 -> 9.3 us; 256 x 1024 x 1024 (8): 11.2 -> 8.3;
// the gated block 2 x 1024 x 1280 x 960: 48 -> 21, 300 x 1024 x 1024 x 1024 (24, then 12): 48 -> 27; not 1000 x 1024 x 768 (32):
// 9.8 / 14.5, nor the second stage of 700 x 1280 x 1280 (30).
int gemm_tc_split_preferred(const mimk_gemm_desc& d, int gated) {
    const int64_t width = gated ? 128 : 256, tiles = ((d.m + BM - 1) / BM) * ((d.n + width - 1) / width) * d.batch;
    if (d.k >= 24 * BK) return tiles <= (d.m <= BM ? 74 : 40);
    return d.m <= 32 ? d.k >= 8 * BK && tiles <= 74 : d.k >= 16 * BK && tiles <= (gated ? 24 : 16);
}

int gemm_tc_split(const mimk_gemm_desc& d, cudaStream_t s, int gated, const void* b2, const mimk_gather_dst* gather, int64_t a_panels,
                  const GemmPitch* pitch) {
    if (a_panels < 1 || (a_panels > 1 && (d.batch != 1 || pitch || d.k % a_panels != 0 || (d.k / a_panels) % BK != 0)) || (gather && d.batch != 1))
        return MIMK_E_UNSUPPORTED;
    int st          = MIMK_OK;
    DeviceInfo* dev = device_info(&st);
    if (!dev) return st;
    const bool b_mn = d.b_layout == MIMK_B_KN;
    const bool a_b = d.batch > 1 && d.stride_a != 0, b_b = d.batch > 1 && d.stride_b != 0;
    const uint64_t na = a_b ? uint64_t(d.batch) : 1, nb = b_b ? uint64_t(d.batch) : 1;
    const uint64_t kp = uint64_t(d.k / a_panels), lda = pitch ? uint64_t(pitch->a) : kp, ldb = pitch ? uint64_t(pitch->b) : uint64_t(b_mn ? d.n : d.k);
    // (the outermost stride of a one-entry operand is never used; it only has to be a legal value)
    const uint64_t sa = a_b ? uint64_t(d.stride_a) * 2 : lda * 2, sb = b_b ? uint64_t(d.stride_b) * 2 : ldb * 2;
    const int64_t tiles_m = (d.m + BM - 1) / BM, kb = (d.k + BK - 1) / BK;
    // 128 columns, or 64 where the result is narrow or eight CTAs for each tile would not fill the chip
    const int bn  = gated || (d.n > 64 && tiles_m * ((d.n + 127) / 128) * d.batch * 8 >= dev->sm_count) ? 128 : 64;
    const int bno = gated ? 64 : bn;
    Params p{};
    p.M = d.m, p.N = d.n, p.K = d.k, p.stride_c = d.batch > 1 ? d.stride_c : 0;
    p.tiles_m = tiles_m, p.tiles_n = (d.n + bno - 1) / bno;
    p.a_batched = a_b, p.b_batched = b_b;
    p.a_rows = int(d.m < BM ? (d.m + 7) & ~int64_t(7) : BM);
    p.stages = STAGE_BUDGET / (p.a_rows * BK * 2 + bn * BK * 2);
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    // the whole chip at two CTAs an SM, but at least four k-blocks for each CTA
    const int64_t items = p.tiles_m * p.tiles_n * d.batch;
    p.split = 1;
    while (p.split < 8 && items * p.split * 2 <= 2 * dev->sm_count && kb >= p.split * 8) p.split *= 2;
    p.a_panel_kb = a_panels > 1 ? int(kp / BK) : int(kb), p.a_panel_rows = a_panels > 1 ? int(d.m) : 0;
    p.n_dst = 1, p.dst[0] = d.c, p.ldc = d.n;
    if (gather) {
        p.n_dst = gather->n_dst, p.ldc = gather->ldc, p.col_off = gather->col_off;
        for (int t = 0; t < gather->n_dst; ++t) p.dst[t] = gather->dst[t];
    }
    p.post_row = static_cast<const float*>(d.post_row), p.post_full = d.post_full, p.post = d.post;
    p.vec_c = d.n % 4 == 0 && p.ldc % 4 == 0 && p.col_off % 4 == 0 && p.stride_c % 4 == 0;
    for (int t = 0; t < p.n_dst; ++t) p.vec_c = p.vec_c && aligned16(p.dst[t]);
    p.status = dev->status_dev;
    const void* B2 = b2 ? b2 : d.b;
    CUtensorMap tA, tB, tB2;
    MIMK_TRY(make_tmap_bf16_3d(&tA, d.a, kp, uint64_t(d.m) * uint64_t(a_panels), na, lda * 2, sa, BK, uint32_t(p.a_rows)));
    if (b_mn) {
        MIMK_TRY(make_tmap_bf16_3d(&tB, d.b, uint64_t(d.n), uint64_t(d.k), nb, ldb * 2, sb, 64, BK));
        MIMK_TRY(make_tmap_bf16_3d(&tB2, B2, uint64_t(d.n), uint64_t(d.k), nb, ldb * 2, sb, 64, BK));
    } else {
        MIMK_TRY(make_tmap_bf16_3d(&tB, d.b, uint64_t(d.k), uint64_t(d.n), nb, ldb * 2, sb, BK, uint32_t(bno)));
        MIMK_TRY(make_tmap_bf16_3d(&tB2, B2, uint64_t(d.k), uint64_t(d.n), nb, ldb * 2, sb, BK, uint32_t(bno)));
    }
    const int64_t ctas = items * p.split;
    if (d.out_dtype == MIMK_BF16)
        return b_mn ? pick<true, __nv_bfloat16>(bn, gated, tA, tB, tB2, p, ctas, s) : pick<false, __nv_bfloat16>(bn, gated, tA, tB, tB2, p, ctas, s);
    return b_mn ? pick<true, float>(bn, gated, tA, tB, tB2, p, ctas, s) : pick<false, float>(bn, gated, tA, tB, tB2, p, ctas, s);
}

}  // namespace mimk
