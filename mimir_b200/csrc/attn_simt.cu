// CUDA-core attention forward: f32 with few keys and every shape the tensor-core kernels do not take.
//
// The reference runs `softmax (q * transpose_2d k) * v` (MimIR lit/tensor/attn_exec.mim:20-22) as seven
// map_reduce_post ops with the full score matrix in memory. Here one warp owns one query row and streams the
// keys in chunks of 32 with a running maximum and sum, so no score matrix exists.
#include <cmath>

#include "attn_row.cuh"
#include "common.cuh"

namespace mimk {
namespace {

constexpr int WARPS = 4, MAX_D = 256;

template <class T>
__global__ void __launch_bounds__(WARPS * 32) attn_simt_kernel(const T* __restrict__ Q, const T* __restrict__ K,
                                                              const T* __restrict__ V, T* __restrict__ O,
                                                              float* __restrict__ lse, int64_t Sq, int64_t Sk, int D,
                                                              float scale, int causal) {
    __shared__ float qs[WARPS][MAX_D];
    const int warp = threadIdx.x >> 5;
    const int64_t h = blockIdx.y;
    const int64_t i = int64_t(blockIdx.x) * WARPS + warp;
    if (i >= Sq) return;  // whole warp leaves together; no block-wide barrier below
    attn_row::row<T, MAX_D>(qs[warp], Q, K, V, O, lse, h, i, Sq, Sk, D, scale, causal);
}

}  // namespace

// f32 with few keys: whether a warp per row beats the 128-row tiles of attn_f32_tc.cu, which do 64 keys' work for one key and start
// later. Both estimated, in us, from measurements (CUDA-graph replays, warp per row / tiles, where the two are close both are near their estimates):
// one row, one key of 64: 4.0 / 8.5; 16 keys: 8.6 / 8.9; 4000 heads x 8 rows x 8 keys x 64: 84 / 149; 500 x 1 x 32 x 128: 20 / 42;
// 500 x 16 x 16 x 16: 15 / 16; the other way 32 x 1 x 512 x 64: 251 / 41, 1 x 4 x 64 x 64: 35 / 9.
int attn_simt_preferred(const mimk_attn_desc& d, int sm_count) {
    if (d.dtype != MIMK_F32 || d.head_dim > MAX_D || d.batch_heads > 65535) return 0;
    const double dim = double(d.head_dim), keys = double(d.seq_k), rows = double(d.batch_heads) * double(d.seq_q);
    const double latency    = 2.2 + 0.025 * dim + keys * (0.2 + 1.4e-3 * dim);
    const double throughput = 2.0 + rows * (2.6e-4 + 5.5e-6 * dim) + rows * (keys - 1) * (1.4e-5 + 3.9e-6 * dim);
    const double tiles = double((d.seq_q + 127) / 128) * double(d.batch_heads), room = sm_count * (d.head_dim <= 64 ? 2.0 : 1.0);
    const double blocks = double((d.seq_k + 63) / 64);
    const double tiled  = std::ceil(tiles / room) * (6.0 + 0.04 * dim + (blocks - 1) * 4.7);
    return (latency > throughput ? latency : throughput) < tiled;
}

int attn_simt(const mimk_attn_desc& d, cudaStream_t s) {
    if (d.head_dim > MAX_D) return MIMK_E_UNSUPPORTED;
    if (d.batch_heads > 65535) return MIMK_E_UNSUPPORTED;
    dim3 grid((unsigned)((d.seq_q + WARPS - 1) / WARPS), (unsigned)d.batch_heads);
    if (d.dtype == MIMK_F32)
        attn_simt_kernel<float><<<grid, WARPS * 32, 0, s>>>(static_cast<const float*>(d.q), static_cast<const float*>(d.k),
                                                           static_cast<const float*>(d.v), static_cast<float*>(d.o), d.lse,
                                                           d.seq_q, d.seq_k, int(d.head_dim), d.scale, d.causal);
    else if (d.dtype == MIMK_BF16)
        attn_simt_kernel<__nv_bfloat16><<<grid, WARPS * 32, 0, s>>>(
            static_cast<const __nv_bfloat16*>(d.q), static_cast<const __nv_bfloat16*>(d.k),
            static_cast<const __nv_bfloat16*>(d.v), static_cast<__nv_bfloat16*>(d.o), d.lse, d.seq_q, d.seq_k,
            int(d.head_dim), d.scale, d.causal);
    else
        return MIMK_E_DTYPE;
    return launch_status();
}

}  // namespace mimk
