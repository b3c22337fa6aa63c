// CUDA-core attention forward: f32 tensors and every shape the tensor-core kernel does not take.
//
// The reference runs `softmax (q * transpose_2d k) * v` (MimIR lit/tensor/attn_exec.mim:20-22) as seven
// map_reduce_post ops with the full score matrix in memory. Here one warp owns one query row and streams the
// keys in chunks of 32 with a running maximum and sum, so no score matrix exists.
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
