// Router tail: fp32 logits -> top-k expert ids (rank order) + normalised weights.
// A warp per token row up to 256 experts and top_k 32; a CTA per token row, one thread per expert, above (n_experts <= 1024,
// top_k <= 64).
// Semantics: src/kernels/exl3/q3rc_router_tail.metal:12-40 (sqrt(softplus)), src/arch/mimo_v2/kernels/mimo_glue_top8.metal
// and src/arch/glm5_next/kernels/glm5n_glue_top8.metal (sigmoid): key = score + bias, rank = number of experts that
// precede (key descending, ties to the lower index, NaN last), ids[rank] = expert, weights from the unbiased score,
// sum folded in rank order (total = w[j] + total), / (sum + 1e-20), x scale.
#include "common.cuh"
#include "kernels.h"
#include "logits_body.cuh"
#include "router_body.cuh"

namespace mlxs {

__global__ void router_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int E, int K,
                              int scoring, int norm, float scale, int32_t* __restrict__ ids,
                              float* __restrict__ weights) {
    extern __shared__ float sm[];
    route_row(logits, bias, E, K, scoring, norm, scale, ids, weights, (int)blockIdx.x, sm, (int)blockDim.x);
}

// a warp per token: 8 tokens per CTA and no barrier (16,384 tokens of 256 experts: 104 -> 37 us against a CTA per token)
__global__ void __launch_bounds__(256) router_warp_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int T,
                                                          int E, int K, int scoring, int norm, float scale,
                                                          int32_t* __restrict__ ids, float* __restrict__ weights) {
    const int t = (int)(blockIdx.x * 8 + (threadIdx.x >> 5));
    if (t < T) route_row_warp<false>(logits + (size_t)t * E, bias, E, K, scoring, norm, scale, ids + (size_t)t * K, weights + (size_t)t * K);
}

// Router logits: the shared device code of logits_body.cuh, two expert rows per CTA of 8 warps, or 8 experts x 8 tokens
constexpr int RL_WARPS = 8;
// H 5120, 256 experts: 1 token 8 us row by row against 10 in tiles, 4 tokens 10 either way, 8 tokens 12 against 10, 16 tokens 20
// against 10, 64 tokens 59 against 12; 64 experts, 8192 tokens 11.6 ms against 0.21
constexpr uint32_t LOGITS_TILE_FROM = 4;
__global__ void __launch_bounds__(RL_WARPS * 32) router_logits_kernel(const __nv_bfloat16* __restrict__ x,
                                                                     const __nv_bfloat16* __restrict__ w, uint32_t T,
                                                                     uint32_t E, uint32_t H, float* __restrict__ logits) {
    extern __shared__ __align__(16) uint8_t rl_sm[];
    logits_rows(x, w, T, E, H, logits, rl_sm, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(256, 2) router_logits_tile_kernel(const __nv_bfloat16* __restrict__ x,
                                                                    const __nv_bfloat16* __restrict__ w, uint32_t T,
                                                                    uint32_t E, uint32_t H, float* __restrict__ logits) {
    logits_tile(x, w, T, E, H, logits, blockIdx.x * LT_CTA_E, blockIdx.y * LT_T);
}

cudaError_t launch_router_logits(const __nv_bfloat16* x, const __nv_bfloat16* w, uint32_t T, uint32_t E, uint32_t H,
                                 float* logits, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    if (H % 8) return cudaErrorInvalidValue;
    if (T > LOGITS_TILE_FROM) {
        router_logits_tile_kernel<<<dim3((E + LT_CTA_E - 1) / LT_CTA_E, (T + LT_T - 1) / LT_T), 256, 0, st>>>(x, w, T, E, H, logits);
        return cudaGetLastError();
    }
    const size_t smem = logits_smem_bytes(H, RL_WARPS);
    cudaError_t err = cudaFuncSetAttribute(router_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    const uint32_t slots = RL_WARPS / LG_PARTS;
    router_logits_kernel<<<(E + slots - 1) / slots, RL_WARPS * 32, smem, st>>>(x, w, T, E, H, logits);
    return cudaGetLastError();
}

cudaError_t launch_router(const float* logits, const float* bias, int T, int E, int K, int scoring, int norm,
                          float scale, int32_t* ids, float* weights, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    if (route_by_warp(E, K)) {
        router_warp_kernel<<<(T + 7) / 8, 256, 0, st>>>(logits, bias, T, E, K, scoring, norm, scale, ids, weights);
        return cudaGetLastError();
    }
    int threads = ((E > K ? E : K) + 31) / 32 * 32;
    size_t smem = router_smem_floats(E, K, threads) * sizeof(float);
    router_kernel<<<T, threads, smem, st>>>(logits, bias, E, K, scoring, norm, scale, ids, weights);
    return cudaGetLastError();
}

}  // namespace mlxs
