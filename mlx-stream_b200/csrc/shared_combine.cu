// The bf16 dense shared expert at decode widths (larger batches: dense_gemm.cu), and the weighted combine.
//
// Shared expert (src/arch/deepseek_v41/graph.zig:2162-2172): h = silu(min(w1 x, lim)) * clip(w3 x, +-lim) in f32,
// rounded to the activation dtype, then w2 h.  Memory-bound on the 3 H I bf16 weights: a CTA owns 16 output features,
// its 8 warps split the reduction dimension, weights stream as 128-bit loads straight into mma A fragments (the k
// order inside a 32-wide chunk is permuted identically for both operands, which a dot product does not see).
//
// Combine (src/arch/deepseek_v41/graph.zig:2182-2184; src/arch/mimo_v2/kernels/mimo_moe_combine.metal;
// src/arch/glm5_next/kernels/glm5n_moe_combine.metal): fixed fold order k = 0..top_k-1, one bf16 rounding.
#include "common.cuh"
#include "kernels.h"

namespace mlxs {

// warps of a CTA (they split the reduction dimension).  The down kernel has 320 row tiles for 148 SMs: with 4 warps
// and about 100 registers every CTA is resident at once (2-3 per SM) instead of running in two waves.
constexpr int sh_warps(int mode) { return mode == 0 ? 8 : 4; }
constexpr int SH_AHEAD = 2;  // weight chunks in flight per warp

// MODE 0: gate/up + activation -> h bf16 [T, N]; 1: down -> out f32 [T, N].  NT = token tiles of 8 per pass: a call of few
// tokens takes the form that holds registers and reduction space for its own tiles only, so that its CTAs fit beside the
// routed kernels' (gate/up at one token 35 -> 27 us; four tiles for 17 .. 32 tokens: the layer of 20 NVFP4 tokens 528 -> 511,
// four EXL3 layers of 32 tokens 1813 -> 1787).
template <int MODE, int NT>
__global__ void __launch_bounds__(sh_warps(MODE) * 32) shared_kernel(const __nv_bfloat16* __restrict__ x, uint32_t T,
                                                               uint32_t Kdim, uint32_t N,
                                                               const __nv_bfloat16* __restrict__ wa,
                                                               const __nv_bfloat16* __restrict__ wb, float limit,
                                                               __nv_bfloat16* __restrict__ h_out,
                                                               float* __restrict__ f_out) {
    extern __shared__ float red[];  // [SH_WARPS][NW][NT tiles][32 lanes][4]
    constexpr int SH_WARPS = sh_warps(MODE);
    constexpr int NW = MODE == 0 ? 2 : 1;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, c = lane & 3u;
    const uint32_t row0 = blockIdx.x * 16;
    for (uint32_t t0 = 0; t0 < T; t0 += NT * 8) {
        const uint32_t nt_n = min((uint32_t)(NT * 8), T - t0);
        const uint32_t ntiles = (nt_n + 7) / 8;
        float acc[NW][NT][4];
#pragma unroll
        for (int w = 0; w < NW; ++w)
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[w][i][q] = 0.f;
        // A warp walks its share of the reduction dimension 32 inputs at a time.  The weights come straight from HBM and
        // are used once, so the loads of the next SH_AHEAD chunks are always in flight (a register ring, statically
        // indexed) while the current chunk's mma run: with one chunk in flight the kernel was bound by the load latency.
        const uint32_t nchunk = Kdim / 32;
        uint4 ring[SH_AHEAD][2 * NW];
        auto load_chunk = [&](uint4 (&dst)[2 * NW], uint32_t kc) {
            if (kc < nchunk) {
                const size_t ko = (size_t)kc * 32 + c * 8;
                dst[0] = __ldcs(reinterpret_cast<const uint4*>(wa + (size_t)(row0 + g) * Kdim + ko));
                dst[1] = __ldcs(reinterpret_cast<const uint4*>(wa + (size_t)(row0 + g + 8) * Kdim + ko));
                if (NW == 2) {
                    dst[2 * NW - 2] = __ldcs(reinterpret_cast<const uint4*>(wb + (size_t)(row0 + g) * Kdim + ko));
                    dst[2 * NW - 1] = __ldcs(reinterpret_cast<const uint4*>(wb + (size_t)(row0 + g + 8) * Kdim + ko));
                }
            }
        };
        // the rows of a chunk's token tiles come from L2: they too are loaded one chunk ahead, all eight at once
        // (predicated, no branch between them)
        static_assert(SH_AHEAD == 2, "the row buffers alternate with the chunk's place in the weight ring");
        uint4 xr[2][NT];
        auto load_rows = [&](uint4 (&dst)[NT], uint32_t kc) {
            const size_t ko = (size_t)kc * 32 + c * 8;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const uint32_t tok = t0 + i * 8 + g;
                dst[i] = make_uint4(0, 0, 0, 0);
                if (kc < nchunk && i < (int)ntiles && tok < T) dst[i] = *reinterpret_cast<const uint4*>(x + (size_t)tok * Kdim + ko);
            }
        };
#pragma unroll
        for (int r = 0; r < SH_AHEAD; ++r) load_chunk(ring[r], warp + r * SH_WARPS);
        load_rows(xr[0], warp);
        for (uint32_t kc0 = warp; kc0 < nchunk; kc0 += SH_AHEAD * SH_WARPS) {
#pragma unroll
            for (int r = 0; r < SH_AHEAD; ++r) {
                const uint32_t kc = kc0 + r * SH_WARPS;
                if (kc < nchunk) {
                    uint4 a[2 * NW];
#pragma unroll
                    for (int q = 0; q < 2 * NW; ++q) a[q] = ring[r][q];
                    load_chunk(ring[r], kc + SH_AHEAD * SH_WARPS);
                    load_rows(xr[r ^ 1], kc + SH_WARPS);
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        if (i < (int)ntiles) {
#pragma unroll
                            for (int w = 0; w < NW; ++w) {
                                const uint32_t a1[4] = {a[2 * w].x, a[2 * w + 1].x, a[2 * w].y, a[2 * w + 1].y};
                                const uint32_t a2[4] = {a[2 * w].z, a[2 * w + 1].z, a[2 * w].w, a[2 * w + 1].w};
                                mma_bf16(acc[w][i], a1, xr[r][i].x, xr[r][i].y);
                                mma_bf16(acc[w][i], a2, xr[r][i].z, xr[r][i].w);
                            }
                        }
                    }
                }
            }
        }
        // cross-warp reduction of the split reduction dimension
#pragma unroll
        for (int w = 0; w < NW; ++w)
#pragma unroll
            for (int i = 0; i < NT; ++i)
                if (i < (int)ntiles)
                    *reinterpret_cast<float4*>(red + ((((size_t)warp * NW + w) * NT + i) * 32 + lane) * 4) =
                        make_float4(acc[w][i][0], acc[w][i][1], acc[w][i][2], acc[w][i][3]);
        __syncthreads();
        for (uint32_t idx = threadIdx.x; idx < ntiles * 128; idx += SH_WARPS * 32) {
            const uint32_t i = idx / 128, ln = (idx / 4) % 32, q = idx % 4;
            float s[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                float v = 0.f;
                for (int ww = 0; ww < SH_WARPS; ++ww) v += red[((((size_t)ww * NW + w) * NT + i) * 32 + ln) * 4 + q];
                s[w] = v;
            }
            const uint32_t row = row0 + (ln >> 2) + ((q & 2) ? 8 : 0);
            const uint32_t tok = t0 + i * 8 + 2 * (ln & 3) + (q & 1);
            if (tok < T) {
                if (MODE == 0) {
                    float gate = s[0], up = s[NW - 1];
                    if (limit > 0.f) {
                        gate = (gate != gate) ? gate : (gate < limit ? gate : limit);
                        up = (up != up) ? up : (up > limit ? limit : (up < -limit ? -limit : up));
                    }
                    const float yv = 1.0f / (1.0f + expf(fabsf(gate)));
                    const float sg = gate < 0.f ? yv : 1.0f - yv;
                    h_out[(size_t)tok * N + row] = __float2bfloat16_rn((gate * sg) * up);
                } else {
                    f_out[(size_t)tok * N + row] = s[0];
                }
            }
        }
        __syncthreads();
    }
}

template <int NT>
static cudaError_t shared_launch(const __nv_bfloat16* x, const __nv_bfloat16* w1, const __nv_bfloat16* w3, const __nv_bfloat16* w2, uint32_t T,
                                 uint32_t H, uint32_t I, float limit, __nv_bfloat16* h_ws, float* out, cudaStream_t st) {
    const size_t smem0 = (size_t)sh_warps(0) * 2 * NT * 32 * 4 * sizeof(float), smem1 = (size_t)sh_warps(1) * NT * 32 * 4 * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(shared_kernel<0, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem0);
    if (e != cudaSuccess) return e;
    // The routed kernels beside it take all of an SM's shared memory: an SM that had to change its split would drain first.
    // (Not from 17 tokens on: the rows then miss the L1, 27 -> 41 us at 64 tokens, four layers of 32 tokens 1787 -> 1804.)
    if (NT < 4 && (e = cudaFuncSetAttribute(shared_kernel<0, NT>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) != cudaSuccess) return e;
    if (NT < 4 && (e = cudaFuncSetAttribute(shared_kernel<1, NT>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)) != cudaSuccess) return e;
    shared_kernel<0, NT><<<I / 16, sh_warps(0) * 32, smem0, st>>>(x, T, H, I, w1, w3, limit, h_ws, nullptr);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    shared_kernel<1, NT><<<H / 16, sh_warps(1) * 32, smem1, st>>>(h_ws, T, I, H, w2, nullptr, 0.f, nullptr, out);
    return cudaGetLastError();
}

cudaError_t launch_shared_expert(const __nv_bfloat16* x, const __nv_bfloat16* w1, const __nv_bfloat16* w3,
                                 const __nv_bfloat16* w2, uint32_t T, uint32_t H, uint32_t I, float limit,
                                 __nv_bfloat16* h_ws, float* out, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    if (T <= 8) return shared_launch<1>(x, w1, w3, w2, T, H, I, limit, h_ws, out, st);
    if (T <= 16) return shared_launch<2>(x, w1, w3, w2, T, H, I, limit, h_ws, out, st);
    if (T <= 32) return shared_launch<4>(x, w1, w3, w2, T, H, I, limit, h_ws, out, st);
    return shared_launch<8>(x, w1, w3, w2, T, H, I, limit, h_ws, out, st);
}

// A thread owns 8 columns of one token and has eight rows' loads in flight (16 or 32 bytes each): the kernel is a read of
// the rows, and with one load of 8 or 16 bytes per step of the fold it ran at half the memory's rate (131,072 bf16 rows of
// 4096: 271 us).  The fold goes in k order whatever the loads do.
template <bool BF16>
__global__ void __launch_bounds__(128) combine_kernel(const void* __restrict__ ro, const float* __restrict__ weights,
                                                      const float* __restrict__ shared, uint32_t nblk, uint32_t K, uint32_t H, int chain,
                                                      __nv_bfloat16* __restrict__ y) {
    const uint32_t t = blockIdx.x / nblk, col = (blockIdx.x % nblk) * 1024 + threadIdx.x * 8;
    grid_dep_wait();
    if (col >= H) return;
    constexpr int V = BF16 ? 1 : 2;   // 16-byte vectors of a row
    float acc[8];
    for (uint32_t k0 = 0; k0 < K; k0 += 8) {
        uint4 r[8][V];
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < K) {
                const size_t row = (size_t)t * K + k0 + j;
                w[j] = weights[row];
                const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(ro) + (row * H + col) * (BF16 ? 2 : 4));
#pragma unroll
                for (int v = 0; v < V; ++v) r[j][v] = __ldcs(p + v);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < K) {
                float f[8];
                if (BF16) {
                    const uint32_t u[4] = {r[j][0].x, r[j][0].y, r[j][0].z, r[j][0].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) { f[2 * q] = __uint_as_float(u[q] << 16); f[2 * q + 1] = __uint_as_float(u[q] & 0xFFFF0000u); }
                } else {
                    const uint32_t u[8] = {r[j][0].x, r[j][0].y, r[j][0].z, r[j][0].w, r[j][V - 1].x, r[j][V - 1].y, r[j][V - 1].z, r[j][V - 1].w};
#pragma unroll
                    for (int q = 0; q < 8; ++q) f[q] = __uint_as_float(u[q]);
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float p = __fadd_rn(__fmul_rn(f[q], w[j]), 0.0f);  // each product rounded, no contraction
                    acc[q] = k0 + j == 0 ? p : __fadd_rn(p, acc[q]);
                }
            }
        }
    }
    float sh[8];
    if (shared) {
        const float4* s4 = reinterpret_cast<const float4*>(shared + (size_t)t * H + col);
        const float4 a = s4[0], b = s4[1];
        sh[0] = a.x; sh[1] = a.y; sh[2] = a.z; sh[3] = a.w; sh[4] = b.x; sh[5] = b.y; sh[6] = b.z; sh[7] = b.w;
    }
    uint32_t o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float a = acc[2 * q + i];
            if (chain) a = bf16_round_f(a);
            if (shared) a = __fadd_rn(a, chain ? bf16_round_f(sh[2 * q + i]) : sh[2 * q + i]);
            v[i] = a;
        }
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[0], v[1]);
        o[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(y + (size_t)t * H + col) = make_uint4(o[0], o[1], o[2], o[3]);
}

cudaError_t launch_combine(const void* ro, int ro_bf16, const float* weights, const float* shared, uint32_t T,
                           uint32_t K, uint32_t H, int chain, __nv_bfloat16* y, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    const uint32_t nblk = (H + 1023) / 1024;
    return launch_dependent(true, ro_bf16 ? combine_kernel<true> : combine_kernel<false>, nblk * T, 128, 0, st, ro, weights, shared, nblk, K, H, chain, y);
}

}  // namespace mlxs
