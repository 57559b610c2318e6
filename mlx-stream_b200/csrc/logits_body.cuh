// The router's logits (device code shared by the logits kernels and the fused front kernel):
// logits[t, e] = sum_k f32(x[t, k]) * f32(W[e, k]), f32 accumulate (src/arch/deepseek_v41/graph.zig:2033; kernels
// q3rc_gate_part.metal, mimo_glue_router_rows.metal).
// Four warps share one expert row: warp s sums the s-th quarter of the inputs (a lane adds its strided products in k
// order, then an xor butterfly), and the four partial sums are folded left, ((p0 + p1) + p2) + p3.  The order is a function
// of the shape only, so all kernels give the same bits.
#pragma once
#include "common.cuh"

namespace mlxs {

constexpr int LG_TOK = 8;     // token rows staged per pass
constexpr int LG_PARTS = 4;   // warps per expert row

// shared memory of a CTA of `nwarps` warps: the staged rows, then the partial sums [nwarps][LG_TOK]
__host__ __device__ inline size_t logits_smem_bytes(uint32_t H, uint32_t nwarps) {
    return (size_t)LG_TOK * H * 2 + (size_t)nwarps * LG_TOK * sizeof(float);
}

// For few tokens: up to LG_TOK token rows are staged in shared memory per pass.  All threads of the CTA call this (it holds
// CTA-wide barriers).  The CTA's warps form nwarps / 4 expert slots; CTA
// `cta` of `n_cta` takes the experts e = (cta * slots + slot), stepping by n_cta * slots.  Where the grid has twice the slots
// that the experts need, neighbouring CTAs share them and take half of the tokens each.
// A lane's first LG_AHEAD vectors of its row are asked for before the rows are staged: one trip to memory for both (a trip per
// vector, after the staging, was 5,600 of 11,400 cycles at one token of H 5120, and 15,000 of 25,000 went to seven tokens of H 6144).
constexpr int LG_AHEAD = 6;
__device__ __forceinline__ void logits_rows(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                            uint32_t T, uint32_t E, uint32_t H, float* __restrict__ logits, uint8_t* sm,
                                            uint32_t cta, uint32_t n_cta) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nwarps = blockDim.x >> 5;
    const uint32_t slots = nwarps / LG_PARTS, slot = warp / LG_PARTS, part = warp % LG_PARTS;
    const bool shared_out = T > 1 && n_cta % 2 == 0 && (n_cta / 2) * slots >= E;
    const uint32_t t_half = (T + 1) / 2, t_begin = shared_out && (cta & 1u) ? t_half : 0u, t_end = shared_out && !(cta & 1u) ? t_half : T;
    if (shared_out) { cta /= 2; n_cta /= 2; }
    const uint32_t nv = H / 8;
    uint4* xs = reinterpret_cast<uint4*>(sm);                                  // [LG_TOK][nv] vectors of 8 bf16
    float* ps = reinterpret_cast<float*>(sm + (size_t)LG_TOK * H * 2);         // [nwarps][LG_TOK]
    const uint32_t v_begin = part * nv / LG_PARTS, v_end = (part + 1) * nv / LG_PARTS;
    const uint32_t e_step = n_cta * slots, rounds = (E + e_step - 1) / e_step;
    uint4 wv[LG_AHEAD];
    auto fetch = [&](uint32_t e, uint32_t v) {
        const uint4* wrow = reinterpret_cast<const uint4*>(w + (size_t)e * H);
#pragma unroll
        for (int i = 0; i < LG_AHEAD; ++i)
            if (v + 32 * i < v_end) wv[i] = wrow[v + 32 * i];
    };
    for (uint32_t t0 = t_begin; t0 < t_end; t0 += LG_TOK) {
        const uint32_t nt = t_end - t0 < (uint32_t)LG_TOK ? t_end - t0 : (uint32_t)LG_TOK;
        const uint32_t e0 = cta * slots + slot;
        if (e0 < E) fetch(e0, v_begin + lane);
        __syncthreads();
        for (uint32_t v = threadIdx.x; v < nt * nv; v += blockDim.x) xs[v] = reinterpret_cast<const uint4*>(x + (size_t)t0 * H)[v];
        __syncthreads();
        for (uint32_t rd = 0; rd < rounds; ++rd) {
            const uint32_t e = rd * e_step + e0;
            const bool live = e < E;
            float acc[LG_TOK];
#pragma unroll
            for (int tt = 0; tt < LG_TOK; ++tt) acc[tt] = 0.f;
            if (live) {
                for (uint32_t v0 = v_begin + lane; v0 < v_end; v0 += 32 * LG_AHEAD) {
                    if (rd || v0 != v_begin + lane) fetch(e, v0);
#pragma unroll 1
                    for (uint32_t v = v0; v < v_end && v < v0 + 32 * LG_AHEAD; v += 32) {
                        // the vectors move up by one: a short loop (unrolled over them, the code alone took longer to fetch)
                        const uint32_t ww[4] = {wv[0].x, wv[0].y, wv[0].z, wv[0].w};
#pragma unroll
                        for (int i = 0; i + 1 < LG_AHEAD; ++i) wv[i] = wv[i + 1];
#pragma unroll
                        for (int tt = 0; tt < LG_TOK; ++tt) {
                            if ((uint32_t)tt >= nt) break;
                            const uint4 xv = xs[tt * nv + v];
                            const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                acc[tt] = __fmaf_rn(__uint_as_float(xw[q] << 16), __uint_as_float(ww[q] << 16), acc[tt]);
                                acc[tt] = __fmaf_rn(__uint_as_float(xw[q] & 0xFFFF0000u), __uint_as_float(ww[q] & 0xFFFF0000u), acc[tt]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int tt = 0; tt < LG_TOK; ++tt) {
                float a = acc[tt];
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, o));
                if (lane == 0) ps[warp * LG_TOK + tt] = a;
            }
            __syncthreads();
            if (live && part == 0 && lane < nt) {
                const float* p0 = ps + (slot * LG_PARTS) * LG_TOK + lane;
                float a = p0[0];
#pragma unroll
                for (int s = 1; s < LG_PARTS; ++s) a = __fadd_rn(a, p0[s * LG_TOK]);
                logits[(size_t)(t0 + lane) * E + e] = a;
            }
            __syncthreads();
        }
    }
}

// For more tokens: a CTA of 8 warps owns 8 experts x 8 tokens, a warp one quarter of the inputs of 4 experts x 8 tokens, so a
// loaded vector serves 4 or 8 products.  With one expert per warp and the rows staged again by every CTA the time went by the
// tokens: 8192 tokens of 64 experts, H 5120, took 11.6 ms.  Issue-bound: 364 instructions for 256 multiply-adds (the rows' and
// the weights' conversion is the rest).
constexpr int LT_E = 4, LT_T = 8;
constexpr int LT_CTA_E = 2 * LT_E;
__device__ __forceinline__ void logits_tile(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, uint32_t T,
                                            uint32_t E, uint32_t H, float* __restrict__ logits, uint32_t e_cta, uint32_t t0) {
    __shared__ float ps[2 * LG_PARTS][32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, part = warp % LG_PARTS, e0 = e_cta + warp / LG_PARTS * LT_E;
    const uint32_t nv = H / 8, v_end = (part + 1) * nv / LG_PARTS;
    const uint4 *wr[LT_E], *xr[LT_T];   // rows beyond the last one are read in its place and not stored
#pragma unroll
    for (int i = 0; i < LT_E; ++i) wr[i] = reinterpret_cast<const uint4*>(w + (size_t)min(e0 + i, E - 1) * H);
#pragma unroll
    for (int i = 0; i < LT_T; ++i) xr[i] = reinterpret_cast<const uint4*>(x + (size_t)min(t0 + i, T - 1) * H);
    float acc[LT_T * LT_E];             // [token][expert]
#pragma unroll
    for (int i = 0; i < LT_T * LT_E; ++i) acc[i] = 0.f;
    for (uint32_t v = part * nv / LG_PARTS + lane; v < v_end; v += 32) {
        uint4 wv[LT_E], xv[LT_T];
#pragma unroll
        for (int i = 0; i < LT_E; ++i) wv[i] = wr[i][v];
#pragma unroll
        for (int i = 0; i < LT_T; ++i) xv[i] = xr[i][v];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float wl[LT_E], wh[LT_E];
#pragma unroll
            for (int i = 0; i < LT_E; ++i) {
                const uint32_t u = q == 0 ? wv[i].x : q == 1 ? wv[i].y : q == 2 ? wv[i].z : wv[i].w;
                wl[i] = __uint_as_float(u << 16); wh[i] = __uint_as_float(u & 0xFFFF0000u);
            }
#pragma unroll
            for (int t = 0; t < LT_T; ++t) {
                const uint32_t u = q == 0 ? xv[t].x : q == 1 ? xv[t].y : q == 2 ? xv[t].z : xv[t].w;
                const float xl = __uint_as_float(u << 16), xh = __uint_as_float(u & 0xFFFF0000u);
#pragma unroll
                for (int i = 0; i < LT_E; ++i) acc[t * LT_E + i] = __fmaf_rn(xh, wh[i], __fmaf_rn(xl, wl[i], acc[t * LT_E + i]));
            }
        }
    }
    // the butterfly of 32 sums at once: at each level two lanes swap half of the sums they still hold, so lane l ends with sum l
    // after 31 shuffles; the same additions as a butterfly per sum
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool hi = lane & (uint32_t)o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float keep = hi ? acc[i + o] : acc[i], give = hi ? acc[i] : acc[i + o];
            acc[i] = __fadd_rn(keep, __shfl_xor_sync(0xFFFFFFFFu, give, o));
        }
    }
    ps[warp][lane] = acc[0];
    __syncthreads();
    const uint32_t t = t0 + lane / LT_E, e = e0 + lane % LT_E;
    if (part == 0 && t < T && e < E) {
        float a = ps[warp][lane];
#pragma unroll
        for (int s = 1; s < LG_PARTS; ++s) a = __fadd_rn(a, ps[warp + s][lane]);
        logits[(size_t)t * E + e] = a;
    }
}

}  // namespace mlxs
