// MXFP4 / NVFP4 expert kernels for experts with many rows: tcgen05 tensor cores, weights decoded into tensor memory.
//
// The reference sends prefill-sized FP4 work to a grouped quantised GEMM over rows sorted by expert
// (src/arch/mimo_v2/math.zig:426-447, src/arch/glm5_next/nvfp4.zig:36-56): bf16 rows times dequantised weights, f32
// accumulate.  The pipeline is lane.cuh's; this file supplies the decode, the row staging and the epilogue:
//   * a decode thread owns one output column and takes 64 of its inputs per stage: 32 codes as one 16-byte word, turned into
//     16-bit values, times the block scale, 16 tensor-memory columns per store (32x32b.x16);
//   * MXFP4: operands are bf16.  The code's 3 magnitude bits placed at bits 6..8 are e2m1 x 2^-126 as bf16 (the 0.5
//     code is a bf16 subnormal); one bf16x2 multiply by 2^(b-1) gives e2m1 x 2^(b-127) exactly, and the rows stay the
//     bf16 they arrived as, so every product is exact.  This needs 2^(b-1) to be a bf16, b <= 128 (block scale <= 2):
//     an expert with a larger scale byte is marked at load and always takes the streaming lane.  The k order inside a group
//     of 8 is the decode's (0,4,1,5,2,6,3,7); the rows are staged in the same order;
//   * NVFP4: operands are f16, weights the exact e2m1 values (one e2m1x2 conversion per two codes) times the block's
//     E4M3 scale (one e4m3x2 conversion; exact in f16, as in the streaming lane), rows rounded bf16 -> f16, the global
//     g/2688 applied in the epilogue (decode_kernels_ref.zig:13-65);
//   * the epilogue works from tensor memory (a thread owns one output column of 16 rows): the reference's bf16 rounding
//     chain for gate/up (mimo_moe_k1_gateup.metal:115-128, glm5n_nvfp4_gateup.metal:109-129), the rounding for down; a warp
//     turns its 32 columns x 16 rows in shared memory so that 16-byte pieces of rows leave (two-byte stores before).
#include <cstdlib>

#include "lane.cuh"

namespace mlxs {

// ------------------------------------------------------------------------------------------------------------
// prep: gather the tile's rows into the B-operand order (bf16 kept for MXFP4, rounded to f16 for NVFP4)
// ------------------------------------------------------------------------------------------------------------
// eight consecutive values of a row in staged order: MXFP4 0,4,1,5,2,6,3,7, NVFP4 natural
template <bool NV>
__device__ __forceinline__ uint4 q_order8(uint4 r) {
    return NV ? r : make_uint4(__byte_perm(r.x, r.z, 0x5410), __byte_perm(r.x, r.z, 0x7632), __byte_perm(r.y, r.w, 0x5410), __byte_perm(r.y, r.w, 0x7632));
}
// a warp moves 32 consecutive inputs of eight rows: four lanes read 64 bytes of a row, eight lanes write one core matrix
template <bool NV>
__global__ void __launch_bounds__(256) q_prep_kernel(const __nv_bfloat16* __restrict__ x, uint32_t top_k, uint32_t H,
                                                     DispatchTables t, const uint32_t* __restrict__ tiles,
                                                     uint16_t* __restrict__ xa) {
    const uint32_t tile = blockIdx.x;
    if (tile >= tiles[0]) return;
    const uint32_t* te = prefill_tile(tiles, tile);
    const uint32_t row0 = te[1], rows = te[2], rows16 = (rows + 15) / 16 * 16;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, r8 = lane >> 2, c = lane & 3u;
    uint16_t* dst = xa + (size_t)te[3] * H;
    for (uint32_t rg = warp; rg < rows16 / 8; rg += 8) {
        const uint32_t r = rg * 8 + r8;
        const bool valid = r < rows;
        const __nv_bfloat16* src = x + (valid ? (size_t)x_row_of(t, t.order[row0 + r], top_k) * H : 0);
        const uint32_t step = gridDim.y * 4;
        for (uint32_t g0 = blockIdx.y * 4 + c; g0 < H / 8; g0 += 4 * step) {   // groups of 8 inputs, four loads in flight
            uint4 raw[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) raw[i] = valid && g0 + i * step < H / 8 ? *reinterpret_cast<const uint4*>(src + (size_t)(g0 + i * step) * 8) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t g = g0 + i * step;
                if (g >= H / 8) break;
                if (NV) {
                    uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const __half2 h = __floats2half2_rn(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xFFFF0000u));
                        w[k] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    raw[i] = make_uint4(w[0], w[1], w[2], w[3]);
                }
                *reinterpret_cast<uint4*>(dst + (size_t)(g / 16) * (rows16 * LN_KST) + ln_row_off(r, g % 16)) = q_order8<NV>(raw[i]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// the bank's part of the lane
// ------------------------------------------------------------------------------------------------------------
// MXFP4: 8 codes of a word -> 4 bf16x2 of e2m1 x 2^-126 (pairs (0,4), (1,5), (2,6), (3,7))
__device__ __forceinline__ void q_decode8_bf16(uint32_t w, uint32_t (&h)[4]) {
    h[0] = ((w << 6) & 0x01C001C0u) | ((w << 12) & 0x80008000u);
    h[1] = ((w << 2) & 0x01C001C0u) | ((w << 8) & 0x80008000u);
    h[2] = ((w >> 2) & 0x01C001C0u) | ((w << 4) & 0x80008000u);
    h[3] = ((w >> 6) & 0x01C001C0u) | (w & 0x80008000u);
}
// NVFP4: 8 codes of a word -> 4 f16x2 of the exact e2m1 values through the conversion instruction (pairs (0,1), (2,3),
// (4,5), (6,7))
__device__ __forceinline__ void q_decode8_f16(uint32_t w, uint32_t (&h)[4]) {
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w));
}
__device__ __forceinline__ uint32_t q_mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t q_mul_f16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// E4M3 byte -> f16x2 (both halves) of its value, exact
__device__ __forceinline__ uint32_t q_e4m3_f16x2(uint32_t b) {
    uint32_t d;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(d) : "h"((uint16_t)(b * 0x0101u)));
    return d;
}
__device__ __forceinline__ float q_sigmoid(float x) {  // src/arch/mimo_v2/moe.zig:341-344
    const float y = sigmoid_tail_fast(x);
    return x < 0.f ? y : 1.0f - y;
}

constexpr uint32_t Q_W_STAGE = 8192;          // code bytes of a projection's (block, stage) in the stream (fp4.cu F4_W_STAGE)
constexpr uint32_t Q_T_STRIDE = 80;           // bytes between two rows of a warp's 16 x 32 staging (conflict-free 16-byte reads)
constexpr uint32_t Q_T_WARP = 16 * Q_T_STRIDE;

template <bool NV>
struct Fp4LaneBank {
    static constexpr uint32_t FORMAT = NV ? UMMA_F16 : UMMA_BF16;
    static constexpr uint32_t S_STAGE = NV ? 1024u : 512u;      // scale bytes of a projection's (block, stage)
    static constexpr uint32_t RAW_BYTES = Q_W_STAGE + S_STAGE;
    static constexpr uint32_t AHEAD = 1;   // pieces of a stage decoded before the operand slot is waited for
    static constexpr int MID = 4;          // MMAs of a stage before the next one's barrier is tested (8: not before the stage)
    static constexpr size_t EPI_SMEM = LN_EPI_WARPS * Q_T_WARP;

    // the stream holds, per stage, the projections' codes, then their scales
    template <int NPASS>
    static __device__ __forceinline__ void copy_stage(uint8_t* dst, const uint8_t* src, uint32_t ks, uint32_t nstage, uint64_t* bar) {
        const uint32_t p = NPASS == 2 && ks >= nstage ? 1u : 0u;
        src += (size_t)(ks - p * nstage) * (NPASS * RAW_BYTES);
        bulk_g2s(dst, src + p * Q_W_STAGE, Q_W_STAGE, bar);
        bulk_g2s(dst + Q_W_STAGE, src + NPASS * Q_W_STAGE + p * S_STAGE, S_STAGE, bar);
    }

    struct Decoder {
        uint32_t w_off, s_off;   // this column's first code word and scale byte of the half stage
        __device__ __forceinline__ Decoder(uint32_t q, uint32_t half, uint32_t lane) {
            const uint32_t m = q * 32u + lane, wr = m >> 4, r = (m >> 3) & 1u, g = m & 7u, sb = half * 2u;
            w_off = (((wr * 4 + sb) * 2 + r) * 32 + g * 4) * 4;                       // words [wr][block][r][g][4]
            s_off = Q_W_STAGE + (NV ? (wr * 4 + sb) * 32 + g * 2 + r : ((wr * 4 + sb) * 8 + g) * 2 + r);
        }
        // piece pc of the stage (or of the constructor's half): a 32-block, 32 codes of this column
        __device__ __forceinline__ void decode(const uint8_t* raw, uint32_t slot_bytes, uint32_t pc, uint32_t (&v)[16]) const {
            const uint4 ww = *reinterpret_cast<const uint4*>(raw + slot_bytes + w_off + pc * 256u);
            const uint8_t* s = raw + slot_bytes + s_off + pc * (NV ? 32u : 16u);
            const uint32_t wds[4] = {ww.x, ww.y, ww.z, ww.w};
            uint32_t s0, s1;
            if (NV) {
                s0 = q_e4m3_f16x2(s[0]);
                s1 = q_e4m3_f16x2(s[16]);
            } else {
                s0 = s1 = ((s[0] + 126u) << 7) * 0x00010001u;   // 2^(b - 1) in both halves
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t h[4];
                if (NV) q_decode8_f16(wds[c], h);
                else q_decode8_bf16(wds[c], h);
#pragma unroll
                for (int i = 0; i < 4; ++i) v[4 * c + i] = NV ? q_mul_f16x2(h[i], c < 2 ? s0 : s1) : q_mul_bf16x2(h[i], s0);
            }
        }
        static __device__ __forceinline__ void store(uint32_t ta, uint32_t pc, const uint32_t (&v)[16]) {
            asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(ta + pc * 16),
                         "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                         "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                         : "memory");
        }
    };

    template <int NPASS, int p>
    static __device__ __forceinline__ bool epilogue(const LaneParams& P, LaneEpi& E, const LanePass& C) {
        const uint32_t lane = E.lane, m = E.q * 32u + lane, nch = C.rows16 / 16;
        float gs = 1.f;
        if (NV) gs = P.gscale[C.expert * 3 + (NPASS == 2 ? p : 2)] / 2688.0f;
        // act(gate), exact in bf16: [CTA][16-row chunk][column][16 rows]
        uint4* act = reinterpret_cast<uint4*>(static_cast<uint8_t*>(P.act) + (size_t)blockIdx.x * LN_ACT_BYTES) + m * 2;
        uint8_t* tw = E.smem + E.ew * Q_T_WARP;
        for (uint32_t c = E.half; c < nch; c += 2) {
            uint32_t v[16];
            tmem_ld16(C.acc + ((E.q * 32u) << 16) + c * 16, v);
            if (NPASS == 2 && p == 0) {
                uint32_t a[8];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    // mimo_moe_k1_gateup.metal:115-128 / glm5n_nvfp4_gateup.metal:109-129
                    float gf = bf16_round_f(__uint_as_float(v[i]) * gs);
                    if (P.limit > 0.f) gf = gf > P.limit ? P.limit : gf;
                    const float y = sigmoid_tail_fast(gf);                        // src/arch/mimo_v2/moe.zig:341-344
                    const uint32_t bits = __bfloat16_as_ushort(__float2bfloat16_rn(gf * (gf < 0.f ? y : 1.0f - y)));
                    if (i & 1) a[i >> 1] |= bits << 16; else a[i >> 1] = bits;
                }
                __stcg(act + c * 256, make_uint4(a[0], a[1], a[2], a[3]));
                __stcg(act + c * 256 + 1, make_uint4(a[4], a[5], a[6], a[7]));
                continue;
            }
            if (NPASS == 2) {
                const uint4 a0 = __ldcg(act + c * 256), a1 = __ldcg(act + c * 256 + 1);
                const uint32_t a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float uf = bf16_round_f(__uint_as_float(v[i]) * gs);
                    if (P.limit > 0.f) uf = uf > P.limit ? P.limit : (uf < -P.limit ? -P.limit : uf);
                    const float hq = bf16_round_f(__uint_as_float(i & 1 ? a[i >> 1] & 0xFFFF0000u : a[i >> 1] << 16) * uf);
                    // the down input: bf16 as is, or rounded to f16; 0 in padding rows (their B rows are 0)
                    *reinterpret_cast<uint16_t*>(tw + i * Q_T_STRIDE + lane * 2) = NV ? __half_as_ushort(__float2half_rn(hq)) : (uint16_t)(__float_as_uint(hq) >> 16);
                }
            } else if (P.out_bf16) {
#pragma unroll
                for (int i = 0; i < 16; ++i) *reinterpret_cast<__nv_bfloat16*>(tw + i * Q_T_STRIDE + lane * 2) = __float2bfloat16_rn(__uint_as_float(v[i]) * gs);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint32_t rr = c * 16 + i;
                    if (rr < C.rows) static_cast<float*>(P.out)[(size_t)P.t.order[C.row0 + rr] * P.H + C.nb * 128 + m] = __uint_as_float(v[i]) * gs;
                }
                continue;
            }
            __syncwarp();
            // 16 rows x 32 columns leave as 16-byte pieces: lane = (row % 8, group of 8 columns)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t i = (lane & 7u) + 8u * j, rr = c * 16 + i, grp = lane >> 3;
                const uint4 w = *reinterpret_cast<const uint4*>(tw + i * Q_T_STRIDE + grp * 16);
                if (NPASS == 2) {
                    uint16_t* xd = P.xd + (size_t)C.srow0 * P.I + (size_t)C.nb * (C.rows16 * LN_KST);
                    *reinterpret_cast<uint4*>(xd + ln_row_off(rr, E.q * 4 + grp)) = q_order8<NV>(w);
                } else if (rr < C.rows) {
                    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(P.out) + (size_t)P.t.order[C.row0 + rr] * P.H + C.nb * 128 + E.q * 32 + grp * 8) = w;
                }
            }
            __syncwarp();
        }
        C.release(lane);
        return true;
    }
};

bool fp4_prefill_supported(uint32_t H, uint32_t I) { return H % 128 == 0 && I % 128 == 0 && (I / 128) % 2 == 0 && (H / 128) % 4 == 0; }

template <bool NV>
static cudaError_t q_launch_all(const Fp4PrefillArgs& a, cudaStream_t st) {
    q_prep_kernel<NV><<<dim3(a.max_tiles, 8), 256, 0, st>>>(a.x, a.top_k, a.H, a.t, a.tiles, a.xa);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    LaneParams P{};
    P.gscale = a.gscale; P.tiles = a.tiles; P.next = a.tiles + 3; P.t = a.t; P.H = a.H; P.I = a.I; P.limit = a.limit;
    P.status = a.status; P.act = a.act;
    P.code = a.gu; P.n_blocks = a.I / 128; P.n_stages = a.H / LN_KST;
    P.expert_stride = (size_t)P.n_blocks * P.n_stages * 2 * Fp4LaneBank<NV>::RAW_BYTES;
    P.xa = a.xa; P.xa_proj_stride = 0; P.xd = a.xd;
    if ((e = lane_launch<Fp4LaneBank<NV>, 2>(P, a.sm_count, st)) != cudaSuccess) return e;
    P.next = a.tiles + 4;
    P.code = a.dn; P.n_blocks = a.H / 128; P.n_stages = a.I / LN_KST;
    P.expert_stride = (size_t)P.n_blocks * P.n_stages * Fp4LaneBank<NV>::RAW_BYTES;
    P.xa = a.xd; P.xd = nullptr; P.out = a.ro; P.out_bf16 = a.ro_bf16;
    return lane_launch<Fp4LaneBank<NV>, 1>(P, a.sm_count, st);
}

cudaError_t launch_fp4_prefill(const Fp4PrefillArgs& a, cudaStream_t st) {
    const cudaError_t e = launch_prefill_plan(a.t, a.n_experts, a.lane_flags, a.min_rows, LN_ROWS, LN_ROWS_NARROW, a.max_tiles, a.tiles, a.status, st);
    if (e != cudaSuccess) return e;
    return a.nv ? q_launch_all<true>(a, st) : q_launch_all<false>(a, st);
}

}  // namespace mlxs
