// EXL3 expert kernels for experts with many rows: tcgen05 tensor cores, the trellis decoded straight into tensor memory.
//
// The reference's prefill lane (src/exl3/quant.zig:1040-1271; texts dsv41_prefill_dig_gemm_*_m128*.metal) decodes
// trellis tiles to f16 in threadgroup memory per K stage and feeds its MMA units with f16 rotated activations and an
// f32 accumulator.  Here the pipeline is lane.cuh's; this file supplies
//   * the decode: a lane (g, c) that has decoded a 16x16 tile holds W[k 2c,2c+1 | 2c+8,2c+9][column g | g+8]: that is one
//     tcgen05.st.16x256b fragment (thread (g, c): lanes g and g + 8, two adjacent 32-bit columns) once the K order inside a
//     16-block is taken as k' = 4c + 2 (k / 8) + k % 2, c = (k % 8) / 2; the rows are staged in the same order.  Four k-tiles of a
//     column tile lie word by word beside each other (common.cuh): two 16-byte loads serve four tiles, and their stores go out
//     together (16x256b.x4);
//   * the row staging: H128(x suh) 128^-0.5, f16, once per projection;
//   * the epilogue: transpose through shared memory, then row-wise Hadamard-128, svh, clamped SwiGLU, suh_d, Hadamard for
//     gate / up (act(gate) waits in an L2-resident scratch between the two passes, read back by the threads that wrote it);
//     Hadamard, svh_d for down.
// What bounds it (54 to 61 warp instructions per decoded tile with the epilogue, about 42 of them the decode by its source; 74 to 80 % of the issue slots): up to about 128 rows per tile the
// decode's instruction issue, above that the MMAs; calls of thousands of tokens run into the 1 kW power cap (1.55 GHz at
// 8192 tokens).  Layer of H 5120, I 2304, 256 experts, calls back to back: 2048 tokens 4.04 -> 3.05 ms, 8192 tokens 10.65 ->
// 7.74 ms against the lane that accumulated gate and up together, 3 % less with uniform MMA operands and wide code loads.
#include <cstdlib>

#include "dispatch_body.cuh"
#include "lane.cuh"

namespace mlxs {

// ------------------------------------------------------------------------------------------------------------
// plan: row tiles per expert from the dispatch tables
// ------------------------------------------------------------------------------------------------------------
// An expert's rows are split evenly over its tiles (a 16-row remainder tile would cost a full decode).
// Staging rows: a tile's rows padded to 16, tiles in sorted order, so tile number n starts at its first row + 16 n.
// narrow: with tiles of up to that many rows the lane has another operand slot (lane.cuh), worth about as much as a
// twentieth of the tiles: taken when the call gets at most one tile in sixteen more.  (300 Zipf-routed tokens, one expert
// above 160 rows: 690 -> 665 us; 4500 tokens, one expert in 23 above: even; 6000 tokens, nearly all above: 5.5 -> 6.5 ms if
// it were taken there.)
// One thread per expert; with one thread adding up the tile counts the kernel took 8 us for 256 experts.
__global__ void __launch_bounds__(DTHREADS) pf_plan_kernel(DispatchTables t, uint32_t E, const uint8_t* __restrict__ flags, uint32_t min_rows,
                                                           uint32_t cap, uint32_t narrow, uint32_t max_tiles, uint32_t* __restrict__ tiles,
                                                           uint32_t* status) {
    __shared__ uint32_t ws[99], s_most;
    const uint32_t e = threadIdx.x;
    if (e == 0) s_most = 0;
    const uint32_t r0 = e < E ? t.offsets[e] : 0u, c = e < E ? t.offsets[e + 1] - r0 : 0u;
    const bool lane = e < E && takes_tensor_lane(c, min_rows, flags, e);
    const uint32_t v[3] = {lane ? (c + cap - 1) / cap : 0u, lane ? (c + narrow - 1) / narrow : 0u, 0u};
    uint32_t base[3], tot[3];
    block_scan3(v, base, tot, ws);
    const int k = tot[1] * 16u <= tot[0] * 17u ? 1 : 0;
    const bool ok = tot[k] <= max_tiles;
    const uint32_t nt = v[k], first = base[k], per = nt ? ((c + nt - 1) / nt + 15) / 16 * 16 : 0u;
    if (nt) atomicMax(&s_most, per);
    if (ok)
        for (uint32_t i = 0; i < nt; ++i)
            *reinterpret_cast<uint4*>(prefill_tile(tiles, first + i)) =
                make_uint4(e, r0 + i * per, min(per, c - i * per), r0 + i * per + 16 * (first + i));
    __syncthreads();
    if (e == 0) {
        if (!ok) atomicMax(status, (uint32_t)ST_WORKLIST_OVERFLOW);
        tiles[0] = ok ? tot[k] : 0u;
        tiles[2] = s_most;
        tiles[3] = tiles[4] = 0;
    }
}

// ------------------------------------------------------------------------------------------------------------
// Hadamard-128 of R rows at once; the levels go in the order of the index bits, as in hadamard128_warp, so the bits of a
// result do not depend on which elements a lane holds.  sg[i] = -1 in lanes with lane bit i set, else +1: a level over a
// lane bit is one shuffle and one exact fused multiply-add per element.
//   SPLIT = false: a lane holds elements 4 lane + {0, 1, 2, 3} (index bits 0, 1 in registers)
//   SPLIT = true:  16 (lane / 4) + 2 (lane % 4) + {0, 1, 8, 9} (index bits 0, 3 in registers)
// ------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void pf_signs(uint32_t lane, float (&sg)[5]) {
#pragma unroll
    for (int i = 0; i < 5; ++i) sg[i] = (lane >> i) & 1u ? -1.0f : 1.0f;
}
template <int R>
__device__ __forceinline__ void pf_level_lane(float (&v)[R][4], float sg, int mask) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) v[r][q] = __fmaf_rn(sg, v[r][q], __shfl_xor_sync(0xFFFFFFFFu, v[r][q], mask));
}
template <int R>
__device__ __forceinline__ void pf_level_reg(float (&v)[R][4], int m) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (!(q & m)) {
                const float lo = v[r][q] + v[r][q | m], hi = v[r][q] - v[r][q | m];
                v[r][q] = lo;
                v[r][q | m] = hi;
            }
}
template <bool SPLIT, bool LEVEL0 = true, int R>
__device__ __forceinline__ void pf_hadamard(float (&v)[R][4], const float (&sg)[5]) {
    if (LEVEL0) pf_level_reg(v, 1);
    if (!SPLIT) pf_level_reg(v, 2);
    pf_level_lane(v, sg[0], 1);
    pf_level_lane(v, sg[1], 2);
    if (SPLIT) pf_level_reg(v, 2);
    pf_level_lane(v, sg[2], 4);
    pf_level_lane(v, sg[3], 8);
    pf_level_lane(v, sg[4], 16);
}

// ------------------------------------------------------------------------------------------------------------
// prep: rows -> rotated f16 activations in the MMA's B-operand order
// ------------------------------------------------------------------------------------------------------------
// The position of input k inside its 16-block is 4 ((k % 8) / 2) + 2 ((k % 16) / 8) + k % 2, the order in which the decode's
// registers fill a tensor-memory fragment.  A lane (t = lane / 4, c = lane % 4) that holds the inputs 16 t + {2c, 2c + 1,
// 2c + 8, 2c + 9} of a 128-block has the four consecutive positions 16 t + 4 c: one 8-byte store at this element offset
// inside the stage.
__device__ __forceinline__ uint32_t pf_lane_off(uint32_t row, uint32_t lane) {
    return ln_row_off(row, (lane >> 2) * 2u + ((lane >> 1) & 1u)) + (lane & 1u) * 4u;
}
__device__ __forceinline__ uint32_t pf_lane_col(uint32_t lane) { return (lane >> 2) * 16u + (lane & 3u) * 2u; }   // and + 1, + 8, + 9
__device__ __forceinline__ uint2 pf_pack4(float v0, float v1, float v2, float v3) {
    const __half2 a = __floats2half2_rn(v0, v1), b = __floats2half2_rn(v2, v3);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ void pf_load_scale4(const __half* p, uint32_t lane, float (&s)[4]) {   // p: the 128-block's scales
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(p + pf_lane_col(lane)));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(p + pf_lane_col(lane) + 8));
    s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
}

// xa: [projection][staging rows][H] (a tile's rows start at its first staging row, padded to 16).  A warp stages eight
// rows of one 128-block: lane = (row, s), with the 32 inputs 32 j + 8 s + i (j < 4, i < 8).  The levels of i and j stay in
// registers.  For a level of s the two lanes swap half their registers: each then has both sides of 16 butterflies, and the
// lane bit has become a bit of i, whose level is done.  The kernel is bound by the L1's data path, which the shuffles share:
// 32 of them per row group and projection (one per input and level, with a last exchange before the stores, was 72).
// After both levels a lane holds exactly the four consecutive positions of pf_lane_off in every 16-block: with c = lane % 4,
// {2 c', 2 c' + 1, 2 c' + 8, 2 c' + 9}, c' = c with its two bits swapped; the 8-byte stores of a warp fill whole lines.
// Two CTAs per SM: with three (80 registers) 60 bytes a thread spilled into the data path that bounds the kernel (300 tokens of
// 64 experts 28.0 -> 26.1 us, 2048 tokens 124 -> 121, 8192 447 -> 451, under ncu).
constexpr int PREP_WARPS = 8;
__global__ void __launch_bounds__(PREP_WARPS * 32, 2) pf_prep_kernel(const __nv_bfloat16* __restrict__ x, uint32_t top_k, uint32_t H,
                                                                  const __half* __restrict__ scales, size_t scales_stride,
                                                                  DispatchTables t, const uint32_t* __restrict__ tiles, size_t proj_stride, __half* __restrict__ xa) {
    const uint32_t tile = blockIdx.x;
    if (tile >= tiles[0]) return;
    const uint32_t* te = prefill_tile(tiles, tile);
    const uint32_t e = te[0], row0 = te[1], rows = te[2];
    const uint32_t rows16 = (rows + 15) / 16 * 16, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nblk = H / 128;
    const uint32_t r8 = lane >> 2, seg = lane & 3u;
    const float S = __uint_as_float(SCALE_BITS);
    const bool odd = seg & 1u, high = seg & 2u;
    // a difference comes out negated in the lane that kept the second halves: made good in the last scaling
    const float S0 = odd ? -S : S, S1 = high ? -S : S, S01 = odd != high ? -S : S;
    const __half* sc_e = scales + (size_t)e * scales_stride + seg * 8;
    for (uint32_t task = blockIdx.y * PREP_WARPS + warp; task < nblk * (rows16 / 8); task += gridDim.y * PREP_WARPS) {
        const uint32_t b = task % nblk, r = task / nblk * 8 + r8;
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = make_uint4(0, 0, 0, 0);
        if (r < rows) {
            const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)x_row_of(t, t.order[row0 + r], top_k) * H + b * 128 + seg * 8);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = src[4 * j];
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const uint4* sp = reinterpret_cast<const uint4*>(sc_e + (size_t)p * H + b * 128);
            float v[32];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 s4 = sp[4 * j];
                const uint32_t xw[4] = {w[j].x, w[j].y, w[j].z, w[j].w}, sw[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&sw[k]));
                    v[8 * j + 2 * k] = __uint_as_float(xw[k] << 16) * sf.x;
                    v[8 * j + 2 * k + 1] = __uint_as_float(xw[k] & 0xFFFF0000u) * sf.y;
                }
            }
            // levels in the order of the index bits: i (registers), s (lanes), j (registers)
            auto level_reg = [&](int m) {
#pragma unroll
                for (int k = 0; k < 32; ++k)
                    if (!(k & m)) {
                        const float lo = v[k] + v[k | m], hi = v[k] - v[k | m];
                        v[k] = lo;
                        v[k | m] = hi;
                    }
            };
            level_reg(1); level_reg(2); level_reg(4);
            auto level_swap = [&](int m, bool second, int lane_mask) {
#pragma unroll
                for (int k = 0; k < 32; ++k)
                    if (!(k & m)) {
                        const float keep = second ? v[k | m] : v[k], got = __shfl_xor_sync(0xFFFFFFFFu, second ? v[k] : v[k | m], lane_mask);
                        v[k] = keep + got;
                        v[k | m] = keep - got;
                    }
            };
            level_swap(4, odd, 1);
            level_swap(2, high, 2);
            level_reg(8); level_reg(16);
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] *= (k & 6) == 6 ? S01 : (k & 4) ? S0 : (k & 2) ? S1 : S;
            // src/kernels/exl3/dsv41_prefill_dig_take2v_5120.metal:57-58: the rotated input is rounded to f16
            const uint32_t c = (seg & 1u) * 2u + (seg >> 1);
            __half* dst = xa + p * proj_stride + (size_t)te[3] * H + (size_t)b * (rows16 * LN_KST) + ln_row_off(r, c >> 1) + (c & 1u) * 4u;
            // registers 8 j + 4 (bit 3 of the input) + 2 (bit 4) + bit 0
#pragma unroll
            for (int t16 = 0; t16 < 8; ++t16) {
                const int k = (t16 >> 1) * 8 + (t16 & 1) * 2;
                *reinterpret_cast<uint2*>(dst + t16 * 128) = pf_pack4(v[k], v[k + 1], v[k + 4], v[k + 5]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// the bank's part of the lane
// ------------------------------------------------------------------------------------------------------------
constexpr int PF_EPI_ROWS = 32;     // rows per epilogue batch
constexpr int PF_ZS_STRIDE = 132;

template <int KB>   // bits per weight
struct Exl3LaneBank {
    static constexpr uint32_t FORMAT = UMMA_F16;
    static constexpr uint32_t TW = 8 * KB, KT_WORDS = 8 * TW;   // words per 16x16 tile, per k-tile of a block
    static constexpr uint32_t RAW_BYTES = (LN_KST / 16) * KT_WORDS * 4;
    static constexpr uint32_t AHEAD = 2;   // pieces of a stage decoded before the operand slot is waited for
    static constexpr int MID = 8;          // MMAs of a stage before the next one's barrier is tested (8: not before the stage)
    static constexpr size_t EPI_SMEM = 2 * PF_EPI_ROWS * PF_ZS_STRIDE * sizeof(float);

    // the passes' k-tiles follow each other in the stream: stage ks of both passes together
    template <int NPASS>
    static __device__ __forceinline__ void copy_stage(uint8_t* dst, const uint8_t* src, uint32_t ks, uint32_t, uint64_t* bar) {
        bulk_g2s(dst, src + (size_t)ks * RAW_BYTES, RAW_BYTES, bar);
    }

    struct Decoder {
        uint32_t wi, wj, lp, off;
        __device__ __forceinline__ Decoder(uint32_t q, uint32_t half, uint32_t lane) {
            exl3_lane_plan_kb<KB>(lane, wi, wj, lp);
            off = half * (LN_KST / 32) * KT_WORDS + 2 * q * (4 * TW);   // lanes 32 q .. hold the 16-column tiles 2 q, 2 q + 1
        }
        // piece pc of the stage (or of the constructor's half): a quad of one of the two tiles
        __device__ __forceinline__ void decode(const uint8_t* raw, uint32_t slot_bytes, uint32_t pc, uint32_t (&v)[16]) const {
            const uint4* w = reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(raw + slot_bytes) + off + (pc >> 1) * ((LN_KST / 32) * KT_WORDS) + (pc & 1u) * (4 * TW));
            const uint4 lo = w[wi], hi = w[wj];
            const uint32_t l4[4] = {lo.x, lo.y, lo.z, lo.w}, h4[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                uint32_t bq[4];
                exl3_decode_lane_kb<KB>(l4[kt], h4[kt], lp, bq);
#pragma unroll
                for (int k = 0; k < 4; ++k) v[4 * kt + k] = bq[k];
            }
        }
        static __device__ __forceinline__ void store(uint32_t ta, uint32_t pc, const uint32_t (&v)[16]) {
            asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(ta + (pc >> 1) * (LN_A_COLS / 2) + ((pc & 1u) << 20)),
                         "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                         "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                         : "memory");
        }
    };

    template <int NPASS, int p>
    static __device__ __forceinline__ bool epilogue(const LaneParams& P, LaneEpi& E, const LanePass& C) {
        const uint32_t lane = E.lane, ew = E.ew, q = E.q, half = E.half, rows = C.rows, rows16 = C.rows16, nb = C.nb;
        const float S = __uint_as_float(SCALE_BITS);
        float sg[5];
        pf_signs(lane, sg);
        float* act = static_cast<float*>(P.act) + (size_t)blockIdx.x * (LN_ROWS * 128) + lane * 4;
        float* zs = reinterpret_cast<float*>(E.smem);   // [2][32 rows][stride]
        const __half* sc = P.scales + (size_t)C.expert * P.scales_stride + 2 * (size_t)P.H + nb * 128;   // svh_g | svh_u | suh_d [I], svh_d [H]
        float svh[4], shd[4] = {0.f, 0.f, 0.f, 0.f};
        if (NPASS == 2) {
            pf_load_scale4(sc + (p ? P.I : 0u), lane, svh);
            if (p == 1) pf_load_scale4(sc + 2 * (size_t)P.I, lane, shd);
        } else {
            const uint2 s0 = *reinterpret_cast<const uint2*>(sc + 3 * (size_t)P.I + lane * 4);
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&s0.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&s0.y));
            svh[0] = a.x; svh[1] = a.y; svh[2] = b.x; svh[3] = b.y;
        }
        for (uint32_t rb = 0; rb < rows16; rb += PF_EPI_ROWS, ++E.batch) {
            float* z = zs + (E.batch & 1u) * (PF_EPI_ROWS * PF_ZS_STRIDE);
            if (rb + half * 16 < rows16) {
                uint32_t v[16];
                tmem_ld16(C.acc + ((q * 32u) << 16) + rb + half * 16, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) z[(half * 16 + i) * PF_ZS_STRIDE + q * 32 + lane] = __uint_as_float(v[i]);
            }
            if (rb + PF_EPI_ROWS >= rows16) C.release(lane);
            // one rendezvous per batch: a staging buffer is written again two batches later, after the next one
            if (!E.sync()) return false;
#pragma unroll
            for (int rr = 0; rr < 4; rr += 2) {
                const uint32_t zr = ew * 4 + rr, r = rb + zr;
                if (r >= rows16) break;
                float v[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float* zp = z + (zr + i) * PF_ZS_STRIDE;
                    if (NPASS == 2) {
                        const float2 a = *reinterpret_cast<const float2*>(zp + pf_lane_col(lane)), b = *reinterpret_cast<const float2*>(zp + pf_lane_col(lane) + 8);
                        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = b.x; v[i][3] = b.y;
                    } else {
                        const float4 a = *reinterpret_cast<const float4*>(zp + lane * 4);
                        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
                    }
                }
                pf_hadamard<NPASS == 2>(v, sg);
                if (NPASS == 2 && p == 0) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float o[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float gm = (v[i][k] * S) * svh[k];
                            float gate = gm;
                            if (P.limit > 0.f) gate = (gm != gm) ? gm : (gm < P.limit ? gm : P.limit);
                            const float yv = sigmoid_tail_fast(gate);
                            o[k] = gate * (gate < 0.f ? yv : 1.0f - yv);
                        }
                        __stcg(reinterpret_cast<float4*>(act + (size_t)(r + i) * 128), make_float4(o[0], o[1], o[2], o[3]));
                    }
                } else if (NPASS == 2) {
                    float4 a4[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) a4[i] = __ldcg(reinterpret_cast<const float4*>(act + (size_t)(r + i) * 128));
                    float h[2][4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float av[4] = {a4[i].x, a4[i].y, a4[i].z, a4[i].w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float um = (v[i][k] * S) * svh[k];
                            float up = um;
                            if (P.limit > 0.f) {
                                const float u0 = (um != um) ? um : (um > -P.limit ? um : -P.limit);
                                up = (u0 != u0) ? u0 : (u0 < P.limit ? u0 : P.limit);
                            }
                            h[i][k] = __fmul_rn(av[k], up);   // 0 in padding rows: their B rows are 0
                        }
                        // x suh_d and the transform's level 0, the first product of a pair unrounded (written out,
                        // so that the bits do not hang on what the compiler contracts)
#pragma unroll
                        for (int k = 0; k < 4; k += 2) {
                            const float t0 = h[i][k], t1 = __fmul_rn(h[i][k + 1], shd[k + 1]);
                            h[i][k] = __fmaf_rn(t0, shd[k], t1);
                            h[i][k + 1] = __fmaf_rn(t0, shd[k], -t1);
                        }
                    }
                    pf_hadamard<true, false>(h, sg);
                    // src/kernels/exl3/header_dig2_x.metal:104: the down input is rounded to f16
                    __half* xd = reinterpret_cast<__half*>(P.xd) + (size_t)C.srow0 * P.I + (size_t)nb * (rows16 * LN_KST);
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        *reinterpret_cast<uint2*>(xd + pf_lane_off(r + i, lane)) = pf_pack4(h[i][0] * S, h[i][1] * S, h[i][2] * S, h[i][3] * S);
                } else {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (r + i >= rows) continue;
                        const uint32_t assign = P.t.order[C.row0 + r + i];
                        *reinterpret_cast<float4*>(static_cast<float*>(P.out) + (size_t)assign * P.H + nb * 128 + lane * 4) =
                            make_float4((v[i][0] * S) * svh[0], (v[i][1] * S) * svh[1], (v[i][2] * S) * svh[2], (v[i][3] * S) * svh[3]);
                    }
                }
            }
        }
        return true;
    }
};

bool exl3_prefill_supported(Exl3Dims d) { return d.I % LN_KST == 0 && d.H % LN_KST == 0; }

size_t lane_act_bytes(int sm_count) { return (size_t)sm_count * LN_ACT_BYTES; }

cudaError_t launch_prefill_plan(DispatchTables t, uint32_t n_experts, const uint8_t* lane_flags, uint32_t min_rows, uint32_t cap,
                                uint32_t narrow, uint32_t max_tiles, uint32_t* tiles, uint32_t* status, cudaStream_t st) {
    if (n_experts > (uint32_t)DTHREADS) return cudaErrorInvalidValue;
    pf_plan_kernel<<<1, DTHREADS, 0, st>>>(t, n_experts, lane_flags, min_rows, cap, narrow, max_tiles, tiles, status);
    return cudaGetLastError();
}

template <int KB>
static cudaError_t pf_launch_all(const Exl3PrefillArgs& a, cudaStream_t st) {
    LaneParams P{};
    P.tiles = a.tiles; P.next = a.tiles + 3; P.t = a.t; P.scales = a.L.scales; P.scales_stride = exl3_scales_per_expert(a.d);
    P.H = a.d.H; P.I = a.d.I; P.limit = a.limit; P.status = a.status; P.act = a.act;
    P.code = reinterpret_cast<const uint8_t*>(a.L.gu_code); P.expert_stride = 8 * exl3_code_words(a.d); P.n_blocks = a.d.I / 128; P.n_stages = a.d.H / LN_KST;
    P.xa = reinterpret_cast<const uint16_t*>(a.xa); P.xa_proj_stride = exl3_prefill_staging_rows(a.rows_cap, a.max_tiles) * a.d.H;
    P.xd = reinterpret_cast<uint16_t*>(a.xd);
    const cudaError_t e = lane_launch<Exl3LaneBank<KB>, 2>(P, a.sm_count, st);
    if (e != cudaSuccess) return e;
    P.next = a.tiles + 4;
    P.code = reinterpret_cast<const uint8_t*>(a.L.d_code); P.expert_stride = 4 * exl3_code_words(a.d); P.n_blocks = a.d.H / 128; P.n_stages = a.d.I / LN_KST;
    P.xa = P.xd; P.xa_proj_stride = 0; P.xd = nullptr; P.out = a.ro;
    return lane_launch<Exl3LaneBank<KB>, 1>(P, a.sm_count, st);
}

cudaError_t launch_exl3_prefill(const Exl3PrefillArgs& a, cudaStream_t st) {
    cudaError_t e = launch_prefill_plan(a.t, a.n_experts, nullptr, a.min_rows, LN_ROWS, LN_ROWS_NARROW, a.max_tiles, a.tiles, a.status, st);
    if (e != cudaSuccess) return e;
    pf_prep_kernel<<<dim3(a.max_tiles, 8), PREP_WARPS * 32, 0, st>>>(a.x, a.top_k, a.d.H, a.L.scales, exl3_scales_per_expert(a.d), a.t,
                                                                     a.tiles,
                                                                     exl3_prefill_staging_rows(a.rows_cap, a.max_tiles) * a.d.H, a.xa);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return a.d.K == 3 ? pf_launch_all<3>(a, st) : pf_launch_all<2>(a, st);
}

}  // namespace mlxs
