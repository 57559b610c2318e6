// EXL3 expert kernels for experts with many rows: tcgen05 tensor cores, the trellis decoded straight into tensor memory.
//
// The reference's prefill lane (src/exl3/quant.zig:1040-1271; texts dsv41_prefill_dig_gemm_*_m128*.metal) decodes
// trellis tiles to f16 in threadgroup memory per K stage and feeds its MMA units with f16 rotated activations and an
// f32 accumulator.  Here a CTA owns (expert, a tile of up to 192 of its rows, a 128-column block) and walks its inputs once
// per projection (a "pass": gate then up, or down alone).  W^T is the MMA's A operand (M = 128 output columns) and lives
// in tensor memory; the rows are the B operand in shared memory (N = rows rounded to 16).
//   * the in-register decode of a 16x16 tile leaves a lane (g, c) with W[k 2c,2c+1 | 2c+8,2c+9][column g | g+8]: that
//     is one tcgen05.st.16x256b fragment (thread (g, c): lanes g and g + 8, two adjacent 32-bit columns) once the K
//     order inside a 16-block is taken as k' = 4c + 2 (k / 8) + k % 2, c = (k % 8) / 2; the rows are staged in the same
//     order, which a dot product does not see;
//   * one pass has one accumulator group of at most 192 tensor-memory columns, so two of them fit (384) beside two decoded
//     stages of 128 inputs (2 x 64): the epilogue of a pass runs on warps of its own under the next pass' decode and MMAs.
//     With gate and up accumulated together (one buffer of 2 x 192) the K loop stood still for the epilogue, a fifth of
//     an item's time, and ragged experts of 65 .. 96 rows paid for it most;
//   * 16 decode warps in two teams take the stages alternately (team = stage parity = operand slot).  A warp decodes its
//     8 tiles of a stage into registers and only then waits for its operand slot: the MMAs of the slot's last stage run
//     under the decode.  The stores go out four k-tiles at a time (16x256b.x4): a store costs the tensor-memory port about
//     the same whatever its width;
//   * the MMA warp runs its loop with all lanes and issues under elect.sync (see elect_one);
//   * one producer warp streams the code, one the rows' rotated f16 activations, which a prep kernel laid out as K-major
//     core matrices with fixed offsets (a row group's 128 inputs are 2 KB), so the MMA descriptors advance by constants;
//   * eight epilogue warps: tcgen05.ld, transpose through shared memory, then row-wise Hadamard-128.  The gate pass leaves
//     act(gate) per CTA in an L2-resident scratch that the same threads read back in the up pass.
// What bounds it: up to about 128 rows per tile the decode (48.5 issue cycles per tile and SM sub-partition, see
// exl3_probe.cu), above that the MMAs.
// Every wait is bounded; on a give-up the CTA sets the status word, skips work and still frees its tensor memory.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

// -DMLXS_LANE_COUNTERS: cycle counters around the waits, the decode and the MMA issue of one CTA, printed once per launch
// (how the lane's bound was found; off in the library)
#ifdef MLXS_LANE_COUNTERS
#include <cstdio>
#define LC(...) __VA_ARGS__
#else
#define LC(...)
#endif

namespace mlxs {

constexpr int PF_KST = 128;         // inputs per operand stage (8 k-tiles)
constexpr int PF_KT = PF_KST / 16;
constexpr int PF_A_COLS = PF_KST / 2;   // tensor-memory columns of a decoded stage
constexpr int PF_ROWS = 192;        // most rows of a tile
constexpr int PF_ACC_COLS = 192;    // columns of one accumulator buffer
constexpr int PF_RAW_STAGES = 4;    // stages of the code ring
constexpr int PF_B_STAGES = 3;      // stages of the rows' ring
constexpr int PF_DONE = 4;          // barriers of the stages in flight: operands complete, MMAs complete
constexpr int PF_EPI_ROWS = 32;     // rows per epilogue batch
constexpr int PF_ZS_STRIDE = 132;
constexpr int PF_DEC_WARPS = 16, PF_EPI_WARPS = 8;
constexpr int PF_THREADS = (PF_DEC_WARPS + PF_EPI_WARPS + 3) * 32;   // + code producer, MMA, rows' producer

// ------------------------------------------------------------------------------------------------------------
// plan: row tiles per expert from the dispatch tables
// ------------------------------------------------------------------------------------------------------------
// Tile table: [0] = tiles of list 0 (experts with up to cap0 rows: one tile each; with cap1 = 0 every expert, in tiles
// of up to cap0 rows), [1] = tiles of list 1 (the other experts, tiles of up to cap1 rows), then the entries {expert,
// first sorted row, rows, first staging row}: list 0 from entry 0, list 1 from entry max_tiles.  An expert's rows are
// split evenly over its tiles (a 16-row remainder tile would cost a full decode).
// Staging rows: a tile's rows padded to 16, tiles in sorted order, so tile number n starts at its first row + 16 n.
__global__ void pf_plan_kernel(DispatchTables t, uint32_t E, const uint8_t* __restrict__ flags, uint32_t min_rows,
                               uint32_t cap0, uint32_t cap1, uint32_t max_tiles, uint32_t* __restrict__ tiles,
                               uint32_t* status) {
    __shared__ uint32_t base0[1025], base1[1025];
    const uint32_t tid = threadIdx.x;
    // tiles per expert in parallel (base0 / base1 hold the counts first), then one thread turns them into offsets
    for (uint32_t e = tid; e < E; e += blockDim.x) {
        const uint32_t c = t.offsets[e + 1] - t.offsets[e];
        const bool lane = takes_tensor_lane(c, min_rows, flags, e), list1 = cap1 && c > cap0;
        base0[e] = lane && !list1 ? (c + cap0 - 1) / cap0 : 0u;
        base1[e] = lane && list1 ? (c + cap1 - 1) / cap1 : 0u;
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t n0 = 0, n1 = 0;
        for (uint32_t e = 0; e < E; ++e) {
            const uint32_t c0 = base0[e], c1 = base1[e];
            base0[e] = n0;
            base1[e] = n1;
            n0 += c0;
            n1 += c1;
        }
        if (n0 > max_tiles || n1 > max_tiles) { atomicMax(status, (uint32_t)ST_WORKLIST_OVERFLOW); n0 = 0; n1 = 0; }
        base0[E] = n0;
        base1[E] = n1;
        tiles[0] = n0;
        tiles[1] = n1;
    }
    __syncthreads();
    if (base0[E] + base1[E] == 0) return;
    for (uint32_t e = tid; e < E; e += blockDim.x) {
        const uint32_t c = t.offsets[e + 1] - t.offsets[e], r0 = t.offsets[e];
        if (!takes_tensor_lane(c, min_rows, flags, e)) continue;
        const bool list1 = cap1 && c > cap0;
        const uint32_t cap = list1 ? cap1 : cap0;
        const uint32_t nt = (c + cap - 1) / cap;
        const uint32_t per = ((c + nt - 1) / nt + 15) / 16 * 16;
        const uint32_t first = list1 ? base1[e] : base0[e], ordinal = base0[e] + base1[e];
        for (uint32_t i = 0; i < nt; ++i) {
            uint32_t* d = prefill_tile(tiles, list1 ? 1 : 0, max_tiles, first + i);
            d[0] = e; d[1] = r0 + i * per; d[2] = min(per, c - i * per); d[3] = r0 + i * per + 16 * (ordinal + i);
        }
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
// Staged rows of a tile with rows16 rows over `width` inputs, as K-major core matrices:
// [k / 128][row / 8][position / 8 of the 128][row % 8][position % 8]: a stage of 128 inputs is rows16 x 256 contiguous
// bytes, core matrices are 128 bytes apart along K and 2 KB along N.  The position of input k inside its 16-block is
// 4 ((k % 8) / 2) + 2 ((k % 16) / 8) + k % 2, the order in which the decode's registers fill a tensor-memory fragment.  A
// lane (t = lane / 4, c = lane % 4) that holds the inputs 16 t + {2c, 2c + 1, 2c + 8, 2c + 9} of a 128-block has the four
// consecutive positions 16 t + 4 c: one 8-byte store at this element offset inside the stage.
constexpr uint32_t PF_LBO = 128, PF_SBO = 2048;   // byte distance of two core matrices along K, along N
__device__ __forceinline__ uint32_t pf_lane_off(uint32_t row, uint32_t lane) {
    return (row >> 3) * 1024u + ((lane >> 2) * 2u + ((lane >> 1) & 1u)) * 64u + (row & 7u) * 8u + (lane & 1u) * 4u;
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
// rows of one 128-block: lane = (row, s), with the 32 inputs 32 j + 8 s + i (j < 4, i < 8).  Five of the transform's seven
// levels then stay in registers and two are shuffles (64 per eight rows; with four inputs per lane it was 160), four lanes
// read 64 contiguous bytes of a row, and the 16-byte stores fill whole lines of core matrices.
constexpr int PREP_WARPS = 8;
__global__ void __launch_bounds__(PREP_WARPS * 32, 3) pf_prep_kernel(const __nv_bfloat16* __restrict__ x, uint32_t top_k, uint32_t H,
                                                                  const __half* __restrict__ scales, size_t scales_stride,
                                                                  DispatchTables t, const uint32_t* __restrict__ tiles, uint32_t max_tiles,
                                                                  size_t proj_stride, __half* __restrict__ xa) {
    const uint32_t tile = blockIdx.x;
    if (tile >= tiles[0]) return;
    const uint32_t* te = prefill_tile(tiles, 0, max_tiles, tile);
    const uint32_t e = te[0], row0 = te[1], rows = te[2];
    const uint32_t rows16 = (rows + 15) / 16 * 16, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nblk = H / 128;
    const uint32_t r8 = lane >> 2, seg = lane & 3u;
    const float S = __uint_as_float(SCALE_BITS);
    const float sg0 = seg & 1u ? -1.0f : 1.0f, sg1 = seg & 2u ? -1.0f : 1.0f;
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
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = __fmaf_rn(sg0, v[k], __shfl_xor_sync(0xFFFFFFFFu, v[k], 1));
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = __fmaf_rn(sg1, v[k], __shfl_xor_sync(0xFFFFFFFFu, v[k], 2));
            level_reg(8); level_reg(16);
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] *= S;
            // src/kernels/exl3/dsv41_prefill_dig_take2v_5120.metal:57-58: the rotated input is rounded to f16
            __half* dst = xa + p * proj_stride + (size_t)te[3] * H + (size_t)b * (rows16 * PF_KST) + (r >> 3) * 1024u + (r & 7u) * 8u;
            // 16-block 2 j + s / 2: an even lane holds its inputs 0 .. 7, the odd one 8 .. 15; the block's first core matrix
            // takes {0, 1, 8, 9, 2, 3, 10, 11}, its second the others, so the two lanes swap half of theirs
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint2 a = pf_pack4(v[8 * j], v[8 * j + 1], v[8 * j + 2], v[8 * j + 3]), c = pf_pack4(v[8 * j + 4], v[8 * j + 5], v[8 * j + 6], v[8 * j + 7]);
                const bool odd = seg & 1u;
                const uint32_t g0 = __shfl_xor_sync(0xFFFFFFFFu, odd ? a.x : c.x, 1), g1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? a.y : c.y, 1);
                *reinterpret_cast<uint4*>(dst + (4 * j + seg) * 64) = odd ? make_uint4(g0, c.x, g1, c.y) : make_uint4(a.x, g0, a.y, g1);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// the kernel
// ------------------------------------------------------------------------------------------------------------
struct PfParams {
    const uint32_t* code;        // layer base of the block stream (8 tiles of 8 K words per k-tile; gate's k-tiles, then up's)
    size_t expert_stride_words;
    uint32_t n_blocks, nkt;      // out / 128, in / 16
    const __half* xa;            // B operand: [projection][staging rows][in]
    size_t xa_proj_stride;       // elements between the projections' staged rows
    const uint32_t* tiles;
    uint32_t max_tiles;
    DispatchTables t;
    const __half* scales;
    size_t scales_stride;
    uint32_t H, I;
    float* act;                  // gate/up: [CTA][192 rows][128] act(gate) between the two passes
    __half* xd;                  // gate/up output = down's B operand, [staging rows][I]
    float* ro;                   // down output [A, H]
    float limit;
    uint32_t* status;
};

__device__ __forceinline__ void tmem_st_16x256_x4(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// NPASS = 2: gate then up of a column block; 1: down.  KB = bits per weight.
template <int NPASS, int KB>
__global__ void __launch_bounds__(PF_THREADS, 1) exl3_prefill_kernel(const PfParams P) {
    constexpr uint32_t TW = 8 * KB;                    // words per 16x16 tile
    constexpr uint32_t KT_WORDS = 8 * TW;              // words per k-tile of a block
    constexpr uint32_t RAW_BYTES = PF_KT * KT_WORDS * 4;
    constexpr uint32_t B_SLOT = PF_ROWS * PF_KST * 2;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t raw_full[PF_RAW_STAGES], raw_empty[PF_RAW_STAGES];
    __shared__ __align__(8) uint64_t full[PF_DONE], done[PF_DONE], acc_full[2], acc_empty[2], epi_bar;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    uint8_t* b_ring = smem_raw;                                          // [stage][rows16 x 256 B]
    uint8_t* raw_ring = b_ring + PF_B_STAGES * B_SLOT;                   // [stage][k-tile][8 tiles]
    float* zs = reinterpret_cast<float*>(raw_ring + PF_RAW_STAGES * RAW_BYTES);   // [2][32 rows][stride]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t n_items = P.tiles[0] * P.n_blocks;
    // a CTA without work leaves before it takes tensor memory (the whole CTA reads the same count)
    if (blockIdx.x >= n_items) return;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PF_RAW_STAGES; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 8); }
        // a stage's operands: the team's warps have stored theirs, the rows have landed
        for (int s = 0; s < PF_DONE; ++s) { mbar_init(&full[s], 8 + 1); mbar_init(&done[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], PF_EPI_WARPS); }
        mbar_init(&epi_bar, PF_EPI_WARPS);
        s_abort = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem, tmem_a = tmem + 2 * PF_ACC_COLS;
    const uint32_t nstage = P.nkt / PF_KT, width = P.nkt * 16;
    const uint32_t my_items = (n_items - blockIdx.x + gridDim.x - 1) / gridDim.x;
    const uint32_t my_stages = my_items * NPASS * nstage;   // stages are numbered through over all passes of the CTA
    auto give_up = [&](uint32_t code) { if (!s_abort) atomicMax(P.status, code); s_abort = 1; };
    // item number i of this CTA -> its tile entry {expert, first sorted row, rows, first staging row} and column block
    auto item_tile = [&](uint32_t i, uint32_t& nb) {
        const uint32_t item = blockIdx.x + i * gridDim.x;
        nb = item % P.n_blocks;
        return prefill_tile(P.tiles, 0, P.max_tiles, item / P.n_blocks);
    };

    if (warp < PF_DEC_WARPS) {
        // ---------------- decode warps: (lane quarter q, half of the stage's k-tiles, team) ----------------
        const uint32_t q = warp & 3u, half = (warp >> 2) & 1u, team = warp >> 3;
        uint32_t wi, wj, lp;
        exl3_lane_plan_kb<KB>(lane, wi, wj, lp);
        const uint32_t* wt0 = reinterpret_cast<const uint32_t*>(raw_ring + team * RAW_BYTES) + half * (PF_KT / 2) * KT_WORDS + 2 * q * TW;
        const uint32_t *tw_i = wt0 + wi, *tw_j = wt0 + wj;
        const uint32_t ta = tmem_a + ((q * 32u) << 16) + team * PF_A_COLS + half * (PF_A_COLS / 2);
        // The team's stages are g = team + 2 i: code slot and barriers alternate between team and team + 2, their phases flip
        // every second stage.  The instructions around the decode count (it is issue-bound), so the addresses advance by an
        // exclusive-or, and the tests of the two barriers that come next (the operand slot, the next stage's code) go out
        // together: a test of a barrier that is ready costs its latency.
        const uint32_t n_i = (my_stages - team + 1) / 2;
        uint32_t b_raw = smem_u32(&raw_full[team]), b_emp = smem_u32(&raw_empty[team]), b_done = smem_u32(&done[team + 2]), b_full = smem_u32(&full[team]);
        const uint32_t x_raw = b_raw ^ smem_u32(&raw_full[team + 2]), x_emp = b_emp ^ smem_u32(&raw_empty[team + 2]),
                       x_done = b_done ^ smem_u32(&done[team]), x_full = b_full ^ smem_u32(&full[team + 2]);
        bool code_ready = false;
        uint32_t i = 0, woff = 0;
        LC(const long long c0 = clock64();)
        for (; i < n_i; ++i) {
            const uint32_t ph = (i >> 1) & 1u;             // phase of this stage's code barrier
            if (!code_ready && !mbar_wait_bounded_at(b_raw, ph, &s_abort)) { give_up(ST_WAIT_FULL); break; }
            uint32_t v[2][16];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                for (int kt = 0; kt < PF_KT / 2; ++kt) {
                    uint32_t bq[4];
                    exl3_decode_lane_kb<KB>(tw_i[woff + kt * KT_WORDS + jj * TW], tw_j[woff + kt * KT_WORDS + jj * TW], lp, bq);
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[jj][kt * 4 + k] = bq[k];
                }
            // this slot's last MMAs are stage g - 2's: barrier team + 2 ((i - 1) % 2), phase ((i - 1) / 2) % 2
            const uint32_t ph_done = ((i + 1) >> 1 & 1u) ^ 1u;
            const bool slot_ready = i == 0 || mbar_try_wait_at(b_done, ph_done);
            b_raw ^= x_raw;
            code_ready = mbar_try_wait_at(b_raw, ((i + 1) >> 1) & 1u);
            if (lane == 0) mbar_arrive_at(b_emp);
            if (!slot_ready && !mbar_wait_bounded_at(b_done, ph_done, &s_abort)) { give_up(ST_WAIT_EMPTY); break; }
            tc_fence_after();
            tmem_st_16x256_x4(ta, v[0]);
            tmem_st_16x256_x4(ta + (16u << 16), v[1]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_at(b_full);
            b_emp ^= x_emp; b_done ^= x_done; b_full ^= x_full; woff ^= 2 * RAW_BYTES / 4;
        }
        LC(if (blockIdx.x == 3 && lane == 0 && warp == 9) printf("LANE<%d> decode warp: %u half stages of %u, cycles per stage: %lld\n", NPASS, n_i, 2 * my_stages, (clock64() - c0) / my_stages);)
    } else if (warp < PF_DEC_WARPS + PF_EPI_WARPS) {
        // ---------------- epilogue warps ----------------
        const uint32_t ew = warp - PF_DEC_WARPS, q = warp & 3u, half = ew >> 2;
        const float S = __uint_as_float(SCALE_BITS);
        float sg[5];
        pf_signs(lane, sg);
        float* act = P.act + ((size_t)blockIdx.x * PF_ROWS) * 128 + lane * 4;
        uint32_t pass_n = 0, epi_ph = 0, batch = 0;
        auto epi_sync = [&]() -> bool {
            __syncwarp();
            if (lane == 0) mbar_arrive(&epi_bar);
            const bool ok = mbar_wait_bounded(&epi_bar, epi_ph, &s_abort);
            epi_ph ^= 1u;
            if (!ok) give_up(ST_WAIT_FULL);
            return ok;
        };
        LC(long long t_wait = 0, t_epi = 0;)
        bool ok = true;
        for (uint32_t it = 0; it < my_items && ok; ++it) {
            uint32_t nb;
            const uint32_t* te = item_tile(it, nb);
            const uint32_t expert = te[0], row0 = te[1], rows = te[2], srow0 = te[3];
            const uint32_t rows16 = (rows + 15) / 16 * 16;
            const __half* sc = P.scales + (size_t)expert * P.scales_stride + 2 * (size_t)P.H + nb * 128;   // svh_g | svh_u | suh_d [I], svh_d [H]
#pragma unroll
            for (int p = 0; p < NPASS && ok; ++p, ++pass_n) {
                const uint32_t buf = pass_n & 1u;
                float svh[4], shd[4] = {0.f, 0.f, 0.f, 0.f};
                if (NPASS == 2) {
                    pf_load_scale4(sc + (p ? P.I : 0u), lane, svh);
                    if (p == 1) pf_load_scale4(sc + 2 * (size_t)P.I, lane, shd);
                } else {
                    const uint2 s0 = *reinterpret_cast<const uint2*>(sc + 3 * (size_t)P.I + lane * 4);
                    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&s0.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&s0.y));
                    svh[0] = a.x; svh[1] = a.y; svh[2] = b.x; svh[3] = b.y;
                }
                LC(const long long e0 = clock64();)
                if (!mbar_wait_bounded(&acc_full[buf], (pass_n >> 1) & 1u, &s_abort, 200)) { give_up(ST_WAIT_FULL); ok = false; break; }
                tc_fence_after();
                LC(const long long e1 = clock64(); t_wait += e1 - e0;)
                for (uint32_t rb = 0; rb < rows16; rb += PF_EPI_ROWS, ++batch) {
                    float* z = zs + (batch & 1u) * (PF_EPI_ROWS * PF_ZS_STRIDE);
                    if (rb + half * 16 < rows16) {
                        uint32_t v[16];
                        tmem_ld16(tmem + ((q * 32u) << 16) + buf * PF_ACC_COLS + rb + half * 16, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) z[(half * 16 + i) * PF_ZS_STRIDE + q * 32 + lane] = __uint_as_float(v[i]);
                    }
                    if (rb + PF_EPI_ROWS >= rows16) {   // the last read of this accumulator buffer
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acc_empty[buf]);
                    }
                    // one rendezvous per batch: a staging buffer is written again two batches later, after the next one
                    if (!epi_sync()) { ok = false; break; }
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
                            __half* xd = P.xd + (size_t)srow0 * P.I + (size_t)nb * (rows16 * PF_KST);
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                *reinterpret_cast<uint2*>(xd + pf_lane_off(r + i, lane)) = pf_pack4(h[i][0] * S, h[i][1] * S, h[i][2] * S, h[i][3] * S);
                        } else {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                if (r + i >= rows) continue;
                                const uint32_t assign = P.t.order[row0 + r + i];
                                *reinterpret_cast<float4*>(P.ro + (size_t)assign * P.H + nb * 128 + lane * 4) =
                                    make_float4((v[i][0] * S) * svh[0], (v[i][1] * S) * svh[1], (v[i][2] * S) * svh[2], (v[i][3] * S) * svh[3]);
                            }
                        }
                    }
                }
                LC(t_epi += clock64() - e1;)
            }
        }
        LC(if (blockIdx.x == 3 && lane == 0 && ew == 1) printf("LANE<%d> epilogue: %u passes, cycles per pass: wait %lld work %lld\n", NPASS, pass_n, t_wait / pass_n, t_epi / pass_n);)
    } else if (warp == PF_DEC_WARPS + PF_EPI_WARPS) {
        // ---------------- code producer ----------------
        if (lane == 0) {
            uint32_t g = 0;
            for (uint32_t it = 0; it < my_items && !s_abort; ++it) {
                uint32_t nb;
                const uint32_t* te = item_tile(it, nb);
                // the passes' k-tiles follow each other in the stream
                const uint32_t* wsrc = P.code + (size_t)te[0] * P.expert_stride_words + (size_t)nb * NPASS * P.nkt * KT_WORDS;
                for (uint32_t ks = 0; ks < NPASS * nstage; ++ks, ++g) {
                    const uint32_t rs = g % PF_RAW_STAGES;
                    if (!mbar_wait_bounded(&raw_empty[rs], ((g / PF_RAW_STAGES) & 1u) ^ 1u, &s_abort, 64)) { give_up(ST_WAIT_EMPTY); break; }
                    mbar_expect_tx(&raw_full[rs], RAW_BYTES);
                    bulk_g2s(raw_ring + rs * RAW_BYTES, wsrc + (size_t)ks * (PF_KT * KT_WORDS), RAW_BYTES, &raw_full[rs]);
                }
            }
            if (s_abort) for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
    } else if (warp == PF_DEC_WARPS + PF_EPI_WARPS + 1) {
        // ---------------- MMA issuer: the whole warp walks the loop, one elected lane issues ----------------
        uint32_t g = 0, bs = 0, pass_n = 0;
        const uint64_t bdesc = umma_smem_desc(smem_u32(b_ring), PF_LBO, PF_SBO);
        const uint32_t bd_lo0 = (uint32_t)bdesc, bd_hi = (uint32_t)(bdesc >> 32);
        bool ok = true;
        LC(long long m_a = 0, m_issue = 0;)
        for (uint32_t it = 0; it < my_items && ok; ++it) {
            uint32_t nb;
            const uint32_t idesc = umma_idesc(UMMA_F16, (item_tile(it, nb)[2] + 15) / 16 * 16);
            for (int p = 0; p < NPASS && ok; ++p, ++pass_n) {
                const uint32_t buf = pass_n & 1u, acc = tmem + buf * PF_ACC_COLS;
                if (!mbar_wait_warp(&acc_empty[buf], ((pass_n >> 1) & 1u) ^ 1u, &s_abort)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
                for (uint32_t ks = 0; ks < nstage; ++ks, ++g) {
                    LC(const long long w1 = clock64();)
                    if (!mbar_wait_warp(&full[g % PF_DONE], (g / PF_DONE) & 1u, &s_abort)) { give_up(ST_WAIT_FULL); ok = false; break; }
                    tc_fence_after();
                    LC(const long long w2 = clock64();)
                    if (elect_one()) {
                        const uint32_t a0 = tmem_a + (g & 1u) * PF_A_COLS, bd_lo = bd_lo0 + bs * (B_SLOT >> 4);
                        umma_f16_ts_lohi(acc, a0, bd_lo, bd_hi, idesc, ks);
#pragma unroll
                        for (int i = 1; i < PF_KT; ++i) umma_f16_ts_lohi(acc, a0 + i * 8, bd_lo + ((i * 2 * PF_LBO) >> 4), bd_hi, idesc, 1u);
                        // one commit per stage frees the operand slot and the rows' slot
                        umma_commit(&done[g % PF_DONE]);
                        if (ks + 1 == nstage) umma_commit(&acc_full[buf]);
                    }
                    __syncwarp();
                    if (++bs == PF_B_STAGES) bs = 0;
                    LC(m_a += w2 - w1; m_issue += clock64() - w2;)
                }
            }
        }
        LC(if (blockIdx.x == 3 && g && lane == 0) printf("LANE<%d> mma warp: %u stages, cycles per stage: operand wait %lld issue %lld\n", NPASS, g, m_a / g, m_issue / g);)
    } else {
        // ---------------- rows' producer ----------------
        if (lane == 0) {
            uint32_t g = 0, bs = 0;
            for (uint32_t it = 0; it < my_items && !s_abort; ++it) {
                uint32_t nb;
                const uint32_t* te = item_tile(it, nb);
                const uint32_t rows16 = (te[2] + 15) / 16 * 16, b_bytes = rows16 * PF_KST * 2;
                for (int p = 0; p < NPASS; ++p) {
                    const __half* xsrc = P.xa + p * P.xa_proj_stride + (size_t)te[3] * width;
                    for (uint32_t ks = 0; ks < nstage; ++ks, ++g) {
                        if (g >= PF_B_STAGES) {
                            const uint32_t d = g - PF_B_STAGES;
                            if (!mbar_wait_bounded(&done[d % PF_DONE], (d / PF_DONE) & 1u, &s_abort, 64)) { give_up(ST_WAIT_EMPTY); break; }
                        }
                        mbar_expect_tx(&full[g % PF_DONE], b_bytes);
                        bulk_g2s(b_ring + bs * B_SLOT, xsrc + (size_t)ks * (rows16 * PF_KST), b_bytes, &full[g % PF_DONE]);
                        if (++bs == PF_B_STAGES) bs = 0;
                    }
                }
            }
            if (s_abort) for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
    }
    // every thread comes here, also after a give-up: the tensor memory is always released
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(tmem, 512);
}

bool exl3_prefill_supported(Exl3Dims d) { return d.I % PF_KST == 0 && d.H % PF_KST == 0; }

size_t exl3_prefill_act_bytes(int sm_count) { return (size_t)sm_count * PF_ROWS * 128 * sizeof(float); }

cudaError_t launch_prefill_plan(DispatchTables t, uint32_t n_experts, const uint8_t* lane_flags, uint32_t min_rows,
                                uint32_t cap0, uint32_t cap1, uint32_t max_tiles, uint32_t* tiles, uint32_t* status,
                                cudaStream_t st) {
    pf_plan_kernel<<<1, 256, 0, st>>>(t, n_experts, lane_flags, min_rows, cap0, cap1, max_tiles, tiles, status);
    return cudaGetLastError();
}

template <int NPASS, int KB>
static cudaError_t pf_launch(const PfParams& P, int sm_count, cudaStream_t st) {
    const size_t smem = (size_t)PF_B_STAGES * PF_ROWS * PF_KST * 2 + (size_t)PF_RAW_STAGES * PF_KT * 64 * KB * 4 + 2 * PF_EPI_ROWS * PF_ZS_STRIDE * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(exl3_prefill_kernel<NPASS, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    exl3_prefill_kernel<NPASS, KB><<<sm_count, PF_THREADS, smem, st>>>(P);
    return cudaGetLastError();
}

template <int KB>
static cudaError_t pf_launch_all(const Exl3PrefillArgs& a, cudaStream_t st) {
    PfParams P{};
    P.tiles = a.tiles; P.max_tiles = a.max_tiles; P.t = a.t; P.scales = a.L.scales; P.scales_stride = exl3_scales_per_expert(a.d);
    P.H = a.d.H; P.I = a.d.I; P.limit = a.limit; P.status = a.status; P.act = a.act;
    P.code = a.L.gu_code; P.expert_stride_words = 2 * exl3_code_words(a.d); P.n_blocks = a.d.I / 128; P.nkt = a.d.H / 16;
    P.xa = a.xa; P.xa_proj_stride = exl3_prefill_staging_rows(a.rows_cap, a.max_tiles) * a.d.H; P.xd = a.xd; P.ro = nullptr;
    const cudaError_t e = pf_launch<2, KB>(P, a.sm_count, st);
    if (e != cudaSuccess) return e;
    P.code = a.L.d_code; P.expert_stride_words = exl3_code_words(a.d); P.n_blocks = a.d.H / 128; P.nkt = a.d.I / 16;
    P.xa = a.xd; P.xa_proj_stride = 0; P.xd = nullptr; P.ro = a.ro;
    return pf_launch<1, KB>(P, a.sm_count, st);
}

cudaError_t launch_exl3_prefill(const Exl3PrefillArgs& a, cudaStream_t st) {
    cudaError_t e = launch_prefill_plan(a.t, a.n_experts, nullptr, a.min_rows, PF_ROWS, 0, a.max_tiles, a.tiles, a.status, st);
    if (e != cudaSuccess) return e;
    pf_prep_kernel<<<dim3(a.max_tiles, 8), PREP_WARPS * 32, 0, st>>>(a.x, a.top_k, a.d.H, a.L.scales, exl3_scales_per_expert(a.d), a.t,
                                                                  a.tiles, a.max_tiles,
                                                                  exl3_prefill_staging_rows(a.rows_cap, a.max_tiles) * a.d.H, a.xa);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return a.d.K == 3 ? pf_launch_all<3>(a, st) : pf_launch_all<2>(a, st);
}

}  // namespace mlxs
