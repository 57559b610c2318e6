// Dense bf16 products on the tcgen05 tensor cores: the shared expert's three linears and the router's logits.
//
// The shared expert (src/arch/deepseek_v41/graph.zig:2162-2172) is h = silu(min(w1 x, lim)) * clip(w3 x, +-lim),
// out = w2 h; the router's logits are f32(x) . W_g^T (graph.zig:2033).  All of them are C[T, N] = X[T, K] . W[N, K]^T
// with bf16 operands and f32 accumulation.  As in the expert lanes W is the MMA's A operand (M = 128 output features per
// accumulator group) and the token rows are the B operand (N = up to 256 rows, rounded to 16): a ragged last tile pads
// to 16 rows, and the epilogue's stores run along the feature dimension.
//   * weights are re-tiled once at load into K-major core matrices, [feature block of 128][k stage of 64][8-row group]
//     ([projection] for gate / up) [8-k group][8 rows x 8 k]: one (block, stage) is one contiguous run for a bulk copy,
//     gate and up of the same block travel together;
//   * rows are staged once per call in the same core-matrix order (dense_rows_kernel); the gate/up epilogue writes h
//     straight into that order for the down product;
//   * a CTA owns (token tile, feature block) with two accumulator groups in tensor memory (gate and up of one block,
//     or two adjacent blocks of a single projection): 2 x 256 columns = all 512;
//   * one producer thread (bulk copies into a ring, mbarriers), one MMA thread (tcgen05.mma.kind::f16 on bf16,
//     K = 16 per instruction, commits free the stage), eight epilogue warps (tcgen05.ld, activation, stores);
//   * calls with few tokens split the reduction into parts (dg_parts): every part is summed by itself and the parts are added
//     in part order, so a sum's bits depend on the part count alone, which is the same for all calls of up to 256 tokens: a
//     row's bits do not depend on the batch around it.  How the parts are spread is free (dg_cost): one CTA takes them in turn
//     with tiles of up to 64 rows, the epilogue warps adding each to their registers under the next part's MMAs; or the CTAs of
//     a cluster leave their parts' f32 tiles in their own shared memory and every CTA folds a slice of the rows over the
//     cluster.  With one CTA folding all parts out of global scratch the fold was most of the time: gate/up at 300 tokens
//     90 us for 42 MB of weights.
// Every wait is bounded; on a give-up the CTA records the status word, skips its work and still frees tensor memory.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace mlxs {

constexpr int DG_KS = 64;                         // inputs per stage
constexpr int DG_NT = 256;                        // most rows per token tile (MMA N)
constexpr int DG_CL_NT = 192;                     // most rows x parts of a CTA in a cluster: the partial tiles have to fit the ring's shared memory
constexpr int DG_CL_MAX = 8;                      // most CTAs of a cluster
constexpr int DG_FOLD_NT = 64;                    // most rows of a tile whose parts one CTA takes in turn: 64 sums per epilogue thread
constexpr int DG_STAGES = 6;                      // most ring stages
constexpr int DG_RING = 192 * 1024;               // ring bytes: 3 stages at 256 rows
constexpr int DG_A_TILE = 128 * DG_KS * 2;        // one projection's (block, stage): 16 KB
constexpr int DG_A_STAGE = 2 * DG_A_TILE;         // two accumulator groups' weights
constexpr int DG_EPI_WARPS = 8;

// ---- load-time re-tiling of a weight matrix W[n_out, K] (row-major bf16) ----
// np = 2: w0 and w1 interleaved per 8-row group ([rc][p][kc][8][8]); np = 1: w0 alone ([rc][kc][8][8])
__global__ void dense_retile_kernel(const __nv_bfloat16* __restrict__ w0, const __nv_bfloat16* __restrict__ w1, uint32_t n_out,
                                    uint32_t K, int np, uint4* __restrict__ dst) {
    const size_t n_vec = (size_t)np * n_out * K / 8;
    const uint32_t nks = K / DG_KS;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += (size_t)gridDim.x * blockDim.x) {
        size_t r = i;
        const uint32_t r8 = r % 8; r /= 8;
        const uint32_t kc = r % 8; r /= 8;
        const uint32_t p = np == 2 ? (uint32_t)(r % 2) : 0u; if (np == 2) r /= 2;
        const uint32_t rc = r % 16; r /= 16;
        const uint32_t ks = r % nks; r /= nks;
        const uint32_t nb = (uint32_t)r;
        const __nv_bfloat16* src = (p ? w1 : w0) + (size_t)(nb * 128 + rc * 8 + r8) * K + (size_t)ks * DG_KS + kc * 8;
        dst[i] = *reinterpret_cast<const uint4*>(src);
    }
}

cudaError_t launch_dense_retile(const __nv_bfloat16* w0, const __nv_bfloat16* w1, uint32_t n_out, uint32_t K, void* dst,
                                cudaStream_t st) {
    if (n_out % (w1 ? 128 : 256) || K % DG_KS) return cudaErrorInvalidValue;
    dense_retile_kernel<<<592, 256, 0, st>>>(w0, w1, n_out, K, w1 ? 2 : 1, static_cast<uint4*>(dst));
    return cudaGetLastError();
}

// ---- rows -> B-operand order ----
// element offset of (row r of tile tt, input k): tiles of nt rows, those before tt are full
__host__ __device__ inline size_t dg_b_off(uint32_t K, uint32_t nt, uint32_t tt, uint32_t rows16, uint32_t r, uint32_t k) {
    return (size_t)tt * nt * K + (size_t)(k / DG_KS) * (rows16 * DG_KS) + (size_t)((k % DG_KS) / 8) * (rows16 * 8) +
           (r / 8) * 64 + (r % 8) * 8 + k % 8;
}
// a warp moves 32 consecutive inputs of eight rows at a time: four lanes read 64 bytes of a row, eight lanes write one core matrix
__global__ void __launch_bounds__(256) dense_rows_kernel(const __nv_bfloat16* __restrict__ x, uint32_t T, uint32_t K, uint32_t nt,
                                                         uint16_t* __restrict__ xb) {
    const uint32_t warp = blockIdx.x * 8 + (threadIdx.x >> 5), n_warps = gridDim.x * 8, lane = threadIdx.x & 31u;
    const uint32_t kq = K / 32, n_tasks = (T + 7) / 8 * kq;
    for (uint32_t task = warp; task < n_tasks; task += n_warps) {
        const uint32_t row = task / kq * 8 + (lane >> 2), k = (task % kq) * 32 + (lane & 3u) * 8;
        const uint32_t tt = row / nt, rows16 = (min(nt, T - tt * nt) + 15) / 16 * 16;
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (row < T) raw = *reinterpret_cast<const uint4*>(x + (size_t)row * K + k);
        *reinterpret_cast<uint4*>(xb + dg_b_off(K, nt, tt, rows16, row - tt * nt, k)) = raw;
        // the last tile's padding to 16 rows
        if (row >= (T + 7) / 8 * 8 - 8 && (row - tt * nt) / 8 % 2 == 0)
            *reinterpret_cast<uint4*>(xb + dg_b_off(K, nt, tt, rows16, row - tt * nt + 8, k)) = make_uint4(0, 0, 0, 0);
    }
}

struct DenseParams {
    const uint8_t* w;          // re-tiled weights
    uint32_t n_blocks;         // output features / 128
    uint32_t n_ks;             // K / 64
    const uint16_t* xb;        // rows in B-operand order
    uint32_t T, K;
    float limit;
    uint16_t* hb;              // gate/up: h in B-operand order over n_out inputs
    float* out;                // plain: [T, n_out] f32
    uint32_t n_out;
    bool out_vec;              // out is 16-byte aligned (the caller's logits need only 4)
    uint32_t nt;               // rows per token tile (a multiple of 16)
    uint32_t n_stages;         // ring stages
    uint32_t k_parts;          // parts of the reduction, each summed by itself
    uint32_t n_cl;             // CTAs of a cluster that share an item's parts (1: no cluster)
    uint32_t* status;
    uint32_t poll_limit;
};

__device__ __forceinline__ float dg_act(float gate, float up, float limit) {
    if (limit > 0.f) {
        gate = (gate != gate) ? gate : (gate < limit ? gate : limit);
        up = (up != up) ? up : (up > limit ? limit : (up < -limit ? -limit : up));
    }
    const float yv = sigmoid_tail_fast(gate);
    const float sg = gate < 0.f ? yv : 1.0f - yv;
    return (gate * sg) * up;
}
// all threads of the cluster's CTAs; what was written to shared memory before is seen by the others after
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t saddr, uint32_t rank) {
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(saddr), "r"(rank));
    return d;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// NPROJ = 2: gate and up of one feature block (activation epilogue -> hb); NPROJ = 1: two adjacent blocks -> out.
// MODE: how an item's parts are spread
constexpr int DG_WHOLE = 0;     // one part; a CTA walks items
constexpr int DG_FOLD = 1;      // a CTA walks items and takes their parts in turn
constexpr int DG_CLUSTER = 2;   // a cluster of n_cl CTAs per item, an even share of its parts each
template <int NPROJ, int MODE>
__global__ void __launch_bounds__(64 + DG_EPI_WARPS * 32, 1) dense_gemm_kernel(const DenseParams P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[DG_STAGES], empty_bar[DG_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    uint8_t* a_ring = smem_raw;                              // [stage][2 groups' tiles]
    uint8_t* b_ring = smem_raw + P.n_stages * DG_A_STAGE;    // [stage][rows16 x 64]
    const uint32_t NT = P.nt, b_stage = NT * DG_KS * 2, NS = P.n_stages;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t n_tt = (P.T + NT - 1) / NT;
    const uint32_t n_fb = NPROJ == 2 ? P.n_blocks : P.n_blocks / 2;     // feature-block groups
    constexpr bool CL = MODE == DG_CLUSTER;
    const uint32_t KP = MODE == DG_WHOLE ? 1u : P.k_parts, NCL = CL ? P.n_cl : 1u;
    const uint32_t n_units = n_tt * n_fb * NCL;
    if (blockIdx.x >= n_units) return;   // before any tensor memory is taken (the whole CTA reads the same count)

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < NS; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], DG_EPI_WARPS); }
        s_abort = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    // part p of the reduction covers stages [p n_ks / KP, (p + 1) n_ks / KP): a function of the shape and the part count
    auto part_begin = [&](uint32_t part) { return (uint32_t)(((uint64_t)part * P.n_ks) / KP); };
    auto give_up = [&](uint32_t code) { if (!s_abort) atomicMax(P.status, code); s_abort = 1; };
    // This CTA's parts: [part0, part1).  In a cluster all of them stay in tensor memory, number l in the columns from 2 l NT;
    // otherwise they alternate between two buffers of 2 NT columns (one where only one fits)
    const uint32_t n_buf = !CL && NT <= 128u ? 2u : 1u;
    auto cl_part = [&](uint32_t rank) { return rank * KP / NCL; };
    const uint32_t cl_rank = CL ? blockIdx.x % NCL : 0u, part0 = cl_part(cl_rank), part1 = cl_part(cl_rank + 1), n_parts = part1 - part0;
    // unit -> (token tile, feature-block group); feature blocks vary fastest so that the CTAs running together share the
    // rows of a few token tiles and the weights in L2
    auto decode_unit = [&](uint32_t unit, uint32_t& tt, uint32_t& fb) {
        const uint32_t item = unit / NCL;
        fb = item % n_fb;
        tt = item / n_fb;
    };

    if (warp == 0) {
        // ---------------- producer ----------------
        if (lane == 0) {
            uint32_t s = 0, ph = 0;
            for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x) {
                uint32_t tt, fb;
                decode_unit(unit, tt, fb);
                const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
                const uint32_t b_bytes = rows16 * DG_KS * 2;
                const uint16_t* xsrc = P.xb + (size_t)tt * NT * P.K;
                bool ok = true;
                for (uint32_t ks = part_begin(part0); ks < part_begin(part1); ++ks) {
                    if (!mbar_wait_bounded(&empty_bar[s], ph ^ 1u, &s_abort, 64, P.poll_limit)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
                    mbar_expect_tx(&full_bar[s], DG_A_STAGE + b_bytes);
                    if (NPROJ == 2) {
                        bulk_g2s(a_ring + s * DG_A_STAGE, P.w + ((size_t)fb * P.n_ks + ks) * DG_A_STAGE, DG_A_STAGE, &full_bar[s]);
                    } else {
                        bulk_g2s(a_ring + s * DG_A_STAGE, P.w + ((size_t)(2 * fb) * P.n_ks + ks) * DG_A_TILE, DG_A_TILE, &full_bar[s]);
                        bulk_g2s(a_ring + s * DG_A_STAGE + DG_A_TILE, P.w + ((size_t)(2 * fb + 1) * P.n_ks + ks) * DG_A_TILE, DG_A_TILE, &full_bar[s]);
                    }
                    bulk_g2s(b_ring + s * b_stage, xsrc + (size_t)ks * (rows16 * DG_KS), b_bytes, &full_bar[s]);
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
            }
            if (s_abort) for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            uint32_t s = 0, ph = 0, n_done = 0;
            const uint32_t a_s = smem_u32(a_ring), b_s = smem_u32(b_ring);
            // gate / up interleave per 8-row group: a projection's core matrices of one K group are 2 KB apart
            constexpr uint32_t A_SBO = NPROJ == 2 ? 2048u : 1024u, A_LBO = 128u, A_GROUP = NPROJ == 2 ? 1024u : (uint32_t)DG_A_TILE;
            for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x) {
                uint32_t tt, fb;
                decode_unit(unit, tt, fb);
                const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
                const uint32_t idesc = umma_idesc(UMMA_BF16, rows16), lbo_b = rows16 * 16;
                bool ok = true;
                for (uint32_t part = part0; part < part1 && ok; ++part) {
                    const uint32_t buf = n_done % n_buf, acc = tmem + (CL ? part - part0 : buf) * 2 * NT;
                    if (!CL && !mbar_wait_bounded(&acc_empty[buf], (n_done / n_buf & 1u) ^ 1u, &s_abort, 64, P.poll_limit)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
                    tc_fence_after();
                    const uint32_t ks0 = part_begin(part), ks1 = part_begin(part + 1);
                    for (uint32_t ks = ks0; ks < ks1; ++ks) {
                        if (!mbar_wait_bounded(&full_bar[s], ph, &s_abort, 0, P.poll_limit)) { give_up(ST_WAIT_FULL); ok = false; break; }
                        tc_fence_after();
                        const uint32_t a0 = a_s + s * DG_A_STAGE, b0 = b_s + s * b_stage;
#pragma unroll
                        for (int gq = 0; gq < 2; ++gq) {
#pragma unroll
                            for (int i = 0; i < DG_KS / 16; ++i)
                                umma_f16(acc + gq * NT, umma_smem_desc(a0 + gq * A_GROUP + i * 2 * A_LBO, A_LBO, A_SBO),
                                         umma_smem_desc(b0 + i * 2 * lbo_b, lbo_b, 128), idesc, ks != ks0 || i ? 1u : 0u);
                        }
                        umma_commit(&empty_bar[s]);
                        if (++s == NS) { s = 0; ph ^= 1u; }
                    }
                    if (ok && (!CL || part + 1 == part1)) { umma_commit(&acc_full[buf]); ++n_done; }
                }
                if (!ok) break;
            }
        }
    } else {
        // ---------------- epilogue warps ----------------
        // warp = (lane quarter q, half): a thread owns output feature 32 q + lane of both groups; the 16-row chunks of
        // the tile alternate between the two halves
        const uint32_t ew = warp - 2, q = warp & 3u, half = ew >> 2;
        uint32_t n_done = 0;
        const uint32_t fl = q * 32u + lane;                     // feature inside the block
        auto wait_acc = [&](uint32_t buf) -> bool {
            if (!mbar_wait_bounded(&acc_full[buf], n_done / n_buf & 1u, &s_abort, 0, P.poll_limit)) { give_up(ST_WAIT_FULL); return false; }
            tc_fence_after();
            return true;
        };
        auto release_acc = [&](uint32_t buf) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            ++n_done;
        };
        for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x) {
            uint32_t tt, fb;
            decode_unit(unit, tt, fb);
            const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16, nch = rows16 / 16;
            // 16 rows (chunk c) of this thread's feature, both groups
            auto emit = [&](uint32_t c, const float (&v0)[16], const float (&v1)[16]) {
                if (NPROJ == 2) {
                    const uint32_t f = fb * 128 + fl;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint32_t r = c * 16 + i;
                        const __nv_bfloat16 hv = __float2bfloat16_rn(dg_act(v0[i], v1[i], P.limit));
                        // padding rows of the tile are written as zeros: the down product reads whole 16-row groups
                        P.hb[dg_b_off(P.n_out, NT, tt, rows16, r, f)] = r < rows ? __bfloat16_as_ushort(hv) : (uint16_t)0;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint32_t r = c * 16 + i;
                        const uint32_t f = 2 * fb * 128 + fl;
                        if (r < rows) {
                            float* o = P.out + (size_t)(tt * NT + r) * P.n_out + f;
                            o[0] = v0[i];
                            o[128] = v1[i];
                        }
                    }
                }
            };
            auto load = [&](uint32_t col, float (&v)[16]) {
                uint32_t r[16];
                tmem_ld16(tmem + ((q * 32u) << 16) + col, r);
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
            };
            if (CL) {
                // the parts' tiles into the ring's memory (all MMAs are complete): [part][group][row][128 features]
                if (!wait_acc(0)) break;
                for (uint32_t c = half; c < nch; c += 2)
                    for (uint32_t l = 0; l < n_parts; ++l) {
                        float v0[16], v1[16];
                        load(2 * l * NT + c * 16, v0);
                        load((2 * l + 1) * NT + c * 16, v1);
                        float* z = reinterpret_cast<float*>(smem_raw) + ((size_t)2 * l * rows16 + c * 16) * 128 + fl;
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            z[i * 128] = v0[i];
                            z[(rows16 + i) * 128] = v1[i];
                        }
                    }
                release_acc(0);
            } else if (MODE == DG_WHOLE) {
                const uint32_t buf = n_done % n_buf;
                if (!wait_acc(buf)) break;
                for (uint32_t c = half; c < nch; c += 2) {
                    float v0[16], v1[16];
                    load(buf * 2 * NT + c * 16, v0);
                    load((buf * 2 + 1) * NT + c * 16, v1);
                    emit(c, v0, v1);
                }
                release_acc(buf);
            } else {
                // at most 64 rows: two chunks per warp; the parts are added in part order
                static_assert(DG_FOLD_NT <= 64, "two chunks of 16 rows per half of the warps");
                float sum[2][2][16];
                bool ok = true;
                for (uint32_t part = 0; part < KP; ++part) {
                    const uint32_t buf = n_done % n_buf;
                    if (!(ok = wait_acc(buf))) break;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int g = 0; g < 2; ++g)
                            if (half + 2 * j < nch) {
                                float v[16];
                                load((buf * 2 + g) * NT + (half + 2 * j) * 16, v);
#pragma unroll
                                for (int i = 0; i < 16; ++i) sum[j][g][i] = part ? __fadd_rn(sum[j][g][i], v[i]) : v[i];
                            }
                    release_acc(buf);
                }
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (half + 2 * j < nch) emit(half + 2 * j, sum[j][0], sum[j][1]);
            }
        }
    }
    // every thread comes here, also after a give-up: the cluster's barriers are always met, the tensor memory is always released
    if (CL) {
        __syncwarp();
        cluster_barrier();
        // the sums of a slice of the tile's rows over the item's parts, in part order
        uint32_t tt, fb;
        decode_unit(blockIdx.x, tt, fb);
        const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
        const uint32_t row0 = cl_rank * rows16 / NCL, n_rows = (cl_rank + 1) * rows16 / NCL - row0, base = smem_u32(smem_raw);
        for (uint32_t i = threadIdx.x; i < n_rows * 16; i += blockDim.x) {
            const uint32_t r = row0 + i / 16, f8 = i % 16;      // eight features of a row, of both groups
            float v[16];
            for (uint32_t rank = 0; rank < NCL; ++rank) {
                const uint32_t src = cluster_addr(base + (r * 128 + f8 * 8) * 4, rank), n = cl_part(rank + 1) - cl_part(rank);
                for (uint32_t l = 0; l < n; ++l) {
                    const bool init = (rank | l) == 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float4 w = ld_cluster4(src + (2 * l + (k >> 1)) * (rows16 * 512) + (k & 1) * 16);
                        v[4 * k] = init ? w.x : __fadd_rn(v[4 * k], w.x);
                        v[4 * k + 1] = init ? w.y : __fadd_rn(v[4 * k + 1], w.y);
                        v[4 * k + 2] = init ? w.z : __fadd_rn(v[4 * k + 2], w.z);
                        v[4 * k + 3] = init ? w.w : __fadd_rn(v[4 * k + 3], w.w);
                    }
                }
            }
            if (NPROJ == 2) {
                uint32_t h[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const __nv_bfloat162 b2 = __floats2bfloat162_rn(dg_act(v[2 * k], v[8 + 2 * k], P.limit), dg_act(v[2 * k + 1], v[9 + 2 * k], P.limit));
                    h[k] = r < rows ? *reinterpret_cast<const uint32_t*>(&b2) : 0u;
                }
                *reinterpret_cast<uint4*>(P.hb + dg_b_off(P.n_out, NT, tt, rows16, r, fb * 128 + f8 * 8)) = make_uint4(h[0], h[1], h[2], h[3]);
            } else if (r < rows) {
                const uint32_t f = 2 * fb * 128 + f8 * 8;
                float* o = P.out + (size_t)(tt * NT + r) * P.n_out + f;
                if (P.out_vec) {
                    float4* o4 = reinterpret_cast<float4*>(o);
                    o4[0] = make_float4(v[0], v[1], v[2], v[3]); o4[1] = make_float4(v[4], v[5], v[6], v[7]);
                    o4[32] = make_float4(v[8], v[9], v[10], v[11]); o4[33] = make_float4(v[12], v[13], v[14], v[15]);
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) { o[k] = v[k]; o[128 + k] = v[8 + k]; }
                }
            }
        }
        __syncwarp();
        cluster_barrier();   // nobody's shared memory goes away under a reader
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(tmem, 512);
}

// ---- how a product is cut ----
struct DgShape { uint32_t n_fb, n_ks; };             // feature-block pairs, stages of 64 inputs
// Parts of the reduction: as many as give every SM a weight stream with tiles of 256 rows, each part at least 4 stages long.
// The bits of a sum go by this count, so it is a function of the item count and the SM count alone and no measurement enters:
// calls of up to 256 tokens always split the same way.
static uint32_t dg_parts(DgShape s, uint32_t T, int sm_count) {
    const uint32_t items = (T + DG_NT - 1) / DG_NT * s.n_fb;
    uint32_t kp = (uint32_t)sm_count / (items ? items : 1u);
    if (kp > s.n_ks / 4) kp = s.n_ks / 4;
    if (kp > 16) kp = 16;
    return kp ? kp : 1u;
}
// Estimated cycles of a product of kp parts cut into tiles of nt rows and spread over clusters of n_cl CTAs: per stage the
// larger of the bytes an SM takes in (55 a cycle) and its eight MMAs with the turn-around of a stage; per wave a constant for
// the pipeline's fill and the epilogue; for a cluster the tiles' way through distributed shared memory.  The constants are a
// fit to 1188 timings at (H, I) = (5120, 2304), (4096, 2048), (6144, 2048), 65 to 8192 tokens, every tile and cluster that
// fits (and 21000 cycles for what all have in common): spread of measured over predicted 11 %, the cut taken 1.01 times the
// best one's time on average and 1.18 times at most.
static double dg_cost(DgShape s, uint32_t T, uint32_t nt, uint32_t kp, uint32_t n_cl, uint32_t max_clusters) {
    const uint32_t rows = nt < T ? nt : (T + 15) / 16 * 16, per = (kp + n_cl - 1) / n_cl;
    const double load = (DG_A_STAGE + rows * 128.0) / 55.0, mma = 8.0 * (rows > 96 ? rows / 2.0 : 48.0) + 140.0;
    const uint32_t items = (T + nt - 1) / nt * s.n_fb, waves = (items + max_clusters - 1) / max_clusters;
    return waves * ((s.n_ks * per + kp - 1) / kp * (load > mma ? load : mma) + 8000.0 + rows * (n_cl > 1 ? per : 1) * 8.0 +
                    (n_cl > 1 ? 4300.0 + rows * per * 60.0 : 0.0));
}
// CTAs per item for tiles of nt rows; 0: the parts' tiles do not fit
static uint32_t dg_pick_cluster(DgShape s, uint32_t T, uint32_t nt, int sm_count, const DenseCaps& caps, double* cost) {
    const uint32_t kp = dg_parts(s, T, sm_count);
    uint32_t best = 0;
    for (uint32_t per = 1; per <= kp; ++per) {            // parts of a CTA
        const uint32_t n_cl = (kp + per - 1) / per;
        if (n_cl > (uint32_t)DG_CL_MAX || (n_cl > 1 ? per * nt > (uint32_t)DG_CL_NT : kp > 1 && nt > (uint32_t)DG_FOLD_NT)) continue;
        const double c = dg_cost(s, T, nt, kp, n_cl, caps.clusters[n_cl]);
        if (!best || c < *cost) { *cost = c; best = n_cl; }
    }
    return best;
}
// rows per tile for one or two products of the same rows; 64 rows and fewer always fit
static uint32_t dg_pick_rows(const DgShape* s, int n, uint32_t T, int sm_count, const DenseCaps& caps) {
    static const uint32_t tiles[] = {DG_NT, DG_CL_NT, 160, 128, 96, 64, 48, 32};
    uint32_t best = 32;
    double c0 = 0;
    bool any = false;
    for (const uint32_t nt : tiles) {
        double c = 0, one = 0;
        bool fits = true;
        for (int i = 0; i < n && fits; ++i) { fits = dg_pick_cluster(s[i], T, nt, sm_count, caps, &one) != 0; c += one; }
        if (fits && (!any || c < c0)) { c0 = c; best = nt; any = true; }
    }
    return best;
}
uint32_t dense_shared_rows(uint32_t T, uint32_t H, uint32_t I, int sm_count, const DenseCaps& caps) {
    const DgShape s[2] = {{I / 128, H / DG_KS}, {H / 256, I / DG_KS}};
    return dg_pick_rows(s, 2, T, sm_count, caps);
}
uint32_t dense_logits_rows(uint32_t T, uint32_t E, uint32_t H, int sm_count, const DenseCaps& caps) {
    const DgShape s{E / 256, H / DG_KS};
    return dg_pick_rows(&s, 1, T, sm_count, caps);
}
// clusters of n CTAs that the device holds at once (an SM holds one CTA; clusters do not cross GPCs)
cudaError_t dense_caps(int sm_count, DenseCaps* caps) {
    const cudaError_t e = cudaFuncSetAttribute(dense_gemm_kernel<2, DG_CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_RING);
    if (e != cudaSuccess) return e;
    caps->clusters[0] = 0;
    caps->clusters[1] = (uint32_t)sm_count;
    for (uint32_t n_cl = 2; n_cl <= (uint32_t)DG_CL_MAX; ++n_cl) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = n_cl; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(n_cl * 64); cfg.blockDim = dim3(64 + DG_EPI_WARPS * 32); cfg.dynamicSmemBytes = DG_RING; cfg.attrs = &attr; cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, dense_gemm_kernel<2, DG_CLUSTER>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = sm_count / (int)n_cl; }
        caps->clusters[n_cl] = (uint32_t)(n > 0 ? n : 1);
    }
    return cudaSuccess;
}

template <int NPROJ>
static cudaError_t dg_launch(DenseParams P, int sm_count, const DenseCaps& caps, cudaStream_t st) {
    const DgShape s{NPROJ == 2 ? P.n_blocks : P.n_blocks / 2, P.n_ks};
    double cost = 0;
    P.out_vec = reinterpret_cast<uintptr_t>(P.out) % 16 == 0;
    P.k_parts = dg_parts(s, P.T, sm_count);
    P.n_cl = dg_pick_cluster(s, P.T, P.nt, sm_count, caps, &cost);
    if (!P.n_cl) return cudaErrorInvalidValue;
    const size_t stage = DG_A_STAGE + (size_t)P.nt * DG_KS * 2;
    P.n_stages = (uint32_t)(DG_RING / stage < (size_t)DG_STAGES ? DG_RING / stage : (size_t)DG_STAGES);
    const uint32_t n_items = (P.T + P.nt - 1) / P.nt * s.n_fb;
    const auto kernel = P.n_cl > 1 ? dense_gemm_kernel<NPROJ, DG_CLUSTER> : P.k_parts > 1 ? dense_gemm_kernel<NPROJ, DG_FOLD> : dense_gemm_kernel<NPROJ, DG_WHOLE>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_RING);
    if (e != cudaSuccess) return e;
    if (P.n_cl == 1) {
        kernel<<<n_items < (uint32_t)sm_count ? n_items : (uint32_t)sm_count, 64 + DG_EPI_WARPS * 32, DG_RING, st>>>(P);
        return cudaGetLastError();
    }
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = P.n_cl; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n_items * P.n_cl); cfg.blockDim = dim3(64 + DG_EPI_WARPS * 32); cfg.dynamicSmemBytes = DG_RING; cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P);
}
static_assert(DG_RING >= 2 * DG_CL_NT * 128 * 4, "a cluster's partial tile in the ring's memory");

static cudaError_t dg_stage_rows(const __nv_bfloat16* x, uint32_t T, uint32_t K, uint32_t nt, uint16_t* xb, int sm_count, cudaStream_t st) {
    const uint32_t tasks = (T + 7) / 8 * (K / 32), want = (tasks + 15) / 16, cap = (uint32_t)sm_count * 8;   // two tasks a warp, or all SMs full
    dense_rows_kernel<<<want < cap ? want : cap, 256, 0, st>>>(x, T, K, nt, xb);
    return cudaGetLastError();
}

cudaError_t launch_dense_shared_expert(const DenseSharedArgs& a, cudaStream_t st) {
    if (a.T == 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (!a.rows_staged && (e = dg_stage_rows(a.x, a.T, a.H, a.nt, a.xb, a.sm_count, st)) != cudaSuccess) return e;
    DenseParams P{};
    P.status = a.status; P.poll_limit = 1u << 20; P.limit = a.limit; P.T = a.T; P.nt = a.nt;
    // gate / up -> h (B-operand order over I inputs)
    P.w = static_cast<const uint8_t*>(a.w_gu); P.n_blocks = a.I / 128; P.n_ks = a.H / DG_KS; P.xb = a.xb; P.K = a.H; P.hb = a.hb; P.out = nullptr; P.n_out = a.I;
    if ((e = dg_launch<2>(P, a.sm_count, *a.caps, st)) != cudaSuccess) return e;
    // down -> out f32 [T, H]
    P.w = static_cast<const uint8_t*>(a.w_d); P.n_blocks = a.H / 128; P.n_ks = a.I / DG_KS; P.xb = a.hb; P.K = a.I; P.hb = nullptr; P.out = a.out; P.n_out = a.H;
    return dg_launch<1>(P, a.sm_count, *a.caps, st);
}

cudaError_t launch_dense_logits(const __nv_bfloat16* x, const void* w_tiled, uint32_t T, uint32_t E, uint32_t H, uint32_t nt, uint16_t* xb,
                                float* logits, uint32_t* status, int sm_count, const DenseCaps& caps, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    const cudaError_t e = dg_stage_rows(x, T, H, nt, xb, sm_count, st);
    if (e != cudaSuccess) return e;
    DenseParams P{};
    P.status = status; P.poll_limit = 1u << 20; P.limit = 0.f; P.T = T; P.nt = nt;
    P.w = static_cast<const uint8_t*>(w_tiled); P.n_blocks = E / 128; P.n_ks = H / DG_KS; P.xb = xb; P.K = H; P.hb = nullptr;
    P.out = logits; P.n_out = E;
    return dg_launch<1>(P, sm_count, caps, st);
}

bool dense_gemm_supported(uint32_t n_out, uint32_t K, int two_blocks) {
    return K % DG_KS == 0 && n_out % (two_blocks ? 256 : 128) == 0;
}

}  // namespace mlxs
