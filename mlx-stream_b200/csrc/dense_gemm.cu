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
//   * calls with too few (token tile, feature block) items for the SMs take smaller token tiles and split the reduction
//     dimension over the CTAs of a cluster (dg_plan): each leaves its f32 partial tile in its own shared memory, and every
//     CTA folds a slice of the rows over the cluster in part order.  With one CTA folding all parts out of global scratch
//     the fold was most of the time: gate/up at 300 tokens 90 us for 42 MB of weights.
// Every wait is bounded; on a give-up the CTA records the status word, skips its work and still frees tensor memory.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace mlxs {

constexpr int DG_KS = 64;                         // inputs per stage
constexpr int DG_NT = 256;                        // most rows per token tile (MMA N)
constexpr int DG_CL_NT = 192;                     // the same in a cluster: the partial tile has to fit the ring's shared memory
constexpr int DG_STAGES = 6;                      // most ring stages
constexpr int DG_RING = 192 * 1024;               // ring bytes: 3 stages at 256 rows
constexpr int DG_A_TILE = 128 * DG_KS * 2;        // one projection's (block, stage): 16 KB
constexpr int DG_A_STAGE = 2 * DG_A_TILE;         // two accumulator groups' weights
constexpr int DG_EPI_WARPS = 8;

// ---- load-time re-tiling of a weight matrix W[n_out, K] (row-major bf16) ----
// np = 2: w0 and w1 interleaved per 8-row group ([rc][p][kc][8][8]); np = 1: w0 alone ([rc][kc][8][8])
__global__ void dense_retile_kernel(const __nv_bfloat16* __restrict__ w0, const __nv_bfloat16* __restrict__ w1, uint32_t n_out,
                                    uint32_t n_valid, uint32_t K, int np, uint4* __restrict__ dst) {
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
        const uint32_t f = nb * 128 + rc * 8 + r8;
        const __nv_bfloat16* src = (p ? w1 : w0) + (size_t)f * K + (size_t)ks * DG_KS + kc * 8;
        dst[i] = f < n_valid ? *reinterpret_cast<const uint4*>(src) : make_uint4(0, 0, 0, 0);
    }
}

cudaError_t launch_dense_retile(const __nv_bfloat16* w0, const __nv_bfloat16* w1, uint32_t n_out, uint32_t K, void* dst,
                                cudaStream_t st) {
    if (K % DG_KS || (w1 && n_out % 128)) return cudaErrorInvalidValue;
    // a single matrix is cut into pairs of blocks: padded with zero features to a whole pair
    const uint32_t n_pad = w1 ? n_out : (n_out + 255) / 256 * 256;
    dense_retile_kernel<<<592, 256, 0, st>>>(w0, w1, n_pad, n_out, K, w1 ? 2 : 1, static_cast<uint4*>(dst));
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
    uint32_t nt;               // rows per token tile (a multiple of 16)
    uint32_t n_stages;         // ring stages
    uint32_t k_parts;          // CTAs of a cluster that share one item's reduction dimension (1: no cluster)
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
// CL: a cluster of k_parts CTAs per item, one part of the reduction each; otherwise a CTA walks whole items.
template <int NPROJ, bool CL>
__global__ void __launch_bounds__(64 + DG_EPI_WARPS * 32, 1) dense_gemm_kernel(const DenseParams P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[DG_STAGES], empty_bar[DG_STAGES], acc_full, acc_empty;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    uint8_t* a_ring = smem_raw;                              // [stage][2 groups' tiles]
    uint8_t* b_ring = smem_raw + P.n_stages * DG_A_STAGE;    // [stage][rows16 x 64]
    const uint32_t NT = P.nt, b_stage = NT * DG_KS * 2, NS = P.n_stages;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t n_tt = (P.T + NT - 1) / NT;
    const uint32_t n_fb = NPROJ == 2 ? P.n_blocks : P.n_blocks / 2;     // feature-block groups
    const uint32_t KP = CL ? P.k_parts : 1u;
    const uint32_t n_units = n_tt * n_fb * KP;
    if (blockIdx.x >= n_units) return;   // before any tensor memory is taken (the whole CTA reads the same count)

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < NS; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(&acc_full, 1);
        mbar_init(&acc_empty, DG_EPI_WARPS);
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
    // unit -> (token tile, feature-block group, part of the reduction); feature blocks vary fastest so that the CTAs
    // running together share the rows of a few token tiles and the weights in L2
    auto decode_unit = [&](uint32_t unit, uint32_t& tt, uint32_t& fb, uint32_t& part) {
        part = unit % KP;
        const uint32_t item = unit / KP;
        fb = item % n_fb;
        tt = item / n_fb;
    };

    if (warp == 0) {
        // ---------------- producer ----------------
        if (lane == 0) {
            uint32_t s = 0, ph = 0;
            for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x) {
                uint32_t tt, fb, part;
                decode_unit(unit, tt, fb, part);
                const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
                const uint32_t b_bytes = rows16 * DG_KS * 2;
                const uint16_t* xsrc = P.xb + (size_t)tt * NT * P.K;
                bool ok = true;
                for (uint32_t ks = part_begin(part); ks < part_begin(part + 1); ++ks) {
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
            for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x, ++n_done) {
                uint32_t tt, fb, part;
                decode_unit(unit, tt, fb, part);
                const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
                const uint32_t idesc = umma_idesc(UMMA_BF16, rows16), lbo_b = rows16 * 16;
                if (!mbar_wait_bounded(&acc_empty, (n_done & 1u) ^ 1u, &s_abort, 64, P.poll_limit)) { give_up(ST_WAIT_EMPTY); break; }
                tc_fence_after();
                bool ok = true;
                const uint32_t nk = part_begin(part + 1) - part_begin(part);
                for (uint32_t kk = 0; kk < nk; ++kk) {
                    if (!mbar_wait_bounded(&full_bar[s], ph, &s_abort, 0, P.poll_limit)) { give_up(ST_WAIT_FULL); ok = false; break; }
                    tc_fence_after();
                    const uint32_t a0 = a_s + s * DG_A_STAGE, b0 = b_s + s * b_stage;
#pragma unroll
                    for (int gq = 0; gq < 2; ++gq) {
#pragma unroll
                        for (int i = 0; i < DG_KS / 16; ++i)
                            umma_f16(tmem + gq * DG_NT, umma_smem_desc(a0 + gq * A_GROUP + i * 2 * A_LBO, A_LBO, A_SBO),
                                     umma_smem_desc(b0 + i * 2 * lbo_b, lbo_b, 128), idesc, (kk | (uint32_t)i) ? 1u : 0u);
                    }
                    umma_commit(&empty_bar[s]);
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                umma_commit(&acc_full);
            }
        }
    } else {
        // ---------------- epilogue warps ----------------
        // warp = (lane quarter q, half): a thread owns output feature 32 q + lane of both groups; the 16-row chunks of
        // the tile alternate between the two halves
        const uint32_t ew = warp - 2, q = warp & 3u, half = ew >> 2;
        uint32_t n_done = 0;
        for (uint32_t unit = blockIdx.x; unit < n_units && !s_abort; unit += gridDim.x, ++n_done) {
            uint32_t tt, fb, part;
            decode_unit(unit, tt, fb, part);
            const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16, nch = rows16 / 16;
            if (!mbar_wait_bounded(&acc_full, n_done & 1u, &s_abort, 0, P.poll_limit)) { give_up(ST_WAIT_FULL); break; }
            tc_fence_after();
            const uint32_t fl = q * 32u + lane;                 // feature inside the block
            for (uint32_t c = half; c < nch; c += 2) {
                uint32_t r0[16], r1[16];
                tmem_ld16(tmem + ((q * 32u) << 16) + 0 * DG_NT + c * 16, r0);
                tmem_ld16(tmem + ((q * 32u) << 16) + 1 * DG_NT + c * 16, r1);
                if (CL) {
                    // this part's tile into the ring's memory (its MMAs are complete): [group][row][128 features]
                    float* z = reinterpret_cast<float*>(smem_raw) + (size_t)c * 16 * 128 + fl;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        z[i * 128] = __uint_as_float(r0[i]);
                        z[(rows16 + i) * 128] = __uint_as_float(r1[i]);
                    }
                } else if (NPROJ == 2) {
                    const uint32_t f = fb * 128 + fl;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint32_t r = c * 16 + i;
                        const __nv_bfloat16 hv = __float2bfloat16_rn(dg_act(__uint_as_float(r0[i]), __uint_as_float(r1[i]), P.limit));
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
                            if (f < P.n_out) o[0] = __uint_as_float(r0[i]);
                            if (f + 128 < P.n_out) o[128] = __uint_as_float(r1[i]);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);
        }
    }
    // every thread comes here, also after a give-up: the cluster's barriers are always met, the tensor memory is always released
    if (CL) {
        __syncwarp();
        cluster_barrier();
        // the sums of a slice of the tile's rows over the cluster's parts, in part order
        uint32_t tt, fb, part;
        decode_unit(blockIdx.x, tt, fb, part);
        const uint32_t rows = min(NT, P.T - tt * NT), rows16 = (rows + 15) / 16 * 16;
        const uint32_t row0 = part * rows16 / KP, n_rows = (part + 1) * rows16 / KP - row0, base = smem_u32(smem_raw);
        for (uint32_t i = threadIdx.x; i < n_rows * 16; i += blockDim.x) {
            const uint32_t r = row0 + i / 16, f8 = i % 16;      // eight features of a row, of both groups
            float v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = 0.f;
            for (uint32_t pp = 0; pp < KP; ++pp) {
                const uint32_t src = cluster_addr(base + (r * 128 + f8 * 8) * 4, pp);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 w = ld_cluster4(src + (k >> 1) * (rows16 * 512) + (k & 1) * 16);
                    v[4 * k] += w.x; v[4 * k + 1] += w.y; v[4 * k + 2] += w.z; v[4 * k + 3] += w.w;
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
                const uint32_t f = 2 * fb * 128 + f8 * 8;           // n_out is a multiple of 8
                float4* o = reinterpret_cast<float4*>(P.out + (size_t)(tt * NT + r) * P.n_out + f);
                if (f < P.n_out) { o[0] = make_float4(v[0], v[1], v[2], v[3]); o[1] = make_float4(v[4], v[5], v[6], v[7]); }
                if (f + 128 < P.n_out) { o[32] = make_float4(v[8], v[9], v[10], v[11]); o[33] = make_float4(v[12], v[13], v[14], v[15]); }
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

// ---- how a product is cut: rows per token tile and CTAs (of a cluster) per item ----
struct DgShape { uint32_t n_fb, n_ks; };             // feature-block pairs, stages of 64 inputs
// clusters of kp CTAs that the device holds at once (an SM holds one CTA; clusters do not cross GPCs)
template <int NPROJ>
static uint32_t dg_max_clusters(uint32_t kp, int sm_count) {
    static uint32_t known[9] = {0};
    if (kp == 1) return (uint32_t)sm_count;
    if (!known[kp]) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kp; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kp * 64); cfg.blockDim = dim3(64 + DG_EPI_WARPS * 32); cfg.dynamicSmemBytes = DG_RING; cfg.attrs = &attr; cfg.numAttrs = 1;
        int n = 0;
        cudaFuncSetAttribute(dense_gemm_kernel<NPROJ, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_RING);
        if (cudaOccupancyMaxActiveClusters(&n, dense_gemm_kernel<NPROJ, true>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = sm_count / (int)kp; }
        known[kp] = (uint32_t)(n > 0 ? n : 1);
    }
    return known[kp];
}
// Estimated cycles of a product cut into tiles of nt rows and kp parts: per stage the larger of the bytes an SM takes in (about
// 50 a cycle) and its eight MMAs with the turn-around of a stage; a constant per wave for the pipeline's fill and the
// epilogue; for a cluster the tile's way through distributed shared memory.  Measured at H 5120, I 2304 (gate/up + down).
static double dg_cost(DgShape s, uint32_t T, uint32_t nt, uint32_t kp, uint32_t max_clusters) {
    const uint32_t rows = nt < T ? nt : (T + 15) / 16 * 16;
    const double load = (DG_A_STAGE + rows * 128.0) / 50.0, mma = 8.0 * (rows / 2.0 > 48.0 ? rows / 2.0 : 48.0) + 120.0;
    const uint32_t items = (T + nt - 1) / nt * s.n_fb, waves = (items + max_clusters - 1) / max_clusters;
    return waves * ((s.n_ks + kp - 1) / kp * (load > mma ? load : mma) + 5000.0 + rows * 16.0) + (kp > 1 ? 3000.0 + rows * 1024.0 / 25.0 : 0.0);
}
template <int NPROJ>
static uint32_t dg_pick_parts(DgShape s, uint32_t T, uint32_t nt, int sm_count, double* cost) {
    uint32_t best = 1;
    double c0 = dg_cost(s, T, nt, 1, (uint32_t)sm_count);
    for (uint32_t kp = 2; kp <= 8 && nt <= (uint32_t)DG_CL_NT && kp * 4 <= s.n_ks; kp *= 2) {
        const double c = dg_cost(s, T, nt, kp, dg_max_clusters<NPROJ>(kp, sm_count));
        if (c < c0) { c0 = c; best = kp; }
    }
    *cost = c0;
    return best;
}
static uint32_t dg_pick_rows(const DgShape* gu, const DgShape* plain, int n_plain, uint32_t T, int sm_count) {
    uint32_t best = DG_NT;
    double c0 = 0;
    for (uint32_t nt = DG_NT; nt >= 64; nt -= nt > (uint32_t)DG_CL_NT ? nt - DG_CL_NT : 32) {
        double c = 0, one = 0;
        if (gu) { dg_pick_parts<2>(*gu, T, nt, sm_count, &one); c += one; }
        for (int i = 0; i < n_plain; ++i) { dg_pick_parts<1>(plain[i], T, nt, sm_count, &one); c += one; }
        if (nt == (uint32_t)DG_NT || c < c0) { c0 = c; best = nt; }
    }
    return best;
}
uint32_t dense_shared_rows(uint32_t T, uint32_t H, uint32_t I, int sm_count) {
    const DgShape gu{I / 128, H / DG_KS}, dn{H / 256, I / DG_KS};
    return dg_pick_rows(&gu, &dn, 1, T, sm_count);
}
uint32_t dense_logits_rows(uint32_t T, uint32_t E, uint32_t H, int sm_count) {
    const DgShape lg{(E + 255) / 256, H / DG_KS};
    return dg_pick_rows(nullptr, &lg, 1, T, sm_count);
}

template <int NPROJ>
static cudaError_t dg_launch(DenseParams P, int sm_count, cudaStream_t st) {
    const DgShape s{NPROJ == 2 ? P.n_blocks : P.n_blocks / 2, P.n_ks};
    double cost = 0;
    P.k_parts = dg_pick_parts<NPROJ>(s, P.T, P.nt, sm_count, &cost);
    const size_t stage = DG_A_STAGE + (size_t)P.nt * DG_KS * 2;
    P.n_stages = (uint32_t)(DG_RING / stage < (size_t)DG_STAGES ? DG_RING / stage : (size_t)DG_STAGES);
    const uint32_t n_items = (P.T + P.nt - 1) / P.nt * s.n_fb;
    cudaError_t e;
    if (P.k_parts == 1) {
        if ((e = cudaFuncSetAttribute(dense_gemm_kernel<NPROJ, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_RING)) != cudaSuccess) return e;
        const uint32_t grid = n_items < (uint32_t)sm_count ? n_items : (uint32_t)sm_count;
        dense_gemm_kernel<NPROJ, false><<<grid, 64 + DG_EPI_WARPS * 32, DG_RING, st>>>(P);
        return cudaGetLastError();
    }
    if ((e = cudaFuncSetAttribute(dense_gemm_kernel<NPROJ, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_RING)) != cudaSuccess) return e;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = P.k_parts; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n_items * P.k_parts); cfg.blockDim = dim3(64 + DG_EPI_WARPS * 32); cfg.dynamicSmemBytes = DG_RING; cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, dense_gemm_kernel<NPROJ, true>, P);
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
    if ((e = dg_launch<2>(P, a.sm_count, st)) != cudaSuccess) return e;
    // down -> out f32 [T, H]
    P.w = static_cast<const uint8_t*>(a.w_d); P.n_blocks = a.H / 128; P.n_ks = a.I / DG_KS; P.xb = a.hb; P.K = a.I; P.hb = nullptr; P.out = a.out; P.n_out = a.H;
    return dg_launch<1>(P, a.sm_count, st);
}

cudaError_t launch_dense_logits(const __nv_bfloat16* x, const void* w_tiled, uint32_t T, uint32_t E, uint32_t H, uint32_t nt, uint16_t* xb,
                                float* logits, uint32_t* status, int sm_count, cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    const cudaError_t e = dg_stage_rows(x, T, H, nt, xb, sm_count, st);
    if (e != cudaSuccess) return e;
    DenseParams P{};
    P.status = status; P.poll_limit = 1u << 20; P.limit = 0.f; P.T = T; P.nt = nt;
    P.w = static_cast<const uint8_t*>(w_tiled); P.n_blocks = (E + 255) / 256 * 2; P.n_ks = H / DG_KS; P.xb = xb; P.K = H; P.hb = nullptr;
    P.out = logits; P.n_out = E;
    return dg_launch<1>(P, sm_count, st);
}

bool dense_gemm_supported(uint32_t n_out, uint32_t K, int two_blocks) {
    return K % DG_KS == 0 && n_out % (two_blocks ? 256 : 128) == 0;
}

}  // namespace mlxs
