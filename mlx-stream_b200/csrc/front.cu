// The front of a decode-sized layer call in one launch: [router logits from x] -> router tail -> dispatch -> row
// staging.  Four dependent kernels of a few microseconds each cost a decode step more in launch gaps than in work
// (at one token: 37 us of a 175 us call); here they are phases of one kernel.
//   phase 0 (only when the layer starts from x): logits = f32(x) . f32(W_g)^T, four warps per expert row, 8 token rows
//            staged in shared memory at a time (src/arch/deepseek_v41/graph.zig:2033; mimo_glue_router_rows.metal), then a
//            grid barrier;
//   phase 1: every CTA routes all tokens: scores by all threads, the selection by a warp per token (router_body.cuh);
//   phase 2: every CTA sorts the assignment rows by expert and builds the work tables in its shared memory (the dispatch
//            kernel's code); CTA 0 writes them out;
//   phase 3: all warps stage the rows for the streaming lane (the prep kernels' code).
// Phases 1 and 2 are a few microseconds whoever does them; done by every CTA for itself they cost no grid barrier (two of
// them, with the round trips of ids and tables through L2, were half of the 17 us this kernel took at one token), and without
// phase 0 the launch is an ordinary one.  More than 256 experts, top_k > 32, or more tokens than shared memory holds scores of
// (165 at 256 experts and top-8): a CTA per token routes, then a barrier.
// The grid barrier is a counter and a generation word in global memory: the last CTA to arrive resets the counter and
// bumps the generation, the others poll the generation with a bound.  A launch with a barrier is cooperative, so all CTAs
// are resident together; a barrier that runs out still records the status word and lets the kernel finish.
#include "common.cuh"
#include "kernels.h"
#include "dispatch_body.cuh"
#include "exl3_prep_body.cuh"
#include "fp4_prep_body.cuh"
#include "logits_body.cuh"
#include "router_body.cuh"

namespace mlxs {

struct FrontParams {
    // phase 0 (w_router == null: the caller supplies logits)
    const __nv_bfloat16* w_router;   // [E, H] bf16
    float* logits_out;               // [T, E] written by phase 0
    // phase 1
    const float* logits;             // [T, E]
    const float* bias;
    int E, K, scoring, norm;
    float scale;
    int32_t* ids;
    float* weights;
    uint32_t T;
    // phase 2
    const uint8_t* loaded;
    DispatchTables t;
    uint32_t chunk_rows, group_chunks, heavy;
    uint32_t* status;
    // phase 3
    const __nv_bfloat16* x;
    uint32_t H;
    int bank_exl3;
    const __half* scales;
    size_t scales_stride;
    uint32_t* xa;
    // grid barrier: [0] arrivals, [1] generation
    uint32_t* bar;
    uint32_t poll_limit;
    int rthreads;
    int by_warp;                     // phases 1 and 2 in every CTA
    uint32_t parts;                  // FP4: warps per staged row
};

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// All CTAs of the grid meet here.  gen: the generation this CTA saw before its first arrival, kept per thread.
__device__ __forceinline__ bool front_grid_sync(uint32_t* bar, uint32_t& gen, uint32_t limit, uint32_t* status) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        bool ok = true;
        __threadfence();
        const uint32_t prev = atomicAdd(&bar[0], 1u);
        if (prev == gridDim.x - 1) {
            bar[0] = 0;
            __threadfence();
            atomicAdd(&bar[1], 1u);
        } else {
            uint32_t i = 0;
            while (ld_acquire_gpu(&bar[1]) == gen) {
                if (++i > limit) { ok = false; atomicMax(status, (uint32_t)ST_WAIT_FULL); break; }
                __nanosleep(32);
            }
        }
        __threadfence();
        s_ok = ok ? 1 : 0;
    }
    gen += 1;
    __syncthreads();
    return s_ok != 0;
}

__global__ void __launch_bounds__(1024, 1) front_kernel(const FrontParams P) {
    extern __shared__ __align__(16) uint8_t fsm[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nwarp = blockDim.x >> 5;
    grid_dep_wait();
    grid_dep_launch();
    // the barrier's generation before this CTA's first arrival (it cannot advance until every CTA, this one too, arrives)
    __shared__ uint32_t s_gen;
    if (threadIdx.x == 0) s_gen = ld_acquire_gpu(&P.bar[1]);
    __syncthreads();
    uint32_t gen = s_gen;
    const uint32_t T = P.T;

    // ---- phase 0: logits from x (the logits kernel's code: four warps per expert row) ----
    if (P.w_router) {
        logits_rows(P.x, P.w_router, T, (uint32_t)P.E, P.H, P.logits_out, fsm, blockIdx.x, gridDim.x);
        front_grid_sync(P.bar, gen, P.poll_limit, P.status);
    }

    // ---- phase 1: the router's tail ----
    // shared memory: ids and weights [A], the tables [E + 1 + 6 A + 16], the dispatch scratch, the scores [T][E + 2]
    const uint32_t A = T * (uint32_t)P.K, E = (uint32_t)P.E;
    int32_t* s_ids = reinterpret_cast<int32_t*>(fsm);
    float* s_w = reinterpret_cast<float*>(s_ids + A);
    DispatchTables S = P.t;
    S.header = reinterpret_cast<uint32_t*>(s_w + A);
    S.offsets = S.header + 16;
    S.order = S.offsets + E + 1;
    S.chunk_expert = S.order + A; S.chunk_row0 = S.chunk_expert + A; S.chunk_rows = S.chunk_row0 + A;
    S.group_chunk0 = S.chunk_rows + A; S.group_mc = S.group_chunk0 + A;
    S.max_chunks = A < P.t.max_chunks ? A : P.t.max_chunks;
    uint32_t* scratch = S.group_mc + A;
    const int32_t* ids = s_ids;
    if (P.by_warp) {
        // one expert per thread: the scoring functions are long, and this kernel's code comes cold from memory
        float* s_sc = reinterpret_cast<float*>(scratch + dispatch_words(A, E));     // [T][E], then per token {max, NaN flag}
        float* s_max = s_sc + (size_t)T * E;
        if (P.scoring == 2) {
            for (uint32_t t = warp; t < T; t += nwarp) {
                float xv[NE], m;
                bool nan;
#pragma unroll
                for (int i = 0; i < NE; ++i) xv[i] = lane + 32 * i < E ? P.logits[(size_t)t * E + lane + 32 * i] : 0.0f;
                route_max_warp(xv, P.E, m, nan);
                if (lane == 0) { s_max[2 * t] = m; s_max[2 * t + 1] = nan ? 1.0f : 0.0f; }
            }
            __syncthreads();
        }
#pragma unroll 1
        for (uint32_t i = threadIdx.x; i < T * E; i += blockDim.x) {
            const float x = P.logits[i];
            if (P.scoring == 2) {
                const float* mx = s_max + 2 * (i / E);
                s_sc[i] = mx[1] != 0.0f ? __int_as_float(0x7FC00000) : det_expf(__fsub_rn(x, mx[0]));
            } else {
                s_sc[i] = route_score(x, P.scoring);
            }
        }
        __syncthreads();
        for (uint32_t t = warp; t < T; t += nwarp)
            route_row_warp<true>(s_sc + t * E, P.bias, P.E, P.K, P.scoring, P.norm, P.scale, s_ids + t * P.K, s_w + t * P.K);
        __syncthreads();
    } else {
        for (uint32_t t = blockIdx.x; t < T; t += gridDim.x)
            route_row(P.logits, P.bias, P.E, P.K, P.scoring, P.norm, P.scale, P.ids, P.weights, (int)t, reinterpret_cast<float*>(fsm), P.rthreads);
        front_grid_sync(P.bar, gen, P.poll_limit, P.status);
        ids = P.ids;
    }

    // ---- phase 2: dispatch, by every CTA for itself ----
    dispatch_body(ids, A, E, P.loaded, S, P.chunk_rows, P.group_chunks, P.heavy, P.status, scratch);
    __syncthreads();
    const uint32_t n_chunks = S.header[HDR_NCHUNKS];
    if (blockIdx.x == 0) {
        const uint32_t n_groups = S.header[HDR_NGROUPS];
        if (threadIdx.x <= HDR_CTR_AUX) P.t.header[threadIdx.x] = S.header[threadIdx.x];
        for (uint32_t i = threadIdx.x; i <= E; i += blockDim.x) P.t.offsets[i] = S.offsets[i];
        for (uint32_t i = threadIdx.x; i < A; i += blockDim.x) {
            P.t.order[i] = S.order[i];
            if (P.by_warp) { P.ids[i] = s_ids[i]; P.weights[i] = s_w[i]; }
        }
        for (uint32_t i = threadIdx.x; i < n_chunks; i += blockDim.x) {
            P.t.chunk_expert[i] = S.chunk_expert[i]; P.t.chunk_row0[i] = S.chunk_row0[i]; P.t.chunk_rows[i] = S.chunk_rows[i];
        }
        for (uint32_t i = threadIdx.x; i < n_groups; i += blockDim.x) { P.t.group_chunk0[i] = S.group_chunk0[i]; P.t.group_mc[i] = S.group_mc[i]; }
    }

    // ---- phase 3: row staging, a warp per (chunk, row, 128-block) or per (chunk, row) ----
    const uint32_t gw = blockIdx.x * nwarp + warp, gstride = gridDim.x * nwarp;
    if (P.bank_exl3) {
        const uint32_t nb = P.H / 128, per_chunk = P.chunk_rows * nb;
        for (uint32_t task = gw; task < n_chunks * per_chunk; task += gstride) {
            const uint32_t chunk = task / per_chunk, rem = task % per_chunk, row = rem / nb, b = rem % nb;
            const uint32_t e = S.chunk_expert[chunk], rows = S.chunk_rows[chunk];
            const bool valid = row < rows;
            const uint32_t assign = valid ? S.order[S.chunk_row0[chunk] + row] : 0u;
            exl3_prep_row_block<false>(P.x, x_row_of(S, assign, (uint32_t)P.K), valid, e, P.H, P.scales, P.scales_stride, chunk, row, b,
                                       lane, P.xa);
        }
    } else {
        // a row's 8-input groups are split over `parts` warps
        const uint32_t parts = P.parts, per_chunk = P.chunk_rows * parts;
        for (uint32_t task = gw; task < n_chunks * per_chunk; task += gstride) {
            const uint32_t chunk = task / per_chunk, rem = task % per_chunk, row = rem / parts, part = rem % parts;
            const bool valid = row < S.chunk_rows[chunk];
            const uint32_t tok = valid ? x_row_of(S, S.order[S.chunk_row0[chunk] + row], (uint32_t)P.K) : 0u;
            fp4_prep_row(P.x, tok, valid, P.H, chunk, row, part * 32u + lane, parts * 32u, P.xa);
        }
    }
}

static int front_route_threads(int E, int K) { return ((E > K ? E : K) + 31) / 32 * 32; }
// smem: the larger of the phases' needs
static size_t front_smem_bytes(int E, int K, uint32_t T, uint32_t H, bool from_x, bool by_warp) {
    size_t s = router_smem_floats(E, K, front_route_threads(E, K)) * sizeof(float);
    const size_t d = ((size_t)8 * T * K + (size_t)E + 17 + dispatch_words(T * (uint32_t)K, (uint32_t)E) + (by_warp ? (size_t)T * (E + 2) : 0)) * sizeof(uint32_t);
    if (d > s) s = d;
    if (from_x) { const size_t l = logits_smem_bytes(H, 32); if (l > s) s = l; }
    return s;
}
static bool front_by_warp(int E, int K, uint32_t T, uint32_t H, bool from_x, size_t smem_max) {
    return route_by_warp(E, K) && front_smem_bytes(E, K, T, H, from_x, true) <= smem_max;
}
bool front_fits(int E, int K, uint32_t T, uint32_t H, bool from_x, size_t smem_max) {
    return front_smem_bytes(E, K, T, H, from_x, front_by_warp(E, K, T, H, from_x, smem_max)) <= smem_max;
}

cudaError_t launch_front(const FrontArgs& a, cudaStream_t st) {
    if (a.T == 0) return cudaSuccess;
    FrontParams P{};
    P.w_router = a.w_router; P.logits_out = a.logits_out; P.logits = a.w_router ? a.logits_out : a.logits; P.bias = a.bias;
    P.E = a.E; P.K = a.K; P.scoring = a.scoring; P.norm = a.norm; P.scale = a.scale; P.ids = a.ids; P.weights = a.weights; P.T = a.T;
    P.loaded = a.loaded; P.t = a.t; P.chunk_rows = a.chunk_rows; P.group_chunks = a.group_chunks; P.heavy = a.heavy; P.status = a.status;
    P.x = a.x; P.H = a.H; P.bank_exl3 = a.bank_exl3; P.scales = a.scales; P.scales_stride = a.scales_stride; P.xa = a.xa;
    P.bar = a.bar; P.poll_limit = 1u << 22;
    P.rthreads = front_route_threads(a.E, a.K);
    P.by_warp = front_by_warp(a.E, a.K, a.T, a.H, a.w_router, a.smem_max) ? 1 : 0;
    const size_t smem = front_smem_bytes(a.E, a.K, a.T, a.H, a.w_router, P.by_warp);
    cudaError_t e = cudaFuncSetAttribute(front_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const bool barrier = a.w_router || !P.by_warp;
    // a warp per staging task (a row's 128-block; for the FP4 banks a sixteenth of a row, or a quarter where that would be more
    // warps than the SMs hold), at most a CTA per SM.  From x, two tokens and more beside the shared expert's kernels, an FP4
    // row always goes by quarters.  The front then ends 2 us later, which is better: gate/up's units belong to its CTAs by
    // number, so while the shared expert's first kernel (35 us, from the front's start on) holds SMs some of them wait, and
    // gate/up takes 60 us from the front's end instead of 53.  NVFP4, H 6144, two tokens, sixteenths -> quarters: of 32 and 128
    // experts 113.9 -> 106.7 and 116.2 -> 108.4 us; handles on whose streams the shared expert's kernel runs before the front
    // or behind gate/up 120.1 -> 121.5 (256 experts).  One token: nothing lost by sixteenths (85.1, 96.9 with 100.8 by quarters).
    const unsigned sms = (unsigned)(a.sm_count > 0 ? a.sm_count : 32);
    const unsigned rows = (unsigned)(a.T * a.K) * a.chunk_rows;
    P.parts = rows * 16u <= 32u * sms && !(a.w_router && a.beside && a.T > 1) ? 16u : 4u;
    unsigned grid = (rows * (a.bank_exl3 ? a.H / 128 : P.parts) + 31u) / 32u;
    // with a barrier 32 to 64 CTAs: one round of expert rows, and room beside the shared expert's kernels; from x two CTAs per set
    // of eight expert rows where that is within the bounds, so that they share out the tokens (logits_body.cuh)
    if (barrier) {
        const unsigned want = a.w_router && a.T > 1 ? 2u * ((unsigned)(a.E + 7) / 8u) : 0u;
        grid = ((grid > want ? grid : want) + 1u) / 2u * 2u;
        grid = grid < 32u ? 32u : grid > 64u ? 64u : grid;
    }
    if (grid > sms) grid = sms;
    if (!barrier) {
        return launch_dependent(true, front_kernel, grid, 1024, smem, st, P);
    }
    void* args[] = {&P};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(front_kernel), dim3(grid), dim3(1024), args, smem, st);
}

}  // namespace mlxs
