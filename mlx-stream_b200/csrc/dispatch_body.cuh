// Device code of the dispatch (stable counting sort + work tables), shared by the dispatch kernels and the fused front
// kernel.
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace mlxs {

constexpr int DTHREADS = 1024;   // one thread per expert in the scans (n_experts <= 1024), one per assignment of a block

// Exclusive prefix sums of three per-thread values over the CTA (1024 threads): warp shuffles, then the 32 warp totals
// by the first warp.  ws: [3][33] words of shared memory; the totals come back in tot[3].
__device__ __forceinline__ void block_scan3(const uint32_t (&v)[3], uint32_t (&excl)[3], uint32_t (&tot)[3], uint32_t* ws) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        uint32_t x = v[k];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        inc[k] = x;
        if (lane == 31) ws[k * 33 + warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t w = ws[k * 33 + lane];
            uint32_t x = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            ws[k * 33 + lane] = x - w;            // exclusive base of each warp
            if (lane == 31) ws[k * 33 + 32] = x;  // total
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        excl[k] = ws[k * 33 + warp] + inc[k] - v[k];
        tot[k] = ws[k * 33 + 32];
    }
}

// Work tables from the per-expert counts (cnt in shared memory, one thread per expert): offsets, chunks of CHUNK_ROWS
// rows, groups of GROUP_CHUNKS chunks.  Experts that take the tensor-core lane get no chunks.  On a table overflow the
// status word is set and no chunk is written.
__device__ __forceinline__ void build_tables(const uint32_t* cnt, uint32_t E, const uint8_t* __restrict__ loaded,
                                             DispatchTables t, uint32_t CHUNK_ROWS, uint32_t GROUP_CHUNKS, uint32_t HEAVY,
                                             uint32_t* ws, uint32_t* status) {
    const uint32_t e = threadIdx.x;
    const uint32_t c = e < E ? cnt[e] : 0u;
    const uint32_t nc = (e >= E || takes_tensor_lane(c, HEAVY, loaded, e)) ? 0u : (c + CHUNK_ROWS - 1) / CHUNK_ROWS;
    const uint32_t ng = (nc + GROUP_CHUNKS - 1) / GROUP_CHUNKS;
    const uint32_t v[3] = {c, nc, ng};
    uint32_t ex[3], tot[3];
    block_scan3(v, ex, tot, ws);
    const uint32_t distinct = (uint32_t)__syncthreads_count(c != 0u);
    if (e < E) t.offsets[e] = ex[0];
    const bool ok = tot[1] <= t.max_chunks;
    if (threadIdx.x == 0) {
        t.offsets[E] = tot[0];
        if (!ok) atomicMax(status, (uint32_t)ST_WORKLIST_OVERFLOW);
        t.header[HDR_NCHUNKS] = ok ? tot[1] : 0u;
        t.header[HDR_NGROUPS] = ok ? tot[2] : 0u;
        t.header[HDR_CTR_GU] = 0;
        t.header[HDR_CTR_DOWN] = 0;
        t.header[HDR_CTR_AUX] = 0;
        t.header[HDR_DISTINCT] = distinct;
    }
    if (ok && e < E) {
        for (uint32_t i = 0; i < nc; ++i) {
            const uint32_t ch = ex[1] + i;
            t.chunk_expert[ch] = e;
            t.chunk_row0[ch] = ex[0] + i * CHUNK_ROWS;
            t.chunk_rows[ch] = min(CHUNK_ROWS, c - i * CHUNK_ROWS);
        }
        for (uint32_t i = 0; i < ng; ++i) {
            t.group_chunk0[ex[2] + i] = ex[1] + i * GROUP_CHUNKS;
            t.group_mc[ex[2] + i] = min(GROUP_CHUNKS, nc - i * GROUP_CHUNKS) | e << 16;
        }
    }
}

// Stable placement of one block of up to DTHREADS assignments (a = first + thread index, all threads call).  Inside a warp
// the lanes with the same expert find each other (match); the warps' counts per expert go through shared memory, a thread per
// expert turns them into the warps' first positions.  (The warps taking turns instead, a barrier each, was 10 of the 12 us
// that 512 rows took.)  pos[id]: the expert's running position; wcnt: place_words(n_warps, E) words.
__host__ __device__ inline uint32_t place_warps(uint32_t rows) { return rows >= (uint32_t)DTHREADS ? DTHREADS / 32u : (rows + 31u) / 32u; }
__host__ __device__ inline size_t place_words(uint32_t n_warps, uint32_t E) { return ((size_t)n_warps * E + 1) / 2; }
__device__ __forceinline__ void place_block(uint32_t id, bool valid, uint32_t a, uint32_t n_warps, uint32_t E, uint32_t* pos,
                                            uint32_t* wcnt, uint32_t* __restrict__ order) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint16_t* wc = reinterpret_cast<uint16_t*>(wcnt);   // [warp][expert]
    for (uint32_t i = threadIdx.x; i < (n_warps * E + 1) / 2; i += DTHREADS) wcnt[i] = 0;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? id : 0xFFFFFFFFu);
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    __syncthreads();
    if (valid && rank == 0) wc[warp * E + id] = (uint16_t)__popc(peers);
    __syncthreads();
    uint32_t sum = 0;
    if (threadIdx.x < E)   // E <= DTHREADS
        for (uint32_t w = 0; w < n_warps; ++w) {
            const uint32_t c = wc[w * E + threadIdx.x];
            wc[w * E + threadIdx.x] = (uint16_t)sum;
            sum += c;
        }
    __syncthreads();
    if (valid) order[pos[id] + wc[warp * E + id] + rank] = a;
    __syncthreads();
    if (threadIdx.x < E) pos[threadIdx.x] += sum;
    __syncthreads();
}

// Few assignments (a decode step of up to four tokens of top-8): a thread per assignment finds its place by looking at all of
// them, a few barriers instead of fourteen.  What the scan and the placement write is written here entry by entry: the thread of
// an expert's rank-th assignment writes the chunk that starts there, if one does, and the group.  The code of a decode step's
// small kernels comes cold, so its length counts: the loops are not unrolled (unrolled, 8 rows took 9,500 cycles).  Inside the
// front kernel, against the scan: 8 rows 7,700 -> 3,600 cycles, 56 rows 7,500 -> 7,400, 128 rows 8,100 -> 13,300.
constexpr uint32_t DISPATCH_FEW = 32;
__device__ __forceinline__ void dispatch_few(const int32_t* __restrict__ ids, uint32_t A, uint32_t E, const uint8_t* __restrict__ loaded,
                                             DispatchTables t, uint32_t CHUNK_ROWS, uint32_t GROUP_CHUNKS, uint32_t HEAVY,
                                             uint32_t* status, uint32_t* dsm) {
    uint4* ids4 = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(dsm) + 15) / 16 * 16);   // [DISPATCH_FEW] ids
    uint4* key4 = ids4 + DISPATCH_FEW / 4;                                                     // [DISPATCH_FEW] id << 2 | starts a group << 1 | starts a chunk
    const uint32_t a = threadIdx.x, n4 = (A + 3) / 4;
    uint32_t id = 0x3FFFFFFFu;   // behind every expert
    if (a < A) {
        const int32_t v = ids[a];
        const bool good = v >= 0 && (uint32_t)v < E;
        id = good ? (uint32_t)v : 0u;
        if (!good) atomicMax(status, (uint32_t)ST_BAD_EXPERT_ID);
        else if (loaded && !loaded[v]) atomicMax(status, (uint32_t)ST_NOT_LOADED);
    }
    if (a < DISPATCH_FEW) reinterpret_cast<uint32_t*>(ids4)[a] = id;
    __syncthreads();
    if (a < E) {   // E <= DTHREADS
        uint32_t less = 0;
#pragma unroll 1
        for (uint32_t i = 0; i < n4; ++i) {
            const uint4 w = ids4[i];
            less += (w.x < a) + (w.y < a) + (w.z < a) + (w.w < a);
        }
        t.offsets[a] = less;
    }
    uint32_t less = 0, rank = 0, c = 0;
    bool chunk = false, group = false;
    if (a < A) {
#pragma unroll 1
        for (uint32_t i = 0; i < n4; ++i) {
            const uint4 q = ids4[i];
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                less += w[k] < id;
                c += w[k] == id;
                rank += w[k] == id && 4 * i + k < a;
            }
        }
        t.order[less + rank] = a;
        chunk = !takes_tensor_lane(c, HEAVY, loaded, id) && rank % CHUNK_ROWS == 0;
        group = chunk && rank % (CHUNK_ROWS * GROUP_CHUNKS) == 0;
    }
    if (a < DISPATCH_FEW) reinterpret_cast<uint32_t*>(key4)[a] = id << 2 | (group ? 2u : 0u) | (chunk ? 1u : 0u);
    const uint32_t n_chunks = (uint32_t)__syncthreads_count(chunk), n_groups = (uint32_t)__syncthreads_count(group);
    const uint32_t distinct = (uint32_t)__syncthreads_count(a < A && rank == 0);
    const bool ok = n_chunks <= t.max_chunks;
    if (a == 0) {
        t.offsets[E] = A;
        if (!ok) atomicMax(status, (uint32_t)ST_WORKLIST_OVERFLOW);
        t.header[HDR_NCHUNKS] = ok ? n_chunks : 0u;
        t.header[HDR_NGROUPS] = ok ? n_groups : 0u;
        t.header[HDR_CTR_GU] = 0;
        t.header[HDR_CTR_DOWN] = 0;
        t.header[HDR_CTR_AUX] = 0;
        t.header[HDR_DISTINCT] = distinct;
    }
    if (chunk && ok) {
        uint32_t ch = rank / CHUNK_ROWS, g = ch / GROUP_CHUNKS;
        const uint32_t in = g * GROUP_CHUNKS, nc = (c + CHUNK_ROWS - 1) / CHUNK_ROWS;
#pragma unroll 1
        for (uint32_t i = 0; i < n4; ++i) {
            const uint4 q = key4[i];
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const bool before = (w[k] >> 2) < id;
                ch += before && (w[k] & 1u);
                g += before && (w[k] & 2u);
            }
        }
        t.chunk_expert[ch] = id;
        t.chunk_row0[ch] = less + rank;
        t.chunk_rows[ch] = min(CHUNK_ROWS, c - rank);
        if (group) {
            t.group_chunk0[g] = ch;
            t.group_mc[g] = min(GROUP_CHUNKS, nc - in) | id << 16;
        }
    }
    __syncthreads();
}

// The whole sort by one CTA of DTHREADS threads (A <= 2048 rows in practice); dsm: dispatch_words(A, E) words of shared memory
__host__ __device__ inline size_t dispatch_words(uint32_t A, uint32_t E) {
    static_assert(2 * DISPATCH_FEW + 3 <= 99, "the short sort's ids and keys fit where the scan's scratch is");
    return (size_t)E + 99 + place_words(place_warps(A), E);
}
__device__ __forceinline__ void dispatch_body(const int32_t* __restrict__ ids, uint32_t A, uint32_t E,
                                              const uint8_t* __restrict__ loaded, DispatchTables t, uint32_t CHUNK_ROWS,
                                              uint32_t GROUP_CHUNKS, uint32_t HEAVY, uint32_t* status, uint32_t* dsm) {
    if (A <= DISPATCH_FEW) return dispatch_few(ids, A, E, loaded, t, CHUNK_ROWS, GROUP_CHUNKS, HEAVY, status, dsm);
    uint32_t* cnt = dsm;                // [E] counts, then running write positions
    uint32_t* ws = dsm + E;             // [99] scan scratch
    const uint32_t tid = threadIdx.x;
    for (uint32_t e = tid; e < E; e += DTHREADS) cnt[e] = 0;
    __syncthreads();
    for (uint32_t a = tid; a < A; a += DTHREADS) {
        int32_t id = ids[a];
        if (id < 0 || (uint32_t)id >= E) { atomicMax(status, (uint32_t)ST_BAD_EXPERT_ID); id = 0; }
        else if (loaded && !loaded[id]) atomicMax(status, (uint32_t)ST_NOT_LOADED);
        atomicAdd(&cnt[id], 1u);
    }
    __syncthreads();
    build_tables(cnt, E, loaded, t, CHUNK_ROWS, GROUP_CHUNKS, HEAVY, ws, status);
    __syncthreads();
    if (tid < E) cnt[tid] = t.offsets[tid];   // the entry this thread wrote
    __syncthreads();
    for (uint32_t a0 = 0; a0 < A; a0 += DTHREADS) {
        const uint32_t a = a0 + tid, left = A - a0;
        uint32_t id = 0;
        if (a < A) {
            const int32_t v = ids[a];
            id = (v < 0 || (uint32_t)v >= E) ? 0u : (uint32_t)v;
        }
        place_block(id, a < A, a, place_warps(left), E, cnt, ws + 99, t.order);
    }
}

}  // namespace mlxs
