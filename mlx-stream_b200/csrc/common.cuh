// Shared device helpers for the routed-MoE kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mlxs {

// Error words kernels may write into the handle's status word (never trap, never spin without a bound).
enum : uint32_t {
    ST_OK = 0,
    ST_BAD_EXPERT_ID = 1,    // a routed id outside [0, n_experts)
    ST_WAIT_FULL = 2,        // a consumer's bounded wait for a staged copy ran out
    ST_WAIT_EMPTY = 3,       // the producer's bounded wait for a free stage ran out
    ST_WORKLIST_OVERFLOW = 4,
    ST_NOT_LOADED = 5,       // a routed expert has no resident record
    ST_EP_OVERFLOW = 6,      // expert parallel: a rank received more rows than its workspace holds
    ST_EP_TIMEOUT = 7        // expert parallel: a peer's epoch word did not arrive within the bound
};

constexpr uint32_t SCALE_BITS = 0x3DB504F3u;  // 128^-0.5 (src/arch/deepseek_v41/experts.zig:428-429)
constexpr uint32_t MUL1 = 0x83DCD12Du;        // src/expert/bank.zig:109

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier + bulk copy (TMA 1-D) ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) {   // by shared-memory address
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { mbar_arrive_at(smem_u32(bar)); }
__device__ __forceinline__ bool mbar_try_wait_at(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// a test that never suspends the warp (try_wait may, for a time that the hardware chooses)
__device__ __forceinline__ bool mbar_test_at(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) { return mbar_try_wait_at(smem_u32(bar), parity); }
// Bounded wait: gives up after `limit` polls (each poll itself blocks for a hardware-defined slice) or as soon as
// *abort_flag is set by another thread of the CTA.  Returns false when it gave up.
// sleep_ns > 0: back off between polls (the single-lane producer / MMA-issuer roles wait most of the time; polling
// flat out would take issue slots from the warps that do the arithmetic).
__device__ __forceinline__ bool mbar_wait_bounded_at(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                     uint32_t sleep_ns = 0, uint32_t limit = (1u << 20)) {
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait_at(bar, parity)) return true;
        if (sleep_ns) __nanosleep(sleep_ns);
        if ((i & 63u) == 63u && *abort_flag) return false;
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  uint32_t sleep_ns = 0, uint32_t limit = (1u << 20)) {
    return mbar_wait_bounded_at(smem_u32(bar), parity, abort_flag, sleep_ns, limit);
}
// global -> this CTA's shared memory, completion counted in bytes on `bar`; 16-byte aligned addresses and size
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Programmatic dependent launch (the chain router -> dispatch -> staging -> gate/up -> down -> combine): a kernel lets the
// next one of the stream start while it still runs; the next one does what needs nothing of it (its prologue, the down
// kernel its first weight copies) and then waits for the whole grid before it and for its memory.  A kernel allows its
// successor only after its own wait, so whatever a successor reads before waiting comes from grids that are complete.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... Params, class... Args>
static inline cudaError_t launch_dependent(bool dependent, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = &attr; cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// ---- tensor-core fragment op: D(16x8 f32) += A(16x16 f16, row) x B(16x8 f16, col) ----
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- EXL3 mul1: two 16-bit trellis states -> half2 (lo = a, hi = b) ----
// value = f16( (1024 + bytesum(state * 0x83DCD12D)) * h(0x1EEE) + h(0xC931) ), one rounding
// (src/exl3/kernels.zig:963-971; src/kernels/exl3/dsv41_exl3_mul1h_k3_2304.metal:27-31)
// The two halves are put together by a byte permute (logic pipe), not a multiply-add: the half-rate multiply pipe has 20 of a
// tile's instructions already (46.8 against 48.5 cycles per tile at K = 3, 43.8 against 45.5 at K = 2; in the tensor-core
// lane, whose epilogue warps use the logic pipe, the two are within 0.7 %).
__device__ __forceinline__ uint32_t mul1_pair(uint32_t sa, uint32_t sb) {
    uint32_t xa = sa * MUL1, xb = sb * MUL1;
    uint32_t ha = __dp4a(xa, 0x01010101u, 0x6400u);  // 0x6400 + byte sum = the half bits of 1024 + s
    uint32_t hb = __dp4a(xb, 0x01010101u, 0x6400u);
    uint32_t pk = __byte_perm(ha, hb, 0x5410);
    const uint32_t kinv = 0x1EEE1EEEu, kbias = 0xC931C931u;
    __half2 r = __hfma2(*reinterpret_cast<__half2*>(&pk), *reinterpret_cast<const __half2*>(&kinv),
                        *reinterpret_cast<const __half2*>(&kbias));
    return *reinterpret_cast<uint32_t*>(&r);
}

// ---- the lane's share of a quad: four k-tiles (64 inputs) of one 16-column tile ----
// A tile's 256 states follow each other in its code (K bits apart, the 16 bits of state i end at stream bit K (i + 1),
// circular; src/exl3/kernels.zig:978-1020).  Lane l = 4 u + j takes the 32 consecutive states 32 u .. 32 u + 31 of k-tile j:
// the 16 inputs of the output columns u and u + 8 (the exllamav3 tensor-core order).  They lie in K whole words and the last
// bits of the word before, so every window has a constant place: no shift by a lane's own distance, no two words per eight
// states.  States 8 c .. 8 c + 7 are b[0..3] = the weights of column u, inputs (2c, 2c+1), (2c+8, 2c+9), then column u + 8's.
// Lanes 4u .. 4u + 3 hold the same columns of four k-tiles, which is one mma A fragment (or one tcgen05.st.16x256b fragment)
// per c with inputs of all four k-tiles; whoever multiplies takes the rows in that order (position 16 c + 4 j + 2 h + b of
// the 64 = input 16 j + 2 c + 8 h + b).
// Against eight states per lane and tile (two words, a funnel shift by the lane) 64 tokens take 1941 -> 1852 us, 16 of K = 2
// 955 -> 887.  In the bare loop with one mma per tile 58.5 -> 55.3 cycles per tile and scheduler (K = 2 57.4 -> 52.5), 46.7 and 43.8
// of them the decode: an mma.sync costs 8.7 whatever its shape.
// The quad in memory: word w of the four k-tiles beside each other, [8 K words][4 k-tiles]: four 4-byte loads here, two 16-byte
// loads for four tiles in the tensor-core lane.  At K = 3 a load's lanes take 32 banks, at K = 2 the lanes u and u + 4 share one.
// (A lane's first two words as one 8-byte load: 1834 and 870 us, but the tensor-core lane would need eight loads again.)
// The tensor-core lane multiplies 16 inputs of one k-tile at a time instead (exl3_decode_lane): with the quad's order the grouping of
// its sums over the inputs changes, and the f16 and bf16 roundings behind them turn that into 2e-4 of a layer's rows and, layer by
// layer, into as much as 1e-2 after four (the streaming kernel's order alone: 5e-6 to 5e-5, 6e-3).
template <int KB>
__device__ __forceinline__ void exl3_quad_words(const uint32_t* __restrict__ quad, uint32_t lane, uint32_t (&z)[4]) {
    // z: the stream's words from its last on, z[KB] = the word before the lane's first (its neighbour's last)
    const uint32_t u = lane >> 2, j = lane & 3u;
    const uint32_t* w = quad + (KB * 4u) * u + j;
#pragma unroll
    for (int i = 0; i < KB; ++i) z[i] = w[4 * (KB - 1 - i)];
    z[KB] = quad[(u ? KB * 4u * u : KB * 32u) - 4u + j];
    if (KB == 2) z[3] = 0u;
}
// 32 stream bits from bit O on (counted from the last)
template <int O>
__device__ __forceinline__ uint32_t exl3_bits(const uint32_t (&z)[4]) {
    return O % 32 == 0 ? z[O / 32] : __funnelshift_r(z[O / 32], z[O / 32 + 1 < 4 ? O / 32 + 1 : 3], O % 32);
}
// the state at bit O: one byte permute or shift where it is byte-aligned inside a word, else a funnel shift and a mask
template <int O>
__device__ __forceinline__ uint32_t exl3_state(const uint32_t (&z)[4]) {
    return O % 32 == 8 ? __byte_perm(z[O / 32], 0u, 0x4421) : O % 32 == 16 ? z[O / 32] >> 16 : exl3_bits<O>(z) & 0xFFFFu;
}
template <int KB, int C>
__device__ __forceinline__ void exl3_decode8(const uint32_t (&z)[4], uint32_t (&b)[4]) {
    constexpr int B = KB * (24 - 8 * C);   // of the group's last state
    if (KB == 3) {
        b[0] = mul1_pair(exl3_state<B + 21>(z), exl3_state<B + 18>(z));
        b[1] = mul1_pair(exl3_state<B + 15>(z), exl3_state<B + 12>(z));
        b[2] = mul1_pair(exl3_state<B + 9>(z), exl3_state<B + 6>(z));
        b[3] = mul1_pair(exl3_state<B + 3>(z), exl3_state<B>(z));
    } else {
        // states four apart are a byte apart: one funnel shift serves both
        const uint32_t f0 = exl3_bits<B>(z), f1 = exl3_bits<B + 2>(z), f2 = exl3_bits<B + 4>(z), f3 = exl3_bits<B + 6>(z);
        b[0] = mul1_pair(__byte_perm(f3, 0u, 0x4421), __byte_perm(f2, 0u, 0x4421));
        b[1] = mul1_pair(__byte_perm(f1, 0u, 0x4421), __byte_perm(f0, 0u, 0x4421));
        b[2] = mul1_pair(f3 & 0xFFFFu, f2 & 0xFFFFu);
        b[3] = mul1_pair(f1 & 0xFFFFu, f0 & 0xFFFFu);
    }
}
// all of it: v[4 c + i] = b[i] of group c
template <int KB>
__device__ __forceinline__ void exl3_decode_quad(const uint32_t (&z)[4], uint32_t (&v)[16]) {
    uint32_t b[4];
    auto put = [&](int c) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * c + i] = b[i];
    };
    exl3_decode8<KB, 0>(z, b); put(0);
    exl3_decode8<KB, 1>(z, b); put(1);
    exl3_decode8<KB, 2>(z, b); put(2);
    exl3_decode8<KB, 3>(z, b); put(3);
}

// ---- one lane's share of one tile (the tensor-core lane) ----
// A 16x16 K=3 tile: lane L owns code positions 8L..8L+7, i.e. the 37 stream bits ending at
// stream bit 24(L+1); `lo` is the tile word holding that last bit, `hi` the word before it (circular), lp the
// distance of the last bit from the word's bit 0.  Returns the two B fragments (k16 x n8) of the tile's column
// halves for mma m16n8k16: b[0], b[1] = columns 0..7, b[2], b[3] = columns 8..15 (the exllamav3 tensor-core order,
// src/exl3/kernels.zig:978-986).
__device__ __forceinline__ void exl3_decode_lane(uint32_t lo, uint32_t hi, uint32_t lp, uint32_t (&b)[4]) {
    uint32_t v0 = __funnelshift_r(lo, hi, lp);  // stream bits, window m at bits [3m, 3m+16)
    uint32_t vh = hi >> lp;
    uint32_t v1 = __funnelshift_r(v0, vh, 18);  // windows 6, 7 at bits 0 and 3
    uint32_t w0 = v0 & 0xFFFFu;
    uint32_t w1 = (v0 >> 3) & 0xFFFFu;
    uint32_t w2 = (v0 >> 6) & 0xFFFFu;
    uint32_t w3 = (v0 >> 9) & 0xFFFFu;
    uint32_t w4 = (v0 >> 12) & 0xFFFFu;
    uint32_t w5 = (v0 >> 15) & 0xFFFFu;
    uint32_t w6 = v1 & 0xFFFFu;
    uint32_t w7 = (v1 >> 3) & 0xFFFFu;
    // code position j = 7 - m; positions (0,1),(2,3) -> columns 0..7 rows (r0,r0+1),(r0+8,r0+9); (4,5),(6,7) -> 8..15
    b[0] = mul1_pair(w7, w6);
    b[1] = mul1_pair(w5, w4);
    b[2] = mul1_pair(w3, w2);
    b[3] = mul1_pair(w1, w0);
}
__device__ __forceinline__ void exl3_lane_plan(uint32_t lane, uint32_t& wi, uint32_t& wj, uint32_t& lp) {
    wi = (3u * lane + 2u) >> 2;        // word of the lane's last stream bit
    wj = (wi + 23u) % 24u;             // the word before it, circular
    lp = 8u * ((lane + 1u) & 3u);
}
// The same for K = 2 (a tile is 16 words): lane L's 8 states end at stream bits 16 L + 2 .. 16 L + 16, i.e. they live in
// the 30 bits ending with halfword L.  `lo` = the word holding halfword L, `hi` = the word before it (circular),
// lp = 0 when halfword L is the word's low half, 16 when it is the high half; window m at bits [2m, 2m + 16).
// Bit-level definition: src/exl3/kernels.zig:988-1020 (tileStates at K = 2), generic window formulas
// scripts/dsv41_exl3_k2_gen.py:96-112.
__device__ __forceinline__ void exl3_decode_lane_k2(uint32_t lo, uint32_t hi, uint32_t lp, uint32_t (&b)[4]) {
    const uint32_t v0 = __funnelshift_r(lo, hi, lp);
    // states four apart are a byte apart: one shift serves both
    const uint32_t v2 = v0 >> 2, v4 = v0 >> 4, v6 = v0 >> 6;
    const uint32_t w0 = v0 & 0xFFFFu, w1 = v2 & 0xFFFFu, w2 = v4 & 0xFFFFu, w3 = v6 & 0xFFFFu;
    const uint32_t w4 = __byte_perm(v0, 0u, 0x4421), w5 = __byte_perm(v2, 0u, 0x4421), w6 = __byte_perm(v4, 0u, 0x4421), w7 = __byte_perm(v6, 0u, 0x4421);
    b[0] = mul1_pair(w7, w6);
    b[1] = mul1_pair(w5, w4);
    b[2] = mul1_pair(w3, w2);
    b[3] = mul1_pair(w1, w0);
}
__device__ __forceinline__ void exl3_lane_plan_k2(uint32_t lane, uint32_t& wi, uint32_t& wj, uint32_t& lp) {
    wi = lane >> 1;
    wj = (wi + 15u) % 16u;
    lp = (lane & 1u) ? 0u : 16u;
}
// by code width
template <int KB>
__device__ __forceinline__ void exl3_decode_lane_kb(uint32_t lo, uint32_t hi, uint32_t lp, uint32_t (&b)[4]) {
    if (KB == 3) exl3_decode_lane(lo, hi, lp, b);
    else exl3_decode_lane_k2(lo, hi, lp, b);
}
template <int KB>
__device__ __forceinline__ void exl3_lane_plan_kb(uint32_t lane, uint32_t& wi, uint32_t& wj, uint32_t& lp) {
    if (KB == 3) exl3_lane_plan(lane, wi, wj, lp);
    else exl3_lane_plan_k2(lane, wi, wj, lp);
}

// ---- 128-point Sylvester-natural Hadamard over a warp: lane holds elements 4*lane .. 4*lane+3 ----
// (unnormalised; src/arch/glm5_next/exl3_forms_ref.zig:116-135)
__device__ __forceinline__ void hadamard128_warp(float (&v)[4], uint32_t lane) {
    float a0 = v[0] + v[1], a1 = v[0] - v[1], a2 = v[2] + v[3], a3 = v[2] - v[3];
    v[0] = a0 + a2; v[1] = a1 + a3; v[2] = a0 - a2; v[3] = a1 - a3;
#pragma unroll
    for (uint32_t m = 1; m < 32; m <<= 1) {
        bool up = (lane & m) != 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float o = __shfl_xor_sync(0xFFFFFFFFu, v[q], m);
            v[q] = up ? (o - v[q]) : (v[q] + o);
        }
    }
}

// split an f32 into f16 hi + f16 lo (hi + lo carries ~22 significant bits)
__device__ __forceinline__ void split_hi_lo(float x, __half& hi, __half& lo) {
    hi = __float2half_rn(x);
    lo = __float2half_rn(x - __half2float(hi));
}
__device__ __forceinline__ uint32_t pack_h2(__half a, __half b) {
    return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}
__device__ __forceinline__ float bf16_round_f(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// 1 / (1 + e^|x|) through the special-function unit (ex2.approx, rcp.approx: a few ulp) for the tensor-core lanes, whose
// results are rounded to 16 bits right after; the streaming lanes keep expf and the IEEE division
__device__ __forceinline__ float sigmoid_tail_fast(float x) { return __fdividef(1.0f, 1.0f + __expf(fabsf(x))); }

// Over how many CTAs (1, 2 or 4, at most lp) the parts of an item's sum are spread in one call of a streaming kernel:
// as many as still give every unit a CTA of its own.  (Splitting further to even out the SMs' shares was measured: the
// extra folds cost more than the balance gains, 0.165 against 0.156 ms at one token.)  cap_items: the items the fold's
// workspace holds.
__device__ __forceinline__ uint32_t ksplit_ctas(uint32_t n_items, uint32_t lp, uint32_t grid, uint32_t cap_items) {
    if (!n_items || n_items > cap_items) return 1u;
    uint32_t np = 1;
    while (np < lp && n_items * (np * 2) <= grid) np *= 2;
    return np;
}

// ---- fixed-sequence exp / log for the router: IEEE +, *, fma, / only, so the host restatement of the same
// statements gives the same bits ----
__device__ __forceinline__ float det_expf(float x) {
    if (x != x) return x;
    if (x > 88.75f) return __int_as_float(0x7F800000);
    if (x < -104.0f) return 0.0f;
    const float magic = 12582912.0f;
    float t = __fmul_rn(x, 1.44269504f);
    float n = __fsub_rn(__fadd_rn(t, magic), magic);
    float r = __fmaf_rn(n, -0.693145752f, x);
    r = __fmaf_rn(n, -1.42860677e-06f, r);
    float p = 1.98412701e-04f;
    p = __fmaf_rn(p, r, 1.38888892e-03f);
    p = __fmaf_rn(p, r, 8.33333377e-03f);
    p = __fmaf_rn(p, r, 4.16666679e-02f);
    p = __fmaf_rn(p, r, 1.66666672e-01f);
    p = __fmaf_rn(p, r, 0.5f);
    p = __fmaf_rn(p, r, 1.0f);
    p = __fmaf_rn(p, r, 1.0f);
    int ni = (int)n;
    int n1 = ni / 2, n2 = ni - n1;
    float s1 = __int_as_float((n1 + 127) << 23), s2 = __int_as_float((n2 + 127) << 23);
    return __fmul_rn(__fmul_rn(p, s1), s2);
}
__device__ __forceinline__ float det_logf(float x) {
    uint32_t b = __float_as_uint(x);
    int e = (int)(b >> 23) - 127;
    float m = __uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
    if (m > 1.41421354f) { m = __fmul_rn(m, 0.5f); e += 1; }
    float f = __fsub_rn(m, 1.0f);
    float s = __fdiv_rn(f, __fadd_rn(2.0f, f));
    float z = __fmul_rn(s, s);
    float R = 9.09090936e-02f;
    R = __fmaf_rn(R, z, 1.11111112e-01f);
    R = __fmaf_rn(R, z, 1.42857149e-01f);
    R = __fmaf_rn(R, z, 0.2f);
    R = __fmaf_rn(R, z, 3.33333343e-01f);
    R = __fmul_rn(R, z);
    float s2 = __fadd_rn(s, s);
    float lo = __fmaf_rn(s2, R, s2);
    float ef = (float)e;
    lo = __fmaf_rn(ef, 1.42860677e-06f, lo);
    return __fmaf_rn(ef, 0.693145752f, lo);
}

}  // namespace mlxs
