// tcgen05 (5th-generation tensor core) wrappers shared by the tensor-core lanes: one CTA per MMA (cta_group::1),
// operands in shared memory as K-major core matrices without swizzle, f32 accumulators in tensor memory.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace mlxs {

enum { UMMA_F16 = 0, UMMA_BF16 = 1 };  // operand format codes of kind::f16

// shared-memory operand descriptor: K-major, no swizzle.  A core matrix is 8 rows x 16 bytes, contiguous (128 B);
// lbo = byte distance of two core matrices along K, sbo = along M / N; addresses and offsets in units of 16 bytes.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor: D f32 (bits 4-5 = 1), A and B format at bits 7-9 / 10-12, both K-major, N >> 3 at bit 17,
// M = 128 (>> 4 at bit 24)
__device__ __forceinline__ uint32_t umma_idesc(uint32_t fmt, uint32_t n) {
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// tensor memory: one warp allocates `cols` columns (a power of two >= 32), writes the base address to shared memory
// and gives up the permit so that a later CTA on the SM can allocate; the same warp frees them
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// One lane of a converged warp (the same one every time).  The MMA warps run their loops with all 32 lanes and put only
// the MMAs and commits of a stage under this predicate: the operands of tcgen05.mma are warp-uniform registers, and with
// the loop inside an `if (lane == 0)` every one of them costs the issuing thread extra instructions.  Measured per MMA
// (M 128, A in tensor memory) beside 16 warps that decode and store operands: one-lane loop 157 cycles whatever N is,
// elected issue 76 / 84 / 98 / 115 cycles at N = 16 / 64 / 128 / 192 (an idle SM: 72 - 97 against 37 / 46 / 65 / 97).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}
// a bounded wait by all lanes of a warp: one answer for the warp
__device__ __forceinline__ bool mbar_wait_warp_at(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (__all_sync(0xFFFFFFFFu, mbar_try_wait_at(bar, parity))) return true;
    return __all_sync(0xFFFFFFFFu, mbar_wait_bounded_at(bar, parity, abort_flag));
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t sleep_ns = 0,
                                               uint32_t limit = (1u << 20)) {
    return __all_sync(0xFFFFFFFFu, mbar_wait_bounded(bar, parity, abort_flag, sleep_ns, limit));
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the same with the A operand in tensor memory: lane = row of A (M = 128), a 32-bit column holds two consecutive K
// elements of a 16-bit type, so one instruction (K = 16) reads 8 columns from a_tmem on
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the same with the shared-memory descriptor as two words: an address step stays inside the low word
__device__ __forceinline__ void umma_f16_ts_lohi(uint32_t tmem_d, uint32_t tmem_a, uint32_t db_lo, uint32_t db_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(db_lo), "r"(db_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_at(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) { umma_commit_at(smem_u32(bar)); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
}  // namespace mlxs
