// The tensor-core lane of the banks that decode their weights on the SM (exl3_prefill.cu, fp4_prefill.cu): the pipeline that
// both share.  A bank supplies its code stream's stages, the decode of a quarter of a stage, and the epilogue of a pass.
//
// A CTA owns (expert, a tile of up to 192 of its rows, a 128-column block) and walks the inputs once per projection (a
// "pass": gate then up, or down alone).  W^T is the MMA's A operand (M = 128 output columns), decoded straight into tensor
// memory; the rows are the B operand in shared memory (N = rows rounded to 16), staged by a prep kernel as K-major core
// matrices with fixed offsets (eight rows' 128 inputs are 2 KB), so the MMA descriptors advance by constants.
//   * One pass has one accumulator group of at most 192 tensor-memory columns, so two of them fit (384) beside two decoded
//     stages of 128 inputs (2 x 64): the epilogue of a pass runs on warps of its own under the next pass' decode and MMAs.
//     Calls whose tiles have at most 160 or 128 rows leave room for three or four decoded stages: the decode then runs
//     further ahead and a stage's round trip (decode, store, MMAs, slot free) no longer shows.
//     With gate and up accumulated together (2 x 192, one buffer) the K loop stood still for the epilogue, a fifth of an
//     item's time, and experts of 65 .. 96 rows paid for it most.
//   * 16 decode warps in teams that take the stages in turn.  A warp decodes a first piece of its 32 columns into registers
//     (BK::AHEAD quarters of a stage) and only then waits for its operand slot: the MMAs of the slot's last stage run under the decode.  With three or four
//     operand slots there are four teams of four warps, a warp decoding both halves of a stage, with two slots two teams of
//     eight (a team of four keeps its slot for twice as long).  The barriers around a stage were a quarter of the instructions
//     of a warp that decoded one half (EXL3: 60 per 16x16 tile, about 42 of them the decode), and their latencies showed where the
//     decode is short: EXL3 8 % at 2048 tokens and 4 % at 8192, MXFP4 20 % at 2048 and 12 % at 3500.
//     (EXL3 with quarters instead of halves between the stores, or with 5 or 6 warps per lane quarter: slower or equal.)
//   * The MMA warp runs its loop with all lanes and issues under elect.sync (see elect_one); one commit per stage frees the
//     operand slot and the rows' slot.  What its operands come from goes through a shuffle from lane 0, so that the compiler
//     knows that the warp has one value: they stay in uniform registers instead of being moved there for every MMA (cycles
//     from a stage's operands to its eight MMAs issued, 64 / 128 / 256 rows: EXL3 659 / 749 / 778 -> 578 / 728 / 703, NVFP4 at
//     128 554 -> 499; the layer at 2048 EXL3 tokens 2.4 %, 8192 3.0 %, NVFP4 at 4093 3033 -> 2974 us).
//     The FP4 banks, whose decode is short, test the next stage's barrier in the middle of a stage's MMAs and decode and store a
//     quarter of a stage at a time (the first waits for the slot): NVFP4 at 4093 tokens 2979 -> 2949 us, MXFP4 at 16384 6280 -> 6150.
//     What is left there is the copy of rows and codes from L2, 55 to 62 bytes per clock and SM (41 and 53 KB per stage of 760
//     and 870 cycles; the MMAs alone are 520 and 700).  EXL3 is bound by the decode: neither helps, half a stage at a time is 1 %
//     faster at 8192 tokens.
//   * One producer lane streams the code, another the rows: bulk copies into rings.
//   * The code producer takes the CTA's items one by one from a counter and passes them on to the other roles.  Beside the
//     streaming lane the CTAs start when SMs come free, up to a third of the kernel apart, and with items dealt out in
//     advance the last CTA to start decided the time.
// Every wait is bounded; on a give-up the CTA sets the status word, skips work and still frees its tensor memory.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

// -DMLXS_LANE_COUNTERS: cycle counters around the waits and the MMA issue of one CTA, printed once per launch (how the
// lane's bound was found; off in the library)
#ifdef MLXS_LANE_COUNTERS
#include <cstdio>
#define LC(...) __VA_ARGS__
#else
#define LC(...)
#endif

namespace mlxs {

constexpr int LN_KST = 128;             // inputs per stage
constexpr int LN_A_COLS = LN_KST / 2;   // tensor-memory columns of a decoded stage
constexpr int LN_ROWS = 192;            // most rows of a tile
constexpr int LN_ROWS_NARROW = 160;     // most rows that leave room for three operand slots
constexpr int LN_RAW_STAGES = 8;        // most stages of the code ring: two per team
constexpr int LN_B_STAGES = 3;          // stages of the rows' ring
// Items announced to the roles.  An entry is written again LN_ITEMS items later: the code ring, the operand slots and the two
// accumulator buffers keep the slowest role (the epilogue) within 8 + 4 + 3 one-stage items of the code producer.
constexpr uint32_t LN_ITEMS = 32, LN_NO_ITEM = 0xFFFFFFFFu;
constexpr int LN_DONE = 4;              // barriers of the stages in flight: operands complete, MMAs complete
constexpr int LN_DEC_WARPS = 16, LN_EPI_WARPS = 8;
// warps 0 .. 3: MMA, code producer, rows' producer, none; then the decode warps, then the epilogue warps.  The scheduler
// favours the older warp, and the few instructions of the MMA warp are the ones that everybody waits for.
constexpr int LN_SERVICE = 4;
constexpr int LN_THREADS = (LN_SERVICE + LN_DEC_WARPS + LN_EPI_WARPS) * 32;
constexpr uint32_t LN_B_SLOT = LN_ROWS * LN_KST * 2;
constexpr uint32_t LN_LBO = 128, LN_SBO = 2048;   // byte distance of two core matrices along K, along N
// Staged rows of a tile with rows16 rows: [input / 128][row / 8][position / 8 of the 128][row % 8][position % 8], 16-bit
// elements; the position of an input inside its 128 is the bank's (a dot product does not see the order).  Element offset of
// (row, group of 8 positions) inside a stage:
__device__ __forceinline__ uint32_t ln_row_off(uint32_t row, uint32_t group) { return (row >> 3) * 1024u + group * 64u + (row & 7u) * 8u; }

struct LaneParams {
    const uint8_t* code;         // layer base of the code stream
    size_t expert_stride;        // bytes per expert
    uint32_t n_blocks, n_stages; // out / 128, in / 128
    const uint16_t* xa;          // staged rows, pass p at p * xa_proj_stride elements
    size_t xa_proj_stride;
    const uint32_t* tiles;       // the tile table
    uint32_t* next;              // items given out so far
    DispatchTables t;
    uint32_t H, I;
    const __half* scales;        // EXL3: the layer's sign / scale vectors
    size_t scales_stride;
    const float* gscale;         // NVFP4: [E][3] global scales
    void* act;                   // gate/up: lane_act_bytes per CTA, act(gate) between the two passes
    uint16_t* xd;                // gate/up output = down's staged rows [staging rows][I]
    void* out;                   // down output [A, H]
    int out_bf16;
    float limit;
    uint32_t* status;
};
constexpr size_t LN_ACT_BYTES = (size_t)LN_ROWS * 128 * sizeof(float);   // per CTA

// what an epilogue works with
struct LaneEpi {
    uint32_t ew, q, half, lane;  // epilogue warp, its tensor-memory lane quarter, which half of the warps of that quarter
    uint8_t* smem;               // the bank's epilogue staging
    uint64_t* sync_bar;
    volatile int* abort_flag;
    uint32_t* status;
    uint32_t sync_ph, batch;     // phase of sync_bar; batches so far (EXL3's two staging buffers)
    // rendezvous of the epilogue warps: a bounded mbarrier wait like every other
    __device__ __forceinline__ bool sync() {
        __syncwarp();
        if (lane == 0) mbar_arrive(sync_bar);
        const bool ok = mbar_wait_bounded(sync_bar, sync_ph, abort_flag);
        sync_ph ^= 1u;
        if (!ok) {
            if (!*abort_flag) atomicMax(status, (uint32_t)ST_WAIT_FULL);
            *abort_flag = 1;
        }
        return ok;
    }
};
// one pass of one item for an epilogue
struct LanePass {
    uint32_t acc;                // tensor-memory address of the accumulators (lane 0)
    uint32_t expert, row0, rows, rows16, srow0, nb;
    uint64_t* acc_empty;
    // after a warp's last read of the accumulators
    __device__ __forceinline__ void release(uint32_t lane) const {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
    }
};

// shared memory of the two rings: four code stages beside tiles of up to 192 rows, eight where four teams decode.  (As many stages of
// rows as fit, up to eight, with a slot of the call's largest tile: no faster, and NVFP4 at 4093 tokens 3004 -> 3045 us.)
template <class BK>
constexpr size_t ln_ring_bytes() {
    constexpr size_t two = (size_t)LN_B_STAGES * LN_B_SLOT + 4 * BK::RAW_BYTES;
    constexpr size_t four = (size_t)LN_B_STAGES * LN_ROWS_NARROW * LN_KST * 2 + 8 * BK::RAW_BYTES;
    return two > four ? two : four;
}

// NPASS = 2: gate then up of a column block; 1: down
template <class BK, int NPASS>
__global__ void __launch_bounds__(LN_THREADS, 1) lane_kernel(const LaneParams P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t raw_full[LN_RAW_STAGES], raw_empty[LN_RAW_STAGES];
    __shared__ __align__(8) uint64_t bar_stage[2 * LN_DONE], acc_full[2], acc_empty[2], epi_bar, item_full[LN_ITEMS];
    __shared__ uint4 s_tile[LN_ITEMS];       // the tile's entry
    __shared__ uint32_t s_nb[LN_ITEMS];      // the column block, LN_NO_ITEM behind the last item
    uint64_t *full = bar_stage, *done = bar_stage + LN_DONE;             // of the stages in flight: operands complete, MMAs complete
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const uint32_t n_items = P.tiles[0] * P.n_blocks;
    // a CTA that cannot get work leaves before it takes tensor memory (the whole CTA reads the same count)
    if (blockIdx.x >= n_items) return;

    const uint32_t most = __shfl_sync(0xFFFFFFFFu, P.tiles[2], 0);
    // columns of an accumulator buffer (the call's largest tile), operand slots in what is left
    const uint32_t acc_cols = most <= 128u ? 128u : most <= (uint32_t)LN_ROWS_NARROW ? (uint32_t)LN_ROWS_NARROW : (uint32_t)LN_ROWS, slots = (512u - 2u * acc_cols) / LN_A_COLS;
    const uint32_t teams = slots >= 3 ? 4u : 2u, raw_stages = 2u * teams, b_slot = acc_cols * (LN_KST * 2u);
    uint8_t* b_ring = smem_raw;                                          // [stage][rows16 x 256 B]
    uint8_t* raw_ring = b_ring + LN_B_STAGES * b_slot;                   // [stage][BK::RAW_BYTES]
    if (threadIdx.x == 0) {
        for (int s = 0; s < LN_RAW_STAGES; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], LN_DEC_WARPS / teams); }
        // a stage's operands: the team's warps have stored theirs, the rows have landed
        for (int s = 0; s < LN_DONE; ++s) { mbar_init(&full[s], LN_DEC_WARPS / teams + 1); mbar_init(&done[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], LN_EPI_WARPS); }
        mbar_init(&epi_bar, LN_EPI_WARPS);
        for (uint32_t s = 0; s < LN_ITEMS; ++s) mbar_init(&item_full[s], 1);
        s_abort = 0;
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    const uint32_t first = threadIdx.x == 32 ? atomicAdd(P.next, 1u) : 0u;   // the code producer's first item
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, s_tmem, 0), tmem_a = tmem + 2 * acc_cols;
    const uint32_t nstage = P.n_stages, width = nstage * LN_KST;
    auto give_up = [&](uint32_t code) { if (!s_abort) atomicMax(P.status, code); s_abort = 1; };
    // item number n of this CTA, once it is known; false: there is none (or the CTA has given up)
    auto next_item = [&](uint32_t n, uint4& tile, uint32_t& nb, uint32_t sleep_ns) -> bool {
        const uint32_t s = n % LN_ITEMS;
        if (!mbar_wait_bounded(&item_full[s], (n / LN_ITEMS) & 1u, &s_abort, sleep_ns)) { give_up(ST_WAIT_FULL); return false; }
        tile = s_tile[s];
        nb = s_nb[s];
        return nb != LN_NO_ITEM;
    };

    // a decode warp (lane quarter q, team; of two teams: half of the stage's inputs)
    auto decode_stages = [&](auto teams_c) {
        constexpr uint32_t TEAMS = decltype(teams_c)::value;
        const uint32_t dw = warp - LN_SERVICE, q = warp & 3u, team = TEAMS == 4 ? dw >> 2 : dw >> 3, half = TEAMS == 4 ? 0u : (dw >> 2) & 1u;
        const typename BK::Decoder dec(q, half, lane);
        const uint8_t* raw = raw_ring + team * BK::RAW_BYTES;
        const uint32_t ta0 = tmem_a + ((q * 32u) << 16) + half * (LN_A_COLS / 2);
        // The team's stages are g = team + TEAMS i: code slot and code barriers alternate between team and team + TEAMS, their
        // phases flip every second stage.  The instructions around the decode count (it is issue-bound), so those addresses
        // advance by an exclusive-or, and the next stage's code is tested for behind this stage's last decode: a test of a
        // barrier that is ready costs its latency, which the stores and the arrivals hide.
        const uint32_t bar0 = smem_u32(&bar_stage[0]);
        uint32_t b_raw = smem_u32(&raw_full[team]), b_emp = smem_u32(&raw_empty[team]);
        const uint32_t x_raw = b_raw ^ smem_u32(&raw_full[team + TEAMS]), x_emp = b_emp ^ smem_u32(&raw_empty[team + TEAMS]);
        bool code_ready = false;
        uint32_t woff = 0, slot = team % slots;            // of stage g: g % slots
        uint32_t items = 0, known = 0;                     // items so far and the stages they have
        LC(long long t_item = 0, t_code = 0, t_slot = 0; uint32_t n_st = 0; long long t0;)
        for (uint32_t i = 0;; ++i) {
            const uint32_t g = team + TEAMS * i;
            bool more = true;
            LC(t0 = clock64(); ++n_st;)
            while (more && g >= known) {
                uint4 tile;
                uint32_t nb;
                more = next_item(items++, tile, nb, 0);
                known += NPASS * nstage;
            }
            if (!more) break;
            LC(t_item += clock64() - t0; t0 = clock64();)
            if (!code_ready && !mbar_wait_bounded_at(b_raw, (i >> 1) & 1u, &s_abort)) { give_up(ST_WAIT_FULL); break; }
            LC(t_code += clock64() - t0;)
            // this slot's last MMAs are stage d = g - slots
            const uint32_t d = g - slots, b_done = bar0 + 8 * LN_DONE + 8 * (d % LN_DONE), ph_done = (d / LN_DONE) & 1u;
            constexpr uint32_t GROUPS = (TEAMS == 4 ? 4u : 2u) / BK::AHEAD;
            bool ok = true;
#pragma unroll
            for (uint32_t gr = 0; gr < GROUPS; ++gr) {
                uint32_t v[BK::AHEAD][16];
#pragma unroll
                for (uint32_t k = 0; k < BK::AHEAD; ++k) dec.decode(raw, woff, gr * BK::AHEAD + k, v[k]);
                if (gr + 1 == GROUPS) {
                    b_raw ^= x_raw;
                    code_ready = mbar_test_at(b_raw, ((i + 1) >> 1) & 1u);
                    __syncwarp();
                    if (lane == 0) mbar_arrive_at(b_emp);
                }
                if (gr == 0) {
                    LC(t0 = clock64();)
                    if (g >= slots && !mbar_wait_bounded_at(b_done, ph_done, &s_abort)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
                    LC(t_slot += clock64() - t0;)
                    tc_fence_after();
                }
#pragma unroll
                for (uint32_t k = 0; k < BK::AHEAD; ++k) BK::Decoder::store(ta0 + slot * LN_A_COLS, gr * BK::AHEAD + k, v[k]);
            }
            if (!ok) break;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_at(bar0 + 8 * (g % LN_DONE));
            b_emp ^= x_emp; woff ^= TEAMS * BK::RAW_BYTES;
            if (TEAMS == 4 && slots == 3) slot = slot == 2 ? 0u : slot + 1;   // else the slot stays the team's
        }
        LC(if (blockIdx.x == 3 && lane == 0 && (warp == 13 || warp == 16) && n_st) printf("LANE<%d> decode warp %u: %u stages, cycles per stage: item %lld code %lld slot %lld\n", NPASS, warp, n_st, t_item / n_st, t_code / n_st, t_slot / n_st);)
    };

    if (warp >= LN_SERVICE && warp < LN_SERVICE + LN_DEC_WARPS) {
        // ---------------- decode warps ----------------
        LC(const long long c0 = clock64();)
        if (teams == 4) decode_stages(std::integral_constant<uint32_t, 4>());
        else decode_stages(std::integral_constant<uint32_t, 2>());
        LC(if (blockIdx.x == 3 && lane == 0 && warp == 13) printf("LANE<%d> decode warp: %lld cycles\n", NPASS, clock64() - c0);)
    } else if (warp >= LN_SERVICE + LN_DEC_WARPS) {
        // ---------------- epilogue warps ----------------
        LaneEpi E;
        E.ew = warp - LN_SERVICE - LN_DEC_WARPS; E.q = warp & 3u; E.half = E.ew >> 2; E.lane = lane;
        E.smem = smem_raw + ln_ring_bytes<BK>();
        E.sync_bar = &epi_bar; E.abort_flag = &s_abort; E.status = P.status; E.sync_ph = 0; E.batch = 0;
        uint32_t pass_n = 0;
        LC(long long t_wait = 0, t_epi = 0;)
        bool ok = true;
        for (uint32_t it = 0; ok; ++it) {
            LanePass C;
            uint4 te;
            if (!next_item(it, te, C.nb, 200)) break;
            C.expert = te.x; C.row0 = te.y; C.rows = te.z; C.srow0 = te.w; C.rows16 = (te.z + 15) / 16 * 16;
#pragma unroll
            for (int p = 0; p < NPASS && ok; ++p, ++pass_n) {
                const uint32_t buf = pass_n & 1u;
                LC(const long long e0 = clock64();)
                if (!mbar_wait_bounded(&acc_full[buf], (pass_n >> 1) & 1u, &s_abort, 200)) { give_up(ST_WAIT_FULL); ok = false; break; }
                tc_fence_after();
                LC(const long long e1 = clock64(); t_wait += e1 - e0;)
                C.acc = tmem + buf * acc_cols;
                C.acc_empty = &acc_empty[buf];
                ok = p == 0 ? BK::template epilogue<NPASS, 0>(P, E, C) : BK::template epilogue<NPASS, NPASS - 1>(P, E, C);
                LC(t_epi += clock64() - e1;)
            }
        }
        LC(if (blockIdx.x == 3 && lane == 0 && E.ew == 1) printf("LANE<%d> epilogue: %u passes, cycles per pass: wait %lld work %lld\n", NPASS, pass_n, t_wait / pass_n, t_epi / pass_n);)
    } else if (warp == 1) {
        // ---------------- code producer ----------------
        if (lane == 0) {
            uint32_t g = 0;
            for (uint32_t it = 0;; ++it) {
                const uint32_t item = it ? atomicAdd(P.next, 1u) : first;
                const bool more = item < n_items && !s_abort;
                const uint32_t nb = more ? item % P.n_blocks : LN_NO_ITEM;
                const uint4 te = *reinterpret_cast<const uint4*>(prefill_tile(P.tiles, more ? item / P.n_blocks : 0u));
                s_tile[it % LN_ITEMS] = te;
                s_nb[it % LN_ITEMS] = nb;
                mbar_arrive(&item_full[it % LN_ITEMS]);
                if (!more) break;
                const uint8_t* src = P.code + (size_t)te.x * P.expert_stride + (size_t)nb * NPASS * nstage * BK::RAW_BYTES;
                for (uint32_t ks = 0; ks < NPASS * nstage; ++ks, ++g) {
                    const uint32_t rs = g & (raw_stages - 1u);
                    if (!mbar_wait_bounded(&raw_empty[rs], ((g >> (teams == 4 ? 3 : 2)) & 1u) ^ 1u, &s_abort, 64)) { give_up(ST_WAIT_EMPTY); break; }
                    mbar_expect_tx(&raw_full[rs], BK::RAW_BYTES);
                    BK::template copy_stage<NPASS>(raw_ring + rs * BK::RAW_BYTES, src, ks, nstage, &raw_full[rs]);
                }
            }
            if (s_abort) for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
    } else if (warp == 0) {
        // ---------------- MMA issuer: the whole warp walks the loop, one elected lane issues ----------------
        // Between a stage's last MMA and the next one's first only a few MMAs are queued, so this warp's own instructions show:
        // everything a stage needs is worked out before the stage before it is issued.
        uint32_t pass_n = 0;
        const uint64_t bdesc = umma_smem_desc(smem_u32(b_ring), LN_LBO, LN_SBO);
        const uint32_t bd_hi = (uint32_t)(bdesc >> 32), bd_lo0 = (uint32_t)bdesc, bd_step = b_slot >> 4, bd_end = bd_lo0 + LN_B_STAGES * bd_step;
        const uint32_t a_end = tmem_a + slots * LN_A_COLS;
        uint32_t bd_lo = bd_lo0, a0 = tmem_a, bars = smem_u32(&bar_stage[0]), par = 0;   // bars: full[g % LN_DONE], done[g % LN_DONE] 8 LN_DONE bytes on
        const uint32_t bars_end = bars + 8 * LN_DONE;
        bool ok = true, ready = false;
        LC(long long m_a = 0, m_issue = 0, m_acc = 0, m_item = 0, m_all = clock64(); uint32_t g = 0;)
        for (uint32_t it = 0; ok; ++it) {
            uint4 te;
            uint32_t nb;
            LC(long long w0 = clock64();)
            if (!__all_sync(0xFFFFFFFFu, next_item(it, te, nb, 0))) break;
            LC(m_item += clock64() - w0;)
            const uint32_t idesc = umma_idesc(BK::FORMAT, __shfl_sync(0xFFFFFFFFu, (te.z + 15) / 16 * 16, 0));
            for (int p = 0; p < NPASS && ok; ++p, ++pass_n) {
                const uint32_t buf = pass_n & 1u, acc = tmem + buf * acc_cols;
                LC(w0 = clock64();)
                if (!mbar_wait_warp(&acc_empty[buf], ((pass_n >> 1) & 1u) ^ 1u, &s_abort)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
                LC(m_acc += clock64() - w0;)
                for (uint32_t ks = 0; ks < nstage; ++ks) {
                    LC(const long long w1 = clock64(); ++g;)
                    if (!ready && !mbar_wait_warp_at(bars, par, &s_abort)) { give_up(ST_WAIT_FULL); ok = false; break; }
                    tc_fence_after();
                    LC(const long long w2 = clock64();)
                    const uint32_t bars_n = bars + 8 == bars_end ? bars_end - 8 * LN_DONE : bars + 8, par_n = bars + 8 == bars_end ? par ^ 1u : par;
                    const uint32_t bd_n = bd_lo + bd_step == bd_end ? bd_lo0 : bd_lo + bd_step;
                    if (elect_one()) {
                        umma_f16_ts_lohi(acc, a0, bd_lo, bd_hi, idesc, ks);
#pragma unroll
                        for (int i = 1; i < BK::MID; ++i) umma_f16_ts_lohi(acc, a0 + i * 8, bd_lo + ((i * 2 * LN_LBO) >> 4), bd_hi, idesc, 1u);
                    }
                    // the test of the next stage's barrier goes out between the MMAs: behind the last one its latency would show
                    bool next = false;
                    if (BK::MID < LN_KST / 16) next = mbar_test_at(bars_n, par_n);
                    if (elect_one()) {
#pragma unroll
                        for (int i = BK::MID; i < LN_KST / 16; ++i) umma_f16_ts_lohi(acc, a0 + i * 8, bd_lo + ((i * 2 * LN_LBO) >> 4), bd_hi, idesc, 1u);
                        // one commit per stage frees the operand slot and the rows' slot
                        umma_commit_at(bars + 8 * LN_DONE);
                        if (ks + 1 == nstage) umma_commit(&acc_full[buf]);
                    }
                    ready = __all_sync(0xFFFFFFFFu, next);
                    bars = bars_n; par = par_n; bd_lo = bd_n; a0 = a0 + LN_A_COLS == a_end ? tmem_a : a0 + LN_A_COLS;
                    LC(m_a += w2 - w1; m_issue += clock64() - w2;)
                }
            }
        }
        LC(if (blockIdx.x == 3 && g && lane == 0) printf("LANE<%d> mma warp: %u stages, cycles per stage: operand wait %lld issue %lld acc %lld item %lld all %lld\n", NPASS, g, m_a / g, m_issue / g, m_acc / g, m_item / g, (clock64() - m_all) / g);)
    } else if (warp == 2) {
        // ---------------- rows' producer ----------------
        if (lane == 0) {
            uint32_t g = 0, bs = 0;
            for (uint32_t it = 0; !s_abort; ++it) {
                uint4 te;
                uint32_t nb;
                if (!next_item(it, te, nb, 64)) break;
                const uint32_t rows16 = (te.z + 15) / 16 * 16, b_bytes = rows16 * LN_KST * 2;
                for (int p = 0; p < NPASS; ++p) {
                    const uint16_t* xsrc = P.xa + p * P.xa_proj_stride + (size_t)te.w * width;
                    for (uint32_t ks = 0; ks < nstage; ++ks, ++g) {
                        if (g >= LN_B_STAGES) {
                            const uint32_t d = g - LN_B_STAGES;
                            if (!mbar_wait_bounded(&done[d % LN_DONE], (d / LN_DONE) & 1u, &s_abort, 64)) { give_up(ST_WAIT_EMPTY); break; }
                        }
                        mbar_expect_tx(&full[g % LN_DONE], b_bytes);
                        bulk_g2s(b_ring + bs * b_slot, xsrc + (size_t)ks * (rows16 * LN_KST), b_bytes, &full[g % LN_DONE]);
                        if (++bs == LN_B_STAGES) bs = 0;
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

template <class BK, int NPASS>
static cudaError_t lane_launch(const LaneParams& P, int sm_count, cudaStream_t st) {
    const size_t smem = ln_ring_bytes<BK>() + BK::EPI_SMEM;
    cudaError_t e = cudaFuncSetAttribute(lane_kernel<BK, NPASS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    lane_kernel<BK, NPASS><<<sm_count, LN_THREADS, smem, st>>>(P);
    return cudaGetLastError();
}

}  // namespace mlxs
