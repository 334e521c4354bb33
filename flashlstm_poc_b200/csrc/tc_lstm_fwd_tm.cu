// Persistent recurrent forward kernel with W_hh in TENSOR MEMORY: one launch runs all T time steps of one layer whose
// slice of W_hh does not fit shared memory.
//
// What bounds the streamed form (tc_lstm_fwd.cu without resident weights) is the slice itself: at H = 2048 every CTA pulls
// 256 KB of W_hh from L2 each step through an SM port of about 60 B per cycle (4.4 k of a 9.8 k-cycle step), at H = 4096 the
// 134 MB come from HBM.  The accumulators need a few dozen of the 512 tensor-memory columns; the others hold the slice as the
// A operand of tcgen05.mma, what does not fit there stays in shared memory, and only what fits neither is streamed.
//
// This form, with a counter per step, runs batch tiles of 64 sequences and everything streamed; tiles of 32 whose slice stays on the
// chip exchange without it (tc_lstm_fwd_tm_direct.cu), and share the split below.
//
// Work split.  CTA pairs (cta_group::2, M = 256): 128 tensor-memory lanes per CTA.
//   S = 2 (H <= 16 x SMs): a CTA owns 64 gate rows (16 units).  Lanes 0-63 hold their first half of K = H, lanes 64-127 the
//         second half, so that the lanes are full; the B operand has 2 BT rows, K half 0 of the BT sequences staged by the
//         leader and K half 1 by its peer.  The accumulator is 128 lanes x 2 BT columns, of which the blocks (half q, columns
//         of half q) are the two partial sums that the epilogue adds; the other two blocks are computed and ignored.
//   S = 1 (wider layers): a CTA owns 128 gate rows (32 units), the pair's B operand is BT sequences, each CTA stages BT / 2.
// Either way a CTA stages half of what its rows need of h, and nothing is multicast.
//
// K runs in chunk-steps of 64 per half: [0, ct) from tensor memory, [ct, ct + cs) from shared memory.  The rest is streamed
// through a ring of slots by a warp of its own, ascending in even steps of the sequence and descending in odd ones: the slots then
// still hold the chunk-steps that the next step starts with, and L2 is asked first for what it was given last (in one direction
// 94 MB per step go round in its 126 MB and mostly miss).  The direction is the order of the sums: it follows the step's number
// in its sequence, so that a sequence cut into ranges or segments gives the bits of one launch.  A step takes the chunk-steps
// that the slots hold first, so that copies start as soon as h is there, then those in tensor and shared memory, then the
// streamed ones.  Roles, step barrier, epilogue and the way out after a bounded wait expired are the other forward kernel's
// (tc_lstm_fwd.cu): producer and UMMA threads break out of their loops, the 256 epilogue threads leave together, an aborted pair
// lingers before its final cluster barrier.
//
// Replaces the same reference launches as tc_lstm_fwd.cu (flashlstm_v2/src/lstm_forward.cu:744-830, src/lstm.cu:1241-1337).
#include <cstdlib>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc_common.cuh"
#include "tc_kernels.h"
#include "tc_recurrent.cuh"

namespace flstm_b200 {
namespace tc {

namespace {

constexpr int kThreads = 352;  // warps 0-3 and 6-9 epilogue, 4 producer of h, 5 UMMA issuer, 10 producer of weights
constexpr int kEpilogueThreads = 256;
constexpr int kStepBytesW = 128 * 128;  // one chunk-step of A: 128 rows x 64 16-bit elements
constexpr int kTmemColumns = 512;
constexpr int kBarrierBytes = 1024, kMinSmemBytes = 120 * 1024;
// Even: a slot always belongs to the same set of warps.  A set that met a slot only every other time could find its first phase
// still open, whose parity reads as that of the phase it waits for.
constexpr int kFillSlots = (kMinSmemBytes - 1024 - kBarrierBytes) / kStepBytesW / 2 * 2;
constexpr int WCH = kFwdTmGroup;

struct Layout {
    int w, wring, h, p, ex, total;
};

__host__ __device__ inline Layout layout_of(const FwdTmPlan &pl) {
    Layout l;
    l.w = pl.cs * kStepBytesW;
    l.wring = pl.wstages * WCH * kStepBytesW;
    l.h = pl.hstages * pl.ch * (pl.S * pl.BT / 2) * 128;
    l.p = 2 * (2 / pl.S) * pl.BT * 128;
    l.ex = 128 * (pl.BT + 4) * 4;
    l.total = kBarrierBytes + l.w + l.wring + l.h + l.p + l.ex + 1024 /*align*/;
    return l;
}

// The order in which a step takes its chunk-steps: up to three runs, each ascending or descending, each fetched in copies of
// ch chunk-steps of h (a last copy brings chunk-steps that are not used).
struct Run {
    int lo, hi;  // chunk-steps [lo, hi)
    __device__ int copies(int ch) const { return (hi - lo + ch - 1) / ch; }
};
template <bool STREAM>
__device__ __forceinline__ Run run_of(const FwdTmPlan &pl, int which, bool down) {
    const int first = pl.ct + pl.cs;  // first streamed chunk-step
    if (!STREAM) return Run{0, which == 0 ? pl.kc : 0};
    if (which == 1) return Run{0, first};
    const int ring = pl.wstages * WCH, held = down ? pl.kc - ring : first;  // what the slots hold when the step begins
    if (which == 0) return Run{held, held + ring};
    return down ? Run{first, pl.kc - ring} : Run{first + ring, pl.kc};
}

template <int S, int BT, bool STREAM, bool BF16, bool ACCURATE>
__global__ void __launch_bounds__(kThreads, 1)
lstm_fwd_tm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_ws, const __grid_constant__ CUtensorMap tm_h,
                   const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ FwdTmPlan pl, FwdParams p) {
    constexpr int ROWS = 128 / S, UT = 2 / S;  // gate rows and 16-unit tiles of this CTA
    constexpr int N = S * BT, BROWS = N / 2;   // UMMA N, B rows a CTA stages
    constexpr int EXS = BT + 4;                // row stride of the exchange buffer (floats), keeps float4 alignment
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const Layout L = layout_of(pl);
    const int KC = pl.kc, CT = pl.ct, CS = pl.cs, CH = pl.ch, HST = pl.hstages, WST = pl.wstages;
    uint8_t *s_w = smem + kBarrierBytes, *s_wr = s_w + L.w, *s_h = s_wr + L.wring, *s_p = s_h + L.h;
    float *s_ex = reinterpret_cast<float *>(s_p + L.p);
    uint64_t *hfull = reinterpret_cast<uint64_t *>(smem), *hempty = hfull + HST;
    uint64_t *wfull = hempty + HST, *wempty = wfull + WST;
    uint64_t *tfull = wempty + WST, *tempty = tfull + 1, *wbar = tempty + 1;
    uint64_t *pfull = wbar + 1, *pempty = pfull + 2;
    uint64_t *ffull = pempty + 2, *fempty = ffull + kFillSlots;  // while W_hh moves into tensor memory
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fempty + kFillSlots);
    volatile uint32_t *abort_w = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ng = blockIdx.x / pl.cta_rows, jr = blockIdx.x % pl.cta_rows;  // batch group, row block
    const int b0 = ng * BT;
    unsigned int *counter = p.counters + ng;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < HST; ++i) {
            mbar_init(&hfull[i], 1);
            mbar_init(&hempty[i], 1);
        }
        for (int i = 0; i < WST; ++i) {
            mbar_init(&wfull[i], 1);
            mbar_init(&wempty[i], 1);
        }
        mbar_init(tfull, 1);
        mbar_init(tempty, 2 * kEpilogueThreads / 32);  // the epilogue warps of both CTAs report to the leader
        mbar_init(wbar, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&pfull[i], 1);
            mbar_init(&pempty[i], kEpilogueThreads / 32);
        }
        for (int i = 0; i < kFillSlots; ++i) {
            mbar_init(&ffull[i], 1);
            mbar_init(&fempty[i], 4);
        }
        *abort_w = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_w);
        if (STREAM) tma_prefetch_desc(&tm_ws);
        tma_prefetch_desc(&tm_h);
        tma_prefetch_desc(&tm_g);
    }
    if (warp == 5) {
        tmem_alloc_pair(tmem_slot, kTmemColumns);
        tmem_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + N;
    const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
    // W_hh into tensor memory, by way of the shared memory that the rings will use: lane l of the CTA takes row l % ROWS, K half
    // l / ROWS, 32 columns of two elements per chunk-step; the warps 0-3 take the even chunk-steps, 6-9 the odd ones (a warp
    // reaches the lane quadrant warp % 4).  Loads straight from global memory, a row of 128 bytes per lane, took 10 us more per
    // launch at H = 1024.  A wait that expires raises the abort word, on which every role below gives up.
    if (warp == 4 && elect_one()) {
        for (int c = 0; c < CT; ++c) {
            const int slot = c % kFillSlots;
            uint8_t *dst = s_w + slot * kStepBytesW;
            if (c >= kFillSlots && !mbar_wait(&fempty[slot], (uint32_t)(c / kFillSlots - 1) & 1u, abort_w, wait_ns)) break;
            mbar_expect_tx(&ffull[slot], kStepBytesW);
            tma_load_2d(dst, &tm_w, c * 64, jr * ROWS, &ffull[slot]);
            tma_load_2d(dst + 8192, &tm_w, (S == 2 ? KC + c : c) * 64, jr * ROWS + (S == 2 ? 0 : 64), &ffull[slot]);
        }
    } else if (warp != 4 && warp != 5 && warp != 10) {
        const int quad = warp & 3, l = quad * 32 + lane;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        for (int c = warp < 4 ? 0 : 1; c < CT; c += 2) {
            const int slot = c % kFillSlots;
            if (!__all_sync(0xffffffffu, mbar_wait(&ffull[slot], (uint32_t)(c / kFillSlots) & 1u, abort_w, wait_ns))) break;
            const uint8_t *row = s_w + slot * kStepBytesW + l * 128;
            uint32_t r[32];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 v = *reinterpret_cast<const uint4 *>(row + ((i ^ (l & 7)) * 16));
                r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
            }
            tmem_st_32x32b_x32(dst + c * 32, r);
            __syncwarp();
            if (lane == 0) mbar_arrive(&fempty[slot]);
        }
        tmem_st_wait();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers and tensor memory exist before anything crosses the pair
    tcgen05_fence_after();
    // barriers the loads of this CTA complete: the leader's at the same offsets
    const uint32_t hfull_c = map_to_rank(smem_u32(hfull), 0), wfull_c = map_to_rank(smem_u32(wfull), 0);
    const uint32_t wbar_c = map_to_rank(smem_u32(wbar), 0), tempty_c = map_to_rank(smem_u32(tempty), 0);
    const uint32_t hstage_bytes = (uint32_t)(CH * BROWS * 128);
    auto load_w = [&](uint8_t *dst, int c, uint32_t bar) {  // chunk-step c of this CTA's rows; beyond K come zeros
        tma_load_2d_pair(dst, &tm_w, c * 64, jr * ROWS, bar);
        tma_load_2d_pair(dst + 8192, &tm_w, (S == 2 ? KC + c : c) * 64, jr * ROWS + (S == 2 ? 0 : 64), bar);
    };

    const bool tracing = p.trace != nullptr && blockIdx.x == 0;
#define FLSTM_STAMP(step, slot)                                                     \
    do {                                                                            \
        if (tracing && (step) < p.trace_steps) p.trace[(step) * 16 + (slot)] = clock64(); \
    } while (0)

    if (warp == 4) {
        // ------------------------------------------------------------ producer: projection tiles and h
        if (elect_one()) {
            bool ok = true;
            int stage = 0;
            uint32_t phase = 0;
            uint32_t h_issued = 0, h_parity = 0, p_issued = 0, p_parity = 0;
            for (int tt = 0; tt < p.T && ok; ++tt) {
                const int t = p.t0 + tt, pb = tt & 1;
                ok = mbar_wait(&pempty[pb], ((tt >> 1) & 1) ^ 1, abort_w, wait_ns);
                if (!ok) break;
                mbar_expect_tx(&pfull[pb], UT * BT * 128);
                for (int r = 0; r < UT; ++r)
                    tma_load_3d(s_p + (pb * UT + r) * BT * 128, &tm_g, (jr * UT + r) * 64, b0, t, &pfull[pb]);
                p_issued |= 1u << pb;
                p_parity = (p_parity & ~(1u << pb)) | (((tt >> 1) & 1u) << pb);
                // Without a ring the copies of a step are announced ahead of its barrier (their phases of the step before are
                // over long since) and follow it back to back: 1814 -> 1762 us a pass at H = 1024, B = 32, T = 512
                const bool whole = !STREAM && !pl.hring;
                for (int i = 0; whole && leader && i < HST; ++i) {
                    if (tt > 0 && !mbar_wait(&hfull[i], (uint32_t)(tt - 1) & 1u, abort_w, wait_ns)) ok = false;
                    if (!ok) break;
                    mbar_expect_tx(&hfull[i], 2 * hstage_bytes);
                }
                if (!ok) break;
                if (tt > 0) {  // h_{t-1} is complete when every CTA of the group has arrived tt times in this launch
                    ok = wait_counter(counter, (unsigned)pl.cta_rows * (unsigned)tt + p.extra_arrivals, p.err, abort_w, 2u, wait_ns);
                    if (!ok) break;
                    fence_proxy_async_global();
                }
                FLSTM_STAMP(tt, 0);
                for (int i = 0; whole && i < HST; ++i)
                    tma_load_4d_pair(s_h + i * hstage_bytes, &tm_h, 0, S == 2 ? b0 : b0 + (int)rank * BROWS,
                                     (S == 2 ? (int)rank * KC : 0) + i * CH, t, hfull_c + 8u * (uint32_t)i);
                if (whole) {
                    h_issued = (1u << HST) - 1u;
                    h_parity = tt & 1 ? h_issued : 0u;
                }
                const bool down = STREAM && ((tt + p.odd) & 1);
                for (int which = 0; !whole && which < (STREAM ? 3 : 1) && ok; ++which) {
                    const Run run = run_of<STREAM>(pl, which, down);
                    const bool desc = down && which != 1;
                    for (int i = 0, n = run.copies(CH); i < n; ++i) {
                        ok = mbar_wait(&hempty[stage], phase ^ 1, abort_w, wait_ns);
                        if (!ok) break;
                        if (leader) mbar_expect_tx(&hfull[stage], 2 * hstage_bytes);
                        h_issued |= 1u << stage;
                        h_parity = (h_parity & ~(1u << stage)) | (phase << stage);
                        // chunks beyond K come as zeros (and are counted)
                        const int c = desc ? run.hi - (i + 1) * CH : run.lo + i * CH;
                        tma_load_4d_pair(s_h + stage * hstage_bytes, &tm_h, 0, S == 2 ? b0 : b0 + (int)rank * BROWS,
                                         (S == 2 ? (int)rank * KC : 0) + c, t, hfull_c + 8u * (uint32_t)stage);
                        if (++stage == HST) { stage = 0; phase ^= 1; }
                    }
                }
                if (!ok) break;
                FLSTM_STAMP(tt, 1);
            }
            // way out: every copy this thread started must have landed before the CTA exits (the peer's copies complete
            // the leader's barriers; after an abort the whole pair lingers, see below)
            for (int i = 0; i < HST && leader; ++i)
                if (h_issued >> i & 1u) mbar_drain(&hfull[i], h_parity >> i & 1u, ok ? wait_ns : kAbortDrainNs);
            for (int i = 0; i < 2; ++i)
                if (p_issued >> i & 1u) mbar_drain(&pfull[i], p_parity >> i & 1u, wait_ns);
        }
    } else if (warp == 10) {
        // ------------------------------------------------------------ producer: weights kept in shared memory, streamed weights
        if (elect_one()) {
            bool ok = true;
            if (CS > 0) {
                if (leader) mbar_expect_tx(wbar, 2u * (uint32_t)(CS * kStepBytesW));
                for (int c = 0; c < CS; ++c) load_w(s_w + c * kStepBytesW, CT + c, wbar_c);
            }
            // group i of wch chunk-steps lives in slot i % WST; a load waits until the group WST before it (in the direction of the
            // step) has been consumed
            uint32_t loaded = 0, parity = 0, eparity = 0;
            const int first = CT + CS, n = STREAM ? (KC - first) / WCH : 0, slot_bytes = WCH * kStepBytesW;
            for (int tt = 0; STREAM && tt < p.T && ok; ++tt) {
                const bool down = (tt + p.odd) & 1;
                for (int k = tt == 0 ? 0 : WST; k < n; ++k) {
                    const int i = down ? n - 1 - k : k, slot = i % WST;
                    if (k >= WST) {
                        ok = mbar_wait(&wempty[slot], eparity >> slot & 1u, abort_w, wait_ns);
                        if (!ok) break;
                        eparity ^= 1u << slot;
                    }
                    if (leader) mbar_expect_tx(&wfull[slot], 2u * (uint32_t)slot_bytes);
                    if (loaded >> slot & 1u) parity ^= 1u << slot;
                    loaded |= 1u << slot;
                    tma_load_4d_pair(s_wr + slot * slot_bytes, &tm_ws, 0, jr * ROWS, first + i * WCH, 0, wfull_c + 8u * (uint32_t)slot);
                }
            }
            if (CS > 0 && leader) mbar_drain(wbar, 0, wait_ns);
            for (int i = 0; i < WST && leader; ++i)
                if (loaded >> i & 1u) mbar_drain(&wfull[i], parity >> i & 1u, ok ? wait_ns : kAbortDrainNs);
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ UMMA issuer (the leader's)
        if (leader && elect_one()) {
            bool ok = CS == 0 || mbar_wait(wbar, 0, abort_w, wait_ns);
            int hs = 0;
            uint32_t hphase = 0, wparity = 0;
            constexpr uint32_t idesc = umma_idesc_f16(256, N, BF16 ? 1 : 0, 0, 0);
            constexpr uint32_t kStepH = (BROWS * 128) >> 4, kStepW = kStepBytesW >> 4;  // descriptor units
            const uint32_t hempty_l = smem_u32(hempty), wempty_l = smem_u32(wempty), tfull_l = smem_u32(tfull);
            const uint32_t dw_res = umma_desc_lo(smem_u32(s_w)), dw_ring = umma_desc_lo(smem_u32(s_wr)), dh_ring = umma_desc_lo(smem_u32(s_h));
            const int first = CT + CS, ngroups = (KC - first) / WCH;
            int committed = 0;
            for (int tt = 0; tt < p.T && ok; ++tt) {
                ok = mbar_wait_cluster(tempty, (tt & 1) ^ 1, abort_w, wait_ns);
                if (!ok) break;
                tcgen05_fence_after();
                const bool down = STREAM && ((tt + p.odd) & 1);
                uint32_t acc = 0;  // the step's first instruction overwrites the accumulator
                for (int which = 0; which < (STREAM ? 3 : 1) && ok; ++which) {
                    const Run run = run_of<STREAM>(pl, which, down);
                    const bool desc = down && which != 1;
                    int grp = desc ? (run.hi - first) / WCH - 1 : (run.lo - first) / WCH, slot = STREAM && which != 1 ? grp % WST : 0;
                    for (int ld = 0, nld = run.copies(CH); ld < nld; ++ld) {
                        ok = mbar_wait(&hfull[hs], hphase, abort_w, wait_ns);
                        if (!ok) break;
                        if (which == 0 && ld == 0) FLSTM_STAMP(tt, 2);
                        FLSTM_STAMP(tt, 3);
                        tcgen05_fence_after();
                        uint32_t dh = dh_ring + (uint32_t)hs * (hstage_bytes >> 4);
                        if (STREAM && which != 1) {
                            const int left = run.hi - run.lo - ld * CH, cnt = (left < CH ? left : CH) / WCH;  // groups of this copy
                            if (desc) dh += (uint32_t)(CH - WCH) * kStepH;
                            for (int e = 0; e < cnt; ++e) {
                                if (which == 2 || tt == 0) {
                                    ok = mbar_wait(&wfull[slot], wparity >> slot & 1u, abort_w, wait_ns);
                                    if (!ok) break;
                                    wparity ^= 1u << slot;
                                    tcgen05_fence_after();
                                }
                                uint32_t dw = dw_ring + (uint32_t)(slot * WCH) * kStepW;
#pragma unroll
                                for (int c = 0; c < WCH; ++c) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) umma_lo_ss<true>(tmem_base, dw + 2 * k, dh + 2 * k, idesc, k ? 1u : acc);
                                    acc = 1u;
                                    dw += kStepW;
                                    dh += kStepH;
                                }
                                // what the next step begins with stays in its slot
                                if (down ? grp >= WST : grp < ngroups - WST) umma_commit_pair_both(wempty_l + 8u * (uint32_t)slot);
                                if (desc) {
                                    dh -= 2u * (uint32_t)WCH * kStepH;
                                    --grp;
                                    slot = slot == 0 ? WST - 1 : slot - 1;
                                } else {
                                    ++grp;
                                    slot = slot + 1 == WST ? 0 : slot + 1;
                                }
                            }
                            if (!ok) break;
                        } else {
                            int c = run.lo + ld * CH;
                            const int c1 = c + CH < run.hi ? c + CH : run.hi, ct1 = c1 < CT ? c1 : CT;
                            uint32_t da = tmem_a + (uint32_t)c * 32;
#pragma unroll 4
                            for (; c < ct1; ++c) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_lo_ts<true>(tmem_base, da + 8 * k, dh + 2 * k, idesc, k ? 1u : acc);
                                acc = 1u;
                                da += 32;
                                dh += kStepH;
                            }
                            uint32_t dw = dw_res + (uint32_t)(c - CT) * kStepW;
#pragma unroll 2
                            for (; c < c1; ++c) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_lo_ss<true>(tmem_base, dw + 2 * k, dh + 2 * k, idesc, k ? 1u : acc);
                                acc = 1u;
                                dw += kStepW;
                                dh += kStepH;
                            }
                        }
                        if (STREAM || pl.hring) umma_commit_pair_both(hempty_l + 8u * (uint32_t)hs);
                        if (++hs == HST) { hs = 0; hphase ^= 1; }
                    }
                }
                if (!ok) break;
                umma_commit_pair_both(tfull_l);
                ++committed;
                FLSTM_STAMP(tt, 4);
            }
            // the tensor memory is freed at the end of the kernel: the last committed batch of UMMAs must be done
            if (committed > 0) mbar_drain(tfull, (uint32_t)(committed - 1) & 1u, wait_ns);
        }
    } else {
        // ------------------------------------------------------------ epilogue (256 threads)
        const int tid = warp < 4 ? threadIdx.x : threadIdx.x - 64;  // 0..255
        const int u = tid & 15, nb = tid >> 4;  // phase-B ownership: unit u of every 16-unit tile, sequences nb + 16 i
        constexpr int PER = BT / 16, PAIRS = UT * PER;
        float c_keep[PAIRS];
        const size_t slab = (size_t)p.B * p.H, G = (size_t)4 * p.H;
        uint16_t *hs = static_cast<uint16_t *>(p.hs);
        uint16_t *y = static_cast<uint16_t *>(p.y);
        uint16_t *gates = static_cast<uint16_t *>(p.gates);
        const int quad = warp & 3, col0 = warp < 4 ? 0 : BT / 2;  // phase A: lane quadrant, half of the columns
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (S == 2 ? (quad >> 1) * BT : 0) + col0;
        const size_t idx0 = (size_t)(b0 + nb) * p.H + jr * UT * 16 + u;
        const int rows_left = p.B - b0 - nb;  // pair (r, i) exists while 16 i < rows_left
        bool ok = true;
#pragma unroll
        for (int r = 0; r < UT; ++r)
#pragma unroll
            for (int i = 0; i < PER; ++i)
                c_keep[r * PER + i] = 16 * i < rows_left ? p.cs[(size_t)p.t0 * slab + idx0 + (size_t)(16 * i) * p.H + r * 16] : 0.f;
        for (int tt = 0; tt < p.T && ok; ++tt) {
            const int t = p.t0 + tt, pb = tt & 1;
            // No thread leaves between here and the named barrier below, whatever its waits return: the barrier ORs the
            // failures, so that all 256 threads go on or give up together.
            bool good = mbar_wait(&pfull[pb], (tt >> 1) & 1, abort_w, wait_ns);
            float proj[PAIRS][4];
            {
                const uint16_t *ptile = reinterpret_cast<const uint16_t *>(s_p + pb * UT * BT * 128) + nb * 64 + u;
#pragma unroll
                for (int r = 0; r < UT; ++r)
#pragma unroll
                    for (int i = 0; i < PER; ++i)
#pragma unroll
                        for (int g = 0; g < 4; ++g) proj[r * PER + i][g] = load16<BF16>(ptile + r * BT * 64 + i * 1024 + g * 16);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&pempty[pb]);
            uint16_t *h_out = hs + (size_t)(t + 1) * slab + idx0;
            // the whole warp or none of it reads the accumulator
            const bool seen = __all_sync(0xffffffffu, mbar_wait(tfull, tt & 1, abort_w, wait_ns));
            good = good && seen;
            if (tid == 0) FLSTM_STAMP(tt, 5);
            tcgen05_fence_after();
            if (seen) {
                uint32_t acc[BT / 2];
                if (BT == 16) tmem_ld_32x32b_x8(taddr, *reinterpret_cast<uint32_t(*)[8]>(&acc[0]));
                else if (BT == 32) tmem_ld_32x32b_x16(taddr, *reinterpret_cast<uint32_t(*)[16]>(&acc[0]));
                else tmem_ld_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&acc[0]));
                tmem_ld_wait();
                float4 *dst = reinterpret_cast<float4 *>(s_ex + (quad * 32 + lane) * EXS + col0);
#pragma unroll
                for (int i = 0; i < BT / 8; ++i)
                    dst[i] = make_float4(__uint_as_float(acc[4 * i]), __uint_as_float(acc[4 * i + 1]),
                                         __uint_as_float(acc[4 * i + 2]), __uint_as_float(acc[4 * i + 3]));
            }
            tcgen05_fence_before();
            __syncwarp();
            // relaxed: it orders the reuse of the accumulator only (a release would wait for the warp's global stores)
            if (lane == 0) mbar_arrive_cluster_relaxed(tempty_c);
            if (named_barrier_or(1, kEpilogueThreads, !good)) {
                ok = false;
                break;
            }
            if (tid == 0) FLSTM_STAMP(tt, 6);
            float act[PAIRS][4];
            uint16_t h16[PAIRS];
#pragma unroll
            for (int r = 0; r < UT; ++r) {
                const bool pad = ACCURATE && (jr * UT + r) * 16 + u >= p.real_units;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int k = r * PER + i;
                    float a[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float *e = s_ex + (r * 64 + g * 16 + u) * EXS + nb + 16 * i;
                        a[g] = (S == 2 ? e[0] + e[64 * EXS] : e[0]) + proj[k][g];
                    }
                    const float gi = sigmoid_sel<ACCURATE>(pad ? 0.f : a[0]), gf = sigmoid_sel<ACCURATE>(pad ? 0.f : a[1]);
                    const float gg = tanh_sel<ACCURATE>(pad ? 0.f : a[2]), go = sigmoid_sel<ACCURATE>(pad ? 0.f : a[3]);
                    const float c = fmaf(gf, c_keep[k], gi * gg);
                    const float h = go * tanh_sel<ACCURATE>(c);
                    c_keep[k] = c;
                    act[k][0] = gi; act[k][1] = gf; act[k][2] = gg; act[k][3] = go;
                    h16[k] = to16<BF16>(h);
                    // h_t first: it is what the other CTAs wait for
                    if (16 * i < rows_left) h_out[(size_t)(16 * i) * p.H + r * 16] = h16[k];
                }
            }
            if (tid == 0) FLSTM_STAMP(tt, 7);
            // publish h_t: after the named barrier thread 0's release is cumulative over every epilogue warp's stores; the
            // generic->async proxy fence is the consumer's.  The barrier also lets the exchange buffer be written again.
            named_barrier_sync(2, kEpilogueThreads);
            if (tid == 0) red_release_gpu_add(counter, 1u);
            if (tid == 0) FLSTM_STAMP(tt, 8);
            // everything nobody waits for: cell state, gate cache, the caller's y
#pragma unroll
            for (int r = 0; r < UT; ++r)
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    if (16 * i >= rows_left) continue;
                    const int k = r * PER + i;
                    const size_t idx = idx0 + (size_t)(16 * i) * p.H + r * 16;
                    p.cs[(size_t)(t + 1) * slab + idx] = c_keep[k];
                    if (y) y[(size_t)t * slab + idx] = h16[k];
                    if (p.store_gates) {
                        uint16_t *grow = gates + ((size_t)t * p.B + b0 + nb + 16 * i) * G + (size_t)(jr * UT + r) * 64 + u;
#pragma unroll
                        for (int g = 0; g < 4; ++g) grow[g * 16] = to16<BF16>(act[k][g]);
                    }
                }
        }
    }
#undef FLSTM_STAMP
    tcgen05_fence_before();
    __syncthreads();
    // after an abort this CTA's own copies may still be landing on barriers it cannot see (the leader's)
    if (*abort_w) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < kAbortDrainNs) {}
    }
    cluster_sync_all();  // the peer's shared and tensor memory stay valid until the leader's last UMMA is consumed
    if (warp == 5) tmem_dealloc_pair(tmem_base, kTmemColumns);
    if (threadIdx.x == 0 && *abort_w) atomicCAS(p.err, 0u, 1u);
    if (threadIdx.x == 0) leave_counters(p.counters, (int)gridDim.x / pl.cta_rows, p.exits);
}

template <int S, int BT, bool STREAM, bool BF16, bool ACC>
int launch_one(const CUtensorMap &tw, const CUtensorMap &tws, const CUtensorMap &th, const CUtensorMap &tg, const FwdTmPlan &pl, const FwdParams &p,
               cudaStream_t s) {
    auto kern = lstm_fwd_tm_kernel<S, BT, STREAM, BF16, ACC>;
    FLSTM_CUDA_TRY(ensure_smem_limit(kern, (size_t)pl.smem_bytes));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;  // all CTAs must be co-resident: they wait on one another
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, tws, th, tg, pl, p);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "recurrent forward launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

}  // namespace

// ------------------------------------------------------------------ host side
// The forms that lstm_forward_tm has kernels for: with the K halves nothing is streamed, without them always something (on the
// widths that take either on 148 SMs; a GPU with fewer may plan others, and those stay with the other kernels).
static bool has_kernel(const FwdTmPlan &pl) {
    if (pl.direct) return true;
    return pl.S == 2 ? pl.wstages == 0 && pl.BT == 64 : pl.wstages > 0 && (pl.BT == 16 || pl.BT == 32 || pl.BT == 64);
}

int plan_fwd_tm(int B, int H, int sms, size_t smem_limit, FwdTmPlan *plan) {
    *plan = FwdTmPlan{};
    if (H % 64 != 0 || H < 64 || smem_limit < 160 * 1024) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_TMEM"), *pair = std::getenv("FLSTM_FWD_PAIR");  // =0: weights in shared memory, lone CTAs
    if ((env && env[0] == '0') || (pair && pair[0] == '0')) return FLSTM_OK;
    FwdTmPlan pl{};
    pl.S = H / 16 <= sms ? 2 : 1;
    pl.cta_rows = pl.S == 2 ? H / 16 : H / 32;
    if (pl.cta_rows > sms || pl.cta_rows % 2) return FLSTM_OK;
    const int groups = sms / pl.cta_rows;
    for (int bt = pl.S == 2 ? 32 : 16; bt <= 64 && !pl.BT; bt *= 2)
        if ((B + bt - 1) / bt <= groups) pl.BT = bt;
    if (!pl.BT) return FLSTM_OK;
    pl.ngroups = (B + pl.BT - 1) / pl.BT;
    pl.kc = (H / 64 + pl.S - 1) / pl.S;
    const int N = pl.S * pl.BT, tmem_steps = (kTmemColumns - N) / 32, step_h = N / 2 * 128;
    pl.ct = pl.kc < tmem_steps ? pl.kc : tmem_steps;
    auto fits = [&]() { return (size_t)layout_of(pl).total <= smem_limit; };
    // h in copies of 16 KB, the whole tile at once if it fits beside the rest of the weights
    const int rest = pl.kc - pl.ct;
    pl.cs = rest;
    pl.direct = fits_direct(pl, smem_limit);
    pl.ch = 16384 / step_h < pl.kc ? 16384 / step_h : pl.kc;
    pl.hstages = (pl.kc + pl.ch - 1) / pl.ch;
    while (!pl.direct && !fits() && pl.hstages > 2) {
        --pl.hstages;
        pl.hring = 1;
    }
    if (!pl.direct && !fits()) {
        // streamed: all the room goes to the slots, which keep what the next step begins with
        pl.cs = 0;
        pl.hring = 1;
        pl.ch = (16384 / step_h) / WCH * WCH;
        pl.hstages = 2;
        if (!fits()) return FLSTM_OK;
        const int room = (int)((smem_limit - (size_t)layout_of(pl).total) / kStepBytesW);
        pl.wstages = (room - rest % WCH) / WCH;  // chunk-steps that make no whole group stay in shared memory
        if (pl.wstages < 2) return FLSTM_OK;
        if (pl.wstages > rest / WCH) pl.wstages = rest / WCH;
        pl.cs = rest % WCH;
    }
    // All of shared memory: a CTA allocates all of tensor memory, so no other kernel that uses some (another engine's, on another
    // stream) may share its SM; two grids that each held what the other's CTAs were waiting for would run into their limits
    pl.smem_bytes = (int)smem_limit;
    pl.grid = pl.cta_rows * pl.ngroups;
    if (!has_kernel(pl)) return FLSTM_OK;
    pl.use = true;
    *plan = pl;
    return FLSTM_OK;
}

int lstm_forward_tm(int dtype, const FwdTmPlan &pl, const CUtensorMap &tw, const CUtensorMap &tws, const CUtensorMap &th, const CUtensorMap &tg,
                    const FwdParams &p, cudaStream_t s) {
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, acc = p.real_units > 0, stream = pl.wstages > 0;
#define FLSTM_TM_CASE(S_, BT_, ST_)                                                                       \
    if (pl.S == S_ && pl.BT == BT_ && stream == ST_) {                                                    \
        if (bf16) return acc ? launch_one<S_, BT_, ST_, true, true>(tw, tws, th, tg, pl, p, s)                 \
                             : launch_one<S_, BT_, ST_, true, false>(tw, tws, th, tg, pl, p, s);               \
        return acc ? launch_one<S_, BT_, ST_, false, true>(tw, tws, th, tg, pl, p, s)                          \
                   : launch_one<S_, BT_, ST_, false, false>(tw, tws, th, tg, pl, p, s);                        \
    }
    FLSTM_TM_CASE(2, 64, false)
    FLSTM_TM_CASE(1, 16, true) FLSTM_TM_CASE(1, 32, true) FLSTM_TM_CASE(1, 64, true)
#undef FLSTM_TM_CASE
    return set_error(FLSTM_ERR_UNSUPPORTED, "no tensor-memory forward kernel for this plan");
}

}  // namespace tc
}  // namespace flstm_b200
