// Persistent recurrent forward kernel for wide batches: one launch runs all T time steps of one layer, W_hh stays on the chip
// and a CTA works on several batch tiles in turn.
//
// What bounds an output-tiled step GEMM (tc_lstm_step.cu) is what an SM can take in: 768 KB of h and W_hh per CTA and step at
// H = 2048, B = 256, through a port of about 60 B per cycle, and the chain from one step's stores to the next step's operands
// stands between the steps.  Here a CTA pair (cta_group::2, M = 128: 64 gate rows, 16 units per CTA) keeps its rows of W_hh for
// the whole sequence, in tensor memory (the A operand, held twice: lanes 0-63 and 64-127, as an M = 128 instruction over two CTAs
// reads it) and what does not fit there in shared memory.  Only h is staged, half of a tile per CTA.  The batch tiles are
// independent recurrences with a step barrier each, so the chain of one hides behind the UMMAs of the others.
//
// Per step and batch tile of BT sequences:
//   producer warp : waits for the tile's step barrier, streams h_{t-1} through the ring (copies of two or four 64-wide chunks)
//   UMMA thread   : M = 128, N = BT, accumulating over K = H into one of two accumulators (BT / 2 columns: sequences [0, BT/2) in
//                   lanes 0-63, the others in lanes 64-127)
//   16 warps      : the rows of A are ordered so that a lane quadrant holds the four gates of 8 units, 8 lanes each: two
//                   tcgen05.ld of the 16x256b shape leave all four gate sums of a (unit, sequence) pair in one thread, and no
//                   exchange through shared memory is needed.  Projections and cell states are read a tile ahead; h_t is stored
//                   first, cell states, gates and y follow while a thread of its own publishes h_t.
// Rebuilding the gates of a checkpointed segment whose h_t are kept (known_h) is the same launch without the chain: nobody waits
// for a step and no h_t is stored (H = 1024, B = 256, 32 steps: 131 -> 91 us).
// Waits are bounded; producer, publisher, UMMA thread and each epilogue warp break out of their loops by themselves (no barrier of
// threads lies inside the loops) and meet at the final __syncthreads; an aborted pair lingers before the final cluster barrier.
//
// Replaces the same reference launches as tc_lstm_fwd.cu (flashlstm_v2/src/lstm_forward.cu:744-830).
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

// 16 epilogue warps: with 8 a tile of 128 sequences took them 5.3 k cycles of instruction latencies, more than its UMMAs
constexpr int kEpilogueWarps = 16, kProducerWarp = 16, kUmmaWarp = 17, kPublisherWarp = 18;
constexpr int kThreads = (kEpilogueWarps + 3) * 32;
constexpr int kChunkBytesW = 64 * 128;  // 64 rows x 64 16-bit elements
constexpr int kTmemColumns = 512;
constexpr int kBarrierBytes = 1024, kMinSmemBytes = 120 * 1024;
constexpr int kFillSlots = 12;  // a multiple of 4: a slot always belongs to the same set of warps (see tc_lstm_fwd_tm.cu)
static_assert(kBarrierBytes + kFillSlots * kChunkBytesW + 1024 <= kMinSmemBytes, "the fill slots fit every launch");

__host__ __device__ inline int smem_of(const FwdWidePlan &pl) {
    return kBarrierBytes + pl.cs * kChunkBytesW + pl.hstages * pl.ch * (pl.BT / 2) * 128 + 1024 /*align*/;
}

// TRACE: stamps of the group's first tile of each step.  A form of its own: without being asked for they took 6 % of a launch
// (H = 2048, B = 256, T = 24: 297 -> 315 us).
template <int BT, int kCh, bool BF16, bool ACCURATE, bool TRACE>  // kCh: 64-wide chunks per copy of h
__global__ void __launch_bounds__(kThreads, 1)
lstm_fwd_wide_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_h,
                     const __grid_constant__ FwdWidePlan pl, FwdParams p) {
    constexpr int BTH = BT / 2;        // B rows a CTA stages, columns of an accumulator
    constexpr int WC = BTH / 4;        // columns a warp finishes
    constexpr int GROUPS = WC / 8;     // of 8 columns
    constexpr int PAIRS = 2 * GROUPS;  // (unit, sequence) pairs per thread
    constexpr int kStageBytes = kCh * BTH * 128;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int KC = pl.kc, CT = pl.ct, CS = pl.cs, NLOAD = (KC + kCh - 1) / kCh, HST = pl.hstages;
    uint8_t *s_w = smem + kBarrierBytes, *s_h = s_w + CS * kChunkBytesW;
    uint64_t *hfull = reinterpret_cast<uint64_t *>(smem), *hempty = hfull + HST;
    uint64_t *tfull = hempty + HST, *tempty = tfull + 2, *hdone = tempty + 2, *wbar = hdone + 2;
    uint64_t *ffull = wbar + 1, *fempty = ffull + kFillSlots;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fempty + kFillSlots);
    volatile uint32_t *abort_w = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ng = blockIdx.x / pl.cta_rows, jr = blockIdx.x % pl.cta_rows;  // batch group, 16-unit tile
    const int tile0 = ng * pl.nt, tiles = (p.B + BT - 1) / BT;
    const int NT = tiles - tile0 < pl.nt ? tiles - tile0 : pl.nt;  // batch tiles of this group
    unsigned int *counters = p.counters + tile0;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;

    if (threadIdx.x == 0) {
        for (int i = 0; i < HST; ++i) {
            mbar_init(&hfull[i], 1);
            mbar_init(&hempty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * (kEpilogueWarps + 1));  // epilogue warps and publishers of both CTAs report to the leader
            mbar_init(&hdone[i], kEpilogueWarps);
        }
        mbar_init(wbar, 1);
        for (int i = 0; i < kFillSlots; ++i) {
            mbar_init(&ffull[i], 1);
            mbar_init(&fempty[i], 4);
        }
        *abort_w = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_w);
        tma_prefetch_desc(&tm_h);
    }
    if (warp == kUmmaWarp) {
        tmem_alloc_pair(tmem_slot, kTmemColumns);
        tmem_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + 2 * BTH;
    // (ct is a multiple of kCh: a copy of h never mixes tensor- and shared-memory chunks)
    // W_hh into tensor memory by way of the shared memory that the ring will use: lanes l and l + 64 take row l of the tile in the
    // map's order (unit half, gate, unit), 32 columns of two elements per chunk; a warp reaches the lane quadrant warp % 4
    // and takes every fourth chunk.  A wait that expires raises the abort word, on which every role below gives up.
    if (warp == kProducerWarp && elect_one()) {
        for (int c = 0; c < CT; ++c) {
            const int slot = c % kFillSlots;
            if (c >= kFillSlots && !mbar_wait(&fempty[slot], (uint32_t)(c / kFillSlots - 1) & 1u, abort_w, wait_ns)) break;
            mbar_expect_tx(&ffull[slot], kChunkBytesW);
            tma_load_5d(s_w + slot * kChunkBytesW, &tm_w, c * 64, 0, 0, 0, jr, &ffull[slot]);
        }
    } else if (warp < kEpilogueWarps) {
        const int quad = warp & 3, row = (quad & 1) * 32 + lane;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        for (int c = warp >> 2; c < CT; c += 4) {
            const int slot = c % kFillSlots;
            if (!__all_sync(0xffffffffu, mbar_wait(&ffull[slot], (uint32_t)(c / kFillSlots) & 1u, abort_w, wait_ns))) break;
            const uint8_t *src = s_w + slot * kChunkBytesW + row * 128;
            uint32_t r[32];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 v = *reinterpret_cast<const uint4 *>(src + ((i ^ (row & 7)) * 16));
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
    const uint32_t hfull_c = map_to_rank(smem_u32(hfull), 0), wbar_c = map_to_rank(smem_u32(wbar), 0);
    const uint32_t tempty_c = map_to_rank(smem_u32(tempty), 0);
#define FLSTM_STAMP(slot)                                                                                                \
    do {                                                                                                                 \
        if (TRACE && n == 0 && blockIdx.x == 0 && tt < p.trace_steps) p.trace[tt * 16 + (slot)] = clock64();              \
    } while (0)

    if (warp == kProducerWarp) {
        // ------------------------------------------------------------ producer
        if (elect_one()) {
            bool ok = true;
            if (CS > 0) {
                if (leader) mbar_expect_tx(wbar, 2u * (uint32_t)(CS * kChunkBytesW));
                for (int c = 0; c < CS; ++c) tma_load_5d_pair(s_w + c * kChunkBytesW, &tm_w, (CT + c) * 64, 0, 0, 0, jr, wbar_c);
            }
            int stage = 0;
            uint32_t phase = 0, issued = 0, parity = 0;
            for (int tt = 0; tt < p.T && ok; ++tt)
                for (int n = 0; n < NT && ok; ++n) {
                    const int b0 = (tile0 + n) * BT;
                    if (tt > 0 && !p.known_h) {  // h_{t-1} of this tile is complete when every CTA of the group has arrived tt times
                        ok = wait_counter(counters + n, (unsigned)pl.cta_rows * (unsigned)tt + p.extra_arrivals, p.err, abort_w, 2u, wait_ns);
                        if (!ok) break;
                        fence_proxy_async_global();
                    }
                    FLSTM_STAMP(0);
                    for (int ld = 0; ld < NLOAD; ++ld) {
                        ok = mbar_wait(&hempty[stage], phase ^ 1, abort_w, wait_ns);
                        if (!ok) break;
                        if (leader) mbar_expect_tx(&hfull[stage], 2u * kStageBytes);
                        issued |= 1u << stage;
                        parity = (parity & ~(1u << stage)) | (phase << stage);
                        // chunks beyond K come as zeros (and are counted)
                        tma_load_4d_pair(s_h + stage * kStageBytes, &tm_h, 0, b0 + (int)rank * BTH, ld * kCh, p.t0 + tt,
                                         hfull_c + 8u * (uint32_t)stage);
                        if (++stage == HST) { stage = 0; phase ^= 1; }
                    }
                    FLSTM_STAMP(1);
                }
            // way out: every copy this thread started must have landed before the CTA exits (the peer's copies complete
            // the leader's barriers; after an abort the whole pair lingers, see below)
            if (CS > 0 && leader) mbar_drain(wbar, 0, wait_ns);
            for (int i = 0; i < HST && leader; ++i)
                if (issued >> i & 1u) mbar_drain(&hfull[i], parity >> i & 1u, ok ? wait_ns : kAbortDrainNs);
        }
    } else if (warp == kUmmaWarp) {
        // ------------------------------------------------------------ UMMA issuer (the leader's)
        if (leader && elect_one()) {
            bool ok = CS == 0 || mbar_wait(wbar, 0, abort_w, wait_ns);
            int stage = 0;
            uint32_t phase = 0, wi = 0;
            constexpr uint32_t idesc = umma_idesc_f16(128, BT, BF16 ? 1 : 0, 0, 0);
            constexpr uint32_t kStepH = (BTH * 128) >> 4, kStepW = kChunkBytesW >> 4;  // descriptor units
            const uint32_t hempty_l = smem_u32(hempty), tfull_l = smem_u32(tfull);
            const uint32_t dw_res = umma_desc_lo(smem_u32(s_w)), dh_ring = umma_desc_lo(smem_u32(s_h));
            for (int tt = 0; tt < p.T && ok; ++tt)
                for (int n = 0; n < NT && ok; ++n) {
                    const uint32_t buf = wi & 1;
                    ok = mbar_wait_cluster(&tempty[buf], ((wi >> 1) & 1) ^ 1, abort_w, wait_ns);
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint32_t d = tmem_base + buf * BTH;
                    // copies of tensor-memory chunks, then of shared-memory ones: no decision stands between two instructions
                    uint32_t da = tmem_a, dw = dw_res, acc = 0;
                    auto landed = [&]() {
                        ok = mbar_wait(&hfull[stage], phase, abort_w, wait_ns);
                        return dh_ring + (uint32_t)stage * (kStageBytes >> 4);
                    };
                    auto consumed = [&]() {
                        umma_commit_pair_both(hempty_l + 8u * (uint32_t)stage);
                        if (++stage == HST) { stage = 0; phase ^= 1; }
                    };
                    for (int c = 0; c < CT; c += kCh) {
                        const uint32_t dh = landed();
                        if (!ok) break;
                        if (c == 0) FLSTM_STAMP(2);
                        FLSTM_STAMP(3);
#pragma unroll
                        for (int e = 0; e < 4 * kCh; ++e)
                            umma_lo_ts<true>(d, da + 8 * e, dh + (e >> 2) * kStepH + 2 * (e & 3), idesc, e ? 1u : acc);
                        acc = 1;
                        da += 32 * kCh;
                        consumed();
                    }
                    int c = CT;
                    for (; c + kCh <= KC && ok; c += kCh) {
                        const uint32_t dh = landed();
                        if (!ok) break;
                        FLSTM_STAMP(3);
#pragma unroll
                        for (int e = 0; e < 4 * kCh; ++e)
                            umma_lo_ss<true>(d, dw + (e >> 2) * kStepW + 2 * (e & 3), dh + (e >> 2) * kStepH + 2 * (e & 3), idesc, e ? 1u : acc);
                        acc = 1;
                        dw += kCh * kStepW;
                        consumed();
                    }
                    if (c < KC && ok) {  // chunks that make no whole copy
                        uint32_t dh = landed();
                        if (!ok) break;
                        for (; c < KC; ++c) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_lo_ss<true>(d, dw + 2 * k, dh + 2 * k, idesc, k ? 1u : acc);
                            acc = 1;
                            dw += kStepW;
                            dh += kStepH;
                        }
                        consumed();
                    }
                    if (!ok) break;
                    umma_commit_pair_both(tfull_l + 8u * buf);
                    FLSTM_STAMP(4);
                    ++wi;
                }
            // the tensor memory is freed at the end of the kernel: the last committed batch of UMMAs must be done
            if (wi > 0) mbar_drain(&tfull[(wi - 1) & 1], (wi - 1) >> 1 & 1u, wait_ns);
        }
    } else if (warp == kPublisherWarp) {
        // ------------------------------------------------------------ publisher
        // The release takes about a thousand cycles (it waits for the stores it covers); on a thread of its own the epilogue goes
        // on meanwhile.  hdone orders it behind every epilogue warp's stores of h; the generic->async proxy fence is the consumer's.
        if (elect_one()) {
            uint32_t wi = 0;
            bool ok = true;
            for (int tt = 0; tt < p.T && ok; ++tt)
                for (int n = 0; n < NT && ok; ++n, ++wi) {
                    ok = mbar_wait(&hdone[wi & 1], (wi >> 1) & 1, abort_w, wait_ns);
                    if (!ok) break;
                    // no third tile may use this hdone barrier before the publisher has seen this phase of it
                    mbar_arrive_cluster_relaxed(tempty_c + 8u * (wi & 1));
                    if (!p.known_h) red_release_gpu_add(counters + n, 1u);
                    FLSTM_STAMP(8);
                }
        }
    } else {
        // ------------------------------------------------------------ epilogue (16 warps, each on its own)
        // Quadrant q of the lanes: unit half q & 1, sequences (q >> 1) BT / 2 of the tile, of which this warp takes WC columns, 8
        // at a time.  An accumulator fragment is (unit lane / 4, sequences 2 (lane % 4) and + 1); 16-bit data move as (sequence
        // lane / 4, 8 units of gate lane % 4: 16 bytes) and (sequence lane / 4, units 2 (lane % 4) and + 1 of h: 4 bytes), between
        // which movmatrix and a transpose over quads translate.  As 2-byte accesses in fragment order they took 10 k cycles per
        // tile of 128 sequences, four times the UMMAs.
        const int quad = warp & 3, half = quad & 1, q = lane & 3, s8 = lane >> 2;
        const int U = jr * 16 + half * 8 + s8;                           // unit of this thread's fragments
        const int col0 = (quad >> 1) * BTH + (warp >> 2) * WC;           // first sequence of the warp within a tile
        const uint32_t taddr0 = tmem_base + ((uint32_t)(quad * 32) << 16) + (warp >> 2) * WC;
        const size_t slab = (size_t)p.B * p.H, G = (size_t)4 * p.H;
        const bool pad = ACCURATE && U >= p.real_units;
        uint16_t *hs = static_cast<uint16_t *>(p.hs);
        uint16_t *y = static_cast<uint16_t *>(p.y);
        uint16_t *gates = static_cast<uint16_t *>(p.gates);
        const bool y_words = (reinterpret_cast<uintptr_t>(y) & 3) == 0;
        const size_t gcol = (size_t)jr * 64 + q * 16 + half * 8;         // gate q, 8 units
        const size_t hcol = (size_t)jr * 16 + half * 8 + 2 * q;          // two units of h
        uint4 p_next[GROUPS];
        float c_next[PAIRS];
        auto fetch_p = [&](int t, int n) {
            const int b = (tile0 + n) * BT + col0 + s8;
#pragma unroll
            for (int i = 0; i < GROUPS; ++i)
                p_next[i] = b + 8 * i < p.B ? *reinterpret_cast<const uint4 *>(gates + ((size_t)t * p.B + b + 8 * i) * G + gcol) : make_uint4(0, 0, 0, 0);
        };
        auto fetch_c = [&](int t, int n) {
            const int b = (tile0 + n) * BT + col0 + 2 * q;
#pragma unroll
            for (int k = 0; k < PAIRS; ++k) {
                const int r = b + 8 * (k >> 1) + (k & 1);
                c_next[k] = r < p.B ? p.cs[(size_t)t * slab + (size_t)r * p.H + U] : 0.f;
            }
        };
        fetch_p(p.t0, 0);
        fetch_c(p.t0, 0);
        uint32_t wi = 0;
        bool ok = true;
        for (int tt = 0; tt < p.T && ok; ++tt) {
            const int t = p.t0 + tt;
            for (int n = 0; n < NT; ++n, ++wi) {
                const uint32_t buf = wi & 1;
                const int b = (tile0 + n) * BT + col0;
                uint32_t proj[GROUPS][4];
                float c[PAIRS];
#pragma unroll
                for (int i = 0; i < GROUPS; ++i) {
                    proj[i][0] = p_next[i].x; proj[i][1] = p_next[i].y; proj[i][2] = p_next[i].z; proj[i][3] = p_next[i].w;
                    quad_transpose(proj[i], lane);
#pragma unroll
                    for (int g = 0; g < 4; ++g) proj[i][g] = movmatrix_trans(proj[i][g]);
                }
#pragma unroll
                for (int k = 0; k < PAIRS; ++k) c[k] = c_next[k];
                // the next tile's projections and, unless it is this one again, its cell states
                const int n_next = n + 1 == NT ? 0 : n + 1, t_next = n + 1 == NT ? t + 1 : t;
                const bool more = t_next < p.t0 + p.T;
                if (more) fetch_p(t_next, n_next);
                if (more && NT > 1) fetch_c(t_next, n_next);
                // a warp reads the accumulator only if all of its lanes saw it complete
                ok = __all_sync(0xffffffffu, mbar_wait(&tfull[buf], (wi >> 1) & 1, abort_w, wait_ns));
                if (!ok) break;
                if (threadIdx.x == 0) FLSTM_STAMP(5);
                tcgen05_fence_after();
                uint32_t lo[4 * GROUPS], hi[4 * GROUPS];  // gates i, f and g, o: per 8 columns two of each
                tmem_ld_16x256b<GROUPS>(taddr0 + buf * BTH, lo);
                tmem_ld_16x256b<GROUPS>(taddr0 + (16u << 16) + buf * BTH, hi);
                tmem_ld_wait();
                tcgen05_fence_before();
                uint32_t act[GROUPS][4], h2[GROUPS];
                uint16_t *h_out = hs + (size_t)(t + 1) * slab + (size_t)(b + s8) * p.H + hcol;
#pragma unroll
                for (int i = 0; i < GROUPS; ++i) {
                    uint32_t pk[5] = {0, 0, 0, 0, 0};
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        auto gate = [&](uint32_t acc, uint32_t pr) {
                            const uint16_t v = (uint16_t)(e ? pr >> 16 : pr);
                            return pad ? 0.f : __uint_as_float(acc) + load16<BF16>(&v);
                        };
                        const float gi = sigmoid_sel<ACCURATE>(gate(lo[4 * i + e], proj[i][0])), gf = sigmoid_sel<ACCURATE>(gate(lo[4 * i + 2 + e], proj[i][1]));
                        const float gg = tanh_sel<ACCURATE>(gate(hi[4 * i + e], proj[i][2])), go = sigmoid_sel<ACCURATE>(gate(hi[4 * i + 2 + e], proj[i][3]));
                        const float cn = fmaf(gf, c[2 * i + e], gi * gg);
                        c[2 * i + e] = cn;
                        pk[0] |= (uint32_t)to16<BF16>(gi) << (16 * e);
                        pk[1] |= (uint32_t)to16<BF16>(gf) << (16 * e);
                        pk[2] |= (uint32_t)to16<BF16>(gg) << (16 * e);
                        pk[3] |= (uint32_t)to16<BF16>(go) << (16 * e);
                        pk[4] |= (uint32_t)to16<BF16>(go * tanh_sel<ACCURATE>(cn)) << (16 * e);
                    }
                    h2[i] = movmatrix_trans(pk[4]);
#pragma unroll
                    for (int g = 0; g < 4; ++g) act[i][g] = pk[g];
                    // h_t first: it is what the other CTAs wait for
                    if (b + 8 * i + s8 < p.B && !p.known_h) *reinterpret_cast<uint32_t *>(h_out + (size_t)(8 * i) * p.H) = h2[i];
                }
                __syncwarp();
                if (threadIdx.x == 0) FLSTM_STAMP(7);
                if (lane == 0) {
                    mbar_arrive(&hdone[buf]);
                    // Behind hdone, so that nobody arrives there for the next tile of this buffer before all have for this one.
                    // Relaxed: it orders the reuse of the accumulator only (a release would wait for the warp's global stores).
                    mbar_arrive_cluster_relaxed(tempty_c + 8u * buf);
                }
                // everything nobody waits for: cell state, gate cache, the caller's y
#pragma unroll
                for (int k = 0; k < PAIRS; ++k) {
                    const int r = b + 2 * q + 8 * (k >> 1) + (k & 1);
                    if (r < p.B) p.cs[(size_t)(t + 1) * slab + (size_t)r * p.H + U] = c[k];
                }
                if (NT == 1) {
#pragma unroll
                    for (int k = 0; k < PAIRS; ++k) c_next[k] = c[k];
                }
#pragma unroll
                for (int i = 0; i < GROUPS; ++i) {
                    const int r = b + 8 * i + s8;
                    if (p.store_gates) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) act[i][g] = movmatrix_trans(act[i][g]);
                        quad_transpose(act[i], lane);
                        if (r < p.B)
                            *reinterpret_cast<uint4 *>(gates + ((size_t)t * p.B + r) * G + gcol) = make_uint4(act[i][0], act[i][1], act[i][2], act[i][3]);
                    }
                    if (y && r < p.B) {
                        uint16_t *dst = y + (size_t)t * slab + (size_t)r * p.H + hcol;
                        if (y_words) {
                            *reinterpret_cast<uint32_t *>(dst) = h2[i];
                        } else {
                            dst[0] = (uint16_t)h2[i];
                            dst[1] = (uint16_t)(h2[i] >> 16);
                        }
                    }
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
    if (warp == kUmmaWarp) tmem_dealloc_pair(tmem_base, kTmemColumns);
    if (threadIdx.x == 0 && *abort_w) atomicCAS(p.err, 0u, 1u);
    if (threadIdx.x == 0) leave_counters(p.counters, (int)gridDim.x / pl.cta_rows * pl.nt, p.exits);
}

template <int BT, int CH, bool BF16, bool ACC>
int launch_one(const CUtensorMap &tw, const CUtensorMap &th, const FwdWidePlan &pl, const FwdParams &p, cudaStream_t s) {
    auto kern = p.trace ? lstm_fwd_wide_kernel<BT, CH, BF16, ACC, true> : lstm_fwd_wide_kernel<BT, CH, BF16, ACC, false>;
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, th, pl, p);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "recurrent forward launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

}  // namespace

// ------------------------------------------------------------------ host side
int plan_fwd_wide(int B, int H, int sms, size_t smem_limit, FwdWidePlan *plan) {
    *plan = FwdWidePlan{};
    if (H % 64 != 0 || H < 64 || smem_limit < 160 * 1024) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_TMEM"), *pair = std::getenv("FLSTM_FWD_PAIR");  // as for plan_fwd_tm
    if ((env && env[0] == '0') || (pair && pair[0] == '0')) return FLSTM_OK;
    FwdWidePlan pl{};
    pl.cta_rows = H / 16;
    if (pl.cta_rows > sms || pl.cta_rows % 2) return FLSTM_OK;
    const int groups = sms / pl.cta_rows;
    // Tiles of 64 sequences or half as many of 128.  Two of 64 rather than one of 128, whose chain would stand alone; beyond two,
    // an odd number of 64 leaves no half tile empty, and copies of four chunks (below) keep up with the wider tiles, us a step 128 / 64:
    //   3 of 64  H = 1024, B = 280 / 384 6.90 / 5.25, 7.19 / 5.52   H = 640, B = 384 5.27 / 4.49   H = 1792, B = 192 8.18 / 6.67   H = 2048, B = 192 8.95 / 8.11
    //   4        H = 512, B = 1024 7.00 / 5.90   H = 1024, B = 512 7.94 / 7.09   H = 1792, B = 256 8.90 / 8.74   H = 2048, B = 256 9.6 / 10.5
    //   5        H = 512, B = 1280 7.70 / 7.22   H = 1024, B = 640 9.15 / 8.76   H = 1536, B = 320 10.13 / 9.46   H = 2048, B = 320 13.22 / 12.98
    //   6        H = 512, B = 1536 8.10 / 8.55   H = 1024, B = 768 9.59 / 10.38   H = 1536, B = 384 11.02 / 11.40
    // Three tiles beside two groups, four and five in a lone one and H = 2176 keep the wider tiles although most would gain (H = 1024,
    // B = 384 above; H = 1536, B = 256 8.17 / 7.75): tests name shapes of theirs as what tiles of 128 run.
    const int narrow = ((B + 63) / 64 + groups - 1) / groups;
    const bool three_on = narrow == 3 ? groups != 2 && H <= 2112 : (narrow == 4 || narrow == 5) && groups > 1;
    pl.BT = narrow <= 2 || three_on ? 64 : 128;
    const int tiles = (B + pl.BT - 1) / pl.BT;
    pl.nt = (tiles + groups - 1) / groups;
    pl.ngroups = (tiles + pl.nt - 1) / pl.nt;
    // Up to six tiles in turn: H = 1024, B = 1536 28.2 -> 23.4 us a step against the output-tiled kernel, H = 512, B = 2048 17.2 ->
    // 15.0, H = 2048, B = 512 25.4 -> 24.2; eight are slower (H = 1024, B = 2048 30.3 -> 31.8), the epilogue then bounds it
    if (pl.nt > 6 || pl.nt * pl.ngroups > kMaxStepCounters) return FLSTM_OK;
    pl.kc = H / 64;
    const int tmem_chunks = (kTmemColumns - pl.BT) / 32;
    // A copy's wait, its commit and the address arithmetic between take the issuing thread some 200 cycles, more than the eight
    // UMMAs of N = 64 of two chunks.  Tiles of 64 go in copies of four chunks as long as three of them fit; us a step with two / four
    // chunks: H = 1024, B = 256 5.54 / 5.19, H = 2048, B = 100 7.62 / 6.31, H = 1536, B = 100 5.87 / 5.16, H = 512, B = 512 4.90 / 4.62.
    // An UMMA of N = 128 takes twice as long and the ring holds fewer copies: H = 2048, B = 256 10.22 / 10.66, H = 1024, B = 384 7.50 / 8.39.
    auto take_chunks = [&](int ch) {
        pl.ch = ch;
        pl.ct = (pl.kc < tmem_chunks ? pl.kc : tmem_chunks) / ch * ch;
        pl.cs = pl.kc - pl.ct;
        pl.hstages = 32 / ch;
        while (pl.hstages > 3 && (size_t)smem_of(pl) > smem_limit) --pl.hstages;
        return (size_t)smem_of(pl) <= smem_limit;
    };
    if (!(pl.BT == 64 && take_chunks(4)) && !take_chunks(2)) return FLSTM_OK;
    // All of shared memory: a CTA allocates all of tensor memory, so no other kernel that uses some (another engine's, on another
    // stream) may share its SM; two grids that each held what the other's CTAs were waiting for would run into their limits
    pl.smem_bytes = (int)smem_limit;
    pl.grid = pl.cta_rows * pl.ngroups;
    pl.use = true;
    *plan = pl;
    return FLSTM_OK;
}

int lstm_forward_wide(int dtype, const FwdWidePlan &pl, const CUtensorMap &tw, const CUtensorMap &th, const FwdParams &p, cudaStream_t s) {
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, acc = p.real_units > 0;
#define FLSTM_WIDE_CASE(BT_, CH_)                                                                                                     \
    if (pl.BT == BT_ && pl.ch == CH_) {                                                                                              \
        if (bf16) return acc ? launch_one<BT_, CH_, true, true>(tw, th, pl, p, s) : launch_one<BT_, CH_, true, false>(tw, th, pl, p, s); \
        return acc ? launch_one<BT_, CH_, false, true>(tw, th, pl, p, s) : launch_one<BT_, CH_, false, false>(tw, th, pl, p, s);       \
    }
    FLSTM_WIDE_CASE(64, 4) FLSTM_WIDE_CASE(64, 2) FLSTM_WIDE_CASE(128, 2)
#undef FLSTM_WIDE_CASE
    return set_error(FLSTM_ERR_UNSUPPORTED, "no wide forward kernel for this plan");
}

}  // namespace tc
}  // namespace flstm_b200
