// Persistent BPTT kernel with W_hh in TENSOR MEMORY: one launch runs the whole reverse recurrence of one layer.
//
// Same split as tc_lstm_bwd.cu: a cluster of four CTAs owns 64 hidden units, CTA kq contracts its quarter of K = 4H, the
// partial sums are reduce-scattered through distributed shared memory, every CTA runs the pointwise backward of 16 units.
// What bounded that kernel beyond H = 1024 was its slice of W_hh (256 KB per CTA and step at H = 2048, through an SM port of
// about 60 B per cycle) and, at every H, UMMAs of M = 64 that read both operands from shared memory.  Here the slice is the A
// operand in tensor memory (what does not fit its columns stays in shared memory, nothing is streamed), and the tiles are
// M = 128: lanes 0-63 hold W_hh^T of the 64 units for the first half of the CTA's K range, lanes 64-127 for the second half.
// The B operand has 2 BT rows (K half 0 and 1 of the BT sequences), the accumulator 128 lanes x 2 BT columns, of which the
// blocks (half q, columns of half q) are partial sums and the other two are ignored.  A K range of an odd number of 64-wide
// chunks leaves one chunk that runs as an instruction of N = BT from shared memory into the first half's block.
//
// Up to H = 1536 one tile of 32 sequences exchanges without a step barrier (tc_lstm_bwd_tm_direct.cu); this form runs wider ones, tiles
// of 64 and tiles in turn.
//
// Per step: the producer waits for the step barrier and fetches dG_{t+1} of the K range (both halves with one copy: a 5-D
// map orders them as the B operand wants); the UMMA thread contracts; the 256 epilogue threads move the accumulator to shared
// memory, add the halves, send them to the owners with st.async, add the four sources and do the pointwise update.
// Every wait is bounded; the way out is that of tc_lstm_bwd.cu.
//
// Replaces the same reference launches (flashlstm_v2/src/lstm_backward.cu:158-227, 1057-1101).
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

constexpr int kThreads = 352;  // warps 0-3 and 6-9 epilogue, 4 producer, 5 UMMA issuer, 10 publisher of dG
constexpr int kEpilogueThreads = 256;
constexpr int kStepBytesW = 2 * 64 * 128;  // one chunk-step of A: two blocks of 64 K rows x 64 units
constexpr int kTmemColumns = 512;
constexpr int kBarrierBytes = 1024, kMinSmemBytes = 120 * 1024;
// Even: a slot always belongs to the same set of warps.  A set that met a slot only every other time could find its first phase
// still open, whose parity reads as that of the phase it waits for.
constexpr int kFillSlots = (kMinSmemBytes - 1024 - kBarrierBytes) / kStepBytesW / 2 * 2;
constexpr int KS = 4, UPO = 64 / KS;

struct Layout {
    int w, left_w, ring, left, ps, red, total;
};

__host__ __device__ inline Layout layout_of(const BwdTmPlan &pl) {
    Layout l;
    l.w = pl.cs * kStepBytesW;
    l.left_w = pl.left ? kStepBytesW : 0;
    l.ring = pl.stages * pl.ch * 2 * pl.BT * 128;
    l.left = pl.left ? pl.BT * 128 : 0;
    l.ps = 128 * (pl.BT + 4) * 4;
    l.red = 2 * KS * UPO * (pl.BT + 4) * 4;
    l.total = kBarrierBytes + l.w + l.left_w + l.ring + l.left + l.ps + l.red + 1024 /*align*/;
    return l;
}

template <int BT, bool BF16, bool ACCURATE>
__global__ void __launch_bounds__(kThreads, 1)
lstm_bwd_tm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ BwdTmMaps maps,
                   const __grid_constant__ BwdTmPlan pl, BwdParams p) {
    constexpr int PAIRS = BT / 16;  // (unit, sequence) pairs per epilogue thread
    constexpr int RS = BT + 4;      // row stride of the exchange and reduce buffers (floats), keeps float4 alignment
    constexpr int N = 2 * BT;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const Layout L = layout_of(pl);
    const int KP = pl.kp, CT = pl.ct, CS = pl.cs, CH = pl.ch, NLOAD = (KP + CH - 1) / CH, ST = pl.stages;
    const int stage_bytes = CH * N * 128;
    uint8_t *s_w = smem + kBarrierBytes, *s_lw = s_w + L.w, *s_ring = s_lw + L.left_w, *s_left = s_ring + L.ring;
    float *s_ps = reinterpret_cast<float *>(s_left + L.left), *s_red = s_ps + L.ps / 4;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + ST;
    uint64_t *lfull = empty + ST, *lempty = lfull + 1, *tfull = lempty + 1, *tempty = tfull + 1, *wbar = tempty + 1;
    uint64_t *rbar = wbar + 1;  // [2] partial sums received
    uint64_t *gdone = rbar + 2, *pdone = gdone + 2;  // [2] dG stored by every warp / seen by the publisher
    uint64_t *ffull = pdone + 2, *fempty = ffull + kFillSlots;  // while W_hh moves into tensor memory
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fempty + kFillSlots);
    volatile uint32_t *abort_w = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kq = (int)cluster_ctarank();
    const int cl = blockIdx.x / KS, ng = cl / pl.jt, j = cl % pl.jt;  // batch group, unit tile [64j, 64j+64)
    const int tile0 = ng * pl.nt, tiles = (p.B + BT - 1) / BT;
    const int NT = tiles - tile0 < pl.nt ? tiles - tile0 : pl.nt;  // batch tiles of this group, taken in turn
    unsigned int *counters = p.counters + tile0;
    const int kcq = 2 * KP + pl.left, c_first = kq * kcq;  // 64-wide K chunks of this CTA
    const CUtensorMap *tm_dg = &maps.half[kq];

    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(lfull, 1);
        mbar_init(lempty, 1);
        mbar_init(tfull, 1);
        mbar_init(tempty, kEpilogueThreads / 32);
        mbar_init(wbar, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&rbar[i], 1);
            mbar_init(&gdone[i], kEpilogueThreads / 32);
            mbar_init(&pdone[i], 1);
        }
        for (int i = 0; i < kFillSlots; ++i) {
            mbar_init(&ffull[i], 1);
            mbar_init(&fempty[i], 4);
        }
        *abort_w = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_w);
        tma_prefetch_desc(tm_dg);
        if (pl.left) tma_prefetch_desc(&maps.chunk);
    }
    if (warp == 5) {
        tmem_alloc(tmem_slot, kTmemColumns);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + N;
    const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
    // W_hh^T into tensor memory, by way of the shared memory that the rings will use (as in tc_lstm_fwd_tm.cu): lane l takes unit
    // l % 64 and K half l / 64, 32 columns of two K elements per chunk-step; the warps 0-3 take the even chunk-steps, 6-9 the
    // odd ones
    if (warp == 4 && elect_one()) {
        for (int c = 0; c < CT; ++c) {
            const int slot = c % kFillSlots;
            if (c >= kFillSlots && !mbar_wait(&fempty[slot], (uint32_t)(c / kFillSlots - 1) & 1u, abort_w, wait_ns)) break;
            mbar_expect_tx(&ffull[slot], kStepBytesW);
            for (int h = 0; h < 2; ++h)
                tma_load_2d(s_w + slot * kStepBytesW + h * 8192, &tm_w, j * 64, (c_first + h * KP + c) * 64, &ffull[slot]);
        }
    } else if (warp != 4 && warp != 5 && warp != 10) {
        const int quad = warp & 3, l = quad * 32 + lane, un = l & 63;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        for (int c = warp < 4 ? 0 : 1; c < CT; c += 2) {
            const int slot = c % kFillSlots;
            if (!__all_sync(0xffffffffu, mbar_wait(&ffull[slot], (uint32_t)(c / kFillSlots) & 1u, abort_w, wait_ns))) break;
            const uint8_t *tile = s_w + slot * kStepBytesW + (l >> 6) * 8192 + (un & 7) * 2;
            uint32_t r[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int k = 2 * i;
                const uint32_t lo = *reinterpret_cast<const uint16_t *>(tile + k * 128 + (((un >> 3) ^ (k & 7)) * 16));
                const uint32_t hi = *reinterpret_cast<const uint16_t *>(tile + (k + 1) * 128 + (((un >> 3) ^ ((k + 1) & 7)) * 16));
                r[i] = lo | hi << 16;
            }
            tmem_st_32x32b_x32(dst + c * 32, r);
            __syncwarp();
            if (lane == 0) mbar_arrive(&fempty[slot]);
        }
        tmem_st_wait();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers exist before any remote arrive
    tcgen05_fence_after();
    const int s_first = p.s0 > 1 ? p.s0 : 1;  // iteration s handles time T-1-s and, from s = 1 on, contracts dG_{T-s}
    const bool tracing = p.trace != nullptr && blockIdx.x == 0;
#define FLSTM_STAMP(step, slot)                                                     \
    do {                                                                            \
        if (tracing && (step) < p.trace_steps) p.trace[(step) * 16 + (slot)] = clock64(); \
    } while (0)

    if (warp == 4) {
        // ------------------------------------------------------------ producer
        if (elect_one()) {
            bool ok = true;
            if (CS > 0 || pl.left) {
                mbar_expect_tx(wbar, (uint32_t)(L.w + L.left_w));
                for (int c = 0; c < CS; ++c)
                    for (int h = 0; h < 2; ++h)
                        tma_load_2d(s_w + c * kStepBytesW + h * 8192, &tm_w, j * 64, (c_first + h * KP + CT + c) * 64, wbar);
                if (pl.left)  // the second block only feeds lanes whose results are ignored
                    for (int h = 0; h < 2; ++h) tma_load_2d(s_lw + h * 8192, &tm_w, j * 64, (c_first + 2 * KP) * 64, wbar);
            }
            int stage = 0;
            uint32_t phase = 0, lphase = 0;
            uint32_t issued = 0, parity = 0;
            bool left_issued = false;
            for (int s = s_first; s < p.s1 && ok; ++s)
                for (int n = 0; n < NT && ok; ++n) {
                    const int t_src = p.T - s, b0 = (tile0 + n) * BT;
                    // Without a ring (one tile) the copies of a step are announced ahead of its barrier and follow it back to back,
                    // see tc_lstm_fwd_tm.cu; the tile is free then: the barrier came after the UMMAs that read it
                    const uint32_t step = (uint32_t)(s - s_first);
                    for (int i = 0; !pl.ring && i < ST + pl.left; ++i) {
                        uint64_t *bar = i < ST ? &full[i] : lfull;
                        if (step > 0 && !mbar_wait(bar, (step - 1) & 1u, abort_w, wait_ns)) ok = false;
                        if (!ok) break;
                        mbar_expect_tx(bar, i < ST ? (uint32_t)stage_bytes : (uint32_t)(BT * 128));
                    }
                    if (!ok) break;
                    if (s > p.s0)
                        ok = wait_counter(counters + n, (unsigned)(pl.jt * KS) * (unsigned)(s - p.s0) + p.extra_arrivals, p.err, abort_w, 3u,
                                          wait_ns);
                    if (!ok) break;
                    fence_proxy_async_global();
                    if (n == 0) FLSTM_STAMP(s - p.s0, 0);
                    for (int ld = 0; ld < NLOAD; ++ld) {
                        if (pl.ring) {
                            ok = mbar_wait(&empty[stage], phase ^ 1, abort_w, wait_ns);
                            if (!ok) break;
                            mbar_expect_tx(&full[stage], (uint32_t)stage_bytes);
                        }
                        issued |= 1u << stage;
                        parity = (parity & ~(1u << stage)) | (phase << stage);
                        // (x, row, K half, chunk of the half, step); chunks beyond the half come as zeros (and are counted)
                        tma_load_5d(s_ring + stage * stage_bytes, tm_dg, 0, b0, 0, ld * CH, t_src, &full[stage]);
                        if (++stage == ST) { stage = 0; phase ^= 1; }
                    }
                    if (ok && pl.left) {
                        if (pl.ring) {
                            ok = mbar_wait(lempty, lphase ^ 1, abort_w, wait_ns);
                            if (!ok) break;
                            mbar_expect_tx(lfull, BT * 128);
                        }
                        tma_load_4d(s_left, &maps.chunk, 0, b0, c_first + 2 * KP, t_src, lfull);
                        left_issued = true;
                        lphase ^= 1;
                    }
                    if (n == 0) FLSTM_STAMP(s - p.s0, 1);
                }
            // way out (normal or aborted): every copy this thread started must have landed before the CTA exits
            if (CS > 0 || pl.left) mbar_drain(wbar, 0, wait_ns);
            for (int i = 0; i < ST; ++i)
                if (issued >> i & 1u) mbar_drain(&full[i], parity >> i & 1u, wait_ns);
            if (left_issued) mbar_drain(lfull, lphase ^ 1, wait_ns);
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ UMMA issuer
        if (elect_one()) {
        bool ok = (CS == 0 && !pl.left) || mbar_wait(wbar, 0, abort_w, wait_ns);
        int stage = 0;
        uint32_t phase = 0;
        constexpr uint32_t idesc_ts = umma_idesc_f16(128, N, BF16 ? 1 : 0, 0, 0), idesc_ss = umma_idesc_f16(128, N, BF16 ? 1 : 0, 1, 0);
        constexpr uint32_t idesc_left = umma_idesc_f16(128, BT, BF16 ? 1 : 0, 1, 0);
        constexpr uint32_t kStepG = (N * 128) >> 4, kStepW = kStepBytesW >> 4;  // descriptor units
        const uint32_t dw_res = umma_desc_lo(smem_u32(s_w), 8192), dw_left = umma_desc_lo(smem_u32(s_lw), 8192);
        const uint32_t dd_ring = umma_desc_lo(smem_u32(s_ring)), dd_left = umma_desc_lo(smem_u32(s_left));
        const uint32_t empty_l = smem_u32(empty), lempty_l = smem_u32(lempty), tfull_l = smem_u32(tfull);
        int committed = 0;
        const uint32_t items = (uint32_t)(p.s1 - s_first) * (uint32_t)NT;
        for (uint32_t wi = 0; wi < items && ok; ++wi) {
            const int s = s_first + (int)(wi / (uint32_t)NT);
            ok = mbar_wait(tempty, (wi & 1) ^ 1, abort_w, wait_ns);
            if (!ok) break;
            tcgen05_fence_after();
            uint32_t acc = 0;  // the step's first instruction overwrites the accumulator
            for (int ld = 0; ld < NLOAD; ++ld) {
                ok = mbar_wait(&full[stage], phase, abort_w, wait_ns);
                if (!ok) break;
                if (ld == 0) FLSTM_STAMP(s - p.s0, 2);
                if (ld == NLOAD - 1) FLSTM_STAMP(s - p.s0, 3);
                tcgen05_fence_after();
                uint32_t dd = dd_ring + (uint32_t)stage * (uint32_t)(stage_bytes >> 4);
                const int c1 = (ld + 1) * CH < KP ? (ld + 1) * CH : KP;
                int c = ld * CH;
                const int ct1 = c1 < CT ? c1 : CT;
                uint32_t da = tmem_a + (uint32_t)c * 32;
#pragma unroll 4
                for (; c < ct1; ++c) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_lo_ts<false>(tmem_base, da + 8 * k, dd + 2 * k, idesc_ts, k ? 1u : acc);
                    acc = 1u;
                    da += 32;
                    dd += kStepG;
                }
                uint32_t dw = dw_res + (uint32_t)(c - CT) * kStepW;
#pragma unroll 2
                for (; c < c1; ++c) {  // K steps of 16: +2048 bytes on the MN-major W_hh, +32 bytes on the K-major dG
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_lo_ss<false>(tmem_base, dw + 128 * k, dd + 2 * k, idesc_ss, k ? 1u : acc);
                    acc = 1u;
                    dw += kStepW;
                    dd += kStepG;
                }
                if (pl.ring) umma_commit_addr(empty_l + 8u * (uint32_t)stage);
                if (++stage == ST) { stage = 0; phase ^= 1; }
            }
            if (!ok) break;
            if (pl.left) {
                ok = mbar_wait(lfull, wi & 1, abort_w, wait_ns);
                if (!ok) break;
                tcgen05_fence_after();
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_lo_ss<false>(tmem_base, dw_left + 128 * k, dd_left + 2 * k, idesc_left, 1u);
                if (pl.ring) umma_commit_addr(lempty_l);
            }
            umma_commit_addr(tfull_l);
            ++committed;
            FLSTM_STAMP(s - p.s0, 4);
        }
        // the tensor memory is freed at the end of the kernel: the last committed batch of UMMAs must be done
        if (committed > 0) mbar_drain(tfull, (uint32_t)(committed - 1) & 1u, wait_ns);
        }
    } else if (warp == 10) {
        // ------------------------------------------------------------ publisher
        // The release takes about a thousand cycles (it waits for the stores it covers), which the epilogue need not spend.  The
        // generic->async proxy fence is the consumer's.
        if (elect_one()) {
            uint32_t gi = 0;
            bool ok = true;
            for (int s = p.s0; s < p.s1 && s < p.T && ok; ++s)
                for (int n = 0; n < NT; ++n, ++gi) {
                    ok = mbar_wait(&gdone[gi & 1], (gi >> 1) & 1, abort_w, wait_ns);
                    if (!ok) break;
                    mbar_arrive(&pdone[gi & 1]);
                    red_release_gpu_add(counters + n, 1u);
                    if (n == 0) FLSTM_STAMP(s - p.s0, 8);
                }
        }
    } else {
        // ------------------------------------------------------------ epilogue (256 threads)
        const int tid = warp < 4 ? threadIdx.x : threadIdx.x - 64;  // 0..255
        const int u16 = tid & 15, nb = tid >> 4;  // unit u16 of the CTA's 16, sequences nb + 16 i
        const int U = j * 64 + kq * UPO + u16;
        const size_t slab = (size_t)p.B * p.H, G = (size_t)4 * p.H;
        const uint16_t *gates = static_cast<const uint16_t *>(p.gates);
        const uint16_t *dy = static_cast<const uint16_t *>(p.dy);
        const uint16_t *dhn = static_cast<const uint16_t *>(p.dhn);
        const uint16_t *dcn = static_cast<const uint16_t *>(p.dcn);
        uint16_t *dg = static_cast<uint16_t *>(p.dg);
        const int quad = warp & 3, col0 = warp < 4 ? 0 : BT / 2;  // lane quadrant, half of the columns
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (quad >> 1) * BT + col0;
        const uint32_t red_local = smem_u32(s_red), rbar_local = smem_u32(rbar);
        // what the pointwise update of a tile reads, fetched a tile ahead
        struct Inputs {
            uint16_t gi, gf, gg, go, dy;
            float ct, cp, dc;
        };
        Inputs next[PAIRS];
        auto fetch = [&](int s, int n) {
            const int t = p.T - 1 - s;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const int b = (tile0 + n) * BT + nb + 16 * i;
                const size_t idx = (size_t)b * p.H + U;
                next[i].gi = next[i].gf = next[i].gg = next[i].go = next[i].dy = 0;
                next[i].ct = next[i].cp = 0.f;
                if (s == p.s0 || NT > 1) next[i].dc = b >= p.B ? 0.f : s > 0 ? p.dc[idx] : dcn ? load16<BF16>(dcn + idx) : 0.f;
                if (b < p.B && t >= 0) {
                    const uint16_t *grow = gates + ((size_t)t * p.B + b) * G + (size_t)(U >> 4) * 64 + (U & 15);
                    next[i].gi = grow[0];
                    next[i].gf = grow[16];
                    next[i].gg = grow[32];
                    next[i].go = grow[48];
                    next[i].ct = p.cs[(size_t)(t + 1) * slab + idx];
                    next[i].cp = p.cs[(size_t)t * slab + idx];
                    next[i].dy = dy[(size_t)t * slab + idx];
                }
            }
        };
        fetch(p.s0, 0);
        uint32_t wi = 0, gi = 0;  // tiles contracted, tiles published
        bool ok = true;
        for (int s = p.s0; s < p.s1 && ok; ++s) {
            const int t = p.T - 1 - s;  // time step whose dG is produced (t = -1: only dh0 / dc0)
            for (int n = 0; n < NT; ++n) {
                const int b0 = (tile0 + n) * BT;
                // dG and the carried dc are linear in dh and dc: everything else is formed ahead of the wait
                struct Factors {
                    float dy, ka, ki, kf, kg, ko, gf, dc;
                };
                Factors fac[PAIRS];
#pragma unroll
                for (int i = 0; i < PAIRS; ++i) {
                    const Inputs &v = next[i];
                    const float g0 = load16<BF16>(&v.gi), g1 = load16<BF16>(&v.gf), g2 = load16<BF16>(&v.gg), g3 = load16<BF16>(&v.go);
                    const float tc = tanh_sel<ACCURATE>(v.ct);
                    fac[i] = Factors{load16<BF16>(&v.dy), g3 * (1.f - tc * tc), g2 * g0 * (1.f - g0), v.cp * g1 * (1.f - g1),
                                     g0 * (1.f - g2 * g2), tc * g3 * (1.f - g3), g1, v.dc};
                }
                const int n_next = n + 1 == NT ? 0 : n + 1, s_next = n + 1 == NT ? s + 1 : s;
                if (s_next < p.s1) fetch(s_next, n_next);
                // dh contribution from the step above: reduce-scattered partial products
                float dh_in[PAIRS];
                if (s == 0) {
#pragma unroll
                    for (int i = 0; i < PAIRS; ++i) {
                        const int b = b0 + nb + 16 * i;
                        dh_in[i] = (dhn && b < p.B) ? load16<BF16>(dhn + (size_t)b * p.H + U) : 0.f;
                    }
                } else {
                    const int rb = wi & 1;
                    // No thread leaves between here and the second named barrier below, whatever its waits return: the barriers
                    // OR the failures, so that all 256 threads go on or give up together.
                    bool good = __all_sync(0xffffffffu, mbar_wait(tfull, wi & 1, abort_w, wait_ns));
                    if (tid == 0 && n == 0) FLSTM_STAMP(s - p.s0, 5);
                    tcgen05_fence_after();
                    if (good) {
                        uint32_t acc[BT / 2];
                        if (BT == 32) tmem_ld_32x32b_x16(taddr, *reinterpret_cast<uint32_t(*)[16]>(&acc[0]));
                        else tmem_ld_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&acc[0]));
                        tmem_ld_wait();
                        float4 *dst = reinterpret_cast<float4 *>(s_ps + (quad * 32 + lane) * RS + col0);
#pragma unroll
                        for (int i = 0; i < BT / 8; ++i)
                            dst[i] = make_float4(__uint_as_float(acc[4 * i]), __uint_as_float(acc[4 * i + 1]),
                                                 __uint_as_float(acc[4 * i + 2]), __uint_as_float(acc[4 * i + 3]));
                    }
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty);
                    const bool failed = named_barrier_or(1, kEpilogueThreads, !good);
                    if (!failed) {
                        // UPO rows of BT sums for this CTA arrive from every CTA of the cluster, its own included
                        if (tid == 0) mbar_expect_tx(&rbar[rb], (uint32_t)(KS * UPO * BT * 4));
                        constexpr int V = BT / 4;  // 16-byte pieces of a row
#pragma unroll
                        for (int i = 0; i < 64 * V / kEpilogueThreads; ++i) {
                            const int e = tid + i * kEpilogueThreads, row = e / V, v = e % V;
                            const float4 a = *reinterpret_cast<const float4 *>(s_ps + row * RS + 4 * v);
                            const float4 b = *reinterpret_cast<const float4 *>(s_ps + (64 + row) * RS + 4 * v);
                            const uint32_t owner = row / UPO, off = (uint32_t)(((rb * KS + kq) * UPO + row % UPO) * RS + 4 * v) * 4u;
                            st_async_v4(map_to_rank(red_local + off, owner), __float_as_uint(a.x + b.x), __float_as_uint(a.y + b.y),
                                        __float_as_uint(a.z + b.z), __float_as_uint(a.w + b.w), map_to_rank(rbar_local + rb * 8, owner));
                        }
                        if (tid == 0 && n == 0) FLSTM_STAMP(s - p.s0, 9);
                        good = mbar_wait_cluster(&rbar[rb], (wi >> 1) & 1, abort_w, wait_ns);
                    } else {
                        good = false;
                    }
                    if (tid == 0 && n == 0) FLSTM_STAMP(s - p.s0, 10);
                    const float *red = s_red + (size_t)rb * KS * UPO * RS;
#pragma unroll
                    for (int i = 0; i < PAIRS; ++i) {
                        float acc = 0.f;
#pragma unroll
                        for (int src = 0; src < KS; ++src) acc += red[(src * UPO + u16) * RS + nb + 16 * i];
                        dh_in[i] = acc;
                    }
                    // one warp's failure is everybody's
                    if (named_barrier_or(1, kEpilogueThreads, !good)) {
                        ok = false;
                        break;
                    }
                    if (tid == 0 && n == 0) FLSTM_STAMP(s - p.s0, 6);
                    ++wi;
                }
                // fused pointwise backward for the owned (unit, sequence) pairs
#pragma unroll
                for (int i = 0; i < PAIRS; ++i) {
                    const int b = b0 + nb + 16 * i;
                    if (b >= p.B) continue;
                    const size_t idx = (size_t)b * p.H + U;
                    const Factors &f = fac[i];
                    if (t < 0) {
                        if (p.dh0) p.dh0[idx] = dh_in[i];
                        if (p.dc0) p.dc0[idx] = f.dc;
                        continue;
                    }
                    const float dh = ACCURATE && U >= p.real_units ? 0.f : f.dy + dh_in[i];
                    const float dcv = fmaf(dh, f.ka, f.dc), dc_out = dcv * f.gf;
                    uint16_t *drow = dg + ((size_t)t * p.B + b) * G + (size_t)(U >> 4) * 64 + (U & 15);
                    drow[0] = to16<BF16>(dcv * f.ki);
                    drow[16] = to16<BF16>(dcv * f.kf);
                    drow[32] = to16<BF16>(dcv * f.kg);
                    drow[48] = to16<BF16>(dh * f.ko);
                    // the carry of a lone tile stays in its thread; a later launch looks for it in memory
                    if (NT == 1) next[i].dc = dc_out;
                    if (NT > 1 || s + 1 == p.s1) p.dc[idx] = dc_out;
                }
                if (t >= 0) {
                    if (tid == 0 && n == 0) FLSTM_STAMP(s - p.s0, 7);
                    // publish dG_t: ONE arrival per CTA by a thread of its own, behind every warp's stores; no third tile may use
                    // a gdone barrier before the publisher has seen this phase of it
                    const bool seen = gi < 2 || mbar_wait(&pdone[gi & 1], ((gi >> 1) - 1) & 1, abort_w, wait_ns);
                    __syncwarp();
                    if (lane == 0 && seen) mbar_arrive(&gdone[gi & 1]);
                    ++gi;
                }
            }
        }
    }
#undef FLSTM_STAMP
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();  // nobody leaves while a peer may still send into its shared memory
    if (*abort_w) {
        // after an abort this CTA may not have waited for partial sums that a peer sent before it reached the barrier
        // above: give those asynchronous stores time to land before the shared memory is released
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < kAbortDrainNs) {}
    }
    if (warp == 5) tmem_dealloc(tmem_base, kTmemColumns);
    if (threadIdx.x == 0 && *abort_w) atomicCAS(p.err, 0u, 1u);
    if (threadIdx.x == 0) leave_counters(p.counters, (int)gridDim.x / (pl.jt * KS) * pl.nt, p.exits);
}

void cluster_attr(cudaLaunchAttribute *a) {
    a->id = cudaLaunchAttributeClusterDimension;
    a->val.clusterDim.x = KS;
    a->val.clusterDim.y = 1;
    a->val.clusterDim.z = 1;
}

template <int BT, bool BF16, bool ACC>
int launch_one(const CUtensorMap &tw, const BwdTmMaps &maps, const BwdTmPlan &pl, const BwdParams &p, cudaStream_t s) {
    auto kern = lstm_bwd_tm_kernel<BT, BF16, ACC>;
    FLSTM_CUDA_TRY(ensure_smem_limit(kern, (size_t)pl.smem_bytes));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;  // co-residency: CTAs wait on one another
    attr[0].val.cooperative = 1;
    cluster_attr(&attr[1]);
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, maps, pl, p);
    if (e == cudaErrorNotSupported || e == cudaErrorInvalidValue) {
        // as in tc_lstm_bwd.cu: planning has proved that every cluster is resident at once
        cudaGetLastError();
        cfg.attrs = attr + 1;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, tw, maps, pl, p);
    }
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "BPTT launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

// clusters of this plan that the current device holds at once, or -1
template <int BT>
int max_clusters(const BwdTmPlan &pl) {
    auto kern = lstm_bwd_tm_kernel<BT, false, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cudaLaunchAttribute attr[1];
    cluster_attr(attr);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (ensure_smem_limit(kern, (size_t)pl.smem_bytes) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return n;
}

}  // namespace

// ------------------------------------------------------------------ host side
static int plan_groups(int B, int H, int groups, size_t smem_limit, BwdTmPlan *plan) {
    BwdTmPlan pl{};
    pl.jt = H / 64;
    // one tile of 32 sequences per group, of 64, or several of 64 in turn: the tiles are independent recurrences with a step
    // barrier each, so the chain of one hides behind the others' contractions
    pl.BT = B <= 32 * groups ? 32 : 64;
    const int tiles = (B + pl.BT - 1) / pl.BT;
    pl.nt = (tiles + groups - 1) / groups;
    pl.ngroups = (tiles + pl.nt - 1) / pl.nt;
    if (pl.BT == 64 && pl.nt == 1 && H <= 1024) return FLSTM_OK;  // a chain that stands alone: the other kernels are as fast
    // Tiles in turn against the step-by-step GEMMs (which exist for H % 128 == 0), backward pass in us a step with its GEMMs:
    //   2 tiles: H = 512, B = 512 12.4 -> 8.7    H = 1024, B = 256 13.8 -> 9.8   H = 1536, B = 128 17.6 -> 10.9   H = 2048, B = 128 17.4 -> 16.0
    //   3 tiles: H = 640, B = 512 16.2 -> 14.0   H = 1024, B = 384 16.4 -> 13.6  H = 1792, B = 192 21.4 -> 16.3   H = 2048, B = 190 21.9 -> 23.2
    //   4 tiles: H = 512, B = 1024 16.3 -> 17.3  H = 1024, B = 512 18.6 -> 18.5  H = 1536, B = 256 20.4 -> 17.9   H = 1792, B = 256 23.1 -> 21.4
    // Every tile brings its dG through the SM's port (H x 128 bytes) and its own pointwise pass, a step GEMM spreads them.  At other
    // H the alternative takes several tiles per step one after the other (H = 1216, B = 200 25.4 -> 15.2).
    const int most = H % 128 != 0 ? 6 : H > 1792 ? 2 : H > 1024 ? 4 : 3;
    if (pl.nt > most || pl.nt * pl.ngroups > kMaxStepCounters) return FLSTM_OK;
    const int kcq = H / 16 / KS;
    pl.kp = kcq / 2;
    pl.left = kcq % 2;
    const int tmem_steps = (kTmemColumns - 2 * pl.BT) / 32, step_bytes = 2 * pl.BT * 128;
    pl.ct = pl.kp < tmem_steps ? pl.kp : tmem_steps;
    pl.cs = pl.kp - pl.ct;
    auto fits = [&]() { return (size_t)layout_of(pl).total <= smem_limit; };
    if (pl.nt > 1) {  // copies of two chunk-steps, as many as fit: the next tile's arrive while this one is contracted
        pl.ch = pl.kp < 2 ? 1 : 2;
        pl.stages = 16;
        while (!fits() && pl.stages > 3) --pl.stages;
    } else {  // dG in copies of up to 64 KB, the whole tile at once if it fits
        pl.ch = 65536 / step_bytes < pl.kp ? 65536 / step_bytes : pl.kp;
        pl.stages = (pl.kp + pl.ch - 1) / pl.ch;
    }
    while (!fits() && pl.ch > 1) {
        pl.ch = pl.ch > 2 ? 2 : 1;
        pl.stages = (pl.kp + pl.ch - 1) / pl.ch;
        while (!fits() && pl.stages > 2) --pl.stages;
    }
    pl.direct = fits_direct(pl, smem_limit);
    if (!pl.direct && !fits()) return FLSTM_OK;
    pl.ring = !pl.direct && (pl.nt > 1 || pl.stages * pl.ch < pl.kp);
    // All of shared memory: a CTA allocates all of tensor memory, so no other kernel that uses some (another engine's, on another
    // stream) may share its SM; two grids that each held what the other's CTAs were waiting for would run into their limits
    pl.smem_bytes = (int)smem_limit;
    pl.grid = pl.jt * KS * pl.ngroups;
    pl.use = true;
    *plan = pl;
    return FLSTM_OK;
}

int plan_bwd_tm(int B, int H, int sms, size_t smem_limit, BwdTmPlan *plan, bool check_device) {
    *plan = BwdTmPlan{};
    if (H % 64 != 0 || H < 256 || smem_limit < 160 * 1024) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_TMEM");
    if (env && env[0] == '0') return FLSTM_OK;
    // as many batch groups as the device holds clusters for at once
    for (int groups = sms / (H / 64 * KS); groups > 0; --groups) {
        FLSTM_TRY(plan_groups(B, H, groups, smem_limit, plan));
        if (!plan->use) return FLSTM_OK;
        if (!check_device || (plan->direct ? max_clusters_direct(*plan) : plan->BT == 32 ? max_clusters<32>(*plan) : max_clusters<64>(*plan)) * KS >= plan->grid) return FLSTM_OK;
        *plan = BwdTmPlan{};
    }
    return FLSTM_OK;
}

int make_bwd_tm_maps(BwdTmMaps *maps, const BwdTmPlan &pl, const void *dg, size_t steps, size_t B, size_t H) {
    for (int kq = 0; kq < KS; ++kq)
        FLSTM_TRY(make_tensor_map_halves(&maps->half[kq], static_cast<const char *>(dg) + (size_t)kq * (2 * pl.kp + pl.left) * 128, steps, B,
                                         4 * H, pl.BT, pl.kp, pl.ch));
    if (pl.left) FLSTM_TRY(make_tensor_map_chunked(&maps->chunk, dg, steps, B, 4 * H, pl.BT, 1));
    return FLSTM_OK;
}

int lstm_backward_tm(int dtype, const BwdTmPlan &pl, const CUtensorMap &tw, const BwdTmMaps &maps, const BwdParams &p, cudaStream_t s) {
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, acc = p.real_units > 0;
#define FLSTM_TM_CASE(BT_)                                                                                                \
    if (pl.BT == BT_) {                                                                                                   \
        if (bf16) return acc ? launch_one<BT_, true, true>(tw, maps, pl, p, s) : launch_one<BT_, true, false>(tw, maps, pl, p, s); \
        return acc ? launch_one<BT_, false, true>(tw, maps, pl, p, s) : launch_one<BT_, false, false>(tw, maps, pl, p, s); \
    }
    FLSTM_TM_CASE(32) FLSTM_TM_CASE(64)
#undef FLSTM_TM_CASE
    return set_error(FLSTM_ERR_UNSUPPORTED, "no tensor-memory BPTT kernel for this plan");
}

}  // namespace tc
}  // namespace flstm_b200
