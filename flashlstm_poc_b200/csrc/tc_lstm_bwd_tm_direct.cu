// The tensor-memory BPTT kernel (tc_lstm_bwd_tm.cu: clusters of four CTAs that split K = 4H, the K halves of each over the lane
// halves) for one batch tile of 32 sequences, without a step barrier: dG_t goes from CTA to CTA through pieces that announce
// themselves (tc_direct.cuh).
//
// What bounds a step is its chain: with a counter per step 7.6 k cycles at H = 1024, B = 64, of which releasing the stores 1.4 k, the
// counter 1.5 k, copying 64 KB 1.4 k, UMMAs 1.2 k, the reduce-scatter of the partial sums in the cluster 1.4 k, the pointwise update
// 0.5 k.  The exchange here replaces the first three: 5.8 k.
//
// Roles.  Warps 0-15 epilogue and gather, 16 weights kept in shared memory, 17 UMMA issuer, 18 the launch's one counter barrier, then
// fences behind resets.  A CTA's part of dG_t is one 64-wide chunk of K, 128 bytes per sequence; a thread has the four gate
// gradients of a (unit, sequence) pair, four shuffles make pieces of eight units of a gate of them, written whole.
//
// A tile of the operand is free when its accumulator has been read, as in the forward kernel (tc_lstm_fwd_tm_direct.cu); so are the
// exits.
//
// Replaces the same reference launches (flashlstm_v2/src/lstm_backward.cu:158-227, 1057-1101).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc_common.cuh"
#include "tc_direct.cuh"
#include "tc_kernels.h"
#include "tc_recurrent.cuh"

namespace flstm_b200 {
namespace tc {

namespace {

constexpr int kEpilogueThreads = kGatherThreads, kThreads = kEpilogueThreads + 96;
constexpr int kStepBytesW = 2 * 64 * 128;  // one chunk-step of A: two blocks of 64 K rows x 64 units
constexpr int kTmemColumns = 512;
constexpr int kBarrierBytes = 1024;
constexpr int kFillSlots = 8;  // a multiple of 4: a slot always belongs to the same set of warps (see tc_lstm_fwd_tm.cu)
constexpr int kMinSmemBytes = kBarrierBytes + kFillSlots * kStepBytesW + 1024;
constexpr int KS = 4, UPO = 64 / KS, BT = 32, N = 2 * BT;
constexpr int kRowStride = BT + 4;               // of the exchange and reduce buffers (floats), keeps float4 alignment
constexpr uint32_t kRound = kGatherThreads * 16;  // a chunk-step of both halves: what the gather threads copy in a round
static_assert(kRound == N * 128, "a round is a chunk-step");

struct Layout {
    int w, left_w, tile, ps, red, total;
};
__host__ __device__ inline Layout layout_of(const BwdTmPlan &pl) {
    Layout l;
    l.w = pl.cs * kStepBytesW;
    l.left_w = pl.left ? kStepBytesW : 0;
    l.tile = pl.kp * (int)kRound + (pl.left ? BT * 128 : 0);  // the chunk that is left lies behind the chunk-steps
    l.ps = 128 * kRowStride * 4;
    l.red = 2 * KS * UPO * kRowStride * 4;
    l.total = kBarrierBytes + l.w + l.left_w + l.tile + l.ps + l.red + 1024 /*align*/;
    if (l.total < kMinSmemBytes) l.total = kMinSmemBytes;
    return l;
}
// of the kernel that a plan takes: H = 1024 and 1536
__host__ __device__ inline int kernel_rounds(const BwdTmPlan &pl) { return pl.kp + pl.left <= 8 ? 8 : 12; }

// Whether the operand tile's row of a sequence holds a word that its CTA had not written yet: lane `part` of 16 looks at a sixteenth of
// it, all words of each piece.
__device__ __forceinline__ bool holds_unwritten(uint32_t row, int part, int kp, int left) {
    const uint32_t mine = row + (part >> 3) * BT * 128 + (part & 7) * 16;
    bool found = false;
#pragma unroll 1
    for (int c = 0; c < kp; ++c) found |= gather_unwritten(mine + (uint32_t)c * kRound);
    if (left && part < 8) found |= gather_unwritten(mine + (uint32_t)kp * kRound);
    return found;
}

template <int ROUNDS, bool BF16, bool ACCURATE, bool LOST>  // LOST: the self-test's form (LostWords)
__global__ void __launch_bounds__(kThreads, 1)
lstm_bwd_tm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ BwdTmPlan pl, BwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const Layout L = layout_of(pl);
    const int KP = pl.kp, CT = pl.ct, CS = pl.cs;
    uint8_t *s_w = smem + kBarrierBytes, *s_lw = s_w + L.w, *s_tile = s_lw + L.left_w;
    float *s_ps = reinterpret_cast<float *>(s_tile + L.tile), *s_red = s_ps + L.ps / 4;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *tfull = full + kGatherStages, *tempty = tfull + 1, *wbar = tempty + 1;
    uint64_t *rbar = wbar + 1;  // [2] partial sums received
    uint64_t *reset = rbar + 2, *ready = reset + kResetBarriers;
    uint64_t *ffull = ready + 1, *fempty = ffull + kFillSlots;  // while W_hh moves into tensor memory
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fempty + kFillSlots);
    volatile uint32_t *abort_w = tmem_slot + 1;
    const uint32_t performed = smem_u32(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kq = (int)cluster_ctarank();
    const int cl = blockIdx.x / KS, ng = cl / pl.jt, j = cl % pl.jt;  // batch group, unit tile [64j, 64j+64)
    const int b0 = ng * BT;
    unsigned int *counter = p.counters + ng;
    const int kcq = 2 * KP + pl.left, c_first = kq * kcq;  // 64-wide K chunks of this CTA
    const int steps = p.s1 - p.s0;                         // iterations of this launch; all but the last send their dG on
    const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;

    // ring: [slot][group][K range of a cluster rank][chunk-step][half][sequence][64 columns], the order of the operand tile: 4 KB per
    // 64-wide chunk of K.  This CTA writes chunk 4j + kq.
    char *const ring = static_cast<char *>(p.ring);
    const uint32_t group_bytes = (uint32_t)(p.H / 16) * BT * 128, slot_bytes = gridDim.x / (pl.jt * KS) * group_bytes;
    const int u16 = threadIdx.x & 15, nb = (threadIdx.x >> 4) & 31, odd = u16 & 1;  // unit u16 of the CTA's 16, sequence nb
    // the piece of this thread: units (u16 & 8) .. + 7 of one gate; the lanes with bit 1 have none
    const bool has_piece = (u16 & 2) == 0;
    const int piece_col = (2 * odd + (u16 >> 2 & 1)) * 16 + (u16 & 8);
    uint32_t my_piece;
    {
        const int c = 4 * j + kq, range = c / kcq, l = c % kcq;
        const int at = l < KP ? 2 * l : l < 2 * KP ? 2 * (l - KP) + 1 : 2 * KP;
        my_piece = (uint32_t)ng * group_bytes + (uint32_t)(range * kcq + at) * (BT * 128) + nb * 128 + piece_col * 2;
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < kGatherStages; ++i) mbar_init(&full[i], 1);
        mbar_init(tfull, 1);
        mbar_init(tempty, kEpilogueThreads / 32);
        mbar_init(wbar, 1);
        for (int i = 0; i < 2; ++i) mbar_init(&rbar[i], 1);
        for (int i = 0; i < kResetBarriers; ++i) mbar_init(&reset[i], kEpilogueThreads / 32);
        mbar_init(ready, 1);
        for (int i = 0; i < kFillSlots; ++i) {
            mbar_init(&ffull[i], 1);
            mbar_init(&fempty[i], 4);
        }
        *abort_w = 0;
        tmem_slot[2] = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_w);
    }
    if (warp == 17) {
        tmem_alloc(tmem_slot, kTmemColumns);
        tmem_relinquish();
    }
    const uint4 unwritten = make_uint4(kUnwritten, kUnwritten, kUnwritten, kUnwritten);
    if (warp < 16 && has_piece && steps > 1)
        for (int s = 0; s < kDirectSlots; ++s) st_relaxed_gpu_16(ring + (size_t)s * slot_bytes + my_piece, unwritten);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + N;
    // W_hh^T into tensor memory, by way of the shared memory that dG will use (as in tc_lstm_bwd_tm.cu): lane l takes unit l % 64 and K
    // half l / 64, 32 columns of two K elements per chunk-step; of four chunk-steps each set of four warps takes one
    if (warp == 16 && elect_one()) {
        for (int c = 0; c < CT; ++c) {
            const int slot = c % kFillSlots;
            if (c >= kFillSlots && !mbar_wait(&fempty[slot], (uint32_t)(c / kFillSlots - 1) & 1u, abort_w, wait_ns)) break;
            mbar_expect_tx(&ffull[slot], kStepBytesW);
            for (int h = 0; h < 2; ++h)
                tma_load_2d(s_w + slot * kStepBytesW + h * 8192, &tm_w, j * 64, (c_first + h * KP + c) * 64, &ffull[slot]);
        }
    } else if (warp < 16) {
        const int quad = warp & 3, l = quad * 32 + lane, un = l & 63;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        for (int c = warp >> 2; c < CT; c += 4) {
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

    if (warp == 16) {
        // ------------------------------------------------------------ weights kept in shared memory
        if ((CS > 0 || pl.left) && elect_one()) {
            mbar_expect_tx(wbar, (uint32_t)(L.w + L.left_w));
            for (int c = 0; c < CS; ++c)
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(s_w + c * kStepBytesW + h * 8192, &tm_w, j * 64, (c_first + h * KP + CT + c) * 64, wbar);
            if (pl.left)  // the second block only feeds lanes whose results are ignored
                for (int h = 0; h < 2; ++h) tma_load_2d(s_lw + h * 8192, &tm_w, j * 64, (c_first + 2 * KP) * 64, wbar);
            mbar_drain(wbar, 0, wait_ns);
        }
    } else if (warp == 18) {
        // ------------------------------------------------------------ the launch's barrier, then fences behind resets
        if (steps > 1 && elect_one() && wait_counter(counter, (unsigned)(pl.jt * KS) + p.extra_arrivals, p.err, abort_w, 3u, wait_ns)) {
            mbar_arrive(ready);
            perform_resets(reset, performed, steps, abort_w, wait_ns, LOST && blockIdx.x == p.lost.cta && (p.lost.what & kLostCount) ? p.lost.step : -1);
        }
    } else if (warp == 17) {
        // ------------------------------------------------------------ UMMA issuer
        if (elect_one()) {
            bool ok = (CS == 0 && !pl.left) || mbar_wait(wbar, 0, abort_w, wait_ns);
            constexpr uint32_t idesc_ts = umma_idesc_f16(128, N, BF16 ? 1 : 0, 0, 0), idesc_ss = umma_idesc_f16(128, N, BF16 ? 1 : 0, 1, 0);
            constexpr uint32_t idesc_left = umma_idesc_f16(128, BT, BF16 ? 1 : 0, 1, 0);
            constexpr uint32_t kStepG = (N * 128) >> 4, kStepW = kStepBytesW >> 4;  // descriptor units
            const uint32_t dw_res = umma_desc_lo(smem_u32(s_w), 8192), dw_left = umma_desc_lo(smem_u32(s_lw), 8192);
            const uint32_t dd_tile = umma_desc_lo(smem_u32(s_tile)), tfull_l = smem_u32(tfull);
            constexpr int kPieces = stage_pieces(ROUNDS);
            int committed = 0;
            const uint32_t items = (uint32_t)(p.s1 - s_first);
            for (uint32_t wi = 0; wi < items && ok; ++wi) {
                const int s = s_first + (int)wi;
                ok = mbar_wait(tempty, (wi & 1) ^ 1, abort_w, wait_ns);
                if (!ok) break;
                tcgen05_fence_after();
                uint32_t acc = 0, dd = dd_tile, da = tmem_a, dw = dw_res;  // the step's first instruction overwrites the accumulator
                int c = 0;
                for (int st = 0; st < (ROUNDS + kPieces - 1) / kPieces; ++st) {
                    ok = mbar_wait(&full[st], wi & 1, abort_w, wait_ns);
                    if (!ok) break;
                    if (st == 0) FLSTM_STAMP(s - p.s0, 2);
                    FLSTM_STAMP(s - p.s0, 3);
                    tcgen05_fence_after();
                    const int c1 = (st + 1) * kPieces < KP ? (st + 1) * kPieces : KP, ct1 = c1 < CT ? c1 : CT;
#pragma unroll 4
                    for (; c < ct1; ++c) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) umma_lo_ts<false>(tmem_base, da + 8 * k, dd + 2 * k, idesc_ts, k ? 1u : acc);
                        acc = 1u;
                        da += 32;
                        dd += kStepG;
                    }
#pragma unroll 2
                    for (; c < c1; ++c) {  // K steps of 16: +2048 bytes on the MN-major W_hh, +32 bytes on the K-major dG
#pragma unroll
                        for (int k = 0; k < 4; ++k) umma_lo_ss<false>(tmem_base, dw + 128 * k, dd + 2 * k, idesc_ss, k ? 1u : acc);
                        acc = 1u;
                        dw += kStepW;
                        dd += kStepG;
                    }
                }
                if (!ok) break;
                if (pl.left) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_lo_ss<false>(tmem_base, dw_left + 128 * k, dd + 2 * k, idesc_left, 1u);
                }
                umma_commit_addr(tfull_l);
                ++committed;
                FLSTM_STAMP(s - p.s0, 4);
            }
            // the tensor memory is freed at the end of the kernel: the last committed batch of UMMAs must be done
            if (committed > 0) mbar_drain(tfull, (uint32_t)(committed - 1) & 1u, wait_ns);
        }
    } else if (warp < 16) {
        // ------------------------------------------------------------ epilogue and gather (512 threads)
        const int tid = threadIdx.x;
        const int U = j * 64 + kq * UPO + u16, b = b0 + nb;
        const bool valid = b < p.B;
        const size_t slab = (size_t)p.B * p.H, G = (size_t)4 * p.H, idx = (size_t)b * p.H + U;
        const uint16_t *gates = static_cast<const uint16_t *>(p.gates);
        const uint16_t *dy = static_cast<const uint16_t *>(p.dy);
        const uint16_t *dhn = static_cast<const uint16_t *>(p.dhn);
        const uint16_t *dcn = static_cast<const uint16_t *>(p.dcn);
        uint16_t *dg = static_cast<uint16_t *>(p.dg);

        // this thread's pieces of the dG tile
        Gather<ROUNDS, kRound, true, false> g;
        const char *from;
        {
            const int half = tid >> 8, n = (tid & 255) >> 3, x = tid & 7;
            g.to = smem_u32(s_tile) + half * BT * 128 + n * 128 + ((x ^ (n & 7)) << 4);
            g.mine = b0 + n < p.B ? KP + (half == 0 ? pl.left : 0) : 0;
            g.full = map_to_rank(smem_u32(full), (uint32_t)kq);
            from = ring + (size_t)ng * group_bytes + (size_t)(c_first * BT * 128 + half * BT * 128 + n * 128 + x * 16);
            if (p.s0 > 0)  // dG of the step that the launch before ended with
                g.first(reinterpret_cast<const char *>(dg) +
                            (((size_t)(p.T - p.s0) * p.B + b0 + n) * G + (size_t)(c_first + half * KP) * 64 + x * 8) * 2,
                        128, KP, (uint32_t)KP * 128);
        }
        const int quad = warp & 3, col0 = (warp >> 2) * (BT / 4);  // lane quadrant, quarter of the columns
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (quad >> 1) * BT + col0;
        const uint32_t red_local = smem_u32(s_red), rbar_local = smem_u32(rbar);
        if (steps > 1) {
            fence_acq_rel_gpu();
            named_barrier_sync(2, kEpilogueThreads);
            if (tid == 0) red_release_gpu_add(counter, 1u);
        }
        // what the pointwise update reads, fetched a step ahead
        struct Inputs {
            uint16_t gi, gf, gg, go, dy;
            float ct, cp;
        } next;
        auto fetch = [&](int s) {
            const int t = p.T - 1 - s;
            next = Inputs{0, 0, 0, 0, 0, 0.f, 0.f};
            if (valid && t >= 0) {
                const uint16_t *grow = gates + ((size_t)t * p.B + b) * G + (size_t)(U >> 4) * 64 + (U & 15);
                next.gi = grow[0];
                next.gf = grow[16];
                next.gg = grow[32];
                next.go = grow[48];
                next.ct = p.cs[(size_t)(t + 1) * slab + idx];
                next.cp = p.cs[(size_t)t * slab + idx];
                next.dy = dy[(size_t)t * slab + idx];
            }
        };
        fetch(p.s0);
        float dc = !valid ? 0.f : p.s0 > 0 ? p.dc[idx] : dcn ? load16<BF16>(dcn + idx) : 0.f;
        const int lost_at = LOST && blockIdx.x == p.lost.cta && (p.lost.what & kLostPart) ? p.lost.step : -1;
        const int torn_at = LOST && blockIdx.x == p.lost.cta && (p.lost.what & kLostWord) ? p.lost.step : -1;
        uint32_t wi = 0;  // steps contracted
        bool gathered = true;
        for (int s = p.s0; s < p.s1; ++s) {
            const int t = p.T - 1 - s, k = s - p.s0;  // time step whose dG is produced (t = -1: only dh0 / dc0); number in the launch
            // dG and the carried dc are linear in dh and dc: everything else is formed ahead of the wait
            const float g0 = load16<BF16>(&next.gi), g1 = load16<BF16>(&next.gf), g2 = load16<BF16>(&next.gg), g3 = load16<BF16>(&next.go);
            const float tc = tanh_sel<ACCURATE>(next.ct), f_dy = load16<BF16>(&next.dy);
            const float ka = g3 * (1.f - tc * tc), ki = g2 * g0 * (1.f - g0), kf = next.cp * g1 * (1.f - g1), kg = g0 * (1.f - g2 * g2),
                        ko = tc * g3 * (1.f - g3);
            if (s + 1 < p.s1) fetch(s + 1);
            bool good = gathered;
            if (k >= kResetSlack && resets_slot(k - kResetSlack, steps))
                good = wait_performed(performed, (uint32_t)(k - kResetSlack + 1), abort_w, wait_ns) && good;
            // dh contribution from the step above: reduce-scattered partial products
            float dh_in = 0.f;
            if (s == 0) {
                if (dhn && valid) dh_in = load16<BF16>(dhn + idx);
            } else {
                const int rb = wi & 1;
                // No thread leaves between here and the second named barrier below, whatever its waits return: the barriers OR the
                // failures, so that all 512 threads go on or give up together.
                const bool seen = __all_sync(0xffffffffu, mbar_wait(tfull, wi & 1, abort_w, wait_ns));
                good = good && seen;
                if (tid == 0) FLSTM_STAMP(k, 5);
                tcgen05_fence_after();
                if (seen) {
                    uint32_t acc[BT / 4];
                    tmem_ld_32x32b_x8(taddr, acc);
                    tmem_ld_wait();
                    float4 *dst = reinterpret_cast<float4 *>(s_ps + (quad * 32 + lane) * kRowStride + col0);
#pragma unroll
                    for (int i = 0; i < BT / 16; ++i)
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
                    static_assert(64 * V == kEpilogueThreads, "a piece per thread");
                    const int row = tid / V, v = tid % V;
                    const float4 a = *reinterpret_cast<const float4 *>(s_ps + row * kRowStride + 4 * v);
                    const float4 c = *reinterpret_cast<const float4 *>(s_ps + (64 + row) * kRowStride + 4 * v);
                    const uint32_t owner = row / UPO, off = (uint32_t)(((rb * KS + kq) * UPO + row % UPO) * kRowStride + 4 * v) * 4u;
                    st_async_v4(map_to_rank(red_local + off, owner), __float_as_uint(a.x + c.x), __float_as_uint(a.y + c.y),
                                __float_as_uint(a.z + c.z), __float_as_uint(a.w + c.w), map_to_rank(rbar_local + rb * 8, owner));
                    if (tid == 0) FLSTM_STAMP(k, 9);
                    good = mbar_wait_cluster(&rbar[rb], (wi >> 1) & 1, abort_w, wait_ns);
                } else {
                    good = false;
                }
                if (tid == 0) FLSTM_STAMP(k, 10);
                const float *red = s_red + (size_t)rb * KS * UPO * kRowStride;
#pragma unroll
                for (int src = 0; src < KS; ++src) dh_in += red[(src * UPO + u16) * kRowStride + nb];
                // A sum that is no number: a piece that came in part would give one (tc_direct.cuh)
                if (dh_in != dh_in && k > 0 && good && holds_unwritten(smem_u32(s_tile) + nb * 128, u16, KP, pl.left)) {
                    *abort_w = 1;
                    atomicExch(p.err, kErrTornPiece);
                    good = false;
                }
                // one warp's failure is everybody's
                if (named_barrier_or(1, kEpilogueThreads, !good)) break;
                if (tid == 0) FLSTM_STAMP(k, 6);
                ++wi;
            }
            // fused pointwise backward for the owned (unit, sequence) pair
            if (t < 0) {
                if (valid) {
                    if (p.dh0) p.dh0[idx] = dh_in;
                    if (p.dc0) p.dc0[idx] = dc;
                }
                continue;
            }
            const float dh = ACCURATE && U >= p.real_units ? 0.f : f_dy + dh_in;
            const float dcv = fmaf(dh, ka, dc);
            dc = dcv * g1;
            const uint32_t d01 = (uint32_t)to16<BF16>(dcv * ki) | (uint32_t)to16<BF16>(dcv * kf) << 16;
            const uint32_t d23 = (uint32_t)to16<BF16>(dcv * kg) | (uint32_t)to16<BF16>(dh * ko) << 16;
            // two units of a gate in a word: gates i and f (A, B) in even lanes, g and o in odd ones; then A in lanes without bit 2, B in
            // those with it, and eight units in lanes without bit 1
            uint4 piece;
            {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? d01 : d23, 1);
                const uint32_t A = odd ? __byte_perm(other, d23, 0x5410) : __byte_perm(d01, other, 0x5410);
                const uint32_t B = odd ? __byte_perm(other, d23, 0x7632) : __byte_perm(d01, other, 0x7632);
                const bool high = u16 & 4;
                const uint32_t got = __shfl_xor_sync(0xffffffffu, high ? A : B, 4);
                piece.x = high ? got : A;
                piece.z = high ? B : got;
                piece.y = __shfl_xor_sync(0xffffffffu, piece.x, 2);
                piece.w = __shfl_xor_sync(0xffffffffu, piece.z, 2);
            }
            const bool store = has_piece && valid, more = s + 1 < p.s1;
            const size_t slot = (size_t)(k & (kDirectSlots - 1)) * slot_bytes;
            if (more) {
                if (store && !(LOST && k == lost_at)) {
                    uint4 sent = piece;
                    if (LOST && k == torn_at && (nb & 3)) sent.x = kUnwritten;  // (the others are looked at by this word: gather_unwritten_whole)
                    st_relaxed_gpu_16(ring + slot + my_piece, sent);
                }
                g.mark_sent();
                if (k == 0) gathered = mbar_wait(ready, 0, abort_w, wait_ns);  // every CTA of the group has reset its pieces
            }
            if (tid == 0) FLSTM_STAMP(k, 7);
            // everything nobody waits for; the carry of dc stays in its thread, a later launch looks for it in memory
            if (store) *reinterpret_cast<uint4 *>(dg + ((size_t)t * p.B + b) * G + (size_t)(U >> 4) * 64 + piece_col) = piece;
            if (!more) {
                if (valid) p.dc[idx] = dc;
                continue;
            }
            if (resets_slot(k, steps)) {
                if (has_piece) st_relaxed_gpu_16(ring + (size_t)((k + kResetAhead) & (kDirectSlots - 1)) * slot_bytes + my_piece, unwritten);
                __syncwarp();
                if (lane == 0) mbar_arrive(&reset[k % kResetBarriers]);
            }
            if (tid == 0) FLSTM_STAMP(k, 8);
            g.issue(from + slot);
            if (tid == 0) FLSTM_STAMP(k, 0);
            gathered = g.finish(from + slot, p.err, abort_w, 3u, wait_ns) && gathered;
            if (tid == 0) FLSTM_STAMP(k, 1);
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
    if (warp == 17) tmem_dealloc(tmem_base, kTmemColumns);
    if (threadIdx.x == 0 && *abort_w) atomicCAS(p.err, 0u, 1u);
    if (threadIdx.x == 0) leave_counters(p.counters, (int)gridDim.x / (pl.jt * KS), p.exits);
}

void cluster_attr(cudaLaunchAttribute *a) {
    a->id = cudaLaunchAttributeClusterDimension;
    a->val.clusterDim.x = KS;
    a->val.clusterDim.y = 1;
    a->val.clusterDim.z = 1;
}

template <int ROUNDS, bool BF16, bool ACC, bool LOST = false>
int launch_one(const CUtensorMap &tw, const BwdTmPlan &pl, const BwdParams &p, cudaStream_t s) {
    auto kern = lstm_bwd_tm_kernel<ROUNDS, BF16, ACC, LOST>;
    FLSTM_CUDA_TRY(ensure_smem_limit(reinterpret_cast<const void *>(kern), pl.smem_bytes));
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, pl, p);
    if (e == cudaErrorNotSupported || e == cudaErrorInvalidValue) {
        // as in tc_lstm_bwd.cu: planning has proved that every cluster is resident at once
        cudaGetLastError();
        cfg.attrs = attr + 1;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, tw, pl, p);
    }
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "BPTT launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

// clusters of this plan that the current device holds at once, or -1
template <int ROUNDS>
int max_clusters(const BwdTmPlan &pl) {
    auto kern = lstm_bwd_tm_kernel<ROUNDS, false, false, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cudaLaunchAttribute attr[1];
    cluster_attr(attr);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (ensure_smem_limit(reinterpret_cast<const void *>(kern), pl.smem_bytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return n;
}

}  // namespace

// Beyond H = 1536 a CTA copies more than 96 KB of dG a step, which takes longer this way than in the four copies behind a barrier; us a
// step, B = 32 unless said otherwise: H = 832, B = 20 4.29 -> 3.49, H = 1024 4.57 -> 3.75 (B = 64 5.02 -> 4.19), H = 1088 4.90 -> 4.47,
// H = 1280 5.26 -> 4.51, H = 1408 5.37 -> 4.79, H = 1536 5.53 -> 4.92, H = 1664 5.80 -> 6.12, H = 1792 5.96 -> 6.30, H = 2048 6.42 -> 6.66.
bool fits_direct(const BwdTmPlan &pl, size_t smem_limit) {
    return pl.BT == BT && pl.nt == 1 && pl.ct + pl.cs == pl.kp && pl.kp + pl.left <= kernel_rounds(pl) &&
           (size_t)layout_of(pl).total <= smem_limit;
}
size_t direct_ring_bytes(const BwdTmPlan &pl) {
    return pl.use && pl.direct ? (size_t)kDirectSlots * pl.ngroups * pl.jt * 4 * BT * 128 : 0;
}
int max_clusters_direct(const BwdTmPlan &pl) {
    return kernel_rounds(pl) == 8 ? max_clusters<8>(pl) : max_clusters<12>(pl);
}

int lstm_backward_tm_direct(int dtype, const BwdTmPlan &pl, const CUtensorMap &tw, const BwdParams &p, cudaStream_t s) {
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, acc = p.real_units > 0;
#define FLSTM_TM_CASE(R_)                                                                                                      \
    if (kernel_rounds(pl) == R_) {                                                                                            \
        if (p.lost.what && !bf16 && !acc) return launch_one<R_, false, false, true>(tw, pl, p, s);                              \
        if (bf16) return acc ? launch_one<R_, true, true>(tw, pl, p, s) : launch_one<R_, true, false>(tw, pl, p, s);           \
        return acc ? launch_one<R_, false, true>(tw, pl, p, s) : launch_one<R_, false, false>(tw, pl, p, s);                   \
    }
    FLSTM_TM_CASE(8) FLSTM_TM_CASE(12)
#undef FLSTM_TM_CASE
    return set_error(FLSTM_ERR_UNSUPPORTED, "no tensor-memory BPTT kernel for this plan");
}

}  // namespace tc
}  // namespace flstm_b200
