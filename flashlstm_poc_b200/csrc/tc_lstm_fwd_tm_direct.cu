// The tensor-memory forward kernel (tc_lstm_fwd_tm.cu: CTA pairs, K split over the lane halves, nothing streamed) for batch tiles of 32
// sequences, without a step barrier: h_t goes from CTA to CTA through words that announce themselves (tc_direct.cuh).
//
// What bounds a step is its chain of L2 round trips.  With a counter per step, H = 1024, B = 64: 5.6 k cycles, of which
// releasing the stores 1.2 k, the counter 1.5 k, copying 32 KB 1.3 k, UMMAs behind the last copy 0.4 k, accumulator to result 1.1 k.
// The exchange here replaces the first three: 4.2 k cycles (H = 2048, B = 32: 6.9 -> 5.9 k, of which the UMMAs' own 2 k); us a step at
// fits_direct.
//
// Roles.  Warps 0-15 epilogue and gather, 16 projections, 17 UMMA issuer, 18 weights kept in shared memory, 19 the launch's one
// counter barrier, then fences behind resets.  A warp that has sent its part of h_t stores what nobody waits for while
// the others' parts are on their way, copies its share of them (the CTA's half of K, for all BT sequences) and looks at what came:
// with warps of their own for the gather each hand-over between roles added some 300 cycles, and the step took 4.7-4.9 k; the stores
// behind the gather, 4.7 k.
//
// The copies may overwrite h_{t-1}: the accumulator of step t, which the epilogue has read, says that the UMMAs have.  The exchange
// buffer is free again when the next accumulator comes: every warp of the CTA has handed over its part of the gather by then.
//
// Every wait is bounded.  The 512 epilogue threads leave together: a gather that fails is reported at the next step's barrier,
// which ORs the failures.  The other roles break out alone; a pair lingers before its final cluster barrier after an abort.
//
// Replaces the same reference launches as tc_lstm_fwd.cu (flashlstm_v2/src/lstm_forward.cu:744-830, src/lstm.cu:1241-1337).
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

constexpr int kEpilogueThreads = kGatherThreads, kThreads = kEpilogueThreads + 128;
constexpr int BT = 32, N = 2 * BT;         // sequences of a tile, UMMA N
constexpr int kRowStride = BT + 4;         // of the exchange buffer (floats), keeps float4 alignment
constexpr int kStepBytesW = 128 * 128;  // one chunk-step of A: 128 rows x 64 16-bit elements
constexpr int kTmemColumns = 512;
constexpr int kBarrierBytes = 1024;
constexpr int kFillSlots = 8;  // a multiple of 4: a slot always belongs to the same set of warps (see tc_lstm_fwd_tm.cu)
constexpr int kMinSmemBytes = kBarrierBytes + kFillSlots * kStepBytesW + 1024;

// the gather threads take a half of K in rounds of two chunk-steps
constexpr int kRoundSteps = kGatherThreads / (8 * BT);
__host__ __device__ inline int gather_rounds(const FwdTmPlan &pl) { return (pl.kc + kRoundSteps - 1) / kRoundSteps; }
// of the kernel that a plan takes: H = 1024, 2048 and 2368
__host__ __device__ inline int kernel_rounds(const FwdTmPlan &pl) {
    const int n = gather_rounds(pl);
    return n <= 4 ? 4 : n <= 8 ? 8 : 10;
}

struct Layout {
    int w, h, p, ex, total;
};
__host__ __device__ inline Layout layout_of(const FwdTmPlan &pl) {
    Layout l;
    l.w = pl.cs * kStepBytesW;
    l.h = gather_rounds(pl) * kRoundSteps * BT * 128;
    l.p = 2 * BT * 128;
    l.ex = 128 * kRowStride * 4;
    l.total = kBarrierBytes + l.w + l.h + l.p + l.ex + 1024 /*align*/;
    if (l.total < kMinSmemBytes) l.total = kMinSmemBytes;
    return l;
}

template <int ROUNDS, bool BF16, bool ACCURATE, bool LOST>  // LOST: the self-test's form (LostWords)
__global__ void __launch_bounds__(kThreads, 1)
lstm_fwd_tm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ FwdTmPlan pl,
                   FwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const Layout L = layout_of(pl);
    const int KC = pl.kc, CT = pl.ct, CS = pl.cs;
    uint8_t *s_w = smem + kBarrierBytes, *s_h = s_w + L.w, *s_p = s_h + L.h;
    float *s_ex = reinterpret_cast<float *>(s_p + L.p);
    uint64_t *hfull = reinterpret_cast<uint64_t *>(smem), *tfull = hfull + kGatherStages, *tempty = tfull + 1, *wbar = tempty + 1;
    uint64_t *reset = wbar + 1, *ready = reset + kResetBarriers, *pfull = ready + 1, *pempty = pfull + 2;
    uint64_t *ffull = pempty + 2, *fempty = ffull + kFillSlots;  // while W_hh moves into tensor memory
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fempty + kFillSlots);
    volatile uint32_t *abort_w = tmem_slot + 1;
    const uint32_t performed = smem_u32(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ng = blockIdx.x / pl.cta_rows, jr = blockIdx.x % pl.cta_rows;  // batch group, row block
    const int b0 = ng * BT;
    unsigned int *counter = p.counters + ng;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    // ring: [slot][group][16 units][sequence][unit].  A CTA's part is contiguous, and the operand tile has the same order (rows of 32
    // bytes, 32-byte swizzle), so that 128 bytes of the one become 128 bytes of the other: with lines that scatter over four rows of
    // 128 bytes, or lines written by four CTAs, a step took 400 (H = 1024) to 850 cycles (H = 2048) more
    char *const ring = static_cast<char *>(p.ring);
    const uint32_t slot_bytes = (uint32_t)gridDim.x * BT * 32u;

    // epilogue ownership: unit u of the CTA's 16 and sequence nb; the even lanes have the word of units u and u + 1
    const int u = threadIdx.x & 15, nb = (threadIdx.x >> 4) & 31, odd = u & 1;
    const uint32_t my_word = (uint32_t)((blockIdx.x * BT + nb) * 32 + (u & ~1) * 2);
    const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kGatherStages; ++i) mbar_init(&hfull[i], 2);  // the leader's: both CTAs report to it
        mbar_init(tfull, 1);
        mbar_init(tempty, 2 * kEpilogueThreads / 32);
        mbar_init(wbar, 1);
        for (int i = 0; i < kResetBarriers; ++i) mbar_init(&reset[i], kEpilogueThreads / 32);
        mbar_init(ready, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&pfull[i], 1);
            mbar_init(&pempty[i], kEpilogueThreads / 32);
        }
        for (int i = 0; i < kFillSlots; ++i) {
            mbar_init(&ffull[i], 1);
            mbar_init(&fempty[i], 4);
        }
        *abort_w = 0;
        tmem_slot[2] = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_w);
        tma_prefetch_desc(&tm_g);
    }
    if (warp == 17) {
        tmem_alloc_pair(tmem_slot, kTmemColumns);
        tmem_relinquish_pair();
    }
    if (warp < 16 && !odd && p.T > 1)
        for (int s = 0; s < kDirectSlots; ++s) st_relaxed_gpu(ring + (size_t)s * slot_bytes + my_word, kUnwritten);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + N;
    // W_hh into tensor memory, by way of the shared memory that h will use (as in tc_lstm_fwd_tm.cu): lane l of the CTA takes row
    // l % 64, K half l / 64, 32 columns of two elements per chunk-step; of four chunk-steps each set of four warps takes one
    if (warp == 16 && elect_one()) {
        for (int c = 0; c < CT; ++c) {
            const int slot = c % kFillSlots;
            uint8_t *dst = s_w + slot * kStepBytesW;
            if (c >= kFillSlots && !mbar_wait(&fempty[slot], (uint32_t)(c / kFillSlots - 1) & 1u, abort_w, wait_ns)) break;
            mbar_expect_tx(&ffull[slot], kStepBytesW);
            tma_load_2d(dst, &tm_w, c * 64, jr * 64, &ffull[slot]);
            tma_load_2d(dst + 8192, &tm_w, (KC + c) * 64, jr * 64, &ffull[slot]);
        }
    } else if (warp < 16) {
        const int quad = warp & 3, l = quad * 32 + lane;
        const uint32_t dst = tmem_a + ((uint32_t)(quad * 32) << 16);
        for (int c = warp >> 2; c < CT; c += 4) {
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
    const uint32_t wbar_c = map_to_rank(smem_u32(wbar), 0), tempty_c = map_to_rank(smem_u32(tempty), 0);

    const bool tracing = p.trace != nullptr && blockIdx.x == 0;
#define FLSTM_STAMP(step, slot)                                                     \
    do {                                                                            \
        if (tracing && (step) < p.trace_steps) p.trace[(step) * 16 + (slot)] = clock64(); \
    } while (0)

    if (warp >= 16) {
        if (warp == 16) {
            // -------------------------------------------------------- projection tiles, two steps ahead
            if (elect_one()) {
                uint32_t issued = 0, parity = 0;
                for (int tt = 0; tt < p.T; ++tt) {
                    const int pb = tt & 1;
                    if (!mbar_wait(&pempty[pb], ((tt >> 1) & 1) ^ 1, abort_w, wait_ns)) break;
                    mbar_expect_tx(&pfull[pb], BT * 128);
                    tma_load_3d(s_p + pb * BT * 128, &tm_g, jr * 64, b0, p.t0 + tt, &pfull[pb]);
                    issued |= 1u << pb;
                    parity = (parity & ~(1u << pb)) | (((tt >> 1) & 1u) << pb);
                }
                // way out: every copy this thread started must have landed before the CTA exits
                for (int i = 0; i < 2; ++i)
                    if (issued >> i & 1u) mbar_drain(&pfull[i], parity >> i & 1u, wait_ns);
            }
        } else if (warp == 18) {
            // -------------------------------------------------------- weights kept in shared memory
            if (CS > 0 && elect_one()) {
                if (leader) mbar_expect_tx(wbar, 2u * (uint32_t)(CS * kStepBytesW));
                for (int c = 0; c < CS; ++c) {
                    tma_load_2d_pair(s_w + c * kStepBytesW, &tm_w, (CT + c) * 64, jr * 64, wbar_c);
                    tma_load_2d_pair(s_w + c * kStepBytesW + 8192, &tm_w, (KC + CT + c) * 64, jr * 64, wbar_c);
                }
                if (leader) mbar_drain(wbar, 0, wait_ns);
            }
        } else if (warp == 19) {
            // -------------------------------------------------------- the launch's barrier, then fences behind resets
            if (p.T > 1 && elect_one() && wait_counter(counter, (unsigned)pl.cta_rows + p.extra_arrivals, p.err, abort_w, 2u, wait_ns)) {
                mbar_arrive(ready);
                perform_resets(reset, performed, p.T, abort_w, wait_ns, LOST && blockIdx.x == p.lost.cta && (p.lost.what & kLostCount) ? p.lost.step : -1);
            }
        } else {
            // -------------------------------------------------------- UMMA issuer (the leader's)
            if (leader && elect_one()) {
                bool ok = CS == 0 || mbar_wait(wbar, 0, abort_w, wait_ns);
                constexpr uint32_t idesc = umma_idesc_f16(256, N, BF16 ? 1 : 0, 0, 0);
                constexpr uint32_t kTileH = (BT * 32) >> 4, kStepW = kStepBytesW >> 4;  // descriptor units
                const uint32_t tfull_l = smem_u32(tfull), dw_res = umma_desc_lo(smem_u32(s_w)), dh_tile = umma_desc_lo(smem_u32(s_h));
                constexpr int stage_steps = stage_pieces(ROUNDS) * kRoundSteps;
                int committed = 0;
                for (int tt = 0; tt < p.T && ok; ++tt) {
                    ok = mbar_wait_cluster(tempty, (tt & 1) ^ 1, abort_w, wait_ns);
                    if (!ok) break;
                    tcgen05_fence_after();
                    uint32_t acc = 0, dh = dh_tile, da = tmem_a, dw = dw_res;  // the step's first instruction overwrites the accumulator
                    int c = 0;
                    for (int st = 0; st < (ROUNDS + stage_pieces(ROUNDS) - 1) / stage_pieces(ROUNDS); ++st) {
                        ok = mbar_wait(&hfull[st], tt & 1, abort_w, wait_ns);
                        if (!ok) break;
                        if (st == 0) FLSTM_STAMP(tt, 2);
                        FLSTM_STAMP(tt, 3);
                        tcgen05_fence_after();
                        const int c1 = c + stage_steps < KC ? c + stage_steps : KC, ct1 = c1 < CT ? c1 : CT;
#pragma unroll 4
                        for (; c < ct1; ++c) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_lo_ts<true, kUmmaDescHi32>(tmem_base, da + 8 * k, dh + kTileH * k, idesc, k ? 1u : acc);
                            acc = 1u;
                            da += 32;
                            dh += 4 * kTileH;
                        }
#pragma unroll 2
                        for (; c < c1; ++c) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_lo_ss<true, kUmmaDescHi32>(tmem_base, dw + 2 * k, dh + kTileH * k, idesc, k ? 1u : acc);
                            acc = 1u;
                            dw += kStepW;
                            dh += 4 * kTileH;
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
        }
    } else {
        // ------------------------------------------------------------ epilogue and gather (512 threads)
        const int tid = threadIdx.x;
        const size_t slab = (size_t)p.B * p.H, G = (size_t)4 * p.H;
        uint16_t *hs = static_cast<uint16_t *>(p.hs);
        uint16_t *y = static_cast<uint16_t *>(p.y);
        uint16_t *gates = static_cast<uint16_t *>(p.gates);

        // this thread's pieces of the h tile
        constexpr int PIECES = 2 * BT, TILES = kGatherThreads / PIECES;  // 16-byte pieces of 16 units, such tiles per round
        constexpr uint32_t ROUND = TILES * BT * 32;                       // bytes, in the ring and in the tile
        Gather<ROUNDS, ROUND, false, true> g;
        const char *from;
        g.full = map_to_rank(smem_u32(hfull), 0);
        g.turn = (uint32_t)(jr >> 3) & (stage_pieces(ROUNDS) - 1);
        {
            const int n = tid % PIECES >> 1, e = tid & 1, j0 = tid / PIECES;
            const int first = (int)rank * KC * 4, tiles = p.H / 16 - first < 4 * KC ? p.H / 16 - first : 4 * KC;
            g.to = smem_u32(s_h) + j0 * BT * 32 + n * 32 + ((e ^ (n >> 2 & 1)) << 4);
            g.mine = n < p.B - b0 && tiles > j0 ? (tiles - j0 + TILES - 1) / TILES : 0;
            for (int i = g.mine; i < gather_rounds(pl); ++i) gather_zero(g.to + (uint32_t)i * ROUND);  // K beyond H, sequences beyond B
            from = ring + (size_t)((ng * pl.cta_rows + first + j0) * BT * 32 + n * 32 + e * 16);
            // the state that the launch starts from
            g.first(reinterpret_cast<const char *>(hs) + (((size_t)p.t0 * p.B + b0 + n) * p.H + (first + j0) * 16 + e * 8) * 2, TILES * 32);
        }
        const bool y_words = (reinterpret_cast<uintptr_t>(y) & 3) == 0;  // the caller's y may start at any element
        const int quad = warp & 3, col0 = (warp >> 2) * (BT / 4);       // lane quadrant, quarter of the columns
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (quad >> 1) * BT + col0;
        const bool valid = b0 + nb < p.B;
        const size_t idx = (size_t)(b0 + nb) * p.H + jr * 16 + u;
        const bool pad = ACCURATE && jr * 16 + u >= p.real_units;
        if (p.T > 1) {
            fence_acq_rel_gpu();
            named_barrier_sync(2, kEpilogueThreads);
            if (tid == 0) red_release_gpu_add(counter, 1u);
        }
        const int lost_at = LOST && blockIdx.x == p.lost.cta && (p.lost.what & kLostPart) ? p.lost.step : -1;
        float c_keep = valid ? p.cs[(size_t)p.t0 * slab + idx] : 0.f;
        bool gathered = true;
        for (int tt = 0; tt < p.T; ++tt) {
            const int t = p.t0 + tt, pb = tt & 1;
            // No thread leaves between here and the named barrier below, whatever its waits return: the barrier ORs the
            // failures, so that all 512 threads go on or give up together.
            bool good = mbar_wait(&pfull[pb], (tt >> 1) & 1, abort_w, wait_ns) && gathered;
            float proj[4];
            {
                const uint16_t *ptile = reinterpret_cast<const uint16_t *>(s_p + pb * BT * 128) + nb * 64 + u;
#pragma unroll
                for (int gt = 0; gt < 4; ++gt) proj[gt] = load16<BF16>(ptile + gt * 16);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&pempty[pb]);
            if (tt >= kResetSlack && resets_slot(tt - kResetSlack, p.T))
                good = wait_performed(performed, (uint32_t)(tt - kResetSlack + 1), abort_w, wait_ns) && good;
            // the whole warp or none of it reads the accumulator
            const bool seen = __all_sync(0xffffffffu, mbar_wait(tfull, tt & 1, abort_w, wait_ns));
            good = good && seen;
            if (tid == 0) FLSTM_STAMP(tt, 5);
            tcgen05_fence_after();
            if (seen) {
                uint32_t acc[BT / 4];
                tmem_ld_32x32b_x8(taddr, acc);
                tmem_ld_wait();
                float4 *dst = reinterpret_cast<float4 *>(s_ex + (quad * 32 + lane) * kRowStride + col0);
#pragma unroll
                for (int i = 0; i < BT / 16; ++i)
                    dst[i] = make_float4(__uint_as_float(acc[4 * i]), __uint_as_float(acc[4 * i + 1]),
                                         __uint_as_float(acc[4 * i + 2]), __uint_as_float(acc[4 * i + 3]));
            }
            tcgen05_fence_before();
            __syncwarp();
            // relaxed: it orders the reuse of the accumulator only (a release would wait for the warp's global stores)
            if (lane == 0) mbar_arrive_cluster_relaxed(tempty_c);
            if (named_barrier_or(1, kEpilogueThreads, !good)) break;
            if (tid == 0) FLSTM_STAMP(tt, 6);
            float a[4];
#pragma unroll
            for (int gt = 0; gt < 4; ++gt) {
                const float *ex = s_ex + (gt * 16 + u) * kRowStride + nb;
                a[gt] = ex[0] + ex[64 * kRowStride] + proj[gt];
            }
            const float gi = sigmoid_sel<ACCURATE>(pad ? 0.f : a[0]), gf = sigmoid_sel<ACCURATE>(pad ? 0.f : a[1]);
            const float gg = tanh_sel<ACCURATE>(pad ? 0.f : a[2]), go = sigmoid_sel<ACCURATE>(pad ? 0.f : a[3]);
            c_keep = fmaf(gf, c_keep, gi * gg);
            const uint32_t h16 = to16<BF16>(go * tanh_sel<ACCURATE>(c_keep));
            const uint32_t word = __byte_perm(h16, __shfl_xor_sync(0xffffffffu, h16, 1), 0x5410);
            const bool word_valid = !odd && valid, more = tt + 1 < p.T;
            const size_t slot = (size_t)(tt & (kDirectSlots - 1)) * slot_bytes;
            if (more) {
                if (word_valid && !(LOST && tt == lost_at)) st_relaxed_gpu(ring + slot + my_word, word);
                g.mark_sent();
                if (tid == 0) FLSTM_STAMP(tt, 7);
                if (tt == 0) gathered = mbar_wait(ready, 0, abort_w, wait_ns);  // every CTA of the group has reset its words
            }
            // everything nobody waits for, while the others' parts are on their way: h_t and the caller's y, cell state, gate cache
            if (word_valid) {
                *reinterpret_cast<uint32_t *>(hs + (size_t)(t + 1) * slab + idx) = word;
                if (y && y_words) *reinterpret_cast<uint32_t *>(y + (size_t)t * slab + idx) = word;
            }
            // gates i and f of two units from the even lane, g and o from the odd one
            const uint32_t g01 = (uint32_t)to16<BF16>(gi) | (uint32_t)to16<BF16>(gf) << 16;
            const uint32_t g23 = (uint32_t)to16<BF16>(gg) | (uint32_t)to16<BF16>(go) << 16;
            const uint32_t mine = odd ? g23 : g01, other = __shfl_xor_sync(0xffffffffu, odd ? g01 : g23, 1);
            if (valid) {
                p.cs[(size_t)(t + 1) * slab + idx] = c_keep;
                if (y && !y_words) y[(size_t)t * slab + idx] = (uint16_t)h16;
                if (p.store_gates) {
                    uint16_t *grow = gates + ((size_t)t * p.B + b0 + nb) * G + (size_t)jr * 64 + odd * 32 + (u & ~1);
                    *reinterpret_cast<uint32_t *>(grow) = odd ? __byte_perm(other, mine, 0x5410) : __byte_perm(mine, other, 0x5410);
                    *reinterpret_cast<uint32_t *>(grow + 16) = odd ? __byte_perm(other, mine, 0x7632) : __byte_perm(mine, other, 0x7632);
                }
            }
            if (resets_slot(tt, p.T)) {
                if (!odd) st_relaxed_gpu(ring + (size_t)((tt + kResetAhead) & (kDirectSlots - 1)) * slot_bytes + my_word, kUnwritten);
                __syncwarp();
                if (lane == 0) mbar_arrive(&reset[tt % kResetBarriers]);
            }
            if (tid == 0) FLSTM_STAMP(tt, 8);
            if (more) {
                g.issue(from + slot);
                if (tid == 0) FLSTM_STAMP(tt, 0);
                gathered = g.finish(from + slot, p.err, abort_w, 2u, wait_ns) && gathered;
                if (tid == 0) FLSTM_STAMP(tt, 1);
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
    if (warp == 17) tmem_dealloc_pair(tmem_base, kTmemColumns);
    if (threadIdx.x == 0 && *abort_w) atomicCAS(p.err, 0u, 1u);
    if (threadIdx.x == 0) leave_counters(p.counters, (int)gridDim.x / pl.cta_rows, p.exits);
}

template <int ROUNDS, bool BF16, bool ACC, bool LOST = false>
int launch_one(const CUtensorMap &tw, const CUtensorMap &tg, const FwdTmPlan &pl, const FwdParams &p, cudaStream_t s) {
    auto kern = lstm_fwd_tm_kernel<ROUNDS, BF16, ACC, LOST>;
    FLSTM_CUDA_TRY(ensure_smem_limit(reinterpret_cast<const void *>(kern), pl.smem_bytes));
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
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, tg, pl, p);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "recurrent forward launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

}  // namespace

// With tiles of 64 sequences the tile of h is 64 KB at H = 1024 and the UMMAs take as long as the exchange; a step with a barrier
// then takes no longer: H = 832, B = 100 4.41 us against 4.53 this way, H = 1152, B = 100 4.82 / 5.07, H = 1280, 1536, 1792, B = 64
// 4.71 / 4.68, 5.13 / 5.16, 5.60 / 5.73.  Tiles of 32, B = 32 unless said otherwise: H = 832, B = 20 3.13 -> 2.47, H = 1024 3.29 -> 2.65
// (B = 64 3.47 -> 2.94), H = 1280 3.53 -> 2.99, H = 1536 3.80 -> 3.27, H = 2048 4.30 -> 3.79 (B = 8 3.94 -> 3.36), H = 2304, B = 8
// 4.27 -> 3.81.
bool fits_direct(const FwdTmPlan &pl, size_t smem_limit) {
    return pl.S == 2 && pl.BT == BT && pl.ct + pl.cs == pl.kc && gather_rounds(pl) <= kernel_rounds(pl) &&
           (size_t)layout_of(pl).total <= smem_limit;
}
size_t direct_ring_bytes(const FwdTmPlan &pl) { return pl.use && pl.direct ? (size_t)kDirectSlots * pl.grid * pl.BT * 32 : 0; }

int lstm_forward_tm_direct(int dtype, const FwdTmPlan &pl, const CUtensorMap &tw, const CUtensorMap &tg, const FwdParams &p, cudaStream_t s) {
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, acc = p.real_units > 0;
#define FLSTM_TM_CASE(R_)                                                                                        \
    if (kernel_rounds(pl) == R_) {                                                                              \
        if (p.lost.what && !bf16 && !acc) return launch_one<R_, false, false, true>(tw, tg, pl, p, s);          \
        if (bf16) return acc ? launch_one<R_, true, true>(tw, tg, pl, p, s) : launch_one<R_, true, false>(tw, tg, pl, p, s); \
        return acc ? launch_one<R_, false, true>(tw, tg, pl, p, s) : launch_one<R_, false, false>(tw, tg, pl, p, s); \
    }
    FLSTM_TM_CASE(4) FLSTM_TM_CASE(8) FLSTM_TM_CASE(10)
#undef FLSTM_TM_CASE
    return set_error(FLSTM_ERR_UNSUPPORTED, "no tensor-memory forward kernel for this plan");
}

}  // namespace tc
}  // namespace flstm_b200
