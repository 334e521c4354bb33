// Exchange of h_t / dG_t between the CTAs of a recurrent kernel without a step barrier: the words announce themselves.
//
// With a counter per step a CTA stores its part, waits until the stores are performed (a release: 1.2-1.4 k cycles), adds to
// the counter, polls it (1.5 k) and only then starts to copy (1.3 k for 32 KB): three round trips to L2, half of a step of
// 5.6 k cycles at H = 1024.  Here a CTA stores its part into a slot of a ring whose every 32-bit word is kUnwritten until then,
// and the CTAs that need it copy the slot at once (cp.async, 16 bytes each: 32 KB in 840 cycles, 64 KB in 1110, against 907
// and 1190 for bulk copies and 1430 and 1980 for loads through registers), look at what came, and copy again what was not
// there yet.  From the first store to the last checked word a step's exchange takes 1.7 k cycles for 32 KB and 2.2 k for 64 KB.
//
// kUnwritten is no pair of 16-bit results: a conversion from fp32 gives NaN as 0x7fff.  Words are stored whole, so a word is
// either unwritten or complete whatever becomes of the copies' order.
//
// What this takes for granted of the GPU, where PTX promises nothing (cp.async is a weak access, no acquire follows it):
//   - an aligned 32-bit word of one store arrives whole in a copy (every word of a piece is looked at in the forward kernel);
//   - a copy past L1 that starts after a reset has been fenced and its count has been seen, through whatever chain of words and
//     barriers, does not bring the word from before the reset;
//   - 16 aligned bytes of one 128-bit store arrive together: the BPTT looks at one word of four, as looking at all took 3 to 10 % of a step
//     (H = 1088, B = 32 3.72 -> 3.82 us, H = 1024, B = 64 3.35 -> 3.66).  This one is watched: halves of an unwritten word are NaN in either
//     type and make the sums they enter NaN, and where a sum is, the BPTT looks at all words of its operand (kErrTornPiece).
//
// Slots.  Results of step t go to slot t % 8.  After its stores of step t a thread resets its words of slot (t + 4) % 8: nobody reads
// that slot any more (it held step t - 4; the results of step t - 1, which this CTA has seen from all others, were sent by CTAs
// that had gathered step t - 2).  The reset has to be performed before anybody looks for step t + 4, that is before this CTA sends
// step t + 3: a warp of its own fences behind the resets of all threads and counts them (`performed`), and a CTA sends step t + 2
// only when the reset of step t has been counted.  The warps report the resets of step t to mbarrier t % kResetBarriers: they report
// those of step t + kResetSlack when the counting warp has seen step t, so that an mbarrier never completes another phase before the
// one that is waited for has been seen (waits go by parity and would miss it), however late the counting warp is.  Fences in the
// threads themselves, behind their other stores, held them for three thousand cycles a step.  A launch resets all slots before its first step; one counter barrier, which the fill of tensor memory
// hides, comes before the first look.  The copies read L2, where the words are: an old one cannot come from L1.
#pragma once

#include <cstdint>

#include "tc_common.cuh"
#include "tc_recurrent.cuh"

namespace flstm_b200 {
namespace tc {

constexpr int kDirectSlots = 8, kResetAhead = 4, kResetSlack = 2, kResetBarriers = 2;
static_assert(kResetBarriers >= kResetSlack, "a phase of its own for every step that may report its resets ahead of the count");
constexpr uint32_t kUnwritten = 0xffffffffu;
constexpr int kGatherWarps = 16, kGatherThreads = kGatherWarps * 32;  // with 8 warps the exchange takes 100 to 400 cycles more
constexpr int kGatherStages = 3;  // parts of a gather that are handed over one by one, at most
// Pieces of a stage: a stage costs some 400 cycles and lets the UMMAs start as much earlier as it is smaller.
__host__ __device__ constexpr int stage_pieces(int rounds) { return rounds <= 4 ? 2 : 4; }
constexpr int kGatherBarrier = 3;  // named barrier
constexpr uint32_t kGatherDelay = 700, kGatherDelayMax = 2000, kGatherLater = 96, kGatherSooner = 8;  // cycles

__device__ __forceinline__ void st_relaxed_gpu(void *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_gpu_16(void *p, uint4 v) {  // one access of 128 bits
    asm volatile("{\n.reg .b64 lo, hi;\n.reg .b128 v;\nmov.b64 lo, {%1, %2};\nmov.b64 hi, {%3, %4};\nmov.b128 v, {lo, hi};\n"
                 "st.relaxed.gpu.global.b128 [%0], v;\n}\n" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_cta_shared(uint32_t smem_addr) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta_shared(uint32_t smem_addr, uint32_t v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_addr), "r"(v) : "memory");
}
// bounded wait until `count` resets have been counted
__device__ __forceinline__ bool wait_performed(uint32_t performed, uint32_t count, volatile uint32_t *abort_w, unsigned long long limit_ns) {
    if (ld_acquire_cta_shared(performed) >= count) return true;
    const unsigned long long t0 = global_timer_ns();
    for (uint32_t spins = 1; ld_acquire_cta_shared(performed) < count; ++spins) {
        if ((spins & 63u) == 0) {
            if (*abort_w) return false;
            if (global_timer_ns() - t0 > limit_ns) {
                *abort_w = 1;
                return false;
            }
        }
    }
    return true;
}
// The steps of a launch of T steps whose results are sent on: all but the last.  Step t resets the slot of step t + kResetAhead if
// that one is sent.
__device__ __forceinline__ bool resets_slot(int t, int T) { return t + kResetAhead + 1 < T; }
// the warp that performs the resets: reset[t % kResetBarriers] gets an arrival of every storing warp in step t
__device__ __forceinline__ void perform_resets(uint64_t *reset, uint32_t performed, int T, volatile uint32_t *abort_w, unsigned long long limit_ns,
                                               int lost_from) {
    for (int t = 0; resets_slot(t, T) && t != lost_from; ++t) {
        if (!mbar_wait(&reset[t % kResetBarriers], (uint32_t)(t / kResetBarriers) & 1u, abort_w, limit_ns)) return;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        st_release_cta_shared(performed, (uint32_t)t + 1u);
    }
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// 16 bytes global -> shared, past L1, asynchronously
__device__ __forceinline__ void gather_copy(uint32_t smem_addr, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(src) : "memory");
}
__device__ __forceinline__ void gather_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the LEFT newest groups have landed
template <int LEFT>
__device__ __forceinline__ void gather_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
// A piece that is written whole is looked at by one word (see above): lanes 0-7 look at the first word of theirs, 8-15 at the second, ..., so
// that a warp reads every bank once (all four words take four times as long).
__device__ __forceinline__ bool gather_unwritten_whole(uint32_t smem_addr) {
    uint32_t a;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(a) : "r"(smem_addr + (threadIdx.x >> 3 & 3) * 4) : "memory");
    return a == kUnwritten;
}
__device__ __forceinline__ bool gather_unwritten(uint32_t smem_addr) {
    uint32_t a, b, c, d;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(smem_addr) : "memory");
    return max(max(a, b), max(c, d)) == kUnwritten;
}
__device__ __forceinline__ void gather_zero(uint32_t smem_addr) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(smem_addr), "r"(0u) : "memory");
}
// Hand-over to a UMMA thread of the cluster, relaxed: what it covers has been performed (read back) and fenced towards the tensor
// core by the threads that wrote it, and they have met at a barrier.  A release, of whatever scope, would wait for the thread's
// stores to global memory and every copy under way: 450 to 1300 cycles.
__device__ __forceinline__ void gather_arrive(uint32_t bar_cluster_addr) { mbar_arrive_cluster_relaxed(bar_cluster_addr); }

// A gather by kGatherThreads threads of up to ROUNDS pieces of 16 bytes each, piece i from src + i STEP to `to` + i STEP, handed over
// in stages of kStagePieces.  What a step waits for is a chain of instructions of single warps, so all of it is unrolled and its
// addresses are constants apart: with run-time loops a stage cost 400 to 800 cycles, be it copied by cp.async or in bulk.  The
// threads meet at a named barrier and one of them hands the stage over: an arrival of every warp on the mbarrier of another CTA
// takes 14 cycles, 450 a stage.
template <int ROUNDS, uint32_t STEP, bool WHOLE, bool TURNS>
struct Gather {
    static constexpr int kStagePieces = stage_pieces(ROUNDS), kStages = (ROUNDS + kStagePieces - 1) / kStagePieces;
    static_assert(kStages <= kGatherStages, "barriers of the stages");
    uint32_t to;
    int mine;       // pieces of this thread
    uint32_t full;  // the UMMA thread's barriers of the stages, a shared::cluster address
    // A copy that comes too early is a round trip lost (800 cycles), one that comes late as many cycles as it is late: each warp
    // starts its copies `delay` cycles after it has sent its own part, more after a step in which it came too early, less otherwise.
    uint32_t sent, delay = kGatherDelay;
    // TURNS: the pieces of a stage are asked for in an order of a group of CTAs' own (turn < stage_pieces), so that not all of them bring
    // the same line across the dies at once.  Forward 1 to 3 % of a step; the BPTT at H = 2048 lost a tenth by it.
    uint32_t turn = 0;

    __device__ __forceinline__ bool unwritten(uint32_t smem_addr) const {
        return WHOLE ? gather_unwritten_whole(smem_addr) : gather_unwritten(smem_addr);
    }
    __device__ __forceinline__ void hand_over(int stage) const {
        fence_proxy_async_smem();
        named_barrier_sync(kGatherBarrier, kGatherThreads);
        if (threadIdx.x == 0) gather_arrive(full + 8u * (uint32_t)stage);
    }
    // the state that a launch starts from, which lies in rows of its own; piece `apart` comes from `apart_by` bytes further on
    __device__ __forceinline__ void first(const char *src, uint32_t src_step, int apart = -1, uint32_t apart_by = 0) {
        for (int i = 0; i < mine; ++i)
            gather_copy(to + (uint32_t)i * STEP, src + (size_t)((uint32_t)i * src_step + (i == apart ? apart_by : 0u)));
        gather_commit();
        gather_wait<0>();
        for (int st = 0; st < kStages; ++st) hand_over(st);
    }
    __device__ __forceinline__ void mark_sent() { sent = (uint32_t)clock(); }
    // starts the copies of a step
    __device__ __forceinline__ void issue(const char *src) const {
        while ((uint32_t)clock() - sent < delay) {}
#pragma unroll
        for (int st = 0; st < kStages; ++st) {
#pragma unroll
            for (int k = 0; k < kStagePieces; ++k) {
                const uint32_t i = st * kStagePieces + (TURNS ? k ^ turn : k);
                if ((int)i < mine) gather_copy(to + i * STEP, src + i * STEP);
            }
            gather_commit();
        }
    }
    // Waits for them and hands them over.  All threads run through all stages whatever becomes of them.  False: a wait expired or
    // another role gave up (the abort word is raised; the copies have landed).
    __device__ __forceinline__ bool finish(const char *src, unsigned int *err_word, volatile uint32_t *abort_w, unsigned int code,
                                           unsigned long long limit_ns) {
        bool complete = false, ok = true;
        stage<0>(src, err_word, abort_w, code, limit_ns, complete, ok);
        if (complete) delay = delay + kGatherLater < kGatherDelayMax ? delay + kGatherLater : kGatherDelayMax;
        else if (delay >= kGatherSooner) delay -= kGatherSooner;
        return ok;
    }

private:
    template <int ST>
    __device__ __forceinline__ void stage(const char *src, unsigned int *err_word, volatile uint32_t *abort_w, unsigned int code,
                                          unsigned long long limit_ns, bool &complete, bool &ok) const {
        if constexpr (ST < kStages) {
            if (!complete) {
                gather_wait<kStages - 1 - ST>();
                bool missing = false;
#pragma unroll
                for (int i = ST * kStagePieces; i < (ST + 1) * kStagePieces && i < ROUNDS; ++i)
                    missing |= i < mine && unwritten(to + i * STEP);
                if (__any_sync(0xffffffffu, missing)) {
                    ok = again(src, err_word, abort_w, code, limit_ns);
                    complete = true;
                }
            }
            hand_over(ST);
            stage<ST + 1>(src, err_word, abort_w, code, limit_ns, complete, ok);
        }
    }

    // what is missing of any stage is copied again together: a round trip for each stage's missing pieces cost 2 k cycles a step
    __device__ __forceinline__ bool again(const char *src, unsigned int *err_word, volatile uint32_t *abort_w, unsigned int code,
                                          unsigned long long limit_ns) const {
        gather_wait<0>();
        uint32_t todo = 0;
#pragma unroll
        for (int i = 0; i < ROUNDS; ++i)
            if (i < mine && unwritten(to + i * STEP)) todo |= 1u << i;
        unsigned long long since = 0;
        for (uint32_t spins = 1; __any_sync(0xffffffffu, todo); ++spins) {
#pragma unroll
            for (int i = 0; i < ROUNDS; ++i)
                if (todo >> i & 1u) gather_copy(to + i * STEP, src + i * STEP);
            gather_commit();
            gather_wait<0>();
#pragma unroll
            for (int i = 0; i < ROUNDS; ++i)
                if ((todo >> i & 1u) && !unwritten(to + i * STEP)) todo &= ~(1u << i);
            if ((spins & 31u) == 0) {
                if (since == 0) since = global_timer_ns();
                bool give_up = *abort_w != 0;
                if (!give_up && *reinterpret_cast<volatile unsigned int *>(err_word)) {
                    *abort_w = 1;
                    give_up = true;
                }
                if (!give_up && global_timer_ns() - since > limit_ns) {
                    *abort_w = 1;
                    atomicExch(err_word, code);
                    give_up = true;
                }
                if (__any_sync(0xffffffffu, give_up)) return false;
            }
        }
        return true;
    }
};

}  // namespace tc
}  // namespace flstm_b200
