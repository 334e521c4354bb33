// Device helpers and plans shared by the cluster-resident recurrent kernels (tc_cluster_fwd.cu, tc_cluster_bwd.cu).
//
// The grid-wide persistent kernels (tc_lstm_fwd.cu, tc_lstm_bwd.cu) exchange h_t / dG_t through global memory: a step
// costs three serialised L2 round trips (release, barrier poll, TMA load), about 3 us whatever the width.  While W_hh
// fits the registers and shared memory of ONE thread-block cluster (H <= 768 with 16 CTAs), a cluster can run the
// recurrence of its own sequences alone: the exchange becomes st.async into the peers' shared memory, whose bytes the
// receiving mbarrier counts, and clusters never wait on one another.  Measured exchange inside a cluster: 570 cycles
// plus the incoming bytes at 9..14 per cycle.
//
// The products are mma.sync with the weights held as operand fragments in REGISTERS for the whole sequence, 8 sequences
// (one n8 tile) at a time.  tcgen05.mma would read its 64..128 KB of weights from shared memory once per step (128 B
// per cycle: 512..1024 cycles) and hand the sums over through tensor memory; with 1..8 sequences per cluster the
// register form needs 512 cycles at most (measured 8 cycles per m16n8k16 and sub-partition) and leaves the four gate
// sums of a (unit, sequence) pair in one thread.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "common.cuh"
#include "tc_common.cuh"
#include "tc_recurrent.cuh"

namespace flstm_b200 {
namespace tc {

// D (16x8, fp32) += A (16x16) B (16x8)
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
    if (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 bytes global -> shared, asynchronously (16-byte aligned on both sides)
__device__ __forceinline__ void cp_async_16(void *smem_dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Steps a kernel's inputs are fetched ahead of their use: a step takes 700..3000 cycles, a fetch from memory more than
// the shortest of them (fetched one step ahead, H = 64 ran at 2300 cycles a step).
constexpr int kClusterAhead = 4;

// shared-memory row of `bytes` (a multiple of 64), padded so that the 16-byte fragment reads of 8 rows do not conflict
__host__ __device__ constexpr int cluster_row_bytes(int bytes) { return bytes % 128 ? bytes : bytes + 64; }

// clock64() stamps of the first CTA's first thread at fixed points of each traced step (see FwdParams::trace)
#define FLSTM_CL_STAMP(step, slot)                                                       \
    do {                                                                                 \
        if (tracing && (step) < p.trace_steps) p.trace[(step) * 16 + (slot)] = clock64(); \
    } while (0)

struct ClusterFwdPlan {
    bool use;
    int C;         // CTAs per cluster
    int peers;     // CTAs of a cluster that own units (the rest of a power of two idles)
    int nub;       // blocks of 8 hidden units (32 gate rows) per CTA
    int ks;        // warps that split the K = H contraction of one block
    int kr, nsm;   // 32-wide K chunks per warp in registers / in shared memory
    int NT;        // tiles of 8 sequences per cluster
    int seqs;      // sequences per cluster
    int clusters;  // clusters launched
    int threads, smem_bytes;
    int cycles;    // estimated cycles per step
};
struct ClusterFwdParams {
    const void *w_hh;  // 16-bit (4H, H), rows tile-interleaved
    float *cs;         // fp32 (T+1, B, H)
    void *hs;          // 16-bit (T+1, B, H)
    void *y;           // optional copy of h_t
    void *gates;       // 16-bit (T, B, 4H): projection in, activated gates out
    unsigned int *err;
    int T, t0, B, H;
    int store_gates;
    int real_units;  // see FwdParams
    long long *trace;
    int trace_steps;
    unsigned long long wait_ns;
    unsigned int extra_arrivals;
    // from the plan
    int C, peers, nub, ks, nsm, seqs;
    int y_aligned;  // y starts on a 16-byte boundary
};

struct ClusterBwdPlan {
    bool use;
    int C, peers, nub;
    int W;          // warps
    int MT, NKB;    // 16-unit tiles and 32-wide K chunks per warp
    int KSB;        // warp groups that split the CTA's K range
    int NT, seqs, clusters, threads, smem_bytes, cycles;
};
struct ClusterBwdParams {
    const void *w_hh;
    const float *cs;
    const void *gates;
    void *dg;
    const void *dy, *dhn, *dcn;
    float *dh0, *dc0, *dc;
    unsigned int *err;
    int T, s0, s1, B, H;
    int real_units;  // see FwdParams
    long long *trace;
    int trace_steps;
    unsigned long long wait_ns;
    unsigned int extra_arrivals;
    int C, peers, seqs;
    int dy_aligned;  // dY starts on a 16-byte boundary
};

// Plans for a shape, or use = false.  With `check` the occupancy calculator is asked how many clusters of the kernel run
// at once; otherwise the numbers measured on a B200 (148 SMs) are used.  Clusters never wait on one another, so a wrong
// number costs a second wave and nothing else.
struct ClusterCheck {
    bool bf16, accurate;  // which kernel will be launched
};
int plan_cluster_fwd(int B, int H, int sms, size_t smem_limit, ClusterFwdPlan *plan, const ClusterCheck *check);
int plan_cluster_bwd(int B, int H, int sms, size_t smem_limit, ClusterBwdPlan *plan, const ClusterCheck *check);
int lstm_forward_cluster(int dtype, const ClusterFwdPlan &plan, ClusterFwdParams p, cudaStream_t s);
int lstm_backward_cluster(int dtype, const ClusterBwdPlan &plan, ClusterBwdParams p, cudaStream_t s);
bool cluster_enabled();  // FLSTM_CLUSTER=0 keeps the grid-wide kernels
int cluster_count(const void *kernel, int C, int threads, int smem_bytes);  // clusters of a kernel that run at once
int cluster_launch(const void *kernel, int C, int grid, int threads, int smem_bytes, void *params, cudaStream_t s, const char *what);

// clusters of C one-CTA-per-SM CTAs that a B200 holds at once
inline int cluster_slots(int C, int sms) {
    switch (C) {
        case 1: return sms;
        case 2: return sms / 2;
        case 4: return sms * 33 / 148;
        case 8: return sms * 15 / 148;
        default: return sms * 7 / 148;
    }
}

}  // namespace tc
}  // namespace flstm_b200
