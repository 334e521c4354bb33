// Cluster-resident fp32 recurrent kernels: like tc_cluster_fwd.cu / tc_cluster_bwd.cu (one launch runs all steps, every
// thread-block cluster for its own sequences, h_t and partial dh exchanged by st.async), but with true fp32 FMA on the
// CUDA cores, for the configurations that must stay in fp32.
//
// The grid-wide kernels (simt_persistent.cu) read weights and state from shared memory for every FMA and exchange through
// global memory: 5.8 / 8.3 us per forward / BPTT step at H = 256, B = 32.  Here the weights sit in registers (16 per unit
// and 64-wide K chunk and thread; shared memory for what does not fit), a 16-byte read of h or dG from shared memory
// feeds 16 FMAs, and a step is bound by the exchange (about 700 cycles) and 16 FMA cycles per chunk, sequence and warp of
// a sub-partition.
//
// Forward: a half warp owns a hidden unit, its 16 lanes split K; a reduce-scatter by shuffles leaves gate (lane / 4) of
// sequence (lane % 4) in each lane, four sequences at a time.  BPTT: a CTA contracts its own units' dG with its rows of
// W_hh; a lane owns four output units and a quarter of the own units, and after the reduce-scatter it holds the partial
// dh of its four units for one sequence: one 16-byte message to their owner, who adds the sources in a fixed order.
// Buffering, arming of the mbarriers, bounded waits and the way out after a timeout are those of the 16-bit kernels.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "tc_cluster.cuh"

namespace flstm_b200 {
namespace simt {

using namespace tc;

namespace {

__device__ __forceinline__ void cp_async_4(void *smem_dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
// inputs fetched `ahead` steps early: 4, or 2 where the ring would take too much shared memory
__device__ __forceinline__ void ring_wait(int ahead, int younger) {
    // the oldest `ahead - younger` of `ahead` groups must have landed
    if (ahead == 4) {
        if (younger == 3) cp_async_wait<3>();
        else cp_async_wait<2>();
    } else {
        if (younger == 1) cp_async_wait<1>();
        else cp_async_wait<0>();
    }
}

// floats per row of the forward kernel's staging: the units of a CTA plus two, which spreads 16 rows over the banks
__host__ __device__ constexpr int f32_out_row(int threads) { return threads / 16 + 2; }
constexpr int f32_fwd_max_threads(int KR) { return KR <= 4 ? 512 : KR <= 6 ? 384 : 256; }
constexpr int f32_bwd_max_threads(int UR) { return UR <= 4 ? 512 : UR <= 6 ? 384 : 256; }

__device__ __forceinline__ float4 fma4(float s, float4 w, float4 a) {
    a.x = fmaf(s, w.x, a.x);
    a.y = fmaf(s, w.y, a.y);
    a.z = fmaf(s, w.z, a.z);
    a.w = fmaf(s, w.w, a.w);
    return a;
}

// KR: 64-wide K chunks of the weights in registers; p.nsm more in shared memory
template <int KR>
__global__ void __launch_bounds__(f32_fwd_max_threads(KR), 1) f32_cluster_fwd_kernel(const ClusterF32FwdParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ volatile uint32_t abort_w;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slice = lane & 15, gl = (lane >> 2) & 3, sq = lane & 3;
    const int threads = blockDim.x, warps = threads >> 5, H = p.H, Kp = (KR + p.nsm) * 64;
    const uint32_t rank = cluster_ctarank();
    const int b0 = (int)(blockIdx.x / (unsigned)p.C) * p.seqs;
    const int nvalid = p.B - b0 < p.seqs ? p.B - b0 : p.seqs, blocks = (nvalid + 3) / 4, max_blocks = (p.seqs + 3) / 4;
    const int u0 = (int)rank * p.nub, own = H - u0 < p.nub ? H - u0 : p.nub;  // units of this CTA
    const int ul = warp * 2 + (lane >> 4), u = u0 + ul;
    const bool active = own > 0, real = ul < own;
    const int h_bytes = p.seqs * Kp * 4;
    uint8_t *s_h = smem;                                                    // 2 x [sequence][Kp]
    float4 *s_w = reinterpret_cast<float4 *>(s_h + 2 * h_bytes);            // [warp][nsm][4 gates][32 lanes]
    float *s_send = reinterpret_cast<float *>(s_w + (size_t)warps * p.nsm * 128);  // 2 x [sequence][nub]
    float *s_p = s_send + 2 * p.seqs * p.nub;                               // [ahead][block][16 rows][unit] projections
    const int nw = threads / 16, row = f32_out_row(threads);                // units per CTA with the partly used warp, floats per row
    float *s_out = s_p + p.ahead * max_blocks * 16 * row;                   // 2 x [block][16 gate rows, 4 cell rows][unit]
    float *s_c = s_out + 2 * max_blocks * 20 * row;                         // [block][thread] cell states

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&full[i], 1);
        abort_w = 0;
        fence_barrier_init();
    }
    for (int o = tid * 16; o < 2 * h_bytes; o += threads * 16) *reinterpret_cast<uint4 *>(s_h + o) = make_uint4(0, 0, 0, 0);
    for (int o = tid; o < 2 * p.seqs * p.nub; o += threads) s_send[o] = 0.f;
    __syncthreads();
    const size_t slab = (size_t)p.B * H;
    for (int e = tid; e < nvalid * H; e += threads)
        reinterpret_cast<float *>(s_h)[(e / H) * Kp + e % H] = p.hs[(size_t)p.t0 * slab + (size_t)(b0 + e / H) * H + e % H];
    auto load_w = [&](int c, int g) {
        const int k = c * 64 + slice * 4;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = real && k + e < H ? p.w_hh[(size_t)(g * H + u) * H + k + e] : 0.f;
        return make_float4(v[0], v[1], v[2], v[3]);
    };
    float4 wr[KR][4];
#pragma unroll
    for (int c = 0; c < KR; ++c)
#pragma unroll
        for (int g = 0; g < 4; ++g) wr[c][g] = load_w(c, g);
    float4 *my_w = s_w + (size_t)warp * p.nsm * 128 + lane;
    for (int c = 0; c < p.nsm; ++c)
#pragma unroll
        for (int g = 0; g < 4; ++g) my_w[(c * 4 + g) * 32] = load_w(KR + c, g);
    const uint32_t step_bytes = (uint32_t)((H + 3) / 4 * 16 * nvalid) + 16u * p.extra_arrivals;
    if (tid == 0 && active) {
        if (p.T > 1) mbar_expect_tx(&full[1], step_bytes);
        if (p.T > 2) mbar_expect_tx(&full[0], step_bytes);
    }
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers and zeroed buffers exist before anything is sent

    if (active) {
        const size_t G = (size_t)4 * H, gate_step = (size_t)p.B * G;
        auto mine = [&](int blk) { return real && blk * 4 + sq < nvalid; };
        // What goes to or comes from global memory moves in rows: thread = unit tid % nw of row (sequence * 4 + gate) tid / nw of a block, so a
        // warp touches one or two runs of neighbouring floats.  (Each lane fetching and storing its own (unit, sequence, gate) took
        // 16 sectors per instruction ahead of the next wait; H = 256, B = 32, T = 128: 936 -> 918 us a training step.)
        // The state a row stores: h, c or y by gate 0, 1, 2.
        const int fu = tid % nw, frow = tid / nw, fg = frow & 3, fsq = frow >> 2;
        const size_t first = (size_t)p.t0 * p.B + b0 + fsq;
        float *g_ptr = p.gates + first * G + (size_t)fg * H + u0 + fu;
        const float *p_src = g_ptr;
        float *s_ptr = fg == 0 ? p.hs + slab : fg == 1 ? p.cs + slab : fg == 2 ? p.y : nullptr;
        if (s_ptr) s_ptr += first * H + u0 + fu;
        auto moved = [&](int blk) { return fu < own && blk * 4 + fsq < nvalid; };
        int slot_in = 0, slot = 0;  // of the next fetch, of this step
        auto fetch = [&](int tt) {
            if (tt < p.T)
                for (int blk = 0; blk < blocks; ++blk)
                    if (moved(blk)) cp_async_4(s_p + ((slot_in * max_blocks + blk) * 16 + frow) * row + fu, p_src + (size_t)blk * 4 * G);
            cp_async_commit();
            p_src += gate_step;
            slot_in = slot_in + 1 == p.ahead ? 0 : slot_in + 1;
        };
        for (int blk = 0; blk < blocks; ++blk)
            s_c[blk * threads + tid] = mine(blk) ? p.cs[(size_t)p.t0 * slab + (size_t)(b0 + blk * 4 + sq) * H + u] : 0.f;
        for (int tt = 0; tt < p.ahead; ++tt) fetch(tt);
        ring_wait(p.ahead, p.ahead - 1);
        named_barrier_sync(1, threads);
        const int quads = (own + 3) / 4, pieces = nvalid * quads;
        const uint32_t h_local = smem_u32(s_h), bar_off = smem_u32(full) - h_local;
        const int e_seq = lane / quads, e_quad = lane % quads;  // this lane's first piece
        const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
        for (int tt = 0; tt < p.T; ++tt) {
            bool ok = true;
            if (tt > 0) {
                ok = mbar_wait_cluster(&full[tt & 1], (uint32_t)(tt - 1) >> 1 & 1u, &abort_w, wait_ns);
                if (ok && tid == 0 && tt + 2 < p.T) mbar_expect_tx(&full[tt & 1], step_bytes);
            }
            ok = __all_sync(0xffffffffu, ok);
            float *send = s_send + (tt & 1) * p.seqs * p.nub, *out = s_out + (tt & 1) * max_blocks * 20 * row;
            const float *hb = reinterpret_cast<const float *>(s_h + (tt & 1) * h_bytes) + slice * 4;
            for (int blk = 0; blk < blocks; ++blk) {
                const int ns = nvalid - blk * 4;
                float acc[4][4];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
#pragma unroll
                    for (int g = 0; g < 4; ++g) acc[s][g] = 0.f;
                    if (s < ns) {
                        const float *row = hb + (blk * 4 + s) * Kp;
#pragma unroll
                        for (int c = 0; c < KR; ++c) {
                            const float4 h = *reinterpret_cast<const float4 *>(row + c * 64);
#pragma unroll
                            for (int g = 0; g < 4; ++g) acc[s][g] = fmaf(h.x, wr[c][g].x, acc[s][g]);
#pragma unroll
                            for (int g = 0; g < 4; ++g) acc[s][g] = fmaf(h.y, wr[c][g].y, acc[s][g]);
#pragma unroll
                            for (int g = 0; g < 4; ++g) acc[s][g] = fmaf(h.z, wr[c][g].z, acc[s][g]);
#pragma unroll
                            for (int g = 0; g < 4; ++g) acc[s][g] = fmaf(h.w, wr[c][g].w, acc[s][g]);
                        }
                    }
                }
#pragma unroll 1
                for (int c = 0; c < p.nsm; ++c) {
                    const float4 w0 = my_w[(c * 4 + 0) * 32], w1 = my_w[(c * 4 + 1) * 32], w2 = my_w[(c * 4 + 2) * 32],
                                 w3 = my_w[(c * 4 + 3) * 32];
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        if (s < ns) {
                            const float4 h = *reinterpret_cast<const float4 *>(hb + (blk * 4 + s) * Kp + (KR + c) * 64);
                            acc[s][0] = fmaf(h.w, w0.w, fmaf(h.z, w0.z, fmaf(h.y, w0.y, fmaf(h.x, w0.x, acc[s][0]))));
                            acc[s][1] = fmaf(h.w, w1.w, fmaf(h.z, w1.z, fmaf(h.y, w1.y, fmaf(h.x, w1.x, acc[s][1]))));
                            acc[s][2] = fmaf(h.w, w2.w, fmaf(h.z, w2.z, fmaf(h.y, w2.y, fmaf(h.x, w2.x, acc[s][2]))));
                            acc[s][3] = fmaf(h.w, w3.w, fmaf(h.z, w3.z, fmaf(h.y, w3.y, fmaf(h.x, w3.x, acc[s][3]))));
                        }
                }
                // reduce-scatter over the 16 lanes of the unit: bits 3, 2 choose the gate, bits 1, 0 the sequence
                const bool b3 = lane & 8, b2 = lane & 4, b1 = lane & 2, b0s = lane & 1;
                float v[4];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float x0 = __shfl_xor_sync(0xffffffffu, b3 ? acc[s][0] : acc[s][2], 8);
                    const float x1 = __shfl_xor_sync(0xffffffffu, b3 ? acc[s][1] : acc[s][3], 8);
                    const float lo = (b3 ? acc[s][2] : acc[s][0]) + x0, hi = (b3 ? acc[s][3] : acc[s][1]) + x1;
                    v[s] = (b2 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b2 ? lo : hi, 4);
                }
                const float y0 = (b1 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, b1 ? v[0] : v[2], 2);
                const float y1 = (b1 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, b1 ? v[1] : v[3], 2);
                const float sum = (b0s ? y1 : y0) + __shfl_xor_sync(0xffffffffu, b0s ? y0 : y1, 1);
                const bool ours = mine(blk);
                const float a = ours ? sum + s_p[((slot * max_blocks + blk) * 16 + sq * 4 + gl) * row + ul] : 0.f;
                const float act = gl == 2 ? tanh_acc(a) : sigmoid_acc(a);
                const int base = lane & 19;  // unit and sequence of this lane, gate 0
                const float gi = __shfl_sync(0xffffffffu, act, base), gf = __shfl_sync(0xffffffffu, act, base + 4);
                const float gg = __shfl_sync(0xffffffffu, act, base + 8), go = __shfl_sync(0xffffffffu, act, base + 12);
                const float c = fmaf(gf, s_c[blk * threads + tid], gi * gg);
                const float h = go * tanh_acc(c);
                s_c[blk * threads + tid] = c;
                out[(blk * 20 + sq * 4 + gl) * row + ul] = act;
                if (gl == 1) out[(blk * 20 + 16 + sq) * row + ul] = c;
                if (ours && gl == 0) send[(blk * 4 + sq) * p.nub + ul] = h;
            }
            ring_wait(p.ahead, p.ahead - 2);  // the projections of the next step; the barrier shows them to the other threads
            if (named_barrier_or(1, threads, !ok)) break;
            if (tt + 1 < p.T) {
                const uint32_t to = (uint32_t)(((tt + 1) & 1) * h_bytes) + (uint32_t)u0 * 4u, bar = bar_off + ((tt + 1) & 1) * 8u;
                for (int r = warp; r < p.peers; r += warps) {
                    const uint32_t peer = map_to_rank(h_local, (uint32_t)r);
                    if (lane < pieces) {
                        const uint4 m = *reinterpret_cast<const uint4 *>(send + e_seq * p.nub + e_quad * 4);
                        st_async_v4(peer + to + (uint32_t)(e_seq * Kp * 4 + e_quad * 16), m.x, m.y, m.z, m.w, peer + bar);
                    }
                    for (int e = lane + 32; e < pieces; e += 32) {
                        const int n = e / quads, qd = e % quads;
                        const uint4 m = *reinterpret_cast<const uint4 *>(send + n * p.nub + qd * 4);
                        st_async_v4(peer + to + (uint32_t)(n * Kp * 4 + qd * 16), m.x, m.y, m.z, m.w, peer + bar);
                    }
                }
            }
            // everything nobody waits for
            for (int blk = 0; blk < blocks; ++blk)
                if (moved(blk)) {
                    if (p.store_gates) g_ptr[(size_t)blk * 4 * G] = out[(blk * 20 + frow) * row + fu];
                    if (s_ptr)
                        s_ptr[(size_t)blk * 4 * H] = fg == 1 ? out[(blk * 20 + 16 + fsq) * row + fu] : send[(blk * 4 + fsq) * p.nub + fu];
                }
            slot = slot + 1 == p.ahead ? 0 : slot + 1;
            g_ptr += gate_step;
            if (s_ptr) s_ptr += slab;
            fetch(tt + p.ahead);
        }
    }
    __syncthreads();
    cluster_sync_all();  // nobody leaves while a peer may still send into its shared memory
    if (abort_w) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < kAbortDrainNs) {}
    }
    if (tid == 0 && abort_w) atomicCAS(p.err, 0u, 1u);
}

// UR: own units per lane quarter whose weights sit in registers (16 each); p.nsm more in shared memory
template <int UR>
__global__ void __launch_bounds__(f32_bwd_max_threads(UR), 1) f32_cluster_bwd_kernel(const ClusterF32BwdParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t rbar[2];
    __shared__ volatile uint32_t abort_w;
    constexpr int EARLY = 2;  // (unit, sequence, gate) lanes per thread whose factors are formed before the wait
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, o = lane & 7, q = lane >> 3;
    const int threads = blockDim.x, H = p.H, nub = p.nub;
    const uint32_t rank = cluster_ctarank();
    const int b0 = (int)(blockIdx.x / (unsigned)p.C) * p.seqs;
    const int nvalid = p.B - b0 < p.seqs ? p.B - b0 : p.seqs, blocks = (nvalid + 3) / 4;
    const int u0 = (int)rank * nub, own = H - u0 < nub ? H - u0 : nub;
    const bool active = own > 0;
    const int stages = p.ahead + 1, items = nvalid * nub * 4;  // item = (sequence, unit, gate)
    const int part_floats = p.peers * p.seqs * nub;
    float *s_part = reinterpret_cast<float *>(smem);                     // 2 x [source][sequence][nub]
    float *s_dg = s_part + 2 * part_floats;                              // 2 x [sequence][nub][4 gates]
    float *s_in = s_dg + 2 * p.seqs * nub * 4;                           // [stage][sequence][nub][8]: gates, c_t, dY
    float *s_dc = s_in + (size_t)stages * p.seqs * nub * 8;              // [item]
    float4 *s_w = reinterpret_cast<float4 *>(s_dc + p.seqs * nub * 4);   // [warp][nsm][4 gates][32 lanes]

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&rbar[i], 1);
        abort_w = 0;
        fence_barrier_init();
    }
    for (int e = tid; e < 2 * p.seqs * nub * 4; e += threads) s_dg[e] = 0.f;
    for (int e = tid; e < stages * p.seqs * nub * 8; e += threads) s_in[e] = 0.f;
    const int j0 = warp * 32 + o * 4;  // this lane's four output units
    auto load_w = [&](int i, int g) {
        const int u = u0 + q + 4 * i;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = q + 4 * i < own && j0 + e < H ? p.w_hh[(size_t)(g * H + u) * H + j0 + e] : 0.f;
        return make_float4(v[0], v[1], v[2], v[3]);
    };
    float4 wr[UR][4];
#pragma unroll
    for (int i = 0; i < UR; ++i)
#pragma unroll
        for (int g = 0; g < 4; ++g) wr[i][g] = load_w(i, g);
    float4 *my_w = s_w + (size_t)warp * p.nsm * 128 + lane;
    for (int i = 0; i < p.nsm; ++i)
#pragma unroll
        for (int g = 0; g < 4; ++g) my_w[(i * 4 + g) * 32] = load_w(UR + i, g);
    const uint32_t step_bytes = (uint32_t)(p.peers * nvalid * ((own + 3) / 4) * 16) + 16u * p.extra_arrivals;
    const int waits = p.s1 - (p.s0 > 1 ? p.s0 : 1);
    if (tid == 0 && active) {
        if (waits > 0) mbar_expect_tx(&rbar[0], step_bytes);
        if (waits > 1) mbar_expect_tx(&rbar[1], step_bytes);
    }
    __syncthreads();
    cluster_sync_all();

    if (active) {
        const size_t slab = (size_t)p.B * H, G = (size_t)4 * H;
        auto unit_of = [&](int e) { return (e >> 2) % nub; };
        auto seq_of = [&](int e) { return (e >> 2) / nub; };
        auto valid = [&](int e) { return e < items && unit_of(e) < own; };
        auto state_off = [&](int e) { return (size_t)(b0 + seq_of(e)) * H + u0 + unit_of(e); };
        auto gate_off = [&](int e) { return (size_t)(b0 + seq_of(e)) * G + (size_t)(e & 3) * H + u0 + unit_of(e); };
        // running offsets of the first EARLY items of this thread
        size_t st_off[EARLY], gt_off[EARLY];
        bool ok_item[EARLY];
#pragma unroll
        for (int k = 0; k < EARLY; ++k) {
            ok_item[k] = valid(tid + k * threads);
            st_off[k] = ok_item[k] ? state_off(tid + k * threads) : 0;
            gt_off[k] = ok_item[k] ? gate_off(tid + k * threads) : 0;
        }
        for (int e = tid; e < items; e += threads)
            s_dc[e] = !valid(e) ? 0.f : p.s0 == 0 ? (p.dc_init ? p.dc_init[state_off(e)] : 0.f) : p.dc[state_off(e)];
        int slot_in = 0;
        auto fetch_item = [&](int e, size_t soff, size_t goff, int t, float *stage) {
            float *dst = stage + (e >> 2) * 8;
            if (t >= 0) cp_async_4(dst + (e & 3), p.gates + (size_t)t * p.B * G + goff);
            if ((e & 3) == 0) cp_async_4(dst + 4, p.cs + (size_t)(t + 1) * slab + soff);
            if ((e & 3) == 1 && t >= 0) cp_async_4(dst + 5, p.dy + (size_t)t * slab + soff);
        };
        // inputs of iteration s (time T-1-s); time -1 only has the cell state entering step 0
        auto fetch = [&](int s) {
            const int t = p.T - 1 - s;
            float *stage = s_in + (size_t)slot_in * p.seqs * nub * 8;
            if (s <= p.s1 && t >= -1) {
#pragma unroll
                for (int k = 0; k < EARLY; ++k)
                    if (ok_item[k]) fetch_item(tid + k * threads, st_off[k], gt_off[k], t, stage);
                for (int e = tid + EARLY * threads; e < items; e += threads)
                    if (valid(e)) fetch_item(e, state_off(e), gate_off(e), t, stage);
            }
            cp_async_commit();
            slot_in = slot_in + 1 == stages ? 0 : slot_in + 1;
        };
        for (int k = 0; k < stages; ++k) fetch(p.s0 + k);
        if (p.ahead == 4) cp_async_wait<3>();
        else cp_async_wait<1>();
        named_barrier_sync(1, threads);

        const uint32_t part_local = smem_u32(s_part), bar_off = smem_u32(rbar) - part_local;
        const int owner = j0 < H ? j0 / nub : 0;
        const uint32_t owner_base = map_to_rank(part_local, (uint32_t)owner);
        const uint32_t my_dst = owner_base + (uint32_t)((((int)rank * p.seqs + q) * nub + j0 - owner * nub) * 4);
        auto contract_and_send = [&](int db, int pb) {
            const float *dgb = s_dg + db * p.seqs * nub * 4 + q * 4;
            for (int blk = 0; blk < blocks; ++blk) {
                const int ns = nvalid - blk * 4;
                float4 acc[4];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    acc[s] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (s < ns) {
                        const float *row = dgb + (blk * 4 + s) * nub * 4;
#pragma unroll
                        for (int i = 0; i < UR; ++i) {
                            const float4 d = *reinterpret_cast<const float4 *>(row + i * 16);
                            acc[s] = fma4(d.x, wr[i][0], acc[s]);
                            acc[s] = fma4(d.y, wr[i][1], acc[s]);
                            acc[s] = fma4(d.z, wr[i][2], acc[s]);
                            acc[s] = fma4(d.w, wr[i][3], acc[s]);
                        }
                    }
                }
#pragma unroll 1
                for (int i = 0; i < p.nsm; ++i) {
                    const float4 w0 = my_w[(i * 4 + 0) * 32], w1 = my_w[(i * 4 + 1) * 32], w2 = my_w[(i * 4 + 2) * 32],
                                 w3 = my_w[(i * 4 + 3) * 32];
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        if (s < ns) {
                            const float4 d = *reinterpret_cast<const float4 *>(dgb + (blk * 4 + s) * nub * 4 + (UR + i) * 16);
                            acc[s] = fma4(d.w, w3, fma4(d.z, w2, fma4(d.y, w1, fma4(d.x, w0, acc[s]))));
                        }
                }
                // reduce-scatter over the four lanes q of the same outputs: lane q keeps sequence q
                const bool hi = lane & 16, odd = lane & 8;
                float4 a, b;
                auto pick = [&](const float4 &keep, const float4 &give, int mask) {
                    return make_float4(keep.x + __shfl_xor_sync(0xffffffffu, give.x, mask), keep.y + __shfl_xor_sync(0xffffffffu, give.y, mask),
                                       keep.z + __shfl_xor_sync(0xffffffffu, give.z, mask), keep.w + __shfl_xor_sync(0xffffffffu, give.w, mask));
                };
                a = pick(hi ? acc[2] : acc[0], hi ? acc[0] : acc[2], 16);
                b = pick(hi ? acc[3] : acc[1], hi ? acc[1] : acc[3], 16);
                const float4 v = pick(odd ? b : a, odd ? a : b, 8);
                if (j0 < H && q < ns)
                    st_async_v4(my_dst + (uint32_t)((pb * part_floats + blk * 4 * nub) * 4), __float_as_uint(v.x), __float_as_uint(v.y),
                                __float_as_uint(v.z), __float_as_uint(v.w), owner_base + bar_off + pb * 8u);
            }
        };
        if (p.s0 > 0) {  // dG of the step above was written by an earlier launch
            const float *src = p.dg + (size_t)(p.T - p.s0) * p.B * G;
            for (int e = tid; e < items; e += threads)
                if (valid(e)) s_dg[p.seqs * nub * 4 + e] = src[gate_off(e)];
            named_barrier_sync(1, threads);
            contract_and_send(1, 0);
        }
        int w = 0, slot = 0;
        const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
        for (int s = p.s0; s < p.s1; ++s) {
            const int t = p.T - 1 - s, db = (s - p.s0) & 1, next = slot + 1 == stages ? 0 : slot + 1;
            const float *in_t = s_in + (size_t)slot * p.seqs * nub * 8, *in_next = s_in + (size_t)next * p.seqs * nub * 8;
            // dG and the carried dc are linear in dh and dc: everything else stands before the wait
            struct Factors {
                float dy, ka, km, gf;
            };
            auto factors = [&](int e) {
                const float *in = in_t + (e >> 2) * 8;
                const float4 g = *reinterpret_cast<const float4 *>(in);  // i, f, g, o
                const float tc = tanh_acc(in[4]), cp = in_next[(e >> 2) * 8 + 4];
                Factors f;
                f.dy = t >= 0 ? in[5] : 0.f;
                f.ka = g.w * (1.f - tc * tc);
                const int gate = e & 3;
                f.km = gate == 0 ? g.z * g.x * (1.f - g.x) : gate == 1 ? cp * g.y * (1.f - g.y) : gate == 2 ? g.x * (1.f - g.z * g.z)
                                                                                               : tc * g.w * (1.f - g.w);
                f.gf = g.y;
                return f;
            };
            Factors early[EARLY];
#pragma unroll
            for (int k = 0; k < EARLY; ++k)
                if (ok_item[k]) early[k] = factors(tid + k * threads);
            bool good = true;
            const float *part = nullptr;
            if (s > 0) {
                good = mbar_wait_cluster(&rbar[w & 1], (uint32_t)w >> 1 & 1u, &abort_w, wait_ns);
                if (good && tid == 0 && w + 2 < waits) mbar_expect_tx(&rbar[w & 1], step_bytes);
                part = s_part + (w & 1) * part_floats;
                ++w;
            }
            auto item = [&](int e, size_t soff, size_t goff, const Factors &f) {
                // the four gate lanes of a pair add a quarter of the sources each; sources in a fixed order
                float dh = 0.f;
                if (s > 0) {
                    const float *src = part + seq_of(e) * nub + unit_of(e);
                    float d1 = 0.f;
                    int r = e & 3;
                    for (; r + 4 < p.peers; r += 8) {
                        dh += src[(size_t)r * p.seqs * nub];
                        d1 += src[(size_t)(r + 4) * p.seqs * nub];
                    }
                    if (r < p.peers) dh += src[(size_t)r * p.seqs * nub];
                    dh += d1;
                    const unsigned group = 0xfu << (lane & ~3);
                    dh += __shfl_xor_sync(group, dh, 1);
                    dh += __shfl_xor_sync(group, dh, 2);
                } else if (p.dhn) {
                    dh = p.dhn[soff];
                }
                if (t < 0) {
                    if (good && (e & 3) == 0) {
                        if (p.dh0) p.dh0[soff] = dh;
                        if (p.dc0) p.dc0[soff] = s_dc[e];
                    }
                    return;
                }
                dh += f.dy;
                const float dcv = fmaf(dh, f.ka, s_dc[e]);
                const float d = ((e & 3) == 3 ? dh : dcv) * f.km;
                s_dc[e] = dcv * f.gf;
                s_dg[db * p.seqs * nub * 4 + e] = d;
                p.dg[(size_t)t * p.B * G + goff] = d;
            };
#pragma unroll
            for (int k = 0; k < EARLY; ++k)
                if (ok_item[k]) item(tid + k * threads, st_off[k], gt_off[k], early[k]);
            for (int e = tid + EARLY * threads; e < items; e += threads)
                if (valid(e)) item(e, state_off(e), gate_off(e), factors(e));
            // the inputs of the next step and the cell state of the one after
            if (p.ahead == 4) cp_async_wait<2>();
            else cp_async_wait<0>();
            if (named_barrier_or(1, threads, !good) || t < 0) break;
            if (s + 1 < p.s1) {
                contract_and_send(db, w & 1);
                fetch(s + stages);  // into the slot this step has read
            }
            slot = next;
        }
        if (!abort_w && p.s1 <= p.T)  // a later launch continues from here
            for (int e = tid; e < items; e += threads)
                if (valid(e) && (e & 3) == 0) p.dc[state_off(e)] = s_dc[e];
    }
    __syncthreads();
    cluster_sync_all();
    if (abort_w) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < kAbortDrainNs) {}
    }
    if (tid == 0 && abort_w) atomicCAS(p.err, 0u, 1u);
}

using FwdKernel = void (*)(ClusterF32FwdParams);
using BwdKernel = void (*)(ClusterF32BwdParams);

FwdKernel fwd_kernel(int kr) {
    switch (kr) {
        case 1: return f32_cluster_fwd_kernel<1>;
        case 2: return f32_cluster_fwd_kernel<2>;
        case 3: return f32_cluster_fwd_kernel<3>;
        case 4: return f32_cluster_fwd_kernel<4>;
        case 6: return f32_cluster_fwd_kernel<6>;
        case 8: return f32_cluster_fwd_kernel<8>;
    }
    return nullptr;
}
BwdKernel bwd_kernel(int ur) {
    switch (ur) {
        case 1: return f32_cluster_bwd_kernel<1>;
        case 2: return f32_cluster_bwd_kernel<2>;
        case 3: return f32_cluster_bwd_kernel<3>;
        case 4: return f32_cluster_bwd_kernel<4>;
        case 6: return f32_cluster_bwd_kernel<6>;
        case 8: return f32_cluster_bwd_kernel<8>;
    }
    return nullptr;
}

// Fills the rest of a plan for C, nub, seqs; false when it does not fit.  `need` chunks of 16 weights per thread.
bool fill(ClusterF32Plan &pl, bool forward, int need, size_t smem_limit) {
    const int blocks = (pl.seqs + 3) / 4;
    for (int ahead : {4, 2})
        for (int kr : {8, 6, 4, 3, 2, 1}) {
            if (kr > need || pl.threads > (forward ? f32_fwd_max_threads(kr) : f32_bwd_max_threads(kr))) continue;
            pl.kr = kr;
            pl.nsm = need - kr;
            pl.ahead = ahead;
            const size_t weights = (size_t)pl.threads / 32 * pl.nsm * 2048;
            const size_t bytes = forward ? 2 * (size_t)pl.seqs * need * 256 + weights + 2 * (size_t)pl.seqs * pl.nub * 4 +
                                               (size_t)blocks * ((16 * ahead + 40) * f32_out_row(pl.threads) + pl.threads) * 4
                                         : 2 * (size_t)pl.peers * pl.seqs * pl.nub * 4 + 2 * (size_t)pl.seqs * pl.nub * 16 +
                                               (size_t)(ahead + 1) * pl.seqs * pl.nub * 32 + (size_t)pl.seqs * pl.nub * 16 + weights;
            pl.smem_bytes = (int)bytes;
            if (bytes + 1024 <= smem_limit) return true;
        }
    return false;
}

}  // namespace

// The cheapest cluster size by estimated cycles per step (see the head of the file), or use = false.
int plan_cluster_f32(bool forward, int B, int H, int sms, size_t smem_limit, ClusterF32Plan *plan) {
    *plan = ClusterF32Plan{};
    if (!cluster_enabled() || H > 512) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_CLUSTER_SIZE");
    const int only = env ? std::atoi(env) : 0;
    int slots[5];
    for (int n = 0; n < 5; ++n) slots[n] = cluster_slots(1 << n, sms);
    for (int tries = 0; tries < 8; ++tries) {
        *plan = ClusterF32Plan{};
        for (int n = 0; n < 5; ++n) {
            ClusterF32Plan pl{};
            pl.C = 1 << n;
            if ((only && pl.C != only) || slots[n] < 1) continue;
            pl.nub = ((H + pl.C - 1) / pl.C + 3) / 4 * 4;
            if (pl.nub > 32) continue;
            pl.peers = (H + pl.nub - 1) / pl.nub;
            pl.seqs = (B + slots[n] - 1) / slots[n];
            pl.clusters = (B + pl.seqs - 1) / pl.seqs;
            const int warps = forward ? pl.nub / 2 : (H + 31) / 32, chunks = forward ? (H + 63) / 64 : pl.nub / 4;
            pl.threads = warps * 32;
            if (!fill(pl, forward, chunks, smem_limit)) continue;
            const int per_sp = (warps + 3) / 4, blocks = (pl.seqs + 3) / 4;
            pl.cycles = per_sp * chunks * pl.seqs * 16 + warps * pl.nsm * blocks * 16 + 600 + 10 * pl.C + H * 4 * pl.seqs / 14 + 400 +
                        per_sp * blocks * 150;
            pl.use = true;
            if (!plan->use || pl.cycles < plan->cycles) *plan = pl;
        }
        if (!plan->use) return FLSTM_OK;
        const void *kernel = forward ? reinterpret_cast<const void *>(fwd_kernel(plan->kr)) : reinterpret_cast<const void *>(bwd_kernel(plan->kr));
        const int have = cluster_count(kernel, plan->C, plan->threads, plan->smem_bytes);
        if (have >= plan->clusters) return FLSTM_OK;
        for (int n = 0; n < 5; ++n)
            if (plan->C == 1 << n) slots[n] = have;
    }
    plan->use = false;
    return FLSTM_OK;
}

int cluster_f32_forward(const ClusterF32Plan &pl, ClusterF32FwdParams p, cudaStream_t s) {
    p.C = pl.C;
    p.peers = pl.peers;
    p.nub = pl.nub;
    p.nsm = pl.nsm;
    p.seqs = pl.seqs;
    p.ahead = pl.ahead;
    return cluster_launch(reinterpret_cast<const void *>(fwd_kernel(pl.kr)), pl.C, pl.clusters * pl.C, pl.threads, pl.smem_bytes, &p, s,
                          "fp32 cluster forward");
}

int cluster_f32_backward(const ClusterF32Plan &pl, ClusterF32BwdParams p, cudaStream_t s) {
    p.C = pl.C;
    p.peers = pl.peers;
    p.nub = pl.nub;
    p.nsm = pl.nsm;
    p.seqs = pl.seqs;
    p.ahead = pl.ahead;
    return cluster_launch(reinterpret_cast<const void *>(bwd_kernel(pl.kr)), pl.C, pl.clusters * pl.C, pl.threads, pl.smem_bytes, &p, s,
                          "fp32 cluster BPTT");
}

}  // namespace simt
}  // namespace flstm_b200
