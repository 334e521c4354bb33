// Cluster-resident recurrent forward kernel: one launch runs all T steps of a layer, every cluster for its own
// sequences (see tc_cluster.cuh for why and when).
//
// Work split.  A CTA of the cluster owns `nub` blocks of 8 hidden units.  A block's 32 gate rows are two m16 tiles,
// rows 0-7 / 8-15 of the first being gates i / f and of the second g / o of the same 8 units, so that the accumulator
// fragments leave all four gate sums of a (unit, sequence) pair in one thread.  `ks` warps split a block's K = H; each
// keeps its W_hh fragments in registers (kr chunks of 32 columns) and, when those do not suffice, the rest in shared
// memory in fragment order.
//
// Per step and warp: wait for h_{t-1} (mbarrier, bytes counted) -> mma over its K range -> partial sums to the block's
// owner warps through shared memory -> gates, c_t, h_t in registers -> through a small staging tile so that h_t of 8
// units leaves as 16 bytes per sequence: by st.async into every CTA of the cluster first, then, like c_t, y_t and the
// activated gates, to global memory (one 16-byte store per lane and slot).  Projections arrive by cp.async
// kClusterAhead steps early.  No CTA-wide barrier lies in the loop.  With one or two warps per scheduler a step is a
// chain of instruction latencies, so addresses are kept as running pointers and everything that does not depend on
// h_{t-1} stands before the wait: H = 64 went from 2040 to about 1000 cycles a step when the seven 2-byte stores per
// slot, the shuffles and the address arithmetic left the chain.
//
// Two buffers of h suffice: a CTA writes h_{t+1} into a peer only after it has received all of h_t, and a peer's part
// of h_t is sent after every warp of that block has read h_{t-1} (partners deliver their partial sums first).
// Every wait is bounded (FwdParams-style wait_ns); on expiry the CTA's abort word is raised, the warps of a block
// leave together (the block's named barrier ORs the verdicts), and all CTAs meet at the final cluster barrier; an
// aborted CTA then lingers so that messages in flight to it land before its shared memory is released.
//
// Replaces, per step, the same reference code as tc_lstm_fwd.cu (flashlstm_v2/src/lstm_forward.cu:744-830).
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "tc_cluster.cuh"

namespace flstm_b200 {
namespace tc {

namespace {

// Threads a kernel may have so that its weights (16 registers per chunk) and working set stay in registers; the
// register file is divided by whole groups of four warps.
constexpr int cluster_fwd_max_threads(int KR, int NT, int KS) {
    const int slots = (2 * NT + KS - 1) / KS;
    const int need = KR * 16 + NT * 8 + slots * 10 + 52;
    return need <= 128 ? 512 : need <= 168 ? 384 : 256;
}

constexpr int kRowSeqs = 4;  // measured at H = 256..512: 3 sequences per cluster are faster direct, 6 by rows

template <int KR, int NT, int KS, bool BF16, bool ACCURATE>
__global__ void __launch_bounds__(cluster_fwd_max_threads(KR, NT, KS), 1)
cluster_fwd_kernel(const ClusterFwdParams p) {
    constexpr int SLOTS = 2 * NT, OWN = (SLOTS + KS - 1) / KS;  // (sequence) slots of a thread, of which it finishes OWN
    constexpr int OWNERS = KS < SLOTS ? KS : SLOTS;             // warps of a block that finish any
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ volatile uint32_t abort_w;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, i8 = lane >> 2, q = lane & 3;
    const int H = p.H, KC = KR + p.nsm;
    const uint32_t rank = cluster_ctarank();
    const int b0 = (int)(blockIdx.x / (unsigned)p.C) * p.seqs;
    const int nvalid = p.B - b0 < p.seqs ? p.B - b0 : p.seqs;
    const int blk = warp / KS, kq = warp % KS;
    const int ub = (int)rank * p.nub + blk;  // global block of 8 units
    const bool active = ub * 8 < H;
    const int nb = H / 8 - (int)rank * p.nub < p.nub ? H / 8 - (int)rank * p.nub : p.nub;  // blocks this CTA owns
    // h is kept as [32-wide K chunk][8 NT sequences][64 B]: a fragment read is 512 contiguous bytes
    constexpr int CHUNK = 8 * NT * 64;
    const int hb_bytes = KS * KC * CHUNK;
    uint8_t *s_h = smem;                                              // 2 x h
    uint8_t *s_w = s_h + 2 * hb_bytes;                                // [warp][nsm][4 gates][32 lanes] x 16 B
    uint8_t *s_red = s_w + (size_t)(blockDim.x >> 5) * p.nsm * 2048;  // 2 x [block][slot][KS][32 lanes] x 16 B
    // projections of the steps ahead: [step % kClusterAhead][warp][own slot][gate][q] x 8 units
    uint8_t *s_p = s_red + (KS > 1 ? (size_t)2 * p.nub * SLOTS * KS * 512 : 0);
    uint8_t *s_out = s_p + (size_t)kClusterAhead * (blockDim.x >> 5) * OWN * 256;  // [warp][own slot] gates and c_t
    uint8_t *s_send = s_out + (size_t)(blockDim.x >> 5) * OWN * 384;                // 2 x [sequence][own block] 16 B: h_t
    int *s_to = reinterpret_cast<int *>(s_send + 2 * 8 * NT * p.nub * 16);          // where piece (sequence, block) goes in s_h

    if (tid == 0) {
        // C = 1: every owner warp arrives once per step; else one arrival announces the bytes of a step
        for (int i = 0; i < 2; ++i) mbar_init(&full[i], p.C == 1 ? (uint32_t)(p.nub * OWNERS) + p.extra_arrivals : 1u);
        abort_w = 0;
        fence_barrier_init();
    }
    for (int o = tid * 16; o < 2 * hb_bytes; o += blockDim.x * 16) *reinterpret_cast<uint4 *>(s_h + o) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const size_t slab = (size_t)p.B * H;
    // the state the launch starts from
    for (int e = tid; e < nvalid * (H / 8); e += blockDim.x) {
        const int n = e / (H / 8), k = (e % (H / 8)) * 8;
        *reinterpret_cast<uint4 *>(s_h + (k >> 5) * CHUNK + n * 64 + (k & 31) * 2) =
            *reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(p.hs) + (size_t)p.t0 * slab + (size_t)(b0 + n) * H + k);
    }
    for (int e = tid; e < nvalid * nb; e += blockDim.x) {
        const int n = e / nb, b = (int)rank * p.nub + e % nb;
        s_to[e] = (b >> 2) * CHUNK + n * 64 + (b & 3) * 16;
    }
    const int u = ub * 8 + i8;  // this thread's unit
    const bool pad = ACCURATE && u >= p.real_units;
    auto load_w = [&](int c, int g) {  // 8 consecutive columns of gate row g of the unit
        const int k0 = (kq * KC + c) * 32 + 8 * q;
        if (!active || k0 >= H) return make_uint4(0, 0, 0, 0);
        return *reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(p.w_hh) +
                                                (size_t)(((u >> 4) * 4 + g) * 16 + (u & 15)) * H + k0);
    };
    uint4 wr[KR][4];
#pragma unroll
    for (int c = 0; c < KR; ++c)
#pragma unroll
        for (int g = 0; g < 4; ++g) wr[c][g] = load_w(c, g);
    uint4 *my_w = reinterpret_cast<uint4 *>(s_w) + (size_t)warp * p.nsm * 128 + lane;
    for (int c = 0; c < p.nsm; ++c)
#pragma unroll
        for (int g = 0; g < 4; ++g) my_w[(c * 4 + g) * 32] = load_w(KR + c, g);
    const uint32_t step_bytes = (uint32_t)H * 2u * (uint32_t)nvalid + 16u * p.extra_arrivals;
    if (p.C > 1 && tid == 0 && active) {
        if (p.T > 1) mbar_expect_tx(&full[1], step_bytes);
        if (p.T > 2) mbar_expect_tx(&full[0], step_bytes);
    }
    __syncthreads();
    if (p.C > 1) cluster_sync_all();  // every CTA's barriers and zeroed buffers exist before anything is sent

    const bool tracing = p.trace != nullptr && blockIdx.x == 0 && tid == 0;
    if (active) {
        // slot sl = 2 nt + s is sequence nt * 8 + 2 q + s; slot sl is finished by warp sl % KS of the block
        const int seq0 = (kq >> 1) * 8 + 2 * q + (kq & 1);  // of this thread's first own slot
        auto seq_of = [&](int j) { return KS == 1 ? (j >> 1) * 8 + 2 * q + (j & 1) : ((j * KS + kq) >> 1) * 8 + 2 * q + (kq & 1); };
        bool mine[OWN];
        float c_keep[OWN];
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            mine[j] = j * KS + kq < SLOTS && seq_of(j) < nvalid;
            c_keep[j] = mine[j] ? p.cs[(size_t)p.t0 * slab + (size_t)(b0 + seq_of(j)) * H + u] : 0.f;
        }
        // projections: lanes 0..15 fetch 16 bytes (8 units of gate lane / 4, sequence q) each
        const int p_stage = (int)(blockDim.x >> 5) * OWN * 256;
        uint8_t *my_p = s_p + warp * OWN * 256;
        const uint32_t row_g = 8u * (uint32_t)H;  // bytes of one sequence's gates
        const char *p_src = static_cast<const char *>(p.gates) + ((size_t)p.t0 * p.B + b0 + seq0) * row_g +
                            ((ub >> 1) * 64 + (lane >> 2) * 16 + (ub & 1) * 8) * 2;
        const size_t step_g = (size_t)p.B * row_g;
        auto fetch = [&](int tt) {
            if (lane < 16 && tt < p.T) {
#pragma unroll
                for (int j = 0; j < OWN; ++j)
                    if (mine[j])
                        cp_async_16(my_p + (tt % kClusterAhead) * p_stage + j * 256 + lane * 16, p_src + (uint32_t)(seq_of(j) - seq0) * row_g);
            }
            cp_async_commit();
            p_src += step_g;
        };
        for (int tt = 0; tt < kClusterAhead; ++tt) fetch(tt);
        // results: this lane stores 16 bytes of sequence q, kind lane / 4 = gates i, f, g, o, h, y, c (two halves)
        uint8_t *my_out = s_out + warp * OWN * 384;
        const int kind = lane >> 2;
        const int out_off = kind < 4 ? kind * 64 + q * 16 : 256 + q * 32 + (kind & 1) * 16;
        const uint32_t row_o = kind < 4 ? row_g : kind < 6 ? row_g / 4 : row_g / 2;
        char *dst = nullptr;
        {
            const size_t seq = (size_t)p.t0 * p.B + b0 + seq0;
            if (kind < 4) {
                if (p.store_gates) dst = static_cast<char *>(p.gates) + seq * row_g + ((ub >> 1) * 64 + kind * 16 + (ub & 1) * 8) * 2;
            } else if (kind == 4) {
                dst = static_cast<char *>(p.hs) + (seq + p.B) * row_o + ub * 16;
            } else if (kind == 5) {
                if (p.y) dst = static_cast<char *>(p.y) + seq * row_o + ub * 16;
            } else {
                dst = reinterpret_cast<char *>(p.cs) + (seq + p.B) * row_o + ub * 32 + (kind - 6) * 16;
            }
        }
        const size_t step_o = (size_t)p.B * row_o;
        const bool store = dst != nullptr, by_element = kind == 5 && !p.y_aligned;
        // How h_t reaches the peers.  Few sequences: every owner warp sends its own 8 units, 16 bytes per sequence, to
        // CTAs i8 and i8 + 8, with no CTA-wide barrier in the step.  From kRowSeqs on the CTA's units are gathered first
        // and every warp sends whole rows to its share of the peers: contiguous st.async messages move 18 bytes per
        // cycle into a CTA, scattered 16-byte ones 6, which outweighs the barrier (about 100 cycles).
        const bool rows = p.C > 1 && nvalid >= kRowSeqs;
        const int send_bytes = 8 * NT * p.nub * 16, pieces = nvalid * nb, warps = nb * KS;
        const uint32_t h_local = smem_u32(s_h), bar_off = smem_u32(full) - h_local;  // same distance in every CTA
        const int r0 = rows ? warp : i8, r1 = rows ? warp + warps : i8 + 8;
        const bool send0 = r0 < p.peers, send1 = r1 < p.peers;
        const uint32_t peer0 = map_to_rank(h_local, send0 ? (uint32_t)r0 : rank), peer1 = map_to_rank(h_local, send1 ? (uint32_t)r1 : rank);
        const int to0 = lane < pieces ? s_to[lane] : -1, to1 = lane + 32 < pieces ? s_to[lane + 32] : -1;
        const uint8_t *h_row = s_h + kq * KC * CHUNK + i8 * 64 + q * 16;  // sequence i8 of a tile as B column
        const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
        for (int tt = 0; tt < p.T; ++tt) {
            float proj[OWN][4];
            cp_async_wait<kClusterAhead - 1>();
            __syncwarp();
            {
                const uint16_t *src = reinterpret_cast<const uint16_t *>(my_p + (tt % kClusterAhead) * p_stage) + q * 8 + i8;
#pragma unroll
                for (int j = 0; j < OWN; ++j)
#pragma unroll
                    for (int g = 0; g < 4; ++g) proj[j][g] = load16<BF16>(src + j * 128 + g * 32);
            }
            bool ok = true;
            if (tt > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait_cluster(&full[tt & 1], (uint32_t)(tt - 1) >> 1 & 1u, &abort_w, wait_ns));
                // arm the buffer for the step after next (never a phase that has not completed: one arrival too many faults)
                if (p.C > 1 && ok && tid == 0 && tt + 2 < p.T) mbar_expect_tx(&full[tt & 1], step_bytes);
            }
            if (KS == 1 && !rows && !ok) break;
            FLSTM_CL_STAMP(tt, 0);
            float acc[NT][2][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[nt][m][e] = 0.f;
            const uint8_t *hb = h_row + (tt & 1) * hb_bytes;
#pragma unroll
            for (int c = 0; c < KR; ++c) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint4 b = *reinterpret_cast<const uint4 *>(hb + c * CHUNK + nt * 512);
                    mma_16816<BF16>(acc[nt][0], wr[c][0].x, wr[c][1].x, wr[c][0].y, wr[c][1].y, b.x, b.y);
                    mma_16816<BF16>(acc[nt][1], wr[c][2].x, wr[c][3].x, wr[c][2].y, wr[c][3].y, b.x, b.y);
                    mma_16816<BF16>(acc[nt][0], wr[c][0].z, wr[c][1].z, wr[c][0].w, wr[c][1].w, b.z, b.w);
                    mma_16816<BF16>(acc[nt][1], wr[c][2].z, wr[c][3].z, wr[c][2].w, wr[c][3].w, b.z, b.w);
                }
            }
#pragma unroll 1
            for (int c = 0; c < p.nsm; ++c) {
                const uint4 w0 = my_w[(c * 4 + 0) * 32], w1 = my_w[(c * 4 + 1) * 32], w2 = my_w[(c * 4 + 2) * 32],
                            w3 = my_w[(c * 4 + 3) * 32];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint4 b = *reinterpret_cast<const uint4 *>(hb + (KR + c) * CHUNK + nt * 512);
                    mma_16816<BF16>(acc[nt][0], w0.x, w1.x, w0.y, w1.y, b.x, b.y);
                    mma_16816<BF16>(acc[nt][1], w2.x, w3.x, w2.y, w3.y, b.x, b.y);
                    mma_16816<BF16>(acc[nt][0], w0.z, w1.z, w0.w, w1.w, b.z, b.w);
                    mma_16816<BF16>(acc[nt][1], w2.z, w3.z, w2.w, w3.w, b.z, b.w);
                }
            }
            FLSTM_CL_STAMP(tt, 4);
            float4 sum[OWN];
            if (KS > 1) {
                // partial sums to the slots' owners; two buffers, so that a fast warp may write the next step's
                float4 *red = reinterpret_cast<float4 *>(s_red) + (size_t)((tt & 1) * p.nub + blk) * SLOTS * KS * 32 + lane;
#pragma unroll
                for (int sl = 0; sl < SLOTS; ++sl) {
                    const float4 v = make_float4(acc[sl >> 1][0][sl & 1], acc[sl >> 1][0][2 + (sl & 1)], acc[sl >> 1][1][sl & 1],
                                                 acc[sl >> 1][1][2 + (sl & 1)]);
                    if (sl % KS == kq) sum[sl / KS] = v;
                    else red[(sl * KS + kq) * 32] = v;
                }
                ok = !named_barrier_or(1 + blk, KS * 32, !ok);
                if (!rows && !ok) break;  // else all warps of the CTA leave together, at the barrier below
#pragma unroll
                for (int j = 0; j < OWN; ++j)
                    if (j * KS + kq < SLOTS) {
#pragma unroll
                        for (int k = 1; k < KS; ++k) {
                            const float4 v = red[((j * KS + kq) * KS + (kq + k) % KS) * 32];
                            sum[j].x += v.x;
                            sum[j].y += v.y;
                            sum[j].z += v.z;
                            sum[j].w += v.w;
                        }
                    }
            } else {
#pragma unroll
                for (int j = 0; j < OWN; ++j)
                    sum[j] = make_float4(acc[j >> 1][0][j & 1], acc[j >> 1][0][2 + (j & 1)], acc[j >> 1][1][j & 1], acc[j >> 1][1][2 + (j & 1)]);
            }
            FLSTM_CL_STAMP(tt, 6);
            const bool more = tt + 1 < p.T;
            uint8_t *send = s_send + (tt & 1) * send_bytes;  // two: a warp may still read the last step's
            if (kq < OWNERS) {
#pragma unroll
                for (int j = 0; j < OWN; ++j) {
                    const float ai = pad ? 0.f : sum[j].x + proj[j][0], af = pad ? 0.f : sum[j].y + proj[j][1];
                    const float ag = pad ? 0.f : sum[j].z + proj[j][2], ao = pad ? 0.f : sum[j].w + proj[j][3];
                    const float gi = sigmoid_sel<ACCURATE>(ai), gf = sigmoid_sel<ACCURATE>(af);
                    const float gg = tanh_sel<ACCURATE>(ag), go = sigmoid_sel<ACCURATE>(ao);
                    c_keep[j] = fmaf(gf, c_keep[j], gi * gg);
                    const uint16_t h16 = to16<BF16>(go * tanh_sel<ACCURATE>(c_keep[j]));
                    if (mine[j]) reinterpret_cast<uint16_t *>(send + (seq_of(j) * nb + blk) * 16)[i8] = h16;
                    uint16_t *st = reinterpret_cast<uint16_t *>(my_out + j * 384) + q * 8 + i8;
                    st[0] = to16<BF16>(gi);
                    st[32] = to16<BF16>(gf);
                    st[64] = to16<BF16>(gg);
                    st[96] = to16<BF16>(go);
                    *reinterpret_cast<float *>(my_out + j * 384 + 256 + q * 32 + i8 * 4) = c_keep[j];
                }
            }
            const uint32_t buf = (uint32_t)((tt + 1) & 1) * hb_bytes, bar = bar_off + ((tt + 1) & 1) * 8u;
            if (rows) {
                if (named_barrier_or(15, warps * 32, !ok)) break;
                if (more) {
                    auto send_row = [&](uint32_t base) {
                        if (to0 >= 0) {
                            const uint4 m = *reinterpret_cast<const uint4 *>(send + lane * 16);
                            st_async_v4(base + buf + to0, m.x, m.y, m.z, m.w, base + bar);
                        }
                        if (to1 >= 0) {
                            const uint4 m = *reinterpret_cast<const uint4 *>(send + lane * 16 + 512);
                            st_async_v4(base + buf + to1, m.x, m.y, m.z, m.w, base + bar);
                        }
                        for (int e = lane + 64; e < pieces; e += 32) {
                            const uint4 m = *reinterpret_cast<const uint4 *>(send + e * 16);
                            st_async_v4(base + buf + s_to[e], m.x, m.y, m.z, m.w, base + bar);
                        }
                    };
                    if (send0) send_row(peer0);
                    if (send1) send_row(peer1);
                    for (int r = r1 + warps; r < p.peers; r += warps) send_row(map_to_rank(h_local, (uint32_t)r));
                }
            } else if (kq < OWNERS) {
                __syncwarp();
                if (more) {
#pragma unroll
                    for (int j = 0; j < OWN; ++j) {
                        const uint4 m = *reinterpret_cast<const uint4 *>(send + (seq_of(j) * nb + blk) * 16);
                        const uint32_t off = buf + (uint32_t)((ub >> 2) * CHUNK + seq_of(j) * 64 + (ub & 3) * 16);
                        if (p.C == 1) {
                            if (i8 == 0 && mine[j]) *reinterpret_cast<uint4 *>(s_h + off) = m;
                        } else {
                            if (mine[j] && send0) st_async_v4(peer0 + off, m.x, m.y, m.z, m.w, peer0 + bar);
                            if (mine[j] && send1) st_async_v4(peer1 + off, m.x, m.y, m.z, m.w, peer1 + bar);
                        }
                    }
                    if (p.C == 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&full[(tt + 1) & 1]);
                    }
                }
            }
            FLSTM_CL_STAMP(tt, 8);
            if (kq < OWNERS) {  // everything nobody waits for
#pragma unroll
                for (int j = 0; j < OWN; ++j) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(kind == 4 || kind == 5 ? send + (seq_of(j) * nb + blk) * 16
                                                                                            : my_out + j * 384 + out_off);
                    char *to = dst + (uint32_t)(seq_of(j) - seq0) * row_o;
                    if (store && mine[j]) {
                        if (!by_element) {
                            *reinterpret_cast<uint4 *>(to) = v;
                        } else {  // the caller's y may start at any element
                            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int e = 0; e < 8; ++e) reinterpret_cast<uint16_t *>(to)[e] = (uint16_t)(w[e >> 1] >> (16 * (e & 1)));
                        }
                    }
                }
                if (store) dst += step_o;
                fetch(tt + kClusterAhead);
            }
        }
    }
    __syncthreads();
    if (p.C > 1) {
        cluster_sync_all();  // nobody leaves while a peer may still send into its shared memory
        if (abort_w) {
            const unsigned long long t0 = global_timer_ns();
            while (global_timer_ns() - t0 < kAbortDrainNs) {}
        }
    }
    if (tid == 0 && abort_w) atomicCAS(p.err, 0u, 1u);
}

using FwdKernel = void (*)(ClusterFwdParams);

template <int NT, int KS, bool BF16, bool ACC>
FwdKernel fwd_kernel_kr(int kr) {
    switch (kr) {
        case 1: return cluster_fwd_kernel<1, NT, KS, BF16, ACC>;
        case 2: return cluster_fwd_kernel<2, NT, KS, BF16, ACC>;
        case 3: return cluster_fwd_kernel<3, NT, KS, BF16, ACC>;
        case 4: return cluster_fwd_kernel<4, NT, KS, BF16, ACC>;
        case 5: return cluster_fwd_kernel<5, NT, KS, BF16, ACC>;
        case 6: return cluster_fwd_kernel<6, NT, KS, BF16, ACC>;
        case 8: return cluster_fwd_kernel<8, NT, KS, BF16, ACC>;
    }
    return nullptr;
}
template <int KS, bool BF16, bool ACC>
FwdKernel fwd_kernel_nt(int kr, int NT) {
    switch (NT) {
        case 1: return fwd_kernel_kr<1, KS, BF16, ACC>(kr);
        case 2: return fwd_kernel_kr<2, KS, BF16, ACC>(kr);
        case 4: return fwd_kernel_kr<4, KS, BF16, ACC>(kr);
    }
    return nullptr;
}
template <bool BF16, bool ACC>
FwdKernel fwd_kernel_ks(int kr, int NT, int ks) {
    switch (ks) {
        case 1: return fwd_kernel_nt<1, BF16, ACC>(kr, NT);
        case 2: return fwd_kernel_nt<2, BF16, ACC>(kr, NT);
    }
    return nullptr;
}
FwdKernel fwd_kernel(int kr, int NT, int ks, bool bf16, bool accurate) {
    if (accurate) return bf16 ? fwd_kernel_ks<true, true>(kr, NT, ks) : fwd_kernel_ks<false, true>(kr, NT, ks);
    return bf16 ? fwd_kernel_ks<true, false>(kr, NT, ks) : fwd_kernel_ks<false, false>(kr, NT, ks);
}

int fwd_smem(const ClusterFwdPlan &pl) {
    const int kc = pl.kr + pl.nsm, own = (2 * pl.NT + pl.ks - 1) / pl.ks, warps = pl.threads / 32;
    return 2 * pl.ks * kc * 8 * pl.NT * 64 + warps * (pl.nsm * 2048 + kClusterAhead * own * 256 + own * 384) +
           (pl.ks > 1 ? 2 * pl.nub * 2 * pl.NT * pl.ks * 512 : 0) + 8 * pl.NT * pl.nub * (2 * 16 + 4);
}

void fill_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr, int C, int grid, int threads, int smem) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(grid);
    cfg->blockDim = dim3(threads);
    cfg->dynamicSmemBytes = smem;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = C;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

}  // namespace

int cluster_prepare_kernel(const void *kernel, int C, int smem_bytes) {
    if (ensure_smem_limit(kernel, smem_bytes) != cudaSuccess) return -1;
    if (C > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return -1;
    return 0;
}

// The occupancy query takes about a millisecond, so its answers are kept per device, kernel and launch shape.
int cluster_count(const void *kernel, int C, int threads, int smem_bytes) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void *, int, int, int>, int> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(dev, kernel, C, threads, smem_bytes);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    fill_config(&cfg, &attr, C, C, threads, smem_bytes);
    int n = 0;
    if (cluster_prepare_kernel(kernel, C, smem_bytes) != 0 || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return known[key] = n;
}

int cluster_launch(const void *kernel, int C, int grid, int threads, int smem_bytes, void *params, cudaStream_t s, const char *what) {
    if (cluster_prepare_kernel(kernel, C, smem_bytes) != 0)
        return set_error(FLSTM_ERR_CUDA, "%s: the kernel's attributes could not be set: %s", what, cudaGetErrorString(cudaGetLastError()));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    fill_config(&cfg, &attr, C, grid, threads, smem_bytes);
    cfg.stream = s;
    void *args[] = {params};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, args);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
    return FLSTM_OK;
}

bool cluster_enabled() {
    const char *env = std::getenv("FLSTM_CLUSTER");
    return !(env && env[0] == '0');
}

// For every cluster size and split of K: the sequences per cluster that one wave of clusters leaves, the chunks of
// weights that fit the registers (shared memory for what is left) and the estimated cycles of a step; the cheapest
// wins.  The terms: 8 cycles per mma and sub-partition or 20 per dependent pair, 4 cycles per 512 B of weights read
// from shared memory, the exchange as measured (tc_cluster.cuh), the gate functions per own slot.
int plan_cluster_fwd(int B, int H, int sms, size_t smem_limit, ClusterFwdPlan *plan, const ClusterCheck *check) {
    *plan = ClusterFwdPlan{};
    if (!cluster_enabled() || H % 64 || H > 768) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_CLUSTER_SIZE");
    const int only = env ? std::atoi(env) : 0;
    const int blocks = H / 8, chunks = H / 32;
    int slots[5];  // clusters of 1, 2, 4, 8, 16 CTAs that run at once
    for (int n = 0; n < 5; ++n) slots[n] = cluster_slots(1 << n, sms);
    for (int tries = 0; tries < 8; ++tries) {
        *plan = ClusterFwdPlan{};
        for (int n = 0; n < 5; ++n) {
            const int C = 1 << n;
            if ((only && C != only) || slots[n] < 1) continue;
        for (int ks = 1; ks <= 2 && ks <= chunks; ks *= 2)  // (4 is the cheapest plan of no shape)
            for (int kr : {8, 6, 5, 4, 3, 2, 1}) {
                ClusterFwdPlan pl{};
                pl.C = C;
                pl.nub = (blocks + C - 1) / C;
                pl.peers = (blocks + pl.nub - 1) / pl.nub;
                pl.seqs = (B + slots[n] - 1) / slots[n];
                const int tiles = (pl.seqs + 7) / 8, kc = (chunks + ks - 1) / ks;
                pl.NT = tiles <= 1 ? 1 : tiles <= 2 ? 2 : 4;
                const int warps = pl.nub * ks;
                if (tiles > 4 || kr > kc || warps > 16 || warps * 32 > cluster_fwd_max_threads(kr, pl.NT, ks)) continue;
                pl.ks = ks;
                pl.kr = kr;
                pl.nsm = kc - kr;
                pl.threads = warps * 32;
                pl.smem_bytes = fwd_smem(pl);
                if ((size_t)pl.smem_bytes + 1024 > smem_limit) continue;
                pl.clusters = (B + pl.seqs - 1) / pl.seqs;
                const int busy = (warps + 3) / 4 * kc * pl.NT * 32, chain = kc * 40, own = (2 * pl.NT + ks - 1) / ks;
                const int incoming = H * 2 * pl.seqs;
                const int exchange = C == 1 ? 600 : 540 + 10 * C + (pl.seqs < kRowSeqs ? incoming / 6 : 250 + incoming / 14);
                pl.cycles = (busy > chain ? busy : chain) + warps * pl.nsm * 16 + exchange + 300 + (warps + 3) / 4 * 100 + 200 * own +
                            (ks > 1 ? 70 + 10 * ks : 0);
                pl.use = true;
                if (!plan->use || pl.cycles < plan->cycles) *plan = pl;
            }
        }
        if (!plan->use || !check) return FLSTM_OK;
        // only the winner's occupancy is asked for: a query loads the kernel and takes about a millisecond
        const int have = cluster_count(reinterpret_cast<const void *>(fwd_kernel(plan->kr, plan->NT, plan->ks, check->bf16, check->accurate)),
                                       plan->C, plan->threads, plan->smem_bytes);
        if (have >= plan->clusters) return FLSTM_OK;
        for (int n = 0; n < 5; ++n)
            if (plan->C == 1 << n) slots[n] = have;  // fewer run at once than assumed: more sequences for each
    }
    plan->use = false;
    return FLSTM_OK;
}

int lstm_forward_cluster(int dtype, const ClusterFwdPlan &pl, ClusterFwdParams p, cudaStream_t s) {
    p.C = pl.C;
    p.peers = pl.peers;
    p.nub = pl.nub;
    p.ks = pl.ks;
    p.nsm = pl.nsm;
    p.seqs = pl.seqs;
    p.y_aligned = reinterpret_cast<uintptr_t>(p.y) % 16 == 0;
    FwdKernel kern = fwd_kernel(pl.kr, pl.NT, pl.ks, dtype == FLSTM_DTYPE_BF16, p.real_units > 0);
    if (!kern) return set_error(FLSTM_ERR_UNSUPPORTED, "no cluster forward kernel for this plan");
    return cluster_launch(reinterpret_cast<const void *>(kern), pl.C, pl.clusters * pl.C, pl.threads, pl.smem_bytes, &p, s,
                          "cluster recurrent forward");
}

}  // namespace tc
}  // namespace flstm_b200
