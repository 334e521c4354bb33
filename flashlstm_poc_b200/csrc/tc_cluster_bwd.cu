// Cluster-resident BPTT kernel: one launch runs the whole reverse recurrence of a layer, every cluster for its own
// sequences (see tc_cluster.cuh for why and when).
//
// Work split.  A CTA owns U = 8 nub hidden units: it forms their dG_t (all four gates) and contracts it with the 4U
// rows of W_hh that belong to them, which yields its PARTIAL dh_{t-1} of all H units; the fp32 partial sums go to the
// units' owners by st.async (16 bytes = four sequences of one unit, counted by the receiving mbarrier) and are added
// there in a fixed order.  Sending partial sums moves H fp32 values per sequence and CTA instead of the 4H 16-bit
// values an all-gather of dG would.  W_hh^T fragments (units x own gate rows) stay in registers, the ones that do not
// fit in shared memory in fragment order.
//
// Per step: wait for the partial sums -> pointwise backward of the own (unit, sequence) pairs, dG_t to shared memory
// -> one CTA barrier -> mma over the own gate rows -> partial sums out.  The
// gate cache, cell states and dY are fetched kClusterAhead steps ahead by cp.async; dG_t goes to
// global memory in 16-byte pieces at the end of the step.
// Two buffers of partial sums and of dG suffice: a CTA sends the partial sums of step s+1 after it has received all of
// step s, which every peer sent after it had read those of step s-1; and every warp of a CTA sends to some peer, so a
// peer that has moved on proves that the warp has left its product.
// Waits are bounded as in the other persistent kernels; the CTA barrier ORs the verdicts, so all threads leave together.
//
// Replaces, per step, the same reference code as tc_lstm_bwd.cu (flashlstm_v2/src/lstm_backward.cu:158-227,1057-1101).
#include <cstdlib>

#include "common.cuh"
#include "tc_cluster.cuh"

namespace flstm_b200 {
namespace tc {

namespace {

// weight fragments (one 16-unit tile x one 32-wide K chunk, 8 registers) that stay in registers
constexpr int cluster_bwd_reg_frags(int W, int MT, int NKB, int NT, int PP) {
    const int regs = W <= 8 ? 255 : W <= 12 ? 168 : 128;
    const int room = (regs - 60 - MT * NT * 4 - MT - PP * 2) / 8;
    return MT * NKB < room ? MT * NKB : room;
}
constexpr int cluster_bwd_pairs(int W, int units, int NT) { return (units * 8 * NT + 32 * W - 1) / (32 * W); }

template <int W, int MT, int NKB, int KSB, int NT, bool BF16, bool ACCURATE>
__global__ void __launch_bounds__(W * 32, 1)
cluster_bwd_kernel(const ClusterBwdParams p) {
    constexpr int NUB = NKB * KSB, U = 8 * NUB, NS = 8 * NT, THREADS = 32 * W, WG = W / KSB;
    constexpr int PP = cluster_bwd_pairs(W, U, NT);  // (unit, sequence) pairs per thread
    constexpr int FRAGS = MT * NKB, FR = cluster_bwd_reg_frags(W, MT, NKB, NT, PP);
    constexpr int ROW = cluster_row_bytes(NUB * 64);  // one sequence's dG of the own units, k' = unit * 4 + gate
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t rbar[2];
    __shared__ volatile uint32_t abort_w;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, i8 = lane >> 2, q = lane & 3;
    const int H = p.H;
    const uint32_t rank = cluster_ctarank();
    const int b0 = (int)(blockIdx.x / (unsigned)p.C) * p.seqs;
    const int nvalid = p.B - b0 < p.seqs ? p.B - b0 : p.seqs;
    const int u0 = (int)rank * U;  // first own unit
    const bool active = u0 < H;
    const int src_count = p.peers * KSB;
    // sequences per row of the partial sums: with at most four of them the rows are half as long and stay contiguous
    const int ns = NT == 1 && nvalid <= 4 ? 4 : NS;
    const int part_bytes = src_count * U * ns * 4;
    uint8_t *s_part = smem;                       // 2 x [source][own unit][ns sequences] fp32
    uint8_t *s_dg = s_part + 2 * part_bytes;      // 2 x [NS sequences][ROW]
    // inputs of the steps ahead, per sequence and block of 8 units: i, f, g, o, dY (16 B each), c_t (32 B); c_{t-1} is
    // the c_t of the step after.  One slot more than steps ahead, for that c_{t-1}.
    constexpr int SLOT = 112, STAGE = NS * NUB * SLOT, STAGES = kClusterAhead + 1;
    constexpr int OUT = NS * NUB * 64;
    uint8_t *s_in = s_dg + 2 * NS * ROW;
    uint8_t *s_out = s_in + STAGES * STAGE;       // 2 x [block][sequence][gate][8 units]: dG_t on its way to global memory
    uint8_t *s_w = s_out + 2 * OUT;               // [warp][fragment][2][32 lanes] x 16 B

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&rbar[i], p.C == 1 ? (uint32_t)W + p.extra_arrivals : 1u);
        abort_w = 0;
        fence_barrier_init();
    }
    for (int o = tid * 16; o < 2 * NS * ROW; o += THREADS * 16) *reinterpret_cast<uint4 *>(s_dg + o) = make_uint4(0, 0, 0, 0);

    const int mg = warp % WG, kp = warp / WG;  // unit-tile group and K group of this warp
    const uint16_t *w16 = static_cast<const uint16_t *>(p.w_hh);
    // fragment f = m * NKB + kc: rows = units of tile mg * MT + m, columns = the 32 gate rows of own block kp * NKB + kc
    auto load_frag = [&](int m, int kc, uint32_t (&a)[8]) {
        const int mt = mg * MT + m, blk = kp * NKB + kc;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int unit = u0 + blk * 8 + 2 * (i8 >> 1) + j, g = 2 * h + (i8 & 1), col = mt * 16 + e * 8 + 2 * q;
                    uint32_t v = 0;
                    if (unit < H && mt * 16 < H)
                        v = *reinterpret_cast<const uint32_t *>(w16 + (size_t)(((unit >> 4) * 4 + g) * 16 + (unit & 15)) * H + col);
                    a[j * 4 + h * 2 + e] = movmatrix_trans(v);
                }
    };
    uint32_t wr[FR > 0 ? FR : 1][8];
    uint4 *my_w = reinterpret_cast<uint4 *>(s_w) + (size_t)warp * (FRAGS - FR) * 64 + lane;
#pragma unroll
    for (int f = 0; f < FRAGS; ++f) {
        if (f < FR) {
            load_frag(f / NKB, f % NKB, wr[f < FR ? f : 0]);
        } else {
            uint32_t a[8];
            load_frag(f / NKB, f % NKB, a);
            my_w[(f - FR) * 64] = make_uint4(a[0], a[1], a[2], a[3]);
            my_w[(f - FR) * 64 + 32] = make_uint4(a[4], a[5], a[6], a[7]);
        }
    }
    const int own_units = H - u0 < U ? H - u0 : U;
    const uint32_t step_bytes = (uint32_t)(src_count * own_units * ((nvalid + 3) / 4) * 16) + 16u * p.extra_arrivals;
    const int waits = p.s1 - (p.s0 > 1 ? p.s0 : 1);  // iterations that wait for partial sums
    if (p.C > 1 && tid == 0 && active) {
        if (waits > 0) mbar_expect_tx(&rbar[0], step_bytes);
        if (waits > 1) mbar_expect_tx(&rbar[1], step_bytes);
    }
    __syncthreads();
    if (p.C > 1) cluster_sync_all();

    const bool tracing = p.trace != nullptr && blockIdx.x == 0 && tid == 0;
    if (active) {
        const size_t slab = (size_t)p.B * H, G = (size_t)4 * H;
        const uint16_t *gates = static_cast<const uint16_t *>(p.gates), *dy = static_cast<const uint16_t *>(p.dy);
        const uint16_t *dhn = static_cast<const uint16_t *>(p.dhn), *dcn = static_cast<const uint16_t *>(p.dcn);
        uint16_t *dg = static_cast<uint16_t *>(p.dg);
        // pair k of this thread: sequence (tid + k THREADS) % NS, own unit (tid + k THREADS) / NS
        auto seq_of = [&](int k) { return (tid + k * THREADS) % NS; };
        auto unit_of = [&](int k) { return (tid + k * THREADS) / NS; };
        auto valid = [&](int k) { return unit_of(k) < own_units && seq_of(k) < nvalid; };
        auto state_off = [&](int k) { return (size_t)(b0 + seq_of(k)) * H + u0 + unit_of(k); };
        auto gate_off = [&](int k) {
            const int u = u0 + unit_of(k);
            return (size_t)(b0 + seq_of(k)) * G + (u >> 4) * 64 + (u & 15);
        };
        // Inputs of the steps ahead: piece e of a step is 16 bytes of (block, sequence): gates i, f, g, o, dY, c_t (two
        // halves).  Threads with few pieces keep a running pointer for each, else the addresses are formed anew.
        constexpr int PIECES = NS * NUB * 7, NP = (PIECES + THREADS - 1) / THREADS;
        constexpr bool RUNNING = NP <= 2;
        auto piece_src = [&](int e, int t, bool *scalar, int *step) -> const char * {
            const int piece = e % 7, n = e / 7 % NS, blk = e / (7 * NS), u = u0 + blk * 8;
            if (n >= nvalid || u >= H) return nullptr;
            const long long row = b0 + n;
            *scalar = false;
            if (piece >= 5) {
                *step = (int)slab * 4;
                return reinterpret_cast<const char *>(p.cs + (t + 1) * (long long)slab + row * H + u + (piece - 5) * 4);
            }
            if (piece == 4) {
                *scalar = !p.dy_aligned;
                *step = (int)slab * 2;
                return reinterpret_cast<const char *>(dy + t * (long long)slab + row * H + u);
            }
            *step = (int)slab * 8;
            return reinterpret_cast<const char *>(gates + (t * (long long)p.B + row) * (long long)G + (u >> 4) * 64 + piece * 16 + (u & 15));
        };
        auto copy_piece = [&](uint8_t *dst, const char *src, bool scalar) {
            if (!scalar) {
                cp_async_16(dst, src);
            } else {  // the caller's dY may start at any element
                for (int k = 0; k < 8; ++k) reinterpret_cast<uint16_t *>(dst)[k] = reinterpret_cast<const uint16_t *>(src)[k];
            }
        };
        const char *in_src[RUNNING ? NP : 1];
        int in_step[RUNNING ? NP : 1];
        bool in_scalar[RUNNING ? NP : 1];
        if (RUNNING) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                in_step[k] = 0;
                in_scalar[k] = false;
                in_src[k] = tid + k * THREADS < PIECES ? piece_src(tid + k * THREADS, p.T - 1 - p.s0, &in_scalar[k], &in_step[k]) : nullptr;
            }
        }
        int slot_in = 0;  // ring slot of the next fetch
        // the inputs of iteration s (time T-1-s); time -1 only has the cell state entering step 0
        auto fetch = [&](int s) {
            const int t = p.T - 1 - s;
            uint8_t *stage = s_in + slot_in * STAGE;
            if (s <= p.s1 && t >= -1) {
                if (RUNNING) {
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const int e = tid + k * THREADS;
                        if (in_src[k] && (t >= 0 || e % 7 >= 5)) copy_piece(stage + (e / 7) * SLOT + e % 7 * 16, in_src[k], in_scalar[k]);
                        if (in_src[k]) in_src[k] -= in_step[k];
                    }
                } else {
                    for (int e = tid; e < PIECES; e += THREADS) {
                        bool scalar;
                        int step;
                        const char *src = piece_src(e, t, &scalar, &step);
                        if (src && (t >= 0 || e % 7 >= 5)) copy_piece(stage + (e / 7) * SLOT + e % 7 * 16, src, scalar);
                    }
                }
            }
            cp_async_commit();
            slot_in = slot_in + 1 == STAGES ? 0 : slot_in + 1;
        };
        // dG_t leaves in 16-byte pieces (block, sequence, gate)
        constexpr int OUTS = NS * NUB * 4, NO = (OUTS + THREADS - 1) / THREADS;
        constexpr bool RUNNING_OUT = NO <= 2;
        auto out_dst = [&](int e, int t) -> char * {
            const int g = e % 4, n = e / 4 % NS, blk = e / (4 * NS), u = u0 + blk * 8;
            if (n >= nvalid || u >= H) return nullptr;
            return reinterpret_cast<char *>(dg + (t * (long long)p.B + b0 + n) * (long long)G + (u >> 4) * 64 + g * 16 + (u & 15));
        };
        char *out_ptr[RUNNING_OUT ? NO : 1];
        if (RUNNING_OUT) {
#pragma unroll
            for (int k = 0; k < NO; ++k)
                out_ptr[k] = tid + k * THREADS < OUTS ? out_dst(tid + k * THREADS, p.T - 1 - p.s0) : nullptr;
        }
        auto write_out = [&](int t, int buf) {
            const uint4 *src = reinterpret_cast<const uint4 *>(s_out + buf * OUT);
            if (RUNNING_OUT) {
#pragma unroll
                for (int k = 0; k < NO; ++k)
                    if (out_ptr[k]) {
                        *reinterpret_cast<uint4 *>(out_ptr[k]) = src[tid + k * THREADS];
                        out_ptr[k] -= slab * 8;
                    }
            } else {
                for (int e = tid; e < OUTS; e += THREADS)
                    if (char *to = out_dst(e, t)) *reinterpret_cast<uint4 *>(to) = src[e];
            }
        };
        float dc[PP];
#pragma unroll
        for (int k = 0; k < PP; ++k) {
            dc[k] = 0.f;
            if (valid(k)) {
                if (p.s0 == 0) dc[k] = dcn ? load16<BF16>(dcn + state_off(k)) : 0.f;
                else dc[k] = p.dc[state_off(k)];
            }
        }
        for (int k = 0; k <= kClusterAhead; ++k) fetch(p.s0 + k);
        cp_async_wait<kClusterAhead - 1>();  // the first two: c_{t-1} comes with the second
        named_barrier_sync(1, THREADS);
        // where the two 8-unit halves of each of this warp's unit tiles go: this lane sends the half q & 1
        const uint32_t part_local = smem_u32(s_part), bar_off = smem_u32(rbar) - part_local;
        uint32_t dst[MT], dst_base[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int unit = (mg * MT + m) * 16 + (q & 1) * 8 + i8;
            const int owner = unit < H ? unit / U : (int)rank;
            dst_base[m] = p.C > 1 ? map_to_rank(part_local, (uint32_t)owner) : part_local;
            dst[m] = dst_base[m] + (uint32_t)(((((int)rank * KSB + kp) * U + unit % U) * ns + (q >> 1) * 4) * 4);
        }
        // partial dh from the dG in buffer `db`, to part buffer `pb` of the owners
        auto contract_and_send = [&](int db, int pb) {
            float acc[MT][NT][4];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[m][nt][e] = 0.f;
            float acc2[4] = {0.f, 0.f, 0.f, 0.f};  // second chain when there is only one tile
            const uint8_t *row = s_dg + db * NS * ROW + i8 * ROW + kp * NKB * 64 + q * 16;
#pragma unroll
            for (int kc = 0; kc < NKB; ++kc) {
                uint4 b[NT];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) b[nt] = *reinterpret_cast<const uint4 *>(row + nt * 8 * ROW + kc * 64);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int f = m * NKB + kc;
                    uint32_t a[8];
                    if (f < FR) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] = wr[f < FR ? f : 0][e];
                    } else {
                        const uint4 x = my_w[(f - FR) * 64], z = my_w[(f - FR) * 64 + 32];
                        a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
                        a[4] = z.x; a[5] = z.y; a[6] = z.z; a[7] = z.w;
                    }
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        mma_16816<BF16>(acc[m][nt], a[0], a[1], a[2], a[3], b[nt].x, b[nt].y);
                        if (MT * NT == 1) mma_16816<BF16>(acc2, a[4], a[5], a[6], a[7], b[nt].z, b[nt].w);
                        else mma_16816<BF16>(acc[m][nt], a[4], a[5], a[6], a[7], b[nt].z, b[nt].w);
                    }
                }
            }
            if (MT * NT == 1) {
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[0][0][e] += acc2[e];
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const bool unit_ok = (mg * MT + m) * 16 < H;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    // even lanes of a pair take the lower half's unit, odd lanes the upper half's, four sequences each
                    const bool odd = q & 1;
                    const float rx = __shfl_xor_sync(0xffffffffu, odd ? acc[m][nt][0] : acc[m][nt][2], 1);
                    const float ry = __shfl_xor_sync(0xffffffffu, odd ? acc[m][nt][1] : acc[m][nt][3], 1);
                    const float v0 = odd ? rx : acc[m][nt][0], v1 = odd ? ry : acc[m][nt][1];
                    const float v2 = odd ? acc[m][nt][2] : rx, v3 = odd ? acc[m][nt][3] : ry;
                    if (unit_ok && nt * 8 + (q >> 1) * 4 < nvalid) {
                        const uint32_t addr = dst[m] + (uint32_t)(pb * part_bytes + nt * 32);
                        if (p.C == 1)
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v0), "f"(v1), "f"(v2), "f"(v3) : "memory");
                        else
                            st_async_v4(addr, __float_as_uint(v0), __float_as_uint(v1), __float_as_uint(v2), __float_as_uint(v3),
                                        dst_base[m] + bar_off + pb * 8u);
                    }
                }
            }
            if (p.C == 1) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&rbar[pb]);
            }
        };
        if (p.s0 > 0) {  // dG of the step above was written by an earlier launch
            const uint16_t *src = dg + (size_t)(p.T - p.s0) * p.B * G;
#pragma unroll
            for (int k = 0; k < PP; ++k)
                if (valid(k)) {
                    const uint16_t *r = src + gate_off(k);
                    *reinterpret_cast<uint2 *>(s_dg + NS * ROW + seq_of(k) * ROW + unit_of(k) * 8) =
                        make_uint2((uint32_t)r[0] | (uint32_t)r[16] << 16, (uint32_t)r[32] | (uint32_t)r[48] << 16);
                }
            named_barrier_sync(1, THREADS);
            contract_and_send(1, 0);
        }
        int w = 0;       // waits made so far
        int slot = 0;    // ring slot of this iteration's inputs
        const unsigned long long wait_ns = p.wait_ns ? p.wait_ns : kWaitLimitNs;
        for (int s = p.s0; s < p.s1; ++s) {
            const int t = p.T - 1 - s;  // t = -1: only dh0 / dc0
            const int db = (s - p.s0) & 1, next = slot + 1 == STAGES ? 0 : slot + 1;
            // everything that does not depend on dh stands before the wait: dG and the carried dc are linear in dh and dc
            float dh[PP], ka[PP], ki[PP], kf[PP], kg[PP], ko[PP], gf[PP];
#pragma unroll
            for (int k = 0; k < PP; ++k) {
                const int cell = (unit_of(k) >> 3) * NS + seq_of(k), ue = unit_of(k) & 7;
                if (unit_of(k) >= U) continue;
                const uint8_t *in = s_in + slot * STAGE + cell * SLOT;
                const uint16_t *in16 = reinterpret_cast<const uint16_t *>(in) + ue;
                const float gi = load16<BF16>(in16), gg = load16<BF16>(in16 + 16), go = load16<BF16>(in16 + 24);
                gf[k] = load16<BF16>(in16 + 8);
                dh[k] = load16<BF16>(in16 + 32);
                const float tc = tanh_sel<ACCURATE>(reinterpret_cast<const float *>(in + 80)[ue]);
                const float cp = reinterpret_cast<const float *>(s_in + next * STAGE + cell * SLOT + 80)[ue];
                ka[k] = go * (1.f - tc * tc);
                ki[k] = gg * gi * (1.f - gi);
                kf[k] = cp * gf[k] * (1.f - gf[k]);
                kg[k] = gi * (1.f - gg * gg);
                ko[k] = tc * go * (1.f - go);
                if (t < 0) dh[k] = 0.f;
                if (s == 0 && dhn && valid(k)) dh[k] += load16<BF16>(dhn + state_off(k));
            }
            bool good = true;
            if (s > 0) {
                good = mbar_wait_cluster(&rbar[w & 1], (uint32_t)w >> 1 & 1u, &abort_w, wait_ns);
                if (p.C > 1 && good && tid == 0 && w + 2 < waits) mbar_expect_tx(&rbar[w & 1], step_bytes);
                const float *part = reinterpret_cast<const float *>(s_part + (w & 1) * part_bytes);
                ++w;
                FLSTM_CL_STAMP(s - p.s0, 0);
#pragma unroll
                for (int k = 0; k < PP; ++k) {
                    if (unit_of(k) >= U) continue;
                    const float *row = part + unit_of(k) * ns + (seq_of(k) & (ns - 1));
                    const int next_src = U * ns;
                    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;  // four chains, added in a fixed order
                    int src = 0;
                    for (; src + 3 < src_count; src += 4, row += 4 * next_src) {
                        d0 += row[0];
                        d1 += row[next_src];
                        d2 += row[2 * next_src];
                        d3 += row[3 * next_src];
                    }
                    for (; src < src_count; ++src, row += next_src) d0 += row[0];
                    dh[k] += (d0 + d1) + (d2 + d3);
                }
            }
            if (ACCURATE) {
#pragma unroll
                for (int k = 0; k < PP; ++k)
                    if (u0 + unit_of(k) >= p.real_units) dh[k] = 0.f;
            }
            if (t < 0) {
                if (good) {
#pragma unroll
                    for (int k = 0; k < PP; ++k)
                        if (valid(k)) {
                            if (p.dh0) p.dh0[state_off(k)] = dh[k];
                            if (p.dc0) p.dc0[state_off(k)] = dc[k];
                        }
                }
                break;
            }
#pragma unroll
            for (int k = 0; k < PP; ++k) {
                if (!valid(k)) continue;
                const float dcv = fmaf(dh[k], ka[k], dc[k]);
                const uint16_t di = to16<BF16>(dcv * ki[k]), df = to16<BF16>(dcv * kf[k]);
                const uint16_t dgg = to16<BF16>(dcv * kg[k]), dgo = to16<BF16>(dh[k] * ko[k]);
                dc[k] = dcv * gf[k];
                *reinterpret_cast<uint2 *>(s_dg + (db * NS + seq_of(k)) * ROW + unit_of(k) * 8) =
                    make_uint2((uint32_t)di | (uint32_t)df << 16, (uint32_t)dgg | (uint32_t)dgo << 16);
                uint16_t *out = reinterpret_cast<uint16_t *>(s_out + db * OUT) + ((unit_of(k) >> 3) * NS + seq_of(k)) * 32 + (unit_of(k) & 7);
                out[0] = di;
                out[8] = df;
                out[16] = dgg;
                out[24] = dgo;
            }
            FLSTM_CL_STAMP(s - p.s0, 6);
            cp_async_wait<kClusterAhead - 2>();  // the inputs of the next step and the cell state of the one after
            if (named_barrier_or(1, THREADS, !good)) break;
            if (s + 1 < p.s1) {
                contract_and_send(db, w & 1);
                FLSTM_CL_STAMP(s - p.s0, 4);
                fetch(s + STAGES);  // into the slot this step has read
            }
            FLSTM_CL_STAMP(s - p.s0, 8);
            write_out(t, db);
            slot = next;
        }
        if (!abort_w && p.s1 <= p.T) {  // a later launch continues from here
#pragma unroll
            for (int k = 0; k < PP; ++k)
                if (valid(k)) p.dc[state_off(k)] = dc[k];
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

using BwdKernel = void (*)(ClusterBwdParams);

struct BwdShape {
    int W, MT, NKB, KSB;
    BwdKernel kernels[2][2][2];  // NT = 1, 2; f16, bf16; fast, accurate gate functions
};
#define FLSTM_CL_K(W, MT, NKB, KSB, NT, BF) \
    {cluster_bwd_kernel<W, MT, NKB, KSB, NT, BF, false>, cluster_bwd_kernel<W, MT, NKB, KSB, NT, BF, true>}
#define FLSTM_CL_ROW(W, MT, NKB, KSB)                                                                \
    {W, MT, NKB, KSB,                                                                                \
     {{FLSTM_CL_K(W, MT, NKB, KSB, 1, false), FLSTM_CL_K(W, MT, NKB, KSB, 1, true)},                 \
      {FLSTM_CL_K(W, MT, NKB, KSB, 2, false), FLSTM_CL_K(W, MT, NKB, KSB, 2, true)}}}
// warps, 16-unit tiles and K chunks per warp, K groups: one row per width (multiple of 64) and cluster size in use
const BwdShape kBwdShapes[] = {
    FLSTM_CL_ROW(8, 1, 4, 2),    // H = 64,  1 CTA
    FLSTM_CL_ROW(8, 1, 16, 1),   // H = 128, 1 CTA
    FLSTM_CL_ROW(8, 1, 8, 1),    // H = 128, 2 CTAs
    FLSTM_CL_ROW(12, 1, 12, 1),  // H = 192, 2 CTAs
    FLSTM_CL_ROW(12, 1, 6, 1),   // H = 192, 4 CTAs
    FLSTM_CL_ROW(8, 2, 8, 1),    // H = 256, 4 CTAs
    FLSTM_CL_ROW(8, 2, 4, 1),    // H = 256, 8 CTAs
    FLSTM_CL_ROW(8, 2, 2, 1),    // H = 256, 16 CTAs
    FLSTM_CL_ROW(10, 2, 5, 1),   // H = 320, 8 CTAs
    FLSTM_CL_ROW(10, 2, 3, 1),   // H = 320, 14 of 16 CTAs
    FLSTM_CL_ROW(12, 2, 6, 1),   // H = 384, 8 CTAs
    FLSTM_CL_ROW(12, 2, 3, 1),   // H = 384, 16 CTAs
    FLSTM_CL_ROW(14, 2, 4, 1),   // H = 448, 14 of 16 CTAs
    FLSTM_CL_ROW(16, 2, 4, 1),   // H = 512, 16 CTAs
    FLSTM_CL_ROW(12, 3, 5, 1),   // H = 576, 15 of 16 CTAs
    FLSTM_CL_ROW(8, 5, 5, 1),    // H = 640, 16 CTAs
    FLSTM_CL_ROW(8, 6, 6, 1),    // H = 704, 768, 15 / 16 of 16 CTAs: with 12 warps fewer fragments fit into registers, too many for shared memory
};

const BwdShape *shape_of(const ClusterBwdPlan &pl) {
    for (const BwdShape &r : kBwdShapes)
        if (r.W == pl.W && r.MT == pl.MT && r.NKB == pl.NKB && r.KSB == pl.KSB) return &r;
    return nullptr;
}

int bwd_smem(const ClusterBwdPlan &pl) {
    const int U = 8 * pl.nub, NS = 8 * pl.NT, PP = cluster_bwd_pairs(pl.W, U, pl.NT);
    const int in_smem = pl.MT * pl.NKB - cluster_bwd_reg_frags(pl.W, pl.MT, pl.NKB, pl.NT, PP);
    return 2 * pl.peers * pl.KSB * U * NS * 4 + 2 * NS * cluster_row_bytes(pl.nub * 64) + (kClusterAhead + 1) * NS * pl.nub * 112 + 2 * NS * pl.nub * 64 +
           pl.W * in_smem * 1024;
}

}  // namespace

// Like plan_cluster_fwd over the rows of kBwdShapes; a step moves H fp32 partial sums per group of four sequences.
int plan_cluster_bwd(int B, int H, int sms, size_t smem_limit, ClusterBwdPlan *plan, const ClusterCheck *check) {
    *plan = ClusterBwdPlan{};
    if (!cluster_enabled() || H % 64 || H > 768) return FLSTM_OK;
    const char *env = std::getenv("FLSTM_CLUSTER_SIZE");
    const int only = env ? std::atoi(env) : 0;
    const int blocks = H / 8, tiles16 = H / 16;
    int slots[5];
    for (int n = 0; n < 5; ++n) slots[n] = cluster_slots(1 << n, sms);
    for (int tries = 0; tries < 8; ++tries) {
        *plan = ClusterBwdPlan{};
        const BwdShape *shape = nullptr;
        for (int n = 0; n < 5; ++n) {
            const int C = 1 << n, nub = (blocks + C - 1) / C;
            if ((only && C != only) || slots[n] < 1) continue;
            for (const BwdShape &r : kBwdShapes) {
                const int cover = r.W / r.KSB * r.MT;
                if (r.NKB * r.KSB != nub || cover < tiles16 || cover > tiles16 + r.MT * 2) continue;
                ClusterBwdPlan pl{};
                pl.C = C;
                pl.nub = nub;
                pl.peers = (blocks + nub - 1) / nub;
                pl.W = r.W;
                pl.MT = r.MT;
                pl.NKB = r.NKB;
                pl.KSB = r.KSB;
                pl.seqs = (B + slots[n] - 1) / slots[n];
                const int tiles = (pl.seqs + 7) / 8;
                if (tiles > 2) continue;  // with more the estimate below exceeds the grid-wide kernels at every width
                pl.NT = tiles <= 1 ? 1 : 2;
                pl.threads = r.W * 32;
                pl.smem_bytes = bwd_smem(pl);
                if ((size_t)pl.smem_bytes + 1024 > smem_limit) continue;
                pl.clusters = (B + pl.seqs - 1) / pl.seqs;
                const int frags = r.MT * r.NKB, chain = r.NKB * 40, pairs = cluster_bwd_pairs(r.W, 8 * nub, pl.NT);
                const int busy = (r.W + 3) / 4 * frags * pl.NT * 16;
                const int in_smem = frags - cluster_bwd_reg_frags(r.W, r.MT, r.NKB, pl.NT, pairs);
                const int incoming = pl.peers * r.KSB * nub * 8 * ((pl.seqs + 3) / 4) * 16;
                pl.cycles = (busy > chain ? busy : chain) + r.W * in_smem * 8 + (C == 1 ? 300 : 580 + 6 * C + incoming / 14) + 500 +
                            pairs * (250 + 6 * pl.peers * r.KSB) + r.MT * pl.NT * 40;
                pl.use = true;
                if (!plan->use || pl.cycles < plan->cycles) {
                    *plan = pl;
                    shape = &r;
                }
            }
        }
        if (!plan->use || !check) return FLSTM_OK;
        const int have = cluster_count(reinterpret_cast<const void *>(shape->kernels[plan->NT - 1][check->bf16][check->accurate]),
                                       plan->C, plan->threads, plan->smem_bytes);
        if (have >= plan->clusters) return FLSTM_OK;
        for (int n = 0; n < 5; ++n)
            if (plan->C == 1 << n) slots[n] = have;
    }
    plan->use = false;
    return FLSTM_OK;
}

int lstm_backward_cluster(int dtype, const ClusterBwdPlan &pl, ClusterBwdParams p, cudaStream_t s) {
    const BwdShape *r = shape_of(pl);
    if (!r) return set_error(FLSTM_ERR_UNSUPPORTED, "no cluster BPTT kernel for this plan");
    p.C = pl.C;
    p.peers = pl.peers;
    p.seqs = pl.seqs;
    p.dy_aligned = reinterpret_cast<uintptr_t>(p.dy) % 16 == 0;
    return cluster_launch(reinterpret_cast<const void *>(r->kernels[pl.NT - 1][dtype == FLSTM_DTYPE_BF16 ? 1 : 0][p.real_units ? 1 : 0]), pl.C,
                          pl.clusters * pl.C, pl.threads, pl.smem_bytes, &p, s, "cluster BPTT");
}

}  // namespace tc
}  // namespace flstm_b200
