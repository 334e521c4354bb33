// Host-side launchers of the tensor-core path kernels (tc_*.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace flstm_b200 {
namespace tc {

// D[M,N] (row pitch ldd, dtype out_dtype) = A B^T (+ bias[N]), fp32 accumulation in TMEM.
//   a_mn == false: A is (M,K) row-major with pitch lda;  a_mn == true: A is stored (K,M) with pitch lda.
//   b_mn == false: B is (N,K) row-major with pitch ldb;  b_mn == true: B is stored (K,N) with pitch ldb.
//   unperm_h != 0: output rows are written through the inverse tile-interleaved gate order (H = unperm_h).
// `err_word` is a device word the kernel sets to 1 if a bounded wait expired.
int gemm(int dtype, int out_dtype, size_t M, size_t N, size_t K, const void *A, size_t lda, bool a_mn, const void *B,
         size_t ldb, bool b_mn, void *D, size_t ldd, const float *bias, int unperm_h, unsigned int *err_word, int sms,
         cudaStream_t s, bool accumulate = false,  // accumulate (fp32 output only): D += A B^T
         float *scratch = nullptr, size_t scratch_floats = 0);  // room for split-K partial products (fp32 output)

int device_sm_count();

// ------------------------------------------------------------------ persistent recurrent forward
struct FwdPlan {
    int BT;        // sequences per batch tile (UMMA N): 32, 64 or 128
    int rt;        // row tiles (64 gate rows = 16 hidden units x 4 gates) per CTA
    int cta_rows;  // CTAs along the row-tile axis = (H/16) / rt
    int ngroups;   // batch groups (each with its own step barrier)
    int nt;        // batch tiles per group
    int stages;    // TMA ring depth
    int ch;        // 64-wide K chunks per ring stage (one TMA copy each)
    bool resident; // W_hh slice stays in shared memory for the whole sequence
    bool pair;     // neighbouring row-tile CTAs form cta_group::2 pairs; the h map then has BT/2 rows per box
    bool halves;   // the two halves of K are summed apart and added last, the order of the kernel that takes longer launches
    int smem_bytes;
    int grid;
};

// Self-test of the kernels without a step barrier: what CTA `cta` leaves out of step `step` of a launch (from 0).  The kernels have
// forms of their own for it (fp16): in the others it took 1 to 2 % of a step.
struct LostWords {
    unsigned int what;
    int step, cta;
};
// the first words of the pieces it sends (BPTT); all it sends; the count of its resets, from that step on
constexpr unsigned int kLostWord = 1, kLostPart = 2, kLostCount = 4;

// error word: a piece of dG was read before all of it was written (1 to 3: waits that expired)
constexpr unsigned int kErrTornPiece = 4;

struct FwdParams {
    float *cs;            // fp32 (T+1, B, H) cell states, slot 0 = c0
    void *hs;             // 16-bit (T+1, B, H) hidden states, slot 0 = h0
    void *y;              // optional 16-bit (T, B, H) copy of h_t for the caller
    void *gates;          // 16-bit (T, B, 4H): holds P on entry, the activated gates on exit
    unsigned int *counters;  // one step counter per batch group, zero between launches
    unsigned int *exits;     // CTAs that have left, zero between launches (leave_counters)
    void *ring;              // slots through which h_t crosses without a step barrier (tc_direct.cuh)
    unsigned int *err;    // error word: non-zero after a bounded wait expired
    int T, B, H;          // T = number of steps this launch runs
    int t0;               // first (absolute) time step of this launch; the state of step t0 is in slot t0 of hs/cs
    int store_gates;      // write the activated gates back (the gate cache)
    int known_h;          // 1: hs holds every h_t of the launch already (lstm_forward_wide only): no step waits for another's
    int odd;              // 1: the first step of this launch has an odd number in its sequence (order of streamed weights)
    // 0: fast gate functions.  > 0: accurate ones (see common.cuh), and the units from this one on are padding
    // (engine_padded.cu): their pre-activations count as zero, whatever 0 * inf made of them
    int real_units;
    long long *trace;     // optional: CTA 0 stamps clock64() at 16 points of each of the first trace_steps steps
    int trace_steps;
    unsigned long long wait_ns;   // limit of every device-side wait (0 = the 2 s default)
    unsigned int extra_arrivals;  // self-test of the timeout path: the step barrier waits for this many arrivals nobody makes
    LostWords lost;
    // filled by the launcher from the plan
    int rt, cta_rows, nt, stages, ch, halves;
    uint32_t idesc;
};

int plan_fwd(int B, int H, int sms, size_t smem_limit, FwdPlan *plan);
bool wide_tile_enabled();   // 33..64 sequences as one 64-wide batch tile when a CTA would otherwise take two
bool wider_tile_enabled();  // 65..128 sequences as one 128-wide batch tile likewise
// tm_w: W_hh rows tile-interleaved (4H, H), box 64x64, 128B swizzle.  tm_h: hidden states as a
// chunked map (make_tensor_map_chunked) with box rows BT (BT/2 for plan.pair) and plan.ch chunks.  tm_g: projection as
// (T, B, 4H), box 1 x BT x 64, no swizzle.
int lstm_forward_persistent(int dtype, const FwdPlan &plan, const CUtensorMap &tm_w, const CUtensorMap &tm_h,
                            const CUtensorMap &tm_g, FwdParams p, cudaStream_t s);

// ------------------------------------------------------------------ the same with W_hh in tensor memory (tc_lstm_fwd_tm.cu)
struct FwdTmPlan {
    bool use;
    int S;         // 2: K split over the lane halves, 64 gate rows per CTA; 1: 128 gate rows per CTA
    int BT;        // sequences per batch group
    int cta_rows;  // CTAs per batch group (row blocks)
    int ngroups;
    int kc;        // chunk-steps of 64 along K (per half for S = 2)
    int ct, cs;    // of these, kept in tensor / shared memory; the others are streamed each step
    int ch, hstages;  // chunk-steps of h per copy, copies in the ring
    int wstages;   // slots for copies of streamed W_hh (0: nothing is streamed)
    int hring;     // 0: the copies of h hold a whole tile, they need no hand-back
    bool direct;   // h_t crosses without a step barrier (tc_lstm_fwd_tm_direct.cu)
    int smem_bytes;
    int grid;
};
constexpr int kFwdTmGroup = 3;  // streamed chunk-steps per copy
int plan_fwd_tm(int B, int H, int sms, size_t smem_limit, FwdTmPlan *plan);
// tm_w: W_hh as for lstm_forward_persistent.  tm_ws: W_hh as a chunked map of one step, box rows 128, kFwdTmGroup chunks.
// tm_h: chunked map with box rows S * BT / 2 and plan.ch chunks.  tm_g: box 1 x BT x 64.
int lstm_forward_tm(int dtype, const FwdTmPlan &plan, const CUtensorMap &tm_w, const CUtensorMap &tm_ws, const CUtensorMap &tm_h,
                    const CUtensorMap &tm_g, const FwdParams &p, cudaStream_t s);

bool fits_direct(const FwdTmPlan &plan, size_t smem_limit);
size_t direct_ring_bytes(const FwdTmPlan &plan);  // FwdParams::ring
int lstm_forward_tm_direct(int dtype, const FwdTmPlan &plan, const CUtensorMap &tm_w, const CUtensorMap &tm_g, const FwdParams &p,
                           cudaStream_t s);

// ------------------------------------------------------------------ wide batches with W_hh on the chip (tc_lstm_fwd_wide.cu)
struct FwdWidePlan {
    int ch;        // 64-wide chunks of h per copy
    bool use;
    int BT;        // sequences per batch tile: 64 or 128
    int cta_rows;  // CTAs per batch group = H / 16
    int ngroups;
    int nt;        // batch tiles that a CTA takes in turn
    int kc;        // 64-wide chunks of K
    int ct, cs;    // of these, kept in tensor / shared memory (all of them)
    int hstages;   // copies of h in the ring
    int smem_bytes;
    int grid;
};
constexpr int kMaxStepCounters = 900;  // words of Engine::sync_words that step barriers may take
int plan_fwd_wide(int B, int H, int sms, size_t smem_limit, FwdWidePlan *plan);
// tm_w: make_tensor_map_gate_rows.  tm_h: chunked map with box rows BT / 2 and plan.ch chunks.
int lstm_forward_wide(int dtype, const FwdWidePlan &plan, const CUtensorMap &tm_w, const CUtensorMap &tm_h, const FwdParams &p,
                      cudaStream_t s);

// ------------------------------------------------------------------ persistent BPTT
struct BwdPlan {
    int BT;        // sequences per batch tile
    int KS;        // cluster size: CTAs that split the K = 4H contraction of one 64-unit tile
    int jt;        // unit tiles = H / 64
    int ngroups, nt, stages;
    int ch;        // 64-wide K chunks per ring stage (one TMA copy each)
    bool resident;
    bool halves;   // as in FwdPlan, of a CTA's part of K
    int smem_bytes;
    int grid;
};

struct BwdParams {
    const float *cs;      // fp32 (T+1, B, H) cell states from the forward
    const void *gates;    // 16-bit (T, B, 4H) post-activation gate cache, tile-interleaved columns
    void *dg;             // 16-bit (T, B, 4H) pre-activation gradients (written), same column order
    const void *dy;       // 16-bit (T, B, H)
    const void *dhn;      // 16-bit (B, H) or null
    const void *dcn;      // 16-bit (B, H) or null
    float *dh0, *dc0;     // fp32 (B, H) or null
    float *dc;            // fp32 (B, H) scratch for the cell-gradient carry (used when nt > 1)
    unsigned int *counters, *exits;  // as in FwdParams
    void *ring;           // as in FwdParams, of dG
    unsigned int *err;
    int real_units;       // as in FwdParams; a padding unit's dh counts as zero
    long long *trace;     // optional per-step clock64() stamps of CTA 0 (see FwdParams)
    int trace_steps;
    int T, B, H;          // T = length of the whole sequence
    int s0, s1;           // reverse iterations [s0, s1) of this launch; iteration s is time T-1-s, s == T writes dh0/dc0
    unsigned long long wait_ns;   // limit of every device-side wait (0 = the 2 s default)
    unsigned int extra_arrivals;  // self-test of the timeout path (see FwdParams)
    LostWords lost;
    int jt, nt, stages, ch, halves;
    uint32_t idesc;
};

// check_device: verify with the occupancy query of the CURRENT device that all clusters of the grid are resident
// at once (shrinking the number of batch groups if need be) and fail when they are not; false = host arithmetic only.
int plan_bwd(int B, int H, int sms, size_t smem_limit, BwdPlan *plan, bool check_device = true);
// tm_w: the same map as the forward's (W_hh rows tile-interleaved, 64x64 boxes): the BPTT reads the
// slice as an MN-major operand.  tm_dg: dG as a chunked map (make_tensor_map_chunked) of width 4H
// with box rows BT and plan.ch chunks.
int lstm_backward_persistent(int dtype, const BwdPlan &plan, const CUtensorMap &tm_w, const CUtensorMap &tm_dg,
                             BwdParams p, cudaStream_t s);

// ------------------------------------------------------------------ the same with W_hh in tensor memory (tc_lstm_bwd_tm.cu)
struct BwdTmPlan {
    bool use;
    int BT;        // sequences per batch group
    int jt;        // unit tiles = H / 64, a cluster of four CTAs each
    int ngroups;
    int nt;        // batch tiles that a cluster takes in turn
    int kp;        // chunk-steps of 64 per half of a CTA's K range
    int left;      // 1: the range has an odd number of chunks, the last one runs by itself
    int ct, cs;    // chunk-steps of W_hh in tensor / shared memory (all of them)
    int ch, stages;  // chunk-steps of dG per copy, copies in the ring
    int ring;      // 0: the copies hold a whole tile, they need no hand-back
    bool direct;   // dG_t crosses without a step barrier (tc_lstm_bwd_tm_direct.cu)
    int smem_bytes;
    int grid;
};
struct BwdTmMaps {
    CUtensorMap half[4];  // dG from the K range of each CTA of a cluster on (make_tensor_map_halves)
    CUtensorMap chunk;    // single chunks of dG (make_tensor_map_chunked)
};
int plan_bwd_tm(int B, int H, int sms, size_t smem_limit, BwdTmPlan *plan, bool check_device);
int make_bwd_tm_maps(BwdTmMaps *maps, const BwdTmPlan &plan, const void *dg, size_t steps, size_t B, size_t H);
int lstm_backward_tm(int dtype, const BwdTmPlan &plan, const CUtensorMap &tm_w, const BwdTmMaps &maps, const BwdParams &p,
                     cudaStream_t s);
bool fits_direct(const BwdTmPlan &plan, size_t smem_limit);
size_t direct_ring_bytes(const BwdTmPlan &plan);  // BwdParams::ring
int max_clusters_direct(const BwdTmPlan &plan);   // that the current device holds at once, or -1
int lstm_backward_tm_direct(int dtype, const BwdTmPlan &plan, const CUtensorMap &tm_w, const BwdParams &p, cudaStream_t s);

// ------------------------------------------------------------------ wide-batch path: one GEMM launch per step
struct StepPlan {
    bool use;     // the engine takes this path instead of the persistent kernels
    int bn_fwd;   // output-tile width of the forward step GEMM (gate columns): 64, 128 or 256
    int bn_bwd;   // output-tile width of the backward step GEMM (hidden units): 128 or 256
    int splits;   // K = 4H splits of the backward step GEMM (fp32 partial sums, added by the pointwise kernel)
    bool pair;    // tiles of 256 sequences on CTA pairs (cta_group::2); the forward W_hh map then has bn_fwd / 2 rows per box
    bool bwd_pair;        // the backward split-K GEMM runs on CTA pairs (256-sequence tiles)
    bool fwd_persistent;  // forward: one cooperative launch per range of steps (lstm_wide_forward) instead of one per step
    bool fwd_pair;        // that launch runs on CTA pairs (256-sequence tiles); the forward W_hh map has bn_fwd / 2 rows per box
};

struct StepFwdParams {
    unsigned int *err;
    int t;            // absolute time step: h_{t-1} / c_{t-1} in slot t of the state tensors, results in slot t+1
    int B, H;
    int store_gates;  // overwrite the projection with the activated gates (the gate cache)
    int real_units;   // as in FwdParams
};

// Tensor maps of the forward step kernel.  Operands: hs (T+1, B, H) as a 3-D map with 1 x 128 x 64 boxes and
// W_hh (rows tile-interleaved, (4H, H)) with plan.bn_fwd x 64 boxes (plan.bn_fwd / 2 x 64 for CTA pairs), both 128B-swizzled.  Epilogue tiles
// (make_tensor_map_3d_tile, 32-row boxes): gates (T, B, 4H) 64 columns wide, cs (T+1, B, H) fp32 16 wide,
// hs_out (T+1, B, H) 16 wide, y = the caller's (T, B, H) output 16 wide or null.
struct StepFwdMaps {
    const CUtensorMap *hs, *w, *gates, *cs, *hs_out, *y;
};

// All steps [t0, t0 + nsteps) of the forward step GEMM in ONE cooperative launch: the CTAs keep their output tiles,
// a counter barrier in global memory separates the steps (same tensor maps as lstm_step_forward).
struct WideFwdParams {
    unsigned int *err;
    unsigned int *counter, *exits;  // zero between launches
    int t0, nsteps;
    int B, H;
    int store_gates;
    int real_units;
    unsigned long long wait_ns;
    unsigned int extra_arrivals;
};
int lstm_wide_forward(int dtype, const StepPlan &plan, const StepFwdMaps &m, const WideFwdParams &p, int sms, cudaStream_t s);

int plan_step(int B, int H, int sms, size_t smem_limit, StepPlan *plan);
int lstm_step_forward(int dtype, const StepPlan &plan, const StepFwdMaps &m, const StepFwdParams &p, int sms,
                      cudaStream_t s);
// parts[s] (B,H) fp32 = dG_t[:, K slice s] W_hh[K slice s, :].  tm_dg: dG (T, B, 4H) as a 3-D map, box
// 1 x 128 x 64, 128B swizzle.  tm_w64: W_hh (4H, H) with 64 x 64 boxes (read as an MN-major operand).
int lstm_step_backward_gemm(int dtype, const StepPlan &plan, const CUtensorMap &tm_dg, const CUtensorMap &tm_w64, int t,
                            int B, int H, float *parts, unsigned int *err, int sms, cudaStream_t s);
// dG_t and the cell-gradient carry from dh = dy_t + sum(parts[0..nparts)), the gate cache and the cell states.
int lstm_step_backward_pointwise(int dtype, const void *gates_t, const float *c_t, const float *c_prev, const void *dy_t,
                                 const float *parts, int nparts, float *dc, void *dg_t, int B, int H, int real_units, cudaStream_t s);
int sum_parts(const float *parts, int nparts, size_t n, float *out, cudaStream_t s);

// One time step of one layer in one launch (tc_cell.cu); B <= 32, 16-byte aligned x and h_prev.
struct CellParams {
    const void *w_ih, *w_hh;  // 16-bit, rows tile-interleaved: (4H, I), (4H, H)
    const float *bias;        // (4H), same order
    const void *x;            // (B, I)
    const void *h_prev;       // (B, H) or null: zeros
    const void *c_prev;       // (B, H) fp32 or 16-bit, or null: zeros
    void *h_out;              // (B, H)
    float *c_out;             // (B, H)
    void *y, *hn, *cn;        // optional further copies for the caller
    void *h_first;            // where the state that enters a sequence is kept, or null
    float *c_first;
    int c_prev_f32, cn_f32;
    int B, I, H;
    int real_units;           // as in FwdParams
    int follows;              // the launch before it in the stream is another cell step of the same call
};
constexpr int kCellBatch = 32;
int lstm_cell_step(int dtype, const CellParams &p, cudaStream_t s);

// One matrix of one layer from fp32 torch order (4H, K) to the 16-bit tile-interleaved order (4Hp, Kp), padding zero;
// with b_ih / b_hh also the layer's summed bias (4Hp).  One launch packs up to kPackJobs of them.
struct PackJob {
    const float *w;
    void *out;
    const float *b_ih, *b_hh;
    float *bias;
    int H, Hp, K, Kp;
};
constexpr int kPackJobs = 16;
int pack_weights(int dtype, const PackJob *jobs, int count, cudaStream_t s);

}  // namespace tc
}  // namespace flstm_b200
