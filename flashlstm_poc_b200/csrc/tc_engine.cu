// Tensor-core (tcgen05 / TMEM / TMA) path of the engine: planning, tensor maps, weight packing in
// the tile-interleaved gate order, and the per-layer forward / backward schedules.
//
// Gate order.  Every 4H-indexed tensor of this path (rows of W_ih and W_hh, the bias, the columns
// of the projection / gate cache and of dG) uses the tile-interleaved order
//     index(g, u) = ((u / 16) * 4 + g) * 16 + u % 16
// so that the 64 rows a recurrent CTA owns are the four gates of 16 hidden units.  Weight and bias
// gradients are written back in torch order (g*H + u) by the GEMM epilogue / a small kernel.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "kernels.h"
#include "tc_cluster.cuh"
#include "tc_common.cuh"
#include "tc_kernels.h"

namespace flstm_b200 {
namespace tc {

namespace {

struct TcLayer {
    CUtensorMap tm_w;   // w_hh (4H, H), 64x64 boxes, 128B swizzle
    CUtensorMap tm_h;   // hs (Tcap+1, B, H), 1 x BT x 64 boxes, 128B swizzle
    CUtensorMap tm_g;   // gates (Tcap, B, 4H), 1 x BT x 64 boxes, no swizzle
    CUtensorMap tm_dg;  // dG (Tcap, B, 4H), 1 x BT x 64 boxes, 128B swizzle (BPTT operand)
    CUtensorMap tm_h_tm, tm_g_tm;  // hs and gates with the boxes of the tensor-memory forward kernels
    CUtensorMap tm_ws;  // w_hh, 128 x 64 boxes (streamed part of the tensor-memory forward), or its gate-row form (wide forward)
    BwdTmMaps dg_tm;    // dG for the tensor-memory BPTT kernel
    // wide-batch path (one GEMM launch per step)
    CUtensorMap tm_hs3;    // hs (Tcap+1, B, H), 1 x 128 x 64 boxes, 128B swizzle
    CUtensorMap tm_wstep;  // w_hh (4H, H), bn_fwd x 64 boxes, 128B swizzle
    CUtensorMap tm_dg3;    // dG (Tcap, B, 4H), 1 x 128 x 64 boxes, 128B swizzle
    CUtensorMap tm_g_ep, tm_c_ep, tm_h_ep;  // 32-row epilogue tiles of gates / cs / hs
};

struct TcState {
    int sms = 0;
    size_t smem_limit = 0;
    FwdPlan fwd{};
    FwdTmPlan fwdtm{};
    FwdWidePlan wide{};
    BwdPlan bwd{};
    BwdTmPlan bwdtm{};
    size_t fwd_from = 0, bwd_from = 0;  // launches of fewer steps run without tensor memory
    bool bwd_ok = false;
    StepPlan step{};
    ClusterFwdPlan cfwd{};
    ClusterBwdPlan cbwd{};
    void *ring = nullptr;       // slots of the kernels that exchange without a step barrier
    float *dh_parts = nullptr;  // wide-batch path: fp32 (L, splits, B, H) partial sums of dG_t W_hh
    float *dw_parts = nullptr;  // split-K partial products of the weight-gradient GEMMs
    size_t dw_floats = 0, dw_layers = 1;
    std::vector<TcLayer> layers;
    unsigned int *err_host = nullptr;  // pinned mirror of the device error word
};

// Estimated cycles per step above which the grid-wide schedules are faster.  Measured crossings: H = 640 at 64 sequences
// in both directions; beyond 64 sequences the grid-wide forward takes a fifth longer itself (512 x 128 still wins).
constexpr int grid_fwd_cycles(int B) { return B <= 64 ? 5600 : 6500; }
constexpr int kGridBwdCycles = 6500;
// The same where the grid-wide kernel exchanges without a step barrier.  us a step in clusters / that way (estimated cycles):
//   forward   H = 448, B = 112 2.16 / 2.40 (below 4000)   H = 512, B = 96 2.16 / 2.40 (3988)   H = 704, B = 48 2.48 / 2.43 (4560)
//             H = 576, B = 56 / 64 / 96 / 112 2.24 / 2.36 (3842), 3.22 / 2.37 (5230), 3.48 / 2.47 (5560), 3.65 / 2.56
//             H = 640, B = 96 3.76 / 2.55 (6040)   H = 768, B = 32 / 40 / 48 2.48 / 2.40 (4692), 2.58 / 2.47 (4802), 2.66 / 2.46 (4912)
//   backward  H = 512, B = 112 3.78 / 3.76 (5302)   H = 576, B = 64 / 80 4.26 / 3.79, 4.44 / 3.94 (6169)   H = 768, B = 48 3.49 / 3.78 (6039)
// The line is drawn up to 112 sequences; above, batches stay with the schedule of several tiles per cluster, whose tests hold shapes
// there (H = 512, B = 128: 3.49 / 2.47).
constexpr int kDirectBatch = 112, kDirectFwdCycles = 4850, kDirectBwdCycles = 6100;

constexpr int kExitsWord = 1000;  // of Engine::sync_words: CTAs of the running launch that have left (see leave_counters)

TcState *state(Engine &e) { return static_cast<TcState *>(e.tc_state); }

// The kernel of a launch of n steps.
enum class Kind { Cluster, Tmem, Wide, Steps, Grid };
Kind fwd_kind(const TcState &st, size_t n) {
    if (st.cfwd.use) return Kind::Cluster;
    if (n >= st.fwd_from && st.wide.use) return Kind::Wide;
    if (n >= st.fwd_from && st.fwdtm.use) return Kind::Tmem;
    return st.step.use && !st.fwdtm.use ? Kind::Steps : Kind::Grid;
}
Kind bwd_kind(const TcState &st, size_t n) {
    if (st.cbwd.use) return Kind::Cluster;
    if (st.bwdtm.use) return n >= st.bwd_from ? Kind::Tmem : Kind::Grid;
    return st.step.use ? Kind::Steps : Kind::Grid;
}

struct PackJobs {
    PackJob job[kPackJobs];
};

// A warp packs one output row: 16-byte stores of 8 columns per lane, 32-byte loads where the source row allows them.
// One launch for both matrices of up to 8 layers: three launches per layer with one element per thread took 14 us per
// 4096 x 1024 matrix and more than the whole recurrence of a small model.
template <typename T>
__global__ void __launch_bounds__(256) pack_weights_kernel(const __grid_constant__ PackJobs jobs) {
    const PackJob &j = jobs.job[blockIdx.y];
    const int lane = threadIdx.x & 31, rows = 4 * j.Hp;
    const bool vec = j.K % 4 == 0 && (reinterpret_cast<uintptr_t>(j.w) & 15) == 0;
    for (int r = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); r < rows; r += (int)(gridDim.x * (blockDim.x >> 5))) {
        const int u = (r >> 6) * 16 + (r & 15), row = ((r >> 4) & 3) * j.H + u;
        const bool real = u < j.H;
        const float *src = j.w + (size_t)row * j.K;
        T *dst = static_cast<T *>(j.out) + (size_t)r * j.Kp;
        for (int k = lane * 8; k < j.Kp; k += 256) {
            float v[8];
            if (real && vec && k + 8 <= j.K) {
                const float4 a = *reinterpret_cast<const float4 *>(src + k), b = *reinterpret_cast<const float4 *>(src + k + 4);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
                v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = real && k + e < j.K ? src[k + e] : 0.f;
            }
            __align__(16) T o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) st(o + e, v[e]);
            *reinterpret_cast<uint4 *>(dst + k) = *reinterpret_cast<const uint4 *>(o);
        }
        if (lane == 0 && j.bias) j.bias[r] = real ? j.b_ih[row] + j.b_hh[row] : 0.f;
    }
}

int check_launch(const char *what) {
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(err));
    return FLSTM_OK;
}

inline char *byte_ptr(void *p) { return static_cast<char *>(p); }
inline const char *byte_ptr(const void *p) { return static_cast<const char *>(p); }

}  // namespace

int pack_weights(int dtype, const PackJob *jobs, int count, cudaStream_t s) {
    for (int first = 0; first < count; first += kPackJobs) {
        PackJobs args{};
        const int n = count - first < kPackJobs ? count - first : kPackJobs;
        int rows = 0;
        for (int i = 0; i < n; ++i) {
            args.job[i] = jobs[first + i];
            if (4 * jobs[first + i].Hp > rows) rows = 4 * jobs[first + i].Hp;
        }
        const dim3 grid((rows + 7) / 8 < 1184 ? (rows + 7) / 8 : 1184, n);
        if (dtype == FLSTM_DTYPE_F16) pack_weights_kernel<__half><<<grid, 256, 0, s>>>(args);
        else pack_weights_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(args);
        FLSTM_TRY(check_launch("pack_weights"));
    }
    return FLSTM_OK;
}

bool supported(const flstm_engine_config &cfg) {
    if (cfg.dtype != FLSTM_DTYPE_F16 && cfg.dtype != FLSTM_DTYPE_BF16) return false;
    if (cfg.hidden_size % 64 || cfg.input_size % 8) return false;
    const char *off = std::getenv("FLSTM_DISABLE_TC");
    if (off && off[0] == '1') return false;
    int dev = 0, major = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (major != 10) return false;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    StepPlan sp;
    if (plan_step((int)cfg.batch, (int)cfg.hidden_size, device_sm_count(), (size_t)optin, &sp) == FLSTM_OK && sp.use) return true;
    FwdPlan fp;
    if (plan_fwd((int)cfg.batch, (int)cfg.hidden_size, device_sm_count(), (size_t)optin, &fp) != FLSTM_OK) return false;
    if (cfg.training) {
        BwdPlan bp;
        if (plan_bwd((int)cfg.batch, (int)cfg.hidden_size, device_sm_count(), (size_t)optin, &bp) != FLSTM_OK) return false;
    }
    return true;
}

// The kernels with W_hh in tensor memory for a shape, and the launches they take.  Moving W_hh there takes 2 us of a launch (BPTT
// 2 to 4 us), which few steps do not repay; where the other kernels exist in a good form (H % 128 == 0, one batch tile) they
// keep short launches.  Those then sum the halves of K apart, so that a sequence cut into ranges or segments of any length
// gives the bits of one launch.  Calls of n steps in us, other kernels -> these:
//   forward, n = 1 / 2 / 4 / 8 / 16 / 24:
//     without a step barrier
//     H = 1024, B = 32   23.5 / 25.7 / 33.3 / 47.2 / 73.8 / 102.5 -> 23.6 / 27.7 / 32.9 / 43.0 / 62.1 / 83.2
//     H = 1024, B = 64   23.6 / 26.5 / 34.9 / 48.3 / 77.9 / 107.3 -> 23.6 / 28.6 / 33.8 / 43.7 / 65.4 / 87.1
//     H = 1152, B = 20   23.6 / 25.7 / 33.9 / 48.3 / 75.8 / 103.1 -> 23.6 / 27.7 / 31.9 / 43.1 / 63.5 / 84.1
//     H = 2048, B = 32   24.6 / 30.8 / 40.7 / 59.7 / 102.2 / 143.8 -> 27.8 / 30.8 / 36.9 / 51.2 / 78.2 / 107.9
//     with one
//     H = 2048, B = 40, one tile of 64   26.7 / 31.4 / 43.1 / 67.6 / 115.0 / 160.9 -> 28.7 / 32.8 / 44.2 / 67.6 / 112.5 / 154.1
//     H = 2048, B = 256, tiles in turn   35.9 / 53.2 / 84.6 / 154 / 282 / 404 -> 37.2 / 48.7 / 71.9 / 125 / 214 / 297
//   backward, n = 1 / 2 / 4 / 8 / 16:
//     without a step barrier
//     H = 896, B = 60    61.2 / 64.1 / 77.2 / 96.1 / 131.4 -> 63.3 / 66.5 / 76.9 / 90.7 / 119.3
//     H = 1024, B = 32   56.3 / 62.0 / 70.1 / 90.8 / 127.0 -> 59.3 / 62.3 / 70.1 / 86.5 / 113.0
//     H = 1024, B = 64   60.2 / 64.1 / 76.3 / 96.7 / 139.2 -> 62.5 / 65.2 / 76.3 / 91.3 / 124.8
//     H = 1280, B = 32   73.3 / 77.6 / 88.0 / 111.7 / 153.7 -> 76.5 / 80.1 / 87.8 / 105.6 / 138.6
//     with one
//     H = 1280, B = 60   73.2 / 81.9 / 95.3 / 127.0 / 184.2 -> 75.3 / 83.8 / 94.7 / 123.0 / 172.6
//     H = 2048, B = 5    103.1 / 106.2 / 120.3 / 144.7 / 196.4 -> 104.1 / 107.5 / 117.6 / 139.3 / 180.2
//     tiles in turn, H = 1024, B = 140   70.7 / 81.5 / 104 / 149 / 238 -> 68.0 / 77.0 / 92.3 / 123 / 182
// The lines below were drawn for the kernels with a step barrier.  Without one the times cross at 3 to 4 steps in either direction:
// launches of 4 steps forward and of 5 to 11 backward (H <= 1024) take 1 to 7 % longer than they would on these kernels.
static int choose_tmem(int B, int H, bool fwd, bool bwd, int sms, size_t smem_limit, bool check_device, TcState *st) {
    const bool good = H % 128 == 0;
    if (fwd) {
        FLSTM_TRY(plan_fwd_tm(B, H, sms, smem_limit, &st->fwdtm));
        // 33 to 64 sequences per batch group: the K halves make an UMMA of N = 128, which takes longer than the other
        // kernel's of N = 64 (H = 512, B = 250: 4.15 against 3.97 us a step; H = 640, B = 130: 4.16 against 3.98), so that one
        // stays where its weights are resident and a CTA has one batch tile; beyond that the gain per step is small
        FwdPlan f{};
        const bool single = plan_fwd(B, H, sms, smem_limit, &f) == FLSTM_OK && f.nt == 1, fits_one = st->fwdtm.use;
        if (st->fwdtm.BT == 64 && single && f.resident && f.BT <= 64) st->fwdtm.use = false;
        if (st->fwdtm.use && st->fwdtm.S == 2 && good && single && f.pair && f.BT <= 64) {
            st->fwd_from = st->fwdtm.BT == 64 ? 12 : 5;
            st->fwd = f;
            st->fwd.halves = true;
        }
        if (!fits_one) {
            FLSTM_TRY(plan_fwd_wide(B, H, sms, smem_limit, &st->wide));
            if (st->wide.use) st->fwd_from = 2;
        }
    }
    if (bwd) {
        FLSTM_TRY(plan_bwd_tm(B, H, sms, smem_limit, &st->bwdtm, check_device));
        BwdPlan b{};
        if (st->bwdtm.use && good && st->bwdtm.nt == 1 && plan_bwd(B, H, sms, smem_limit, &b, check_device) == FLSTM_OK &&
            b.nt == 1 && b.KS == 4 && b.BT <= 64) {
            st->bwd_from = H <= 1024 ? 12 : 4;
            st->bwd = b;
            st->bwd.halves = true;
        }
    }
    return FLSTM_OK;
}

int init(Engine &e) {
    TcState *st = new TcState();
    e.tc_state = st;
    st->sms = device_sm_count();
    int optin = 0;
    FLSTM_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, e.device));
    st->smem_limit = (size_t)optin;
    const int B = (int)e.cfg.batch, H = (int)e.cfg.hidden_size;
    // Each direction takes the cluster-resident kernel while its estimated step is shorter than the grid-wide ones'.
    // FLSTM_STEP_MIN_BATCH asks for one of the grid-wide schedules by name.
    if (!std::getenv("FLSTM_STEP_MIN_BATCH")) {
        // the cross-layer wavefront would put two cooperative grids side by side
        const char *wave = std::getenv("FLSTM_WAVE_CHUNK");
        const bool wavefront = wave && std::atoi(wave) > 0;
        const ClusterCheck check{e.cfg.dtype == FLSTM_DTYPE_BF16, e.logical_h > 0};
        // (the other plan is made only where it decides: it asks the device about its kernel, which loads it)
        const bool direct = !wavefront && B <= kDirectBatch;
        FLSTM_TRY(plan_cluster_fwd(B, H, st->sms, st->smem_limit, &st->cfwd, &check));
        if (st->cfwd.cycles > grid_fwd_cycles(B)) st->cfwd.use = false;
        if (st->cfwd.use && st->cfwd.cycles > kDirectFwdCycles && direct) {
            FwdTmPlan other{};
            FLSTM_TRY(plan_fwd_tm(B, H, st->sms, st->smem_limit, &other));
            if (other.use && other.direct) st->cfwd.use = false;
        }
        if (e.cfg.training) {
            FLSTM_TRY(plan_cluster_bwd(B, H, st->sms, st->smem_limit, &st->cbwd, &check));
            if (st->cbwd.cycles > kGridBwdCycles) st->cbwd.use = false;
            if (st->cbwd.use && st->cbwd.cycles > kDirectBwdCycles && direct) {
                BwdTmPlan other{};
                FLSTM_TRY(plan_bwd_tm(B, H, st->sms, st->smem_limit, &other, /*check_device=*/true));
                if (other.use && other.direct) st->cbwd.use = false;
            }
        }
        if (!wavefront)
            FLSTM_TRY(choose_tmem(B, H, !st->cfwd.use, e.cfg.training && !st->cbwd.use, st->sms, st->smem_limit, /*check_device=*/true, st));
    }
    const bool tm_fwd = st->fwdtm.use || st->wide.use;
    const bool grid_fwd = !st->cfwd.use && !tm_fwd, grid_bwd = e.cfg.training && !st->cbwd.use && !st->bwdtm.use;
    const bool short_wide = st->wide.use && st->fwd_from > 1;
    st->bwd_ok = e.cfg.training != 0;
    if (grid_fwd || grid_bwd || short_wide) FLSTM_TRY(plan_step(B, H, st->sms, st->smem_limit, &st->step));
    if (short_wide && !st->step.use && plan_fwd(B, H, st->sms, st->smem_limit, &st->fwd) != FLSTM_OK) st->fwd_from = 0;
    if (st->step.use && grid_bwd) {
        const size_t n = e.layers.size() * (size_t)st->step.splits * e.cfg.batch * e.cfg.hidden_size;
        e.fixed.want(&st->dh_parts, n * sizeof(float));
    }
    if (!st->step.use && grid_fwd) FLSTM_TRY(plan_fwd(B, H, st->sms, st->smem_limit, &st->fwd));
    if (!st->step.use && grid_bwd) FLSTM_TRY(plan_bwd(B, H, st->sms, st->smem_limit, &st->bwd));
    if (e.cfg.training) {  // a split GEMM has at most one 128 x 128 tile per SM
        st->dw_floats = (size_t)st->sms * 128 * 128;
        // one per layer where the cross-layer wavefront can run two layers' GEMMs at once
        st->dw_layers = st->step.use && !tm_fwd && !st->bwdtm.use ? e.layers.size() : 1;
        e.fixed.want(&st->dw_parts, st->dw_layers * st->dw_floats * sizeof(float));
    }
    if (const size_t bytes = std::max(direct_ring_bytes(st->fwdtm), direct_ring_bytes(st->bwdtm))) e.fixed.want(&st->ring, bytes);
    st->layers.resize(e.layers.size());
    // one bias-gradient scratch per layer: with the cross-layer wavefront two layers may reduce at once
    if (e.cfg.training) e.fixed.want(&e.db_part, e.layers.size() * (size_t)simt::column_sum_scratch_floats(4 * e.cfg.hidden_size) * sizeof(float));
    st->err_host = host_word_acquire();
    if (!st->err_host) return set_error(FLSTM_ERR_CUDA, "pinned allocation failed");
    return FLSTM_OK;
}

void destroy(Engine &e) {
    TcState *st = state(e);
    if (!st) return;
    host_word_release(st->err_host);
    delete st;
    e.tc_state = nullptr;
}

int on_capacity_change(Engine &e) {
    TcState *st = state(e);
    // time extent of the gate-sized buffers (one segment with activation checkpoints); dG has one slot more then
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, cap = e.buf_steps, dg_steps = cap + (e.recompute ? 1 : 0);
    for (size_t li = 0; li < e.layers.size(); ++li) {
        auto &l = e.layers[li];
        auto &t = st->layers[li];
        const bool bwd = e.cfg.training && l.dg;
        const bool grid_fwd = st->fwd.BT > 0, grid_bwd = bwd && st->bwd.BT > 0, step_bwd = bwd && bwd_kind(*st, 1) == Kind::Steps;
        if (st->cfwd.use && (!e.cfg.training || st->cbwd.use)) continue;  // the cluster kernels use plain loads
        FLSTM_TRY(make_tensor_map_2d(&t.tm_w, l.w_hh, 4 * H, H, H, 64, 64, true));
        if (bwd && st->bwdtm.use && !st->bwdtm.direct) FLSTM_TRY(make_bwd_tm_maps(&t.dg_tm, st->bwdtm, l.dg, dg_steps, B, H));
        if (st->wide.use) {
            FLSTM_TRY(make_tensor_map_gate_rows(&t.tm_ws, l.w_hh, H));
            FLSTM_TRY(make_tensor_map_chunked(&t.tm_h_tm, l.hs, cap + 1, B, H, st->wide.BT / 2, st->wide.ch));
        }
        if (st->fwdtm.use) {
            if (!st->fwdtm.direct)
                FLSTM_TRY(make_tensor_map_chunked(&t.tm_h_tm, l.hs, cap + 1, B, H, st->fwdtm.S * st->fwdtm.BT / 2, st->fwdtm.ch));
            FLSTM_TRY(make_tensor_map_3d(&t.tm_g_tm, l.gates, cap, B, 4 * H, 4 * H, B * 4 * H, st->fwdtm.BT, 64, false));
            if (st->fwdtm.wstages) FLSTM_TRY(make_tensor_map_chunked(&t.tm_ws, l.w_hh, 1, 4 * H, H, 128, kFwdTmGroup));
        }
        if (st->step.use) {
            FLSTM_TRY(make_tensor_map_3d(&t.tm_hs3, l.hs, cap + 1, B, H, H, B * H, 128, 64, true));
            FLSTM_TRY(make_tensor_map_2d(&t.tm_wstep, l.w_hh, 4 * H, H, H, (st->step.pair || st->step.fwd_pair) ? st->step.bn_fwd / 2 : st->step.bn_fwd, 64, true));
            FLSTM_TRY(make_tensor_map_3d_tile(&t.tm_g_ep, l.gates, 2, cap, B, 4 * H, 32, 64));
            FLSTM_TRY(make_tensor_map_3d_tile(&t.tm_c_ep, l.cs, 4, cap + 1, B, H, 32, 16));
            FLSTM_TRY(make_tensor_map_3d_tile(&t.tm_h_ep, l.hs, 2, cap + 1, B, H, 32, 16));
            if (step_bwd)
                FLSTM_TRY(make_tensor_map_3d(&t.tm_dg3, l.dg, dg_steps, B, 4 * H, 4 * H, B * 4 * H, 128, 64, true));
        }
        if (grid_fwd) {
            FLSTM_TRY(make_tensor_map_chunked(&t.tm_h, l.hs, cap + 1, B, H, st->fwd.pair ? st->fwd.BT / 2 : st->fwd.BT, st->fwd.ch));
            FLSTM_TRY(make_tensor_map_3d(&t.tm_g, l.gates, cap, B, 4 * H, 4 * H, B * 4 * H, st->fwd.BT, 64, false));
        }
        if (grid_bwd)
            FLSTM_TRY(make_tensor_map_chunked(&t.tm_dg, l.dg, dg_steps, B, 4 * H, st->bwd.BT, st->bwd.ch));
    }
    return FLSTM_OK;
}

int set_weights(Engine &e, int first, int count, const float *const *params, cudaStream_t s) {
    std::vector<PackJob> jobs;
    const int Hp = (int)e.cfg.hidden_size, H = e.logical_h ? e.logical_h : Hp;
    for (int li = first; li < first + count; ++li, params += 4) {
        auto &l = e.layers[li];
        const int Kp = (int)l.in_size, K = !e.logical_h ? Kp : li == 0 ? e.logical_in : H;
        jobs.push_back({params[0], l.w_ih, params[2], params[3], l.bias, H, Hp, K, Kp});
        jobs.push_back({params[1], l.w_hh, nullptr, nullptr, nullptr, H, Hp, H, Hp});
    }
    e.launches += (jobs.size() + kPackJobs - 1) / kPackJobs;
    return pack_weights(e.cfg.dtype, jobs.data(), (int)jobs.size(), s);
}

// Deferred error reporting: the device error word is mirrored into pinned host memory at the end of every call (by the
// launch that copies the final states, see CopyBatch); a non-zero mirror fails the NEXT call.
static int check_async_error(Engine &e) {
    TcState *st = state(e);
    if (st && *st->err_host) {
        const unsigned int code = *st->err_host;
        *st->err_host = 0;
        cudaMemset(e.sync_words, 0, sizeof(unsigned int));
        return set_error(FLSTM_ERR_TIMEOUT, code == kErrTornPiece ? "a piece of dG was read before all of it was written (code %u)"
                                                                  : "a bounded device-side wait expired in a persistent kernel (code %u)", code);
    }
    return FLSTM_OK;
}

int poll_error(Engine &e) { return check_async_error(e); }

unsigned int *error_mirror(Engine &e) { return state(e)->err_host; }

int recurrent_path(const Engine &e, bool backward, int *ctas, int *seqs) {
    const TcState *st = static_cast<const TcState *>(e.tc_state);
    const bool cluster = backward ? st->cbwd.use : st->cfwd.use;
    *ctas = !cluster ? 0 : backward ? st->cbwd.C : st->cfwd.C;
    *seqs = !cluster ? 0 : backward ? st->cbwd.seqs : st->cfwd.seqs;
    if (cluster) return FLSTM_PATH_CLUSTER;
    if (!st->step.use || (backward ? st->bwdtm.use : st->fwdtm.use || st->wide.use)) return FLSTM_PATH_GRID;
    return !backward && st->step.fwd_persistent && wavefront_chunk(e, (size_t)-1) == 0 ? FLSTM_PATH_GRID : FLSTM_PATH_STEPS;
}

void recurrent_kernel(const Engine &e, bool backward, size_t steps, flstm_kernel_info *out) {
    const TcState &st = *static_cast<const TcState *>(e.tc_state);
    if (!backward) {
        switch (fwd_kind(st, steps)) {
            case Kind::Cluster: *out = {"cluster_fwd_kernel", 0, st.cfwd.seqs, 1, 0, 0}; break;
            case Kind::Wide: *out = {"lstm_fwd_wide_kernel", 0, st.wide.BT, st.wide.nt, st.wide.ngroups, 0}; break;
            case Kind::Tmem: *out = {"lstm_fwd_tm_kernel", 0, st.fwdtm.BT, 1, st.fwdtm.ngroups, st.fwdtm.wstages > 0}; break;
            case Kind::Steps:
                if (st.step.fwd_persistent && wavefront_chunk(e, (size_t)-1) == 0) *out = {"wide_fwd_kernel", 0, 0, 1, 0, 1};
                else *out = {"step_kernel", 1, 0, 1, 0, 1};
                break;
            case Kind::Grid: *out = {"lstm_fwd_kernel", 0, st.fwd.BT, st.fwd.nt, st.fwd.ngroups, !st.fwd.resident}; break;
        }
    } else {
        switch (bwd_kind(st, steps)) {
            case Kind::Cluster: *out = {"cluster_bwd_kernel", 0, st.cbwd.seqs, 1, 0, 0}; break;
            case Kind::Steps: *out = {"step_kernel", 2, 0, 1, 0, 1}; break;  // step_bwd_pointwise_kernel and the GEMM
            case Kind::Grid: *out = {"lstm_bwd_kernel", 0, st.bwd.BT, st.bwd.nt, st.bwd.ngroups, !st.bwd.resident}; break;
            default: *out = {"lstm_bwd_tm_kernel", 0, st.bwdtm.BT, st.bwdtm.nt, st.bwdtm.ngroups, 0}; break;
        }
    }
}

bool exchanges_directly(const Engine &e, bool backward, size_t steps) {
    const TcState &st = *static_cast<const TcState *>(e.tc_state);
    return backward ? bwd_kind(st, steps) == Kind::Tmem && st.bwdtm.direct : fwd_kind(st, steps) == Kind::Tmem && st.fwdtm.direct;
}

bool takes_known_h(const Engine &e, size_t steps) {
    return fwd_kind(*static_cast<const TcState *>(e.tc_state), steps) == Kind::Wide;
}

int forward_layer(Engine &e, int li, size_t t0, size_t t1, const void *x_l, void *y_out, cudaStream_t s) {
    TcState *st = state(e);
    FLSTM_TRY(check_async_error(e));
    auto &l = e.layers[li];
    auto &t = st->layers[li];
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, es = dtype_size(e.cfg.dtype), n = t1 - t0;
    unsigned int *err = e.sync_words;
    size_t m0 = e.timer.mark(s);
    // P = X W_ih^T + (b_ih + b_hh) for the steps of the range, 16-bit, columns tile-interleaved
    FLSTM_TRY(gemm(e.cfg.dtype, e.cfg.dtype, n * B, 4 * H, l.in_size, byte_ptr(x_l) + t0 * B * l.in_size * es, l.in_size, false,
                   l.w_ih, l.in_size, false, byte_ptr(l.gates) + t0 * B * 4 * H * es, 4 * H, l.bias, 0, err, st->sms, s));
    size_t m1 = e.timer.mark(s);
    const Kind kind = fwd_kind(*st, n);
    if (kind == Kind::Cluster) {
        ClusterFwdParams cp{};
        cp.w_hh = l.w_hh;
        cp.cs = l.cs;
        cp.hs = l.hs;
        cp.y = y_out;
        cp.gates = l.gates;
        cp.err = err;
        cp.T = (int)n;
        cp.t0 = (int)t0;
        cp.B = (int)B;
        cp.H = (int)H;
        cp.store_gates = (e.cfg.training && e.seg.keep_gates) ? 1 : 0;
        cp.real_units = e.logical_h;
        cp.trace = (li == 0 && t0 == 0) ? e.trace : nullptr;
        cp.trace_steps = e.trace_steps;
        cp.wait_ns = e.wait_limit_ns;
        cp.extra_arrivals = e.selftest_missing_arrivals;
        FLSTM_TRY(lstm_forward_cluster(e.cfg.dtype, st->cfwd, cp, s));
        size_t m2 = e.timer.mark(s);
        e.timer.span(PH_PROJ, m0, m1);
        e.timer.span(PH_RECUR_FWD, m1, m2);
        e.launches += 2;
        return FLSTM_OK;
    }
    if (kind == Kind::Steps) {
        CUtensorMap tm_y;
        if (y_out) FLSTM_TRY(make_tensor_map_3d_tile(&tm_y, y_out, 2, t1, B, H, 32, 16));
        const StepFwdMaps maps{&t.tm_hs3, &t.tm_wstep, &t.tm_g_ep, &t.tm_c_ep, &t.tm_h_ep, y_out ? &tm_y : nullptr};
        // one cooperative launch for the whole range, unless layers run concurrently on their own streams (the
        // cross-layer wavefront): two cooperative grids that each need most of the machine must not be in flight
        // at once, each could hold SMs the other is waiting for
        if (st->step.fwd_persistent && wavefront_chunk(e, (size_t)-1) == 0) {
            WideFwdParams wp{};
            wp.err = err;
            wp.counter = e.sync_words + 1;
            wp.exits = e.sync_words + kExitsWord;
            wp.t0 = (int)t0;
            wp.nsteps = (int)n;
            wp.B = (int)B;
            wp.H = (int)H;
            wp.store_gates = (e.cfg.training && e.seg.keep_gates) ? 1 : 0;
            wp.real_units = e.logical_h;
            wp.wait_ns = e.wait_limit_ns;
            wp.extra_arrivals = e.selftest_missing_arrivals;
            FLSTM_TRY(lstm_wide_forward(e.cfg.dtype, st->step, maps, wp, st->sms, s));
            size_t m2 = e.timer.mark(s);
            e.timer.span(PH_PROJ, m0, m1);
            e.timer.span(PH_RECUR_FWD, m1, m2);
            e.launches += 2;
            return FLSTM_OK;
        }
        for (size_t step = t0; step < t1; ++step) {
            StepFwdParams sp{};
            sp.err = err;
            sp.t = (int)step;
            sp.B = (int)B;
            sp.H = (int)H;
            sp.store_gates = (e.cfg.training && e.seg.keep_gates) ? 1 : 0;
            sp.real_units = e.logical_h;
            FLSTM_TRY(lstm_step_forward(e.cfg.dtype, st->step, maps, sp, st->sms, s));
        }
        size_t m2 = e.timer.mark(s);
        e.timer.span(PH_PROJ, m0, m1);
        e.timer.span(PH_RECUR_FWD, m1, m2);
        e.launches += 1 + n;
        return FLSTM_OK;
    }
    FwdParams p{};
    p.cs = l.cs;
    p.hs = l.hs;
    p.y = y_out;
    p.gates = l.gates;
    p.counters = e.sync_words + 1;
    p.exits = e.sync_words + kExitsWord;
    p.ring = st->ring;
    p.err = err;
    p.T = (int)n;
    p.t0 = (int)t0;
    p.B = (int)B;
    p.H = (int)H;
    p.store_gates = (e.cfg.training && e.seg.keep_gates) ? 1 : 0;
    p.known_h = e.seg.known_h ? 1 : 0;
    p.odd = (int)((e.seq_start + e.seg.start + t0) & 1);
    p.real_units = e.logical_h;
    p.trace = (li == 0 && t0 == 0) ? e.trace : nullptr;
    p.trace_steps = e.trace_steps;
    p.wait_ns = e.wait_limit_ns;
    p.extra_arrivals = e.selftest_missing_arrivals;
    p.lost = {e.selftest_lost.what, (int)e.selftest_lost.step, (int)e.selftest_lost.sequence / 32 * st->fwdtm.cta_rows};
    if (kind == Kind::Wide) FLSTM_TRY(lstm_forward_wide(e.cfg.dtype, st->wide, t.tm_ws, t.tm_h_tm, p, s));
    else if (kind == Kind::Tmem && st->fwdtm.direct) FLSTM_TRY(lstm_forward_tm_direct(e.cfg.dtype, st->fwdtm, t.tm_w, t.tm_g_tm, p, s));
    else if (kind == Kind::Tmem) FLSTM_TRY(lstm_forward_tm(e.cfg.dtype, st->fwdtm, t.tm_w, t.tm_ws, t.tm_h_tm, t.tm_g_tm, p, s));
    else FLSTM_TRY(lstm_forward_persistent(e.cfg.dtype, st->fwd, t.tm_w, t.tm_h, t.tm_g, p, s));
    size_t m2 = e.timer.mark(s);
    e.timer.span(PH_PROJ, m0, m1);
    e.timer.span(PH_RECUR_FWD, m1, m2);
    e.launches += 2;
    return FLSTM_OK;
}

// Inference over a few steps: a launch per layer and step reads the layer's weights once, against projection GEMM, state copies
// and the weight loads of a persistent kernel, all of which a few steps do not repay.  One call, cells / other path, us (I = H;
// - where the rule below does not take cells):
//   2 layers, H = 128, B = 32:   T = 1 10 / 33    T = 2 16 / 33    T = 3 23 / 36    T = 4  - / 37
//   4 layers, H = 512, B = 8:    T = 1 16 / 74    T = 2 30 / 82    T = 3 44 / 82    T = 4  - / 87
//   3 layers, H = 1024, B = 24:  T = 1 21 / 70    T = 2 41 / 78    T = 3 60 / 86    T = 4  - / 91
//   1 layer, H = 1024, B = 16:   T = 1  7 / 29    T = 2 12 / 32    T = 3 16 / 35    T = 4 22 / 35
//   1 layer, H = 1152, B = 24:   T = 1 10 / 29    T = 2 16 / 33    T = 3 24 / 34    T = 4 31 / 38
//   1 layer, H = 1216, B = 16:   T = 1 12 / 31    T = 2 22 / 33    T = 3 32 / 35    T = 4 41 / 39
//   1 layer, H = 1280, B = 32:   T = 1 16 / 31    T = 2 31 / 33    T = 3  - / 36
//   1 layer, H = 1536, B = 16:   T = 1 12 / 35    T = 2 25 / 37    T = 3 35 / 37    T = 4  - / 40
//   1 layer, H = 2048, B = 16:   T = 1 15 / 39    T = 2 29 / 37    T = 3 44 / 41    T = 4  - / 44
//   1 layer, H = 2048, B = 32:   T = 1 21 / 33    T = 2  - / 37
//   1 layer, B = 24, T = 1:      H = 3072 46 / 58   H = 3584 - / 66
// From the second step on weights that stay in L2 (half of its 126 MB) are what pays, and for a third step 48 MB of them; beyond
// that only T = 1 does.  More than 16 sequences take twice the operand loads per step, which wide layers do not repay.  Beyond
// H = 1184 (8 units per CTA) there are more CTAs than SMs, which a fourth step does not repay.  Up to 16 sequences it goes to
// stacks of 512 units altogether or where the other path is the grid-wide kernel (H > 512 at these batches), beyond 16 to a
// single layer; larger stacks, with a launch per layer and step to prepare, are left to the other path.
// A result that overlaps an input keeps to the other path, which has read all of x, h0 and c0 before it writes any.
bool cell_path(const Engine &e, size_t T, const void *x, const void *h0, const void *c0, const void *y, const void *hn, const void *cn) {
    if (e.backend != FLSTM_BACKEND_TC || e.cfg.training || T > 4 || e.cfg.batch > (size_t)kCellBatch || e.trace) return false;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(h0)) & 15) return false;
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, L = e.layers.size(), states = L * B * H, ces = e.cell_io_f32 ? sizeof(float) : 2;
    const struct { const void *p; size_t bytes; } in[] = {{x, T * B * e.cfg.input_size * 2}, {h0, states * 2}, {c0, states * ces}},
                                                  out[] = {{y, T * B * H * 2}, {hn, states * 2}, {cn, states * ces}};
    for (const auto &o : out)
        for (const auto &i : in) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(o.p), b = reinterpret_cast<uintptr_t>(i.p);
            if (a && b && a < b + i.bytes && b < a + o.bytes) return false;
        }
    size_t weights = 0;
    for (const auto &l : e.layers) weights += 8 * H * (l.in_size + H);
    const bool wide = B > 16;
    if (T == 1) return !wide || H <= 3072;
    if (weights > ((size_t)64 << 20)) return false;
    if (T == 4) return H <= 1152 && (wide ? L == 1 : H > 512 || L * H <= 512);
    if (T == 3 && weights > ((size_t)48 << 20)) return false;
    return !wide || H <= (T == 2 ? 1280 : 1152);
}

int forward_cells(Engine &e, size_t T, const void *x, const void *h0, const void *c0, void *y, void *hn, void *cn, cudaStream_t s) {
    FLSTM_TRY(check_async_error(e));
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, slab = B * H, L = e.layers.size();
    const size_t ces = e.cell_io_f32 ? sizeof(float) : 2;
    size_t m0 = e.timer.mark(s);
    for (size_t t = 0; t < T; ++t)
        for (size_t li = 0; li < L; ++li) {
            auto &l = e.layers[li];
            CellParams p{};
            p.w_ih = l.w_ih;
            p.w_hh = l.w_hh;
            p.bias = l.bias;
            p.x = li == 0 ? byte_ptr(x) + t * B * l.in_size * 2 : byte_ptr(e.layers[li - 1].hs) + (t + 1) * slab * 2;
            if (t > 0) {
                p.h_prev = byte_ptr(l.hs) + t * slab * 2;
                p.c_prev = l.cs + t * slab;
                p.c_prev_f32 = 1;
            } else {
                p.h_prev = h0 ? byte_ptr(h0) + li * slab * 2 : nullptr;
                p.c_prev = c0 ? byte_ptr(c0) + li * slab * ces : nullptr;
                p.c_prev_f32 = e.cell_io_f32 ? 1 : 0;
                p.h_first = l.hs;
                p.c_first = l.cs;
            }
            p.h_out = byte_ptr(l.hs) + (t + 1) * slab * 2;
            p.c_out = l.cs + (t + 1) * slab;
            p.y = (li == L - 1 && y) ? byte_ptr(y) + t * slab * 2 : nullptr;
            if (t == T - 1) {
                p.hn = hn ? byte_ptr(hn) + li * slab * 2 : nullptr;
                p.cn = cn ? byte_ptr(cn) + li * slab * ces : nullptr;
                p.cn_f32 = e.cell_io_f32 ? 1 : 0;
            }
            p.B = (int)B;
            p.I = (int)l.in_size;
            p.H = (int)H;
            p.real_units = e.logical_h;
            p.follows = t > 0 || li > 0;
            FLSTM_TRY(lstm_cell_step(e.cfg.dtype, p, s));
            ++e.launches;
        }
    e.timer.span(PH_RECUR_FWD, m0, e.timer.mark(s));
    return FLSTM_OK;
}

// Wide-batch BPTT over the steps [t0, t1), descending: per step one pointwise kernel (dG_t, cell-gradient
// carry) and one split-K GEMM (the fp32 partial sums of dG_t W_hh that step t-1 adds to its dy).
static int backward_steps(Engine &e, int li, size_t T, size_t t0, size_t t1, const void *dy_l, const void *dhn_l,
                          const void *dcn_l, float *dh0_l, float *dc0_l, bool finalize, cudaStream_t s) {
    TcState *st = state(e);
    auto &l = e.layers[li];
    auto &t = st->layers[li];
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, es = dtype_size(e.cfg.dtype), slab = B * H;
    const int splits = st->step.splits;
    float *parts = st->dh_parts + (size_t)li * splits * slab;
    float *dc = e.dc_layers + (size_t)li * slab;
    if (t1 == T) {
        // gradients entering the last step: dh_n in partial buffer 0, dc_n in the carry
        if (dhn_l) { FLSTM_TRY(simt::convert(e.cfg.dtype, dhn_l, FLSTM_DTYPE_F32, parts, slab, s)); ++e.launches; }
        else FLSTM_CUDA_TRY(cudaMemsetAsync(parts, 0, slab * sizeof(float), s));
        if (dcn_l) { FLSTM_TRY(simt::convert(e.cfg.dtype, dcn_l, FLSTM_DTYPE_F32, dc, slab, s)); ++e.launches; }
        else FLSTM_CUDA_TRY(cudaMemsetAsync(dc, 0, slab * sizeof(float), s));
    }
    for (size_t step = t1; step-- > t0;) {
        const int nparts = (step == T - 1) ? 1 : splits;
        FLSTM_TRY(lstm_step_backward_pointwise(e.cfg.dtype, byte_ptr(l.gates) + step * B * 4 * H * es, l.cs + (step + 1) * slab,
                                               l.cs + step * slab, byte_ptr(dy_l) + step * slab * es, parts, nparts, dc,
                                               byte_ptr(l.dg) + step * B * 4 * H * es, (int)B, (int)H, e.logical_h, s));
        ++e.launches;
        if (step > 0 || dh0_l || !finalize) {  // the product at step 0 is dh0, or the carry into the segment before
            FLSTM_TRY(lstm_step_backward_gemm(e.cfg.dtype, st->step, t.tm_dg3, t.tm_w, (int)step, (int)B, (int)H, parts,
                                              e.sync_words, st->sms, s));
            ++e.launches;
        }
    }
    if (t0 == 0 && finalize) {
        if (dh0_l) { FLSTM_TRY(sum_parts(parts, splits, slab, dh0_l, s)); ++e.launches; }
        if (dc0_l) FLSTM_CUDA_TRY(cudaMemcpyAsync(dc0_l, dc, slab * sizeof(float), cudaMemcpyDeviceToDevice, s));
    }
    return FLSTM_OK;
}

// Opt-in (FLSTM_WAVE_CHUNK=<steps per chunk>): measured neutral on configs 3 and 5, which already run at the
// board's power cap -- the overlap only lowers the SM clock (1.9 -> 1.6 GHz) -- so the default stays the
// layer-by-layer schedule.
size_t wavefront_chunk(const Engine &e, size_t n) {
    TcState *st = static_cast<TcState *>(e.tc_state);
    if (!st || !st->step.use || st->fwdtm.use || st->wide.use || st->bwdtm.use || e.layers.size() < 2 || e.timer.enabled) return 0;
    const char *env = std::getenv("FLSTM_WAVE_CHUNK");
    if (!env) return 0;
    const long v = std::atol(env);
    if (v <= 0) return 0;
    return (size_t)v < n ? (size_t)v : 0;  // a single chunk is the plain layer-by-layer schedule
}

int backward_layer(Engine &e, int li, size_t T, size_t t0, size_t t1, const void *x_l, const void *dy_l, const void *dhn_l,
                   const void *dcn_l, void *dx_l, float *dh0_l, float *dc0_l, cudaStream_t s, cudaEvent_t dx_ready) {
    TcState *st = state(e);
    FLSTM_TRY(check_async_error(e));
    if (!st->bwd_ok) return set_error(FLSTM_ERR_UNSUPPORTED, "tensor-core backward is not planned for this engine");
    auto &l = e.layers[li];
    auto &t = st->layers[li];
    const size_t B = e.cfg.batch, H = e.cfg.hidden_size, es = dtype_size(e.cfg.dtype), n = t1 - t0;
    unsigned int *err = e.sync_words;
    size_t m0 = e.timer.mark(s);
    // with activation checkpoints `T` and the range are segment-local; only the segment that starts the sequence
    // finishes the recurrence (dh0 / dc0) and the layer's gradients
    const bool finalize = t0 == 0 && (!e.seg.active || e.seg.final_segment);
    const Kind kind = bwd_kind(*st, n);
    if (kind == Kind::Cluster) {
        ClusterBwdParams cp{};
        cp.w_hh = l.w_hh;
        cp.cs = l.cs;
        cp.gates = l.gates;
        cp.dg = l.dg;
        cp.dy = dy_l;
        cp.dhn = dhn_l;
        cp.dcn = dcn_l;
        cp.dh0 = dh0_l;
        cp.dc0 = dc0_l;
        cp.dc = e.dc_layers + (size_t)li * B * H;
        cp.real_units = e.logical_h;
        cp.err = err;
        cp.T = (int)T;
        cp.s0 = (int)(T - t1);
        cp.s1 = (int)(T - t0) + (finalize ? 1 : 0);
        cp.B = (int)B;
        cp.H = (int)H;
        cp.trace = (li == 0 && e.trace && t1 == T) ? e.trace + (size_t)e.trace_steps * 16 : nullptr;
        cp.trace_steps = e.trace_steps;
        cp.wait_ns = e.wait_limit_ns;
        cp.extra_arrivals = e.selftest_missing_arrivals;
        FLSTM_TRY(lstm_backward_cluster(e.cfg.dtype, st->cbwd, cp, s));
        e.launches += 1;
    } else if (kind == Kind::Steps) {
        FLSTM_TRY(backward_steps(e, li, T, t0, t1, dy_l, dhn_l, dcn_l, dh0_l, dc0_l, finalize, s));
    } else {
    BwdParams p{};
    p.cs = l.cs;
    p.gates = l.gates;
    p.dg = l.dg;
    p.dy = dy_l;
    p.dhn = dhn_l;
    p.dcn = dcn_l;
    p.dh0 = dh0_l;
    p.dc0 = dc0_l;
    p.dc = e.dc_layers + (size_t)li * B * H;
    p.real_units = e.logical_h;
    p.trace = (li == 0 && e.trace && t1 == T) ? e.trace + (size_t)e.trace_steps * 16 : nullptr;
    p.trace_steps = e.trace_steps;
    p.counters = e.sync_words + 1;
    p.exits = e.sync_words + kExitsWord;
    p.ring = st->ring;
    p.err = err;
    p.T = (int)T;
    p.s0 = (int)(T - t1);
    p.s1 = (int)(T - t0) + (finalize ? 1 : 0);  // the last range also runs the iteration that writes dh0 / dc0
    p.B = (int)B;
    p.H = (int)H;
    p.wait_ns = e.wait_limit_ns;
    p.extra_arrivals = e.selftest_missing_arrivals;
    p.lost = {e.selftest_lost.what, (int)e.selftest_lost.step, (int)e.selftest_lost.sequence / 32 * st->bwdtm.jt * 4};
    if (kind == Kind::Tmem && st->bwdtm.direct) FLSTM_TRY(lstm_backward_tm_direct(e.cfg.dtype, st->bwdtm, t.tm_w, p, s));
    else if (kind == Kind::Tmem) FLSTM_TRY(lstm_backward_tm(e.cfg.dtype, st->bwdtm, t.tm_w, t.dg_tm, p, s));
    else FLSTM_TRY(lstm_backward_persistent(e.cfg.dtype, st->bwd, t.tm_w, t.tm_dg, p, s));
    e.launches += 1;
    }
    size_t m1 = e.timer.mark(s);
    auto input_grad = [&]() -> int {
        if (!dx_l) return FLSTM_OK;
        // dX = dG W_ih for the steps of the range: W_ih (rows tile-interleaved, like dG's columns) is read as stored
        FLSTM_TRY(gemm(e.cfg.dtype, e.cfg.dtype, n * B, l.in_size, 4 * H, byte_ptr(l.dg) + t0 * B * 4 * H * es, 4 * H, false,
                       l.w_ih, l.in_size, true, byte_ptr(dx_l) + t0 * B * l.in_size * es, l.in_size, nullptr, 0, err, st->sms,
                       s));
        ++e.launches;
        return FLSTM_OK;
    };
    auto weight_grads = [&]() -> int {
        if (t0 != 0) return FLSTM_OK;
        // dW = dG^T [X | H_prev] over the whole sequence: both operands read as stored (reduction dim
        // T*B outermost); rows of the product are written back in torch gate order.  With a communicator
        // each block of the layer's gradients starts its allreduce as soon as it is complete.
        // With activation checkpoints the sum runs segment by segment (the n steps in the buffers now),
        // accumulating from the second segment on, and the allreduce follows the last one.
        const size_t steps = e.seg.active ? n : T;
        const bool acc = e.seg.active && !e.seg.first_segment, last = !e.seg.active || e.seg.final_segment;
        const size_t n_ih = 4 * H * l.in_size;
        float *parts = st->dw_parts + (st->dw_layers > 1 ? (size_t)li * st->dw_floats : 0);
        // Opt-in (FLSTM_DW_SIDE_BY_SIDE=1, without a communicator): the two GEMMs run SIDE BY SIDE, each on its share of
        // the SMs.  Their 128 x 256 tiles run for milliseconds (K = T*B), so a last, partly filled round of tiles is
        // expensive -- config 3: 512 tiles each, 4 + 4 rounds on 148 SMs one after the other, 7 rounds on 74 + 74 SMs.
        // Measured: the phase drops from 27.7 to 26.0 ms, the whole step does not (122.2 against 120.7 ms): the board
        // is at its power cap in this phase, and SMs that idle through a partial round let the others clock higher.
        const size_t tiles_ih = ((4 * H + 127) / 128) * ((l.in_size + 255) / 256), tiles_hh = ((4 * H + 127) / 128) * ((H + 255) / 256);
        int sms_ih = (int)((size_t)st->sms * tiles_ih / (tiles_ih + tiles_hh));
        if (sms_ih < 1) sms_ih = 1;
        if (sms_ih > st->sms - 1) sms_ih = st->sms - 1;
        const int sms_hh = st->sms - sms_ih;
        auto rounds = [](size_t tiles, int sms) { return (tiles + sms - 1) / sms; };
        const size_t seq_rounds = rounds(tiles_ih, st->sms) + rounds(tiles_hh, st->sms);
        // a round = the time of one tile, whatever the number of CTAs working
        const size_t par_rounds = std::max(rounds(tiles_ih, sms_ih), rounds(tiles_hh, sms_hh));
        const char *sbs = std::getenv("FLSTM_DW_SIDE_BY_SIDE");
        const bool side_by_side = !e.comm && st->sms >= 2 && sbs && sbs[0] == '1' && par_rounds < seq_rounds;
        if (side_by_side) {
            FLSTM_TRY(e.ensure_aux_stream());
            FLSTM_CUDA_TRY(cudaEventRecord(e.aux_fork, s));
            FLSTM_CUDA_TRY(cudaStreamWaitEvent(e.aux_stream, e.aux_fork, 0));
            FLSTM_TRY(gemm(e.cfg.dtype, FLSTM_DTYPE_F32, 4 * H, H, steps * B, l.dg, 4 * H, true, l.hs, H, true, l.dw_hh, H,
                           nullptr, (int)H, err, sms_hh, e.aux_stream, acc));
            FLSTM_TRY(gemm(e.cfg.dtype, FLSTM_DTYPE_F32, 4 * H, l.in_size, steps * B, l.dg, 4 * H, true, x_l, l.in_size, true,
                           l.dw_ih, l.in_size, nullptr, (int)H, err, sms_ih, s, acc));
            FLSTM_CUDA_TRY(cudaEventRecord(e.aux_join, e.aux_stream));
            FLSTM_CUDA_TRY(cudaStreamWaitEvent(s, e.aux_join, 0));
        } else {
            FLSTM_TRY(gemm(e.cfg.dtype, FLSTM_DTYPE_F32, 4 * H, l.in_size, steps * B, l.dg, 4 * H, true, x_l, l.in_size, true,
                           l.dw_ih, l.in_size, nullptr, (int)H, err, st->sms, s, acc, parts, st->dw_floats));
            if (last) FLSTM_TRY(e.reduce_grads(l.grad_offset, n_ih, s));
            FLSTM_TRY(gemm(e.cfg.dtype, FLSTM_DTYPE_F32, 4 * H, H, steps * B, l.dg, 4 * H, true, l.hs, H, true, l.dw_hh, H,
                           nullptr, (int)H, err, st->sms, s, acc, parts, st->dw_floats));
        }
        FLSTM_TRY(simt::column_sum_two_pass(e.cfg.dtype, l.dg, steps * B, 4 * H,
                                            e.db_part + (size_t)li * simt::column_sum_scratch_floats(4 * H), l.db, (int)H, s,
                                            acc));
        if (last) FLSTM_TRY(e.reduce_grads(l.grad_offset + n_ih, l.grad_count - n_ih, s));
        e.launches += 4;
        return FLSTM_OK;
    };
    size_t m2, m3;
    if (dx_ready) {
        // wavefront: the layer below waits for dX of this range, so it goes first
        FLSTM_TRY(input_grad());
        FLSTM_CUDA_TRY(cudaEventRecord(dx_ready, s));
        m2 = e.timer.mark(s);
        FLSTM_TRY(weight_grads());
        m3 = e.timer.mark(s);
        e.timer.span(PH_XGRAD, m1, m2);
        e.timer.span(PH_WGRAD, m2, m3);
    } else {
        // weight gradients first: their allreduce then hides behind the input-gradient GEMM
        FLSTM_TRY(weight_grads());
        m2 = e.timer.mark(s);
        FLSTM_TRY(input_grad());
        m3 = e.timer.mark(s);
        e.timer.span(PH_WGRAD, m1, m2);
        e.timer.span(PH_XGRAD, m2, m3);
    }
    e.timer.span(PH_BPTT, m0, m1);
    return FLSTM_OK;
}

// A device word per device for the stand-alone entry points (never freed; 4 bytes).
static unsigned int *standalone_error_word() {
    static unsigned int *words[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!words[dev]) {
        if (cudaMalloc((void **)&words[dev], sizeof(unsigned int)) != cudaSuccess) return nullptr;
        cudaMemset(words[dev], 0, sizeof(unsigned int));
    }
    return words[dev];
}

int device_sm_count() {
    static int sms[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return sms[dev] > 0 ? sms[dev] : 1;
}

}  // namespace tc
}  // namespace flstm_b200

extern "C" int flstm_tc_plan(size_t batch, size_t hidden_size, int training, int sm_count, size_t smem_limit,
                             flstm_tc_plan_info *out) {
    using namespace flstm_b200;
    if (!out || sm_count < 1) return set_error(FLSTM_ERR_INVALID, "bad argument");
    *out = flstm_tc_plan_info{};
    tc::StepPlan sp{};
    FLSTM_TRY(tc::plan_step((int)batch, (int)hidden_size, sm_count, smem_limit, &sp));
    out->step_path = sp.use ? 1 : 0;
    out->step_bn_fwd = sp.bn_fwd;
    out->step_bn_bwd = sp.bn_bwd;
    out->step_splits = sp.splits;
    out->step_pair = sp.pair ? 1 : 0;
    out->step_fwd_pair = sp.fwd_pair ? 1 : 0;
    if (sp.use) return FLSTM_OK;
    tc::FwdPlan f{};
    FLSTM_TRY(tc::plan_fwd((int)batch, (int)hidden_size, sm_count, smem_limit, &f));
    out->fwd_batch_tile = f.BT;
    out->fwd_pair = f.pair ? 1 : 0;
    out->fwd_row_tiles_per_cta = f.rt;
    out->fwd_grid = f.grid;
    out->fwd_batch_groups = f.ngroups;
    out->fwd_tiles_per_group = f.nt;
    out->fwd_stages = f.stages;
    out->fwd_chunks_per_stage = f.ch;
    out->fwd_weights_resident = f.resident ? 1 : 0;
    out->fwd_smem_bytes = f.smem_bytes;
    if (training) {
        tc::BwdPlan b{};
        FLSTM_TRY(tc::plan_bwd((int)batch, (int)hidden_size, sm_count, smem_limit, &b, /*check_device=*/false));
        out->bwd_batch_tile = b.BT;
        out->bwd_cluster_size = b.KS;
        out->bwd_grid = b.grid;
        out->bwd_batch_groups = b.ngroups;
        out->bwd_tiles_per_group = b.nt;
        out->bwd_stages = b.stages;
        out->bwd_chunks_per_stage = b.ch;
        out->bwd_weights_resident = b.resident ? 1 : 0;
        out->bwd_smem_bytes = b.smem_bytes;
    }
    return FLSTM_OK;
}

extern "C" int flstm_tmem_plan(size_t batch, size_t hidden_size, int training, int sm_count, size_t smem_limit,
                               flstm_tmem_plan_info *out) {
    using namespace flstm_b200;
    if (!out || sm_count < 1) return set_error(FLSTM_ERR_INVALID, "bad argument");
    *out = flstm_tmem_plan_info{};
    tc::TcState st;
    FLSTM_TRY(tc::choose_tmem((int)batch, (int)hidden_size, true, training != 0, sm_count, smem_limit, /*check_device=*/false, &st));
    if (st.wide.use) {
        out->fwd_kernel = 2;
        out->fwd_batch_tile = st.wide.BT;
        out->fwd_batch_groups = st.wide.ngroups;
        out->fwd_tiles_in_turn = st.wide.nt;
        out->fwd_grid = st.wide.grid;
        out->fwd_smem_bytes = st.wide.smem_bytes;
    } else if (st.fwdtm.use) {
        out->fwd_kernel = 1;
        out->fwd_k_halves = st.fwdtm.S == 2;
        out->fwd_batch_tile = st.fwdtm.BT;
        out->fwd_batch_groups = st.fwdtm.ngroups;
        out->fwd_tiles_in_turn = 1;
        out->fwd_weights_streamed = st.fwdtm.wstages > 0;
        out->fwd_grid = st.fwdtm.grid;
        out->fwd_smem_bytes = st.fwdtm.smem_bytes;
    }
    out->fwd_from_steps = (int)st.fwd_from;
    if (st.bwdtm.use) {
        out->bwd_kernel = 1;
        out->bwd_batch_tile = st.bwdtm.BT;
        out->bwd_batch_groups = st.bwdtm.ngroups;
        out->bwd_tiles_in_turn = st.bwdtm.nt;
        out->bwd_grid = st.bwdtm.grid;
        out->bwd_smem_bytes = st.bwdtm.smem_bytes;
        out->bwd_from_steps = (int)st.bwd_from;
    }
    return FLSTM_OK;
}

extern "C" int flstm_tc_gemm(int dtype, int out_dtype, size_t M, size_t N, size_t K, const void *A, const void *B,
                             void *D, size_t ldd, const float *bias, int layout, void *stream) {
    using namespace flstm_b200;
    if (!A || !B || !D) return set_error(FLSTM_ERR_INVALID, "null pointer argument");
    if (layout < 0 || layout > 2) return set_error(FLSTM_ERR_INVALID, "layout must be 0, 1 or 2");
    unsigned int *err = tc::standalone_error_word();
    if (!err) return set_error(FLSTM_ERR_CUDA, "could not allocate the error word");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool a_mn = layout == 1, b_mn = layout >= 1;
    const size_t lda = a_mn ? M : K, ldb = b_mn ? N : K;
    FLSTM_TRY(tc::gemm(dtype, out_dtype, M, N, K, A, lda, a_mn, B, ldb, b_mn, D, ldd, bias, 0, err,
                       tc::device_sm_count(), s));
    unsigned int h = 0;
    FLSTM_CUDA_TRY(cudaMemcpyAsync(&h, err, sizeof(h), cudaMemcpyDeviceToHost, s));
    FLSTM_CUDA_TRY(cudaStreamSynchronize(s));
    if (h) {
        cudaMemsetAsync(err, 0, sizeof(h), s);
        return set_error(FLSTM_ERR_TIMEOUT, "tensor-core GEMM: a bounded device-side wait expired");
    }
    return FLSTM_OK;
}
