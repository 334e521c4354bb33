// Internal C++ view of the engine handle (the C ABI in include/flashlstm_b200/engine.h wraps it).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "flashlstm_b200/engine.h"
#include "kernels.h"

namespace flstm_b200 {

struct Comm;  // data-parallel communicator (comm.cu)

// Device-time accounting per phase with CUDA events; records only when enabled, never syncs
// until the totals are read.
enum Phase { PH_PROJ = 0, PH_RECUR_FWD, PH_BPTT, PH_WGRAD, PH_XGRAD, PH_ALLREDUCE, PH_COUNT };
struct PhaseTimer {
    bool enabled = false;
    std::vector<cudaEvent_t> pool;
    size_t used = 0;
    struct Span { int phase; size_t a, b; };
    std::vector<Span> spans;
    void reset() { used = 0; spans.clear(); }
    size_t mark(cudaStream_t s);
    void span(int phase, size_t a, size_t b) { if (enabled) spans.push_back({phase, a, b}); }
    int totals(float *out);
    ~PhaseTimer();
};

// Per-layer device buffers.  "T" below is the engine's storage type.
struct LayerBuffers {
    size_t in_size = 0;      // I_l
    void *w_ih = nullptr;    // T (4H, I_l)   SIMT: torch row order; TC: tile-interleaved rows
    void *w_hh = nullptr;    // T (4H, H)     same row order as w_ih
    float *bias = nullptr;   // fp32 (4H)     b_ih + b_hh, same order as the rows of w_ih
    void *gates = nullptr;   // T (Tcap, B, 4H)  input projection, overwritten by the gate cache
    void *hs = nullptr;      // T (Tcap+1, B, H) slot 0 = h0, slot t+1 = h_t
    float *cs = nullptr;     // fp32 (Tcap+1, B, H)
    void *dg = nullptr;      // T (Tcap, B, 4H)  pre-activation gradients (training)
    void *dx = nullptr;      // T (Tcap, B, I_l) gradient w.r.t. this layer's input (layers > 0)
    // activation-checkpoint mode (Engine::recompute > 0): the time-sized buffers above hold one segment
    void *y_all = nullptr;   // T (Tcap, B, H)  layers below the top: h_t for every step = the next layer's input
    void *ck_h = nullptr;    // T (K, B, H)     hidden state entering segment k
    float *ck_c = nullptr;   // fp32 (K, B, H)  cell state entering segment k
    float *dw_ih = nullptr;  // views into the flat gradient buffer
    float *dw_hh = nullptr;
    float *db = nullptr;
    size_t grad_offset = 0;  // element offset of this layer's [dW_ih | dW_hh | db] slice
    size_t grad_count = 0;
    bool weights_set = false;
};

// Copies of small strided matrices (states in and out of the engine's buffers, padding, the error word), collected and
// run as one launch: with one memcpy / memset / conversion per state and layer a call of a small model spent more time
// on its launches than on its recurrence.
struct CopyJob {
    const void *src;  // null: zeros
    void *dst;
    size_t rows, src_pitch, dst_pitch;  // pitches in elements
    int src_cols, dst_cols;             // columns [src_cols, dst_cols) of the destination become zero
    int src_dtype, dst_dtype;
};
struct CopyBatch {
    std::vector<CopyJob> jobs;
    const unsigned int *err = nullptr;  // device error word, mirrored to err_host by the next launch when non-zero
    unsigned int *err_host = nullptr;
    void add(const void *src, int src_dtype, size_t src_pitch, int src_cols, void *dst, int dst_dtype, size_t dst_pitch,
             int dst_cols, size_t rows);
    void dense(const void *src, int src_dtype, void *dst, int dst_dtype, size_t rows, size_t cols) {
        add(src, src_dtype, cols, (int)cols, dst, dst_dtype, cols, (int)cols, rows);
    }
    int run(cudaStream_t s, unsigned long long *launches);
};

// Buffers that live and die together come from ONE cudaMalloc: each costs about 0.4 ms here, and an engine has dozens.
struct Arena {
    struct Request { void **p; size_t bytes; };
    std::vector<Request> requests;
    void *base = nullptr;
    template <typename P>
    void want(P **p, size_t bytes) { requests.push_back({reinterpret_cast<void **>(p), bytes}); }
    template <typename P>
    void forget(P **p) {  // a request that is not committed
        for (size_t i = requests.size(); i-- > 0;)
            if (requests[i].p == reinterpret_cast<void **>(p)) requests.erase(requests.begin() + i);
    }
    int commit();   // allocates what was asked for since the last commit (at most one allocation at a time)
    void release();
};
// A pinned host word for an engine's error mirror, from a small process-wide slab (cudaMallocHost takes milliseconds).
unsigned int *host_word_acquire();
void host_word_release(unsigned int *word);

struct Engine {
    flstm_engine_config cfg{};
    Arena fixed, timed;  // weights, gradients, scratch; buffers sized by the sequence length
    int backend = FLSTM_BACKEND_SIMT;
    int device = 0;
    size_t t_cap = 0;  // longest sequence the engine is currently sized for
    // Activation checkpoints (the reference's recompute interval R, flashlstm_v2/src/lstm_forward.cu:727-783,
    // lstm_backward.cu:975-1054): with recompute = R > 0 the forward keeps only the h/c state entering every
    // R-th step, and the backward re-runs the forward of one R-step segment at a time to rebuild its gate
    // cache.  gates / hs / cs / dg then span buf_steps = min(R, t_cap) steps instead of t_cap.
    size_t recompute = 0;
    size_t buf_steps = 0;
    size_t workspace_bytes = 0;  // bytes of the time-sized buffers currently allocated
    struct SegmentMode {
        bool active = false;         // the layer backward works on one segment with segment-local time indices
        bool final_segment = true;   // the segment that starts at t = 0: dh0/dc0 and the gradient allreduce follow it
        bool first_segment = true;   // the first one processed (the end of the sequence): weight gradients start from zero
        bool keep_gates = true;      // forward writes the activated gates back (off in the checkpointing forward pass)
        bool known_h = false;        // the segment's h_t stand in hs: the forward only rebuilds gates and cell states
        size_t start = 0;            // number of the segment's first step within the call's sequence
    } seg;
    std::vector<LayerBuffers> layers;
    float *grads = nullptr;  // flat fp32: per layer [dW_ih | dW_hh | db]
    size_t grad_count = 0;
    float *dc_layers = nullptr;  // fp32 (L,B,H) cell-gradient carry, kept between backward ranges
    float *db_part = nullptr;  // TC: per batch-tile partial bias gradients
    unsigned int *sync_words = nullptr;  // TC: grid-barrier counters + error word
    size_t last_T = 0;       // sequence length of the last complete forward (0 = none)
    size_t fwd_progress = 0; // steps of the current forward already enqueued
    size_t bwd_progress = 0; // backward has been enqueued down to this step
    unsigned long long launches = 0;
    // Limit of every device-side wait of the persistent kernels in nanoseconds (0 = the kernels' 2 s default) and
    // the timeout self-test: a step barrier that waits for this many arrivals which nobody makes.
    unsigned long long wait_limit_ns = 0;
    unsigned int selftest_missing_arrivals = 0;
    struct {
        unsigned int what = 0;
        size_t step = 0, sequence = 0;
    } selftest_lost;  // tc::LostWords
    // A 16-bit shape that the tensor-core path cannot tile runs there zero-padded (engine_padded.cu): this engine then
    // only owns the logical gradients and staging tensors, `inner` has the padded sizes and does the work.
    Engine *inner = nullptr;
    int logical_h = 0, logical_in = 0;  // of an inner engine: the sizes of the parameters it is given (0: not one)
    struct Padding {
        void *x = nullptr, *dy = nullptr, *dx = nullptr;            // (T, B, .) padded
        void *h0 = nullptr, *dhn = nullptr, *dcn = nullptr;         // (L, B, Hp) engine dtype
        float *c0 = nullptr, *dh0 = nullptr, *dc0 = nullptr;        // (L, B, Hp) fp32
        void *gates = nullptr, *hs = nullptr;                       // logical copies behind flstm_engine_cache_ptrs
        float *cs = nullptr;
        size_t t_cap = 0, t_mirror = 0;
        size_t time_bytes = 0, state_bytes = 0, mirror_bytes = 0;
    } pad;
    Engine &core() { return inner ? *inner : *this; }
    int padded_create();
    void padded_release();
    void padded_drop();  // back to the CUDA-core path, before anything has run
    int padded_reserve(size_t T);
    int padded_forward_range(size_t T, size_t t0, size_t t1, const void *x, const void *h0, const void *c0, void *y, void *hn,
                             void *cn, cudaStream_t s);
    int padded_backward_range(size_t T, size_t t0, size_t t1, const void *dy, const void *dhn, const void *dcn, void *dx,
                              float *dh0, float *dc0, cudaStream_t s);
    int padded_cache_ptrs(int layer, void **gates, float **cells, void **hiddens);
    int padded_mirror(size_t t0, size_t t1, cudaStream_t s);
    bool cell_io_f32 = false;       // c0 / c_n cross the API as fp32 instead of the engine dtype
    size_t seq_start = 0;           // number of the calls' first step within a sequence that is streamed from outside in segments
    const void *x_saved = nullptr;  // layer-0 input of the last forward (caller keeps it alive)
    PhaseTimer timer;
    Comm *comm = nullptr;
    bool comm_aborted = false;  // the watchdog gave up on a step: no collective until a new communicator is attached
    cudaStream_t comm_stream = nullptr;
    cudaEvent_t comm_fork = nullptr, comm_join = nullptr;
    // second compute stream (created on first use): the two weight-gradient GEMMs of a layer run side by side on
    // disjoint halves of the SMs when that saves a round of tiles
    cudaStream_t aux_stream = nullptr;
    cudaEvent_t aux_fork = nullptr, aux_join = nullptr;
    int ensure_aux_stream();
    long long *trace = nullptr;  // device: [2 (fwd,bwd)][trace_steps][16] clock stamps of CTA 0
    int trace_steps = 0;
    void *tc_state = nullptr;  // tensor-core path: cached tensor maps etc. (tc_engine.cu)
    // CUDA-core path: persistent recurrent kernels when the shape fits (simt_persistent.cu)
    simt::ClusterF32Plan f32_fwd{}, f32_bwd{};  // fp32: recurrences inside thread-block clusters (simt_cluster.cu)
    int simt_grid = 0;                       // 0: one launch per step
    unsigned int *simt_err_host = nullptr;   // pinned mirror of the error word
    int simt_check_error();
    float *simt_scratch = nullptr;           // split-K partial products of the weight-gradient GEMMs
    size_t simt_scratch_floats = 0;
    // Cross-layer wavefront (wide-batch path with stacked layers): layer l > 0 runs its time chunks on
    // lanes[l] one chunk behind layer l-1, so independent per-step kernels of different layers share the GPU.
    std::vector<cudaStream_t> lanes;        // lanes[0] is the caller's stream (not owned)
    std::vector<cudaEvent_t> lane_events;   // pool, reused call after call in stream order
    size_t lane_events_used = 0;
    // sum `count` floats of the flat gradient buffer at `offset` over the ranks, on the communication stream,
    // after everything enqueued on `from` so far (no-op without a communicator)
    int reduce_grads(size_t offset, size_t count, cudaStream_t from);
    int ensure_lanes(cudaStream_t s);
    cudaEvent_t next_lane_event();

    ~Engine();
    int allocate(size_t t_cap);
    void release_time_buffers();
    int ensure_capacity(size_t T);
    int reserve(size_t T);  // the same, padded or not; buffers handed out before (cache_ptrs) are gone when they grow
    int init();  // workspace, plans and backend state for cfg / backend / device
    // parameters of layers [first, first + count): w_ih, w_hh, b_ih, b_hh of each
    int set_weights(int first, int count, const float *const *params, cudaStream_t s);
    int forward(size_t T, const void *x, const void *h0, const void *c0, void *y, void *hn, void *cn,
                cudaStream_t s);
    int backward(size_t T, const void *dy, const void *dhn, const void *dcn, void *dx, float *dh0,
                 float *dc0, cudaStream_t s);
    int forward_range(size_t T, size_t t0, size_t t1, const void *x, const void *h0, const void *c0, void *y, void *hn,
                      void *cn, cudaStream_t s);
    int forward_checkpointed(size_t T, const void *x, const void *h0, const void *c0, void *y, void *hn, void *cn,
                             cudaStream_t s);
    int backward_checkpointed(size_t T, const void *dy, const void *dhn, const void *dcn, void *dx, float *dh0, float *dc0,
                              cudaStream_t s);
    int backward_segment(size_t n, bool last_in_time, bool first_in_time, const void *x_seg, const void *h_in,
                         const float *c_in, const void *dy_seg, const void *dhn, const void *dcn, void *dx_seg, float *dh0,
                         float *dc0, cudaStream_t s);
    int set_recompute(size_t R);
    int backward_range(size_t T, size_t t0, size_t t1, const void *dy, const void *dhn, const void *dcn, void *dx,
                       float *dh0, float *dc0, cudaStream_t s);
};

}  // namespace flstm_b200

// The opaque handle of the C ABI.
struct flstm_engine {
    flstm_b200::Engine impl;
};

namespace flstm_b200 {

// Tensor-core path entry points (tc_engine.cu).  `supported` decides AUTO resolution.
namespace tc {
constexpr size_t kSyncWords = 1024;  // step counters, exit counter and error word of an engine
bool supported(const flstm_engine_config &cfg);
int init(Engine &e);
void destroy(Engine &e);
int on_capacity_change(Engine &e);
int poll_error(Engine &e);  // reports (and clears) a device-side wait that expired in an earlier launch
int set_weights(Engine &e, int first, int count, const float *const *params, cudaStream_t s);
unsigned int *error_mirror(Engine &e);
int recurrent_path(const Engine &e, bool backward, int *ctas, int *seqs);  // flstm_path
void recurrent_kernel(const Engine &e, bool backward, size_t steps, flstm_kernel_info *out);
bool exchanges_directly(const Engine &e, bool backward, size_t steps);  // flstm_engine_direct
// whether a launch of this many steps runs without waiting from step to step where SegmentMode::known_h
bool takes_known_h(const Engine &e, size_t steps);
int forward_layer(Engine &e, int layer, size_t t0, size_t t1, const void *x_l, void *y_out, cudaStream_t s);
// `dx_ready` (optional) is recorded on `s` once dx_l of the range is complete, before the weight gradients
int backward_layer(Engine &e, int layer, size_t T, size_t t0, size_t t1, const void *x_l, const void *dy_l,
                   const void *dhn_l, const void *dcn_l, void *dx_l, float *dh0_l, float *dc0_l, cudaStream_t s,
                   cudaEvent_t dx_ready = nullptr);
// steps per wavefront chunk for a range of n steps; 0 = no cross-layer wavefront for this engine
size_t wavefront_chunk(const Engine &e, size_t n);
// whether a T-step inference call runs step by step (tc_cell.cu), and that call
bool cell_path(const Engine &e, size_t T, const void *x, const void *h0, const void *c0, const void *y, const void *hn, const void *cn);
int forward_cells(Engine &e, size_t T, const void *x, const void *h0, const void *c0, void *y, void *hn, void *cn, cudaStream_t s);
}  // namespace tc

// Communicator (comm.cu): NCCL loaded at run time with dlopen.
int comm_unique_id(void *id128);
int comm_create(const void *id128, int rank, int world, Comm **out);
void comm_destroy(Comm *c);
void comm_abort(Comm *c);  // ncclCommAbort (falls back to destroy when the library lacks it), frees c
int comm_allreduce_sum_f32(Comm *c, float *buf, size_t count, cudaStream_t s);

}  // namespace flstm_b200
