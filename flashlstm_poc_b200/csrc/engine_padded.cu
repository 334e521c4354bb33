// 16-bit shapes that the tensor-core path cannot tile (hidden size not a multiple of 64 or input width not a multiple of
// 8) run on it zero-padded: an inner engine has the padded sizes Hp and Ip, this one copies the caller's tensors in and
// out.  A padded hidden unit starts from zero states and the kernels take its pre-activations and its dh as zero, so it
// stays at c = h = 0 (its gates are sigmoid(0) and tanh(0) = 0) and passes no gradient on.  Its zero weights alone would
// not do: one infinite input, which leaves the real units' gates saturated and finite, made it 0 * inf = NaN and from
// the next step on the whole sequence.  Padded input columns meet zero weights.  The weights are packed straight into
// the padded layout.
//
// Before, such shapes ran in the CUDA-core kernels, one launch per step once W_hh outgrew shared memory: two layers of
// H = I = 650, B = 20, T = 35 forward + backward took 6.9 ms.
#include <algorithm>
#include <new>

#include "common.cuh"
#include "engine.h"

namespace flstm_b200 {

namespace {

inline char *bytes(void *p) { return static_cast<char *>(p); }
inline const char *bytes(const void *p) { return static_cast<const char *>(p); }
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename P>
int grab(P **p, size_t n, size_t *total) {
    void *raw = nullptr;
    if (n == 0) return FLSTM_OK;
    const cudaError_t e = cudaMalloc(&raw, n);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "cudaMalloc(%zu bytes) failed: %s", n, cudaGetErrorString(e));
    *p = static_cast<P *>(raw);
    *total += n;
    return FLSTM_OK;
}
template <typename P>
void drop(P *&p) {
    if (p) cudaFree(p);
    p = nullptr;
}

// gate cache (steps, B, 4Hp) tile-interleaved -> (steps, B, 4H) torch order
__global__ void unpad_gates_kernel(const uint16_t *__restrict__ in, int H, int Hp, size_t rows, uint16_t *__restrict__ out) {
    const size_t total = rows * 4 * H;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (4 * H);
        const int col = (int)(i % (4 * H)), g = col / H, u = col % H;
        out[i] = in[r * 4 * Hp + (size_t)(u >> 4) * 64 + g * 16 + (u & 15)];
    }
}

}  // namespace

int Engine::padded_create() {
    if (cfg.dtype != FLSTM_DTYPE_F16 && cfg.dtype != FLSTM_DTYPE_BF16) return FLSTM_OK;
    flstm_engine_config padded = cfg;
    padded.hidden_size = (cfg.hidden_size + 63) / 64 * 64;
    padded.input_size = (cfg.input_size + 7) / 8 * 8;
    padded.backend = FLSTM_BACKEND_TC;
    if (!tc::supported(padded)) return FLSTM_OK;  // the CUDA-core path takes it
    inner = new (std::nothrow) Engine();
    if (!inner) return set_error(FLSTM_ERR_INVALID, "out of host memory");
    inner->cfg = padded;
    inner->device = device;
    inner->backend = FLSTM_BACKEND_TC;
    inner->logical_h = (int)cfg.hidden_size;
    inner->logical_in = (int)cfg.input_size;
    backend = FLSTM_BACKEND_TC;
    const size_t n = cfg.layers * cfg.batch * padded.hidden_size;
    if (padded.hidden_size != cfg.hidden_size) {
        fixed.want(&pad.h0, n * 2);
        fixed.want(&pad.c0, n * sizeof(float));
        if (cfg.training) {
            fixed.want(&pad.dhn, n * 2);
            fixed.want(&pad.dcn, n * 2);
            fixed.want(&pad.dh0, n * sizeof(float));
            fixed.want(&pad.dc0, n * sizeof(float));
        }
        pad.state_bytes = n * (cfg.training ? 18 : 6);
    }
    return inner->init();
}

void Engine::padded_release() {
    drop(pad.gates);
    drop(pad.hs);
    drop(pad.cs);
}

void Engine::padded_drop() {
    padded_release();
    timed.release();
    fixed.release();
    delete inner;
    inner = nullptr;
    pad = Padding{};
    backend = FLSTM_BACKEND_SIMT;
}

// Staging tensors for sequences of up to T steps: for max_seq_len steps when the engine is made, so that a call within it
// allocates nothing (it may be captured).  A tensor whose width needs no padding has one too: the caller's may start off a
// 16-byte boundary.
int Engine::padded_reserve(size_t T) {
    if (T <= pad.t_cap) return FLSTM_OK;
    if (pad.t_cap) FLSTM_CUDA_TRY(cudaDeviceSynchronize());
    timed.release();
    pad.t_cap = 0;
    const size_t cap = std::max(T, cfg.max_seq_len), B = cfg.batch;
    const size_t x_bytes = cap * B * inner->cfg.input_size * 2, y_bytes = cfg.training ? cap * B * inner->cfg.hidden_size * 2 : 0;
    timed.want(&pad.x, x_bytes);
    timed.want(&pad.dx, cfg.training ? x_bytes : 0);
    timed.want(&pad.dy, y_bytes);
    FLSTM_TRY(timed.commit());
    pad.time_bytes = x_bytes * (cfg.training ? 2 : 1) + y_bytes;
    pad.t_cap = cap;
    return FLSTM_OK;
}

int Engine::padded_forward_range(size_t T, size_t t0, size_t t1, const void *x, const void *h0, const void *c0, void *y, void *hn,
                                 void *cn, cudaStream_t s) {
    Engine &in = *inner;
    const int dt = cfg.dtype, L = cfg.layers, c_dtype = cell_io_f32 ? (int)FLSTM_DTYPE_F32 : dt;
    const size_t B = cfg.batch, H = cfg.hidden_size, Hp = in.cfg.hidden_size, I = cfg.input_size, Ip = in.cfg.input_size, es = 2;
    const bool pad_h = Hp != H, pad_x = Ip != I || !aligned16(x), pad_y = pad_h || !aligned16(y);
    if (t0 == 0) {
        for (auto &l : layers)
            if (!l.weights_set) return set_error(FLSTM_ERR_INVALID, "weights have not been set for every layer");
        FLSTM_TRY(padded_reserve(T));
    } else if (in.fwd_progress != t0 || t1 > pad.t_cap) {
        return set_error(FLSTM_ERR_INVALID, "forward ranges must be contiguous and ascending (expected start %zu, got %zu)", in.fwd_progress, t0);
    }
    CopyBatch batch;
    if (pad_x)
        batch.add(bytes(x) + t0 * B * I * es, dt, I, (int)I, bytes(pad.x) + t0 * B * Ip * es, dt, Ip, (int)Ip, (t1 - t0) * B);
    if (pad_h && t0 == 0) {
        if (h0) batch.add(h0, dt, H, (int)H, pad.h0, dt, Hp, (int)Hp, L * B);
        if (c0) batch.add(c0, c_dtype, H, (int)H, pad.c0, FLSTM_DTYPE_F32, Hp, (int)Hp, L * B);
    }
    FLSTM_TRY(batch.run(s, &launches));
    in.cell_io_f32 = pad_h || cell_io_f32;
    FLSTM_TRY(in.forward_range(T, t0, t1, pad_x ? pad.x : x, pad_h && h0 ? pad.h0 : h0, pad_h && c0 ? pad.c0 : c0,
                               pad_y ? nullptr : y, pad_h ? nullptr : hn, pad_h ? nullptr : cn, s));
    if (y && pad_y)
        batch.add(bytes(in.layers.back().hs) + (t0 + 1) * B * Hp * es, dt, Hp, (int)H, bytes(y) + t0 * B * H * es, dt, H, (int)H,
                  (t1 - t0) * B);
    if (pad_h && t1 == T) {
        const size_t ces = cell_io_f32 ? sizeof(float) : es;
        for (int li = 0; li < L; ++li) {
            if (hn) batch.add(bytes(in.layers[li].hs) + T * B * Hp * es, dt, Hp, (int)H, bytes(hn) + li * B * H * es, dt, H, (int)H, B);
            if (cn) batch.add(in.layers[li].cs + T * B * Hp, FLSTM_DTYPE_F32, Hp, (int)H, bytes(cn) + li * B * H * ces, c_dtype, H, (int)H, B);
        }
    }
    FLSTM_TRY(batch.run(s, &launches));
    return padded_mirror(t0, t1, s);
}

int Engine::padded_backward_range(size_t T, size_t t0, size_t t1, const void *dy, const void *dhn, const void *dcn, void *dx,
                                  float *dh0, float *dc0, cudaStream_t s) {
    Engine &in = *inner;
    const int dt = cfg.dtype, L = cfg.layers;
    const size_t B = cfg.batch, H = cfg.hidden_size, Hp = in.cfg.hidden_size, I = cfg.input_size, Ip = in.cfg.input_size, es = 2;
    if (!dy) return set_error(FLSTM_ERR_INVALID, "dy is null");
    const bool pad_h = Hp != H, pad_dy = pad_h || !aligned16(dy), pad_dx = dx && (Ip != I || !aligned16(dx));
    CopyBatch batch;
    // the inner engine checks the order of the ranges; a wrong one must not write past the staging tensors
    if (cfg.training && in.last_T == T && t0 < t1 && t1 <= T) {
        if (pad_dy)
            batch.add(bytes(dy) + t0 * B * H * es, dt, H, (int)H, bytes(pad.dy) + t0 * B * Hp * es, dt, Hp, (int)Hp, (t1 - t0) * B);
        if (pad_h && dhn && t1 == T) batch.add(dhn, dt, H, (int)H, pad.dhn, dt, Hp, (int)Hp, L * B);
        if (pad_h && dcn && t1 == T) batch.add(dcn, dt, H, (int)H, pad.dcn, dt, Hp, (int)Hp, L * B);
        FLSTM_TRY(batch.run(s, &launches));
    }
    FLSTM_TRY(in.backward_range(T, t0, t1, pad_dy ? pad.dy : dy, pad_h && dhn ? pad.dhn : dhn, pad_h && dcn ? pad.dcn : dcn,
                                pad_dx ? pad.dx : dx, pad_h && dh0 ? pad.dh0 : dh0, pad_h && dc0 ? pad.dc0 : dc0, s));
    if (pad_dx)
        batch.add(bytes(pad.dx) + t0 * B * Ip * es, dt, Ip, (int)I, bytes(dx) + t0 * B * I * es, dt, I, (int)I, (t1 - t0) * B);
    if (t0 == 0) {
        if (pad_h && dh0) batch.add(pad.dh0, FLSTM_DTYPE_F32, Hp, (int)H, dh0, FLSTM_DTYPE_F32, H, (int)H, L * B);
        if (pad_h && dc0) batch.add(pad.dc0, FLSTM_DTYPE_F32, Hp, (int)H, dc0, FLSTM_DTYPE_F32, H, (int)H, L * B);
        // gradients: rows g * Hp + u of the padded matrices -> g * H + u, without the padded columns
        for (int li = 0; li < L; ++li) {
            auto &l = layers[li], &p = in.layers[li];
            for (size_t g = 0; g < 4; ++g) {
                batch.add(p.dw_ih + g * Hp * p.in_size, FLSTM_DTYPE_F32, p.in_size, (int)l.in_size, l.dw_ih + g * H * l.in_size,
                          FLSTM_DTYPE_F32, l.in_size, (int)l.in_size, H);
                batch.add(p.dw_hh + g * Hp * Hp, FLSTM_DTYPE_F32, Hp, (int)H, l.dw_hh + g * H * H, FLSTM_DTYPE_F32, H, (int)H, H);
                batch.add(p.db + g * Hp, FLSTM_DTYPE_F32, Hp, (int)H, l.db + g * H, FLSTM_DTYPE_F32, H, (int)H, 1);
            }
        }
    }
    FLSTM_TRY(batch.run(s, &launches));
    if (comm && t0 == 0) {
        FLSTM_TRY(reduce_grads(0, grad_count, s));
        FLSTM_CUDA_TRY(cudaEventRecord(comm_join, comm_stream));
        FLSTM_CUDA_TRY(cudaStreamWaitEvent(s, comm_join, 0));
    }
    return FLSTM_OK;
}

// Logical copies of the caches for flstm_engine_cache_ptrs: made when they are first asked for, kept up to date by the
// forward calls after that.
int Engine::padded_cache_ptrs(int layer, void **gates, float **cells, void **hiddens) {
    Engine &in = *inner;
    const size_t cap = in.t_cap, B = cfg.batch, H = cfg.hidden_size, L = cfg.layers;
    if (pad.t_mirror != cap) {
        FLSTM_CUDA_TRY(cudaDeviceSynchronize());
        drop(pad.gates);
        drop(pad.hs);
        drop(pad.cs);
        pad.mirror_bytes = 0;
        pad.t_mirror = cap;
    }
    bool fresh = false;
    if (gates && !pad.gates) {
        FLSTM_TRY(grab(&pad.gates, L * cap * B * 4 * H * 2, &pad.mirror_bytes));
        fresh = true;
    }
    if (cells && !pad.cs) {
        FLSTM_TRY(grab(&pad.cs, L * (cap + 1) * B * H * sizeof(float), &pad.mirror_bytes));
        fresh = true;
    }
    if (hiddens && !pad.hs) {
        FLSTM_TRY(grab(&pad.hs, L * (cap + 1) * B * H * 2, &pad.mirror_bytes));
        fresh = true;
    }
    if (fresh) {
        FLSTM_CUDA_TRY(cudaDeviceSynchronize());
        FLSTM_TRY(padded_mirror(0, cap, nullptr));
        FLSTM_CUDA_TRY(cudaDeviceSynchronize());
    }
    if (gates) *gates = bytes(pad.gates) + layer * cap * B * 4 * H * 2;
    if (cells) *cells = pad.cs + layer * (cap + 1) * B * H;
    if (hiddens) *hiddens = bytes(pad.hs) + layer * (cap + 1) * B * H * 2;
    return FLSTM_OK;
}

int Engine::padded_mirror(size_t t0, size_t t1, cudaStream_t s) {
    if ((!pad.gates && !pad.hs && !pad.cs) || pad.t_mirror != inner->t_cap) return FLSTM_OK;
    const size_t cap = pad.t_mirror, B = cfg.batch, H = cfg.hidden_size, Hp = inner->cfg.hidden_size;
    CopyBatch batch;
    for (size_t li = 0; li < layers.size(); ++li) {
        auto &p = inner->layers[li];
        const size_t from = t0 == 0 ? 0 : t0 + 1, n = t1 + 1 - from;  // slots of the state tensors
        if (pad.hs)
            batch.add(bytes(p.hs) + from * B * Hp * 2, cfg.dtype, Hp, (int)H, bytes(pad.hs) + (li * (cap + 1) + from) * B * H * 2, cfg.dtype,
                      H, (int)H, n * B);
        if (pad.cs)
            batch.add(p.cs + from * B * Hp, FLSTM_DTYPE_F32, Hp, (int)H, pad.cs + (li * (cap + 1) + from) * B * H, FLSTM_DTYPE_F32, H,
                      (int)H, n * B);
        if (pad.gates && t1 > t0) {
            const uint16_t *src = static_cast<const uint16_t *>(p.gates) + t0 * B * 4 * Hp;
            unpad_gates_kernel<<<1184, 256, 0, s>>>(src, (int)H, (int)Hp, (t1 - t0) * B,
                                                    static_cast<uint16_t *>(pad.gates) + (li * cap + t0) * B * 4 * H);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "gate copy launch failed: %s", cudaGetErrorString(e));
        }
    }
    return batch.run(s, &launches);
}

}  // namespace flstm_b200
