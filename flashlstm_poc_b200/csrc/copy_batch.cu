// One launch for a batch of small strided copies (engine.h, CopyBatch): initial and final states of every layer, zero
// padding of tensors whose widths the tensor-core path cannot tile, and the mirror of the error word.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace flstm_b200 {

namespace {

constexpr int kCopyJobs = 24;
struct CopyArgs {
    CopyJob job[kCopyJobs];
    const unsigned int *err;  // device error word and its host mirror (null: not with this launch)
    unsigned int *err_host;
};

template <int BYTES>
struct Piece;
template <> struct Piece<16> { using type = uint4; };
template <> struct Piece<8> { using type = uint2; };
template <> struct Piece<4> { using type = uint32_t; };
template <> struct Piece<2> { using type = uint16_t; };

// V consecutive elements of a row, converted; columns from src_cols on (or all, without a source) are zero
template <typename TI, typename TO, int V>
__device__ __forceinline__ void copy_job(const CopyJob &j) {
    const TI *src = static_cast<const TI *>(j.src);
    TO *dst = static_cast<TO *>(j.dst);
    const unsigned per_row = (unsigned)(j.dst_cols + V - 1) / V;
    const size_t total = j.rows * per_row, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += stride) {
        const size_t r = total <= 0xffffffffu ? (unsigned)i / per_row : i / per_row;
        const int c = (int)(i - r * per_row) * V;
        const TI *from = src + r * j.src_pitch + c;
        TO *to = dst + r * j.dst_pitch + c;
        using In = typename Piece<V * sizeof(TI)>::type;
        using Out = typename Piece<V * sizeof(TO)>::type;
        __align__(16) TI in[V];
        if (!src || c >= j.src_cols) *reinterpret_cast<In *>(in) = In{};
        else *reinterpret_cast<In *>(in) = *reinterpret_cast<const In *>(from);
        __align__(16) TO out[V];
#pragma unroll
        for (int e = 0; e < V; ++e) st(out + e, ld(in + e));
        *reinterpret_cast<Out *>(to) = *reinterpret_cast<const Out *>(out);
    }
}

template <typename TI, typename TO>
__device__ __forceinline__ void copy_any(const CopyJob &j) {
    // four or two elements at a time where columns, pitches and addresses allow it
    auto allows = [&](int v) {
        return (((size_t)j.src_cols | (size_t)j.dst_cols | j.src_pitch | j.dst_pitch) & (v - 1)) == 0 &&
               (reinterpret_cast<uintptr_t>(j.src) & (v * sizeof(TI) - 1)) == 0 &&
               (reinterpret_cast<uintptr_t>(j.dst) & (v * sizeof(TO) - 1)) == 0;
    };
    if (allows(4)) copy_job<TI, TO, 4>(j);
    else if (allows(2)) copy_job<TI, TO, 2>(j);
    else copy_job<TI, TO, 1>(j);
}

__global__ void __launch_bounds__(256) copy_batch_kernel(const __grid_constant__ CopyArgs args) {
    // the host word lies across PCIe: it is written only when there is something to report
    if (args.err && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        const unsigned int code = *args.err;
        if (code) *args.err_host = code;
    }
    const CopyJob &j = args.job[blockIdx.y];
    switch (j.src_dtype * 3 + j.dst_dtype) {
        case FLSTM_DTYPE_F32 * 3 + FLSTM_DTYPE_F32: copy_any<float, float>(j); break;
        case FLSTM_DTYPE_F32 * 3 + FLSTM_DTYPE_F16: copy_any<float, __half>(j); break;
        case FLSTM_DTYPE_F32 * 3 + FLSTM_DTYPE_BF16: copy_any<float, __nv_bfloat16>(j); break;
        case FLSTM_DTYPE_F16 * 3 + FLSTM_DTYPE_F32: copy_any<__half, float>(j); break;
        case FLSTM_DTYPE_F16 * 3 + FLSTM_DTYPE_F16: copy_any<__half, __half>(j); break;
        case FLSTM_DTYPE_BF16 * 3 + FLSTM_DTYPE_F32: copy_any<__nv_bfloat16, float>(j); break;
        case FLSTM_DTYPE_BF16 * 3 + FLSTM_DTYPE_BF16: copy_any<__nv_bfloat16, __nv_bfloat16>(j); break;
    }
}

}  // namespace

void CopyBatch::add(const void *src, int src_dtype, size_t src_pitch, int src_cols, void *dst, int dst_dtype, size_t dst_pitch,
                    int dst_cols, size_t rows) {
    if (rows == 0 || dst_cols == 0) return;
    jobs.push_back({src, dst, rows, src_pitch, dst_pitch, src_cols, dst_cols, src_dtype, dst_dtype});
}

int CopyBatch::run(cudaStream_t s, unsigned long long *launches) {
    for (size_t first = 0; first < jobs.size() || err; first += kCopyJobs) {
        CopyArgs args{};
        const size_t n = jobs.size() - first < (size_t)kCopyJobs ? jobs.size() - first : (size_t)kCopyJobs;
        size_t units = 1;
        for (size_t i = 0; i < n; ++i) {
            const CopyJob &j = args.job[i] = jobs[first + i];
            units = std::max(units, j.rows * (size_t)(j.dst_cols + 3) / 4);
        }
        args.err = err;
        args.err_host = err_host;
        err = nullptr;
        const size_t blocks = std::min<size_t>((units + 255) / 256, 1184);
        copy_batch_kernel<<<dim3((unsigned)blocks, (unsigned)std::max<size_t>(n, 1)), 256, 0, s>>>(args);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "copy batch launch failed: %s", cudaGetErrorString(e));
        if (launches) ++*launches;
    }
    jobs.clear();
    return FLSTM_OK;
}

}  // namespace flstm_b200
