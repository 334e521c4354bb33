// One time step of one layer in one launch: gates = x W_ih^T + h W_hh^T + b, cell update, for at most 32 sequences.
//
// Generation step by step reads every weight once and multiplies it with a handful of columns.  The projection GEMM pads
// M = 1 to 128 rows on a few CTAs (10 us for 4096 x 1024) and the persistent recurrent kernel loads its 128 KB weight slice
// per CTA before its first step (7 us); with the state copies a two-layer step at H = 1024 took 6 launches and 50 us for
// 34 MB of weights (5 us of HBM time).  Here a CTA owns 8 hidden units (32 gate rows: two m16 tiles holding gates i / f and
// g / o of the same units), its warps take 32-wide K chunks of [x | h] in turn straight from global memory into mma.sync
// operand fragments (16-byte loads, four chunks in flight per warp), and the warps' sums meet in shared memory once.
// States are read where the caller has them and written where the caller wants them.  Two layers, H = 1024, one sequence: 50 -> 8.2 us
// on the device, 97 -> 12 us a call (host work is what is left); bound by the latency of four rounds of loads per warp.
#include "common.cuh"
#include "tc_cluster.cuh"
#include "tc_kernels.h"

namespace flstm_b200 {
namespace tc {

namespace {

template <int NT, bool BF16, bool ACCURATE>
__global__ void __launch_bounds__(512, 1) cell_step_kernel(const CellParams p) {
    extern __shared__ float red[];  // [warp][NT][4 gates][8 units][8 sequences], then the sums of the gates
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, i8 = lane >> 2, q = lane & 3, warps = blockDim.x >> 5;
    const int H = p.H, I = p.I, u = blockIdx.x * 8 + i8;
    const size_t row0 = (size_t)((u >> 4) * 64 + (u & 15));  // gate g of the unit is 16 g rows further
    const int x_chunks = (I + 31) / 32, chunks = x_chunks + (p.h_prev ? H / 32 : 0);
    const uint16_t *w_ih = static_cast<const uint16_t *>(p.w_ih), *w_hh = static_cast<const uint16_t *>(p.w_hh);
    const uint16_t *x = static_cast<const uint16_t *>(p.x), *h = static_cast<const uint16_t *>(p.h_prev);
    float acc[NT][2][4] = {};
    constexpr int DEPTH = NT == 1 ? 4 : 2;
    uint4 w[DEPTH][4];
    auto load_w = [&](int c0) {
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
            const int c = c0 + d * warps;
            const bool of_x = c < x_chunks;
            const int k = (of_x ? c : c - x_chunks) * 32 + 8 * q, K = of_x ? I : H;
            const uint16_t *wrow = (of_x ? w_ih : w_hh) + row0 * K + k;
#pragma unroll
            for (int g = 0; g < 4; ++g)
                w[d][g] = c < chunks && k < K ? __ldg(reinterpret_cast<const uint4 *>(wrow + (size_t)(16 * g) * K)) : make_uint4(0, 0, 0, 0);
        }
    };
    // Weights do not come from the launch before: the first rounds of them are under way before its results are waited for.  The
    // next launch may start once this one has waited, so that whatever it finds here was complete before the first of them.
    load_w(warp);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int c0 = warp; c0 < chunks; c0 += warps * DEPTH) {
        if (c0 != warp) load_w(c0);
        uint4 b[DEPTH][NT];
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
            const int c = c0 + d * warps;
            const bool of_x = c < x_chunks;
            const int k = (of_x ? c : c - x_chunks) * 32 + 8 * q, K = of_x ? I : H;
            const uint16_t *brow = (of_x ? x : h) + k;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int n = nt * 8 + i8;
                b[d][nt] = c < chunks && k < K && n < p.B ? *reinterpret_cast<const uint4 *>(brow + (size_t)n * K) : make_uint4(0, 0, 0, 0);
            }
        }
#pragma unroll
        for (int d = 0; d < DEPTH; ++d)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                mma_16816<BF16>(acc[nt][0], w[d][0].x, w[d][1].x, w[d][0].y, w[d][1].y, b[d][nt].x, b[d][nt].y);
                mma_16816<BF16>(acc[nt][1], w[d][2].x, w[d][3].x, w[d][2].y, w[d][3].y, b[d][nt].x, b[d][nt].y);
                mma_16816<BF16>(acc[nt][0], w[d][0].z, w[d][1].z, w[d][0].w, w[d][1].w, b[d][nt].z, b[d][nt].w);
                mma_16816<BF16>(acc[nt][1], w[d][2].z, w[d][3].z, w[d][2].w, w[d][3].w, b[d][nt].z, b[d][nt].w);
            }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int g = 0; g < 4; ++g)
            *reinterpret_cast<float2 *>(red + ((warp * NT + nt) * 4 + g) * 64 + i8 * 8 + 2 * q) =
                make_float2(acc[nt][g >> 1][(g & 1) * 2], acc[nt][g >> 1][(g & 1) * 2 + 1]);
    __syncthreads();
    float *sums = red + warps * NT * 256;
    for (int e = tid; e < NT * 256; e += blockDim.x) {  // e = (nt, gate, unit, sequence)
        float s = 0.f;
        for (int w = 0; w < warps; ++w) s += red[w * NT * 256 + e];
        const int g = (e >> 6) & 3, uu = blockIdx.x * 8 + ((e >> 3) & 7);
        sums[e] = s + p.bias[(size_t)((uu >> 4) * 64 + g * 16 + (uu & 15))];
    }
    __syncthreads();
    for (int e = tid; e < NT * 64; e += blockDim.x) {  // e = (sequence, unit): neighbouring threads store neighbouring units
        const int n = e >> 3, uu = blockIdx.x * 8 + (e & 7);
        if (n >= p.B) continue;
        const float *v = sums + (n >> 3) * 256 + (e & 7) * 8 + (n & 7);
        const bool pad = ACCURATE && uu >= p.real_units;
        const float gi = sigmoid_sel<ACCURATE>(pad ? 0.f : v[0]), gf = sigmoid_sel<ACCURATE>(pad ? 0.f : v[64]);
        const float gg = tanh_sel<ACCURATE>(pad ? 0.f : v[128]), go = sigmoid_sel<ACCURATE>(pad ? 0.f : v[192]);
        const size_t idx = (size_t)n * H + uu;
        const float c_prev = !p.c_prev ? 0.f : p.c_prev_f32 ? static_cast<const float *>(p.c_prev)[idx]
                                                            : load16<BF16>(static_cast<const uint16_t *>(p.c_prev) + idx);
        if (p.h_first) {
            static_cast<uint16_t *>(p.h_first)[idx] = h ? h[idx] : (uint16_t)0;
            p.c_first[idx] = c_prev;
        }
        const float c = fmaf(gf, c_prev, gi * gg);
        const uint16_t h16 = to16<BF16>(go * tanh_sel<ACCURATE>(c));
        static_cast<uint16_t *>(p.h_out)[idx] = h16;
        p.c_out[idx] = c;
        if (p.y) static_cast<uint16_t *>(p.y)[idx] = h16;
        if (p.hn) static_cast<uint16_t *>(p.hn)[idx] = h16;
        if (p.cn) {
            if (p.cn_f32) static_cast<float *>(p.cn)[idx] = c;
            else static_cast<uint16_t *>(p.cn)[idx] = to16<BF16>(c);
        }
    }
}

}  // namespace

int lstm_cell_step(int dtype, const CellParams &p, cudaStream_t s) {
    const int NT = p.B <= 8 ? 1 : p.B <= 16 ? 2 : 4, chunks = (p.I + 31) / 32 + p.H / 32;
    const int warps = chunks >= 32 ? 16 : 8;
    const bool bf16 = dtype == FLSTM_DTYPE_BF16, accurate = p.real_units > 0;
#define FLSTM_CELL(NT_) \
    (bf16 ? (accurate ? cell_step_kernel<NT_, true, true> : cell_step_kernel<NT_, true, false>) \
          : (accurate ? cell_step_kernel<NT_, false, true> : cell_step_kernel<NT_, false, false>))
    auto kern = NT == 1 ? FLSTM_CELL(1) : NT == 2 ? FLSTM_CELL(2) : FLSTM_CELL(4);
#undef FLSTM_CELL
    const size_t smem = (size_t)(warps + 1) * NT * 256 * sizeof(float);
    FLSTM_CUDA_TRY(ensure_smem_limit(kern, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.H / 8);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.follows ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e != cudaSuccess) return set_error(FLSTM_ERR_CUDA, "cell step launch failed: %s", cudaGetErrorString(e));
    return FLSTM_OK;
}

}  // namespace tc
}  // namespace flstm_b200
