// The training losses' pass over the posteriors: S[row] = sum over the row of softplus(-x), and its adjoint.
// Both losses (mean bit cross-entropy against the all-zero codeword, and the stopping loss) are functions of
// the row sums, one row per frame and iteration.
//
// Bound by memory: the forward reads every posterior once, the backward reads it again and writes its
// gradient.  One warp per row, four float4 loads in flight per lane.  r1/2 K=1024, 4096 frames, 20 iterations
// (839 MB of posteriors): forward 0.19 ms, backward 0.31 ms (B200), where the chain of library kernels it replaces
// (negate, softplus, reduce; expand, softplus backward, negate) took 0.86 and 1.04 ms in passes of 0.84 or 1.7 GB.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ldpc_loss.cuh"

namespace ldpcb200 {

constexpr int LOSS_WARPS = 8;

// softplus(-x) is linear below x = -20, as the library's softplus.  Four values take one logarithm: with z = e^-x
// the sum of log(1 + z) is log(1 + w), w = the product of the 1 + z less 1, built from sums and products of
// nonnegative terms (no cancellation, at most e^80).  minus the derivative by x is sigmoid(-x), 1 below -20 in
// float.
__device__ __forceinline__ float sp_neg4(const float4& v) {
    auto term = [](float x, float& lin) {
        const bool far = x < -20.0f;
        lin += far ? -x : 0.0f;
        return far ? 0.0f : expf(-x);
    };
    auto join = [](float a, float b) { return __fmaf_rn(a, b, a) + b; };  // (1 + a)(1 + b) - 1
    float lin = 0.0f;
    const float a = term(v.x, lin), b = term(v.y, lin), c = term(v.z, lin), d = term(v.w, lin);
    return log1pf(join(join(a, b), join(c, d))) + lin;
}
__device__ __forceinline__ float sig_neg(float x) { return __frcp_rn(1.0f + expf(x)); }

__global__ void __launch_bounds__(32 * LOSS_WARPS) softplus_rows_kernel(const float* __restrict__ x, uint64_t rows, int n4,
                                                                        float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const uint64_t step = (uint64_t)gridDim.x * LOSS_WARPS;
    for (uint64_t r = (uint64_t)blockIdx.x * LOSS_WARPS + (threadIdx.x >> 5); r < rows; r += step) {
        const float4* p = reinterpret_cast<const float4*>(x) + r * (uint64_t)n4;
        float s = 0.0f;
        int i = lane;
        for (; i + 96 < n4; i += 128) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = __ldcs(p + i + 32 * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) s += sp_neg4(v[k]);
        }
        for (; i < n4; i += 32) {
            const float4 v = __ldcs(p + i);
            s += sp_neg4(v);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        if (lane == 0) out[r] = s;
    }
}

__global__ void __launch_bounds__(32 * LOSS_WARPS) softplus_rows_grad_kernel(const float* __restrict__ x,
                                                                             const float* __restrict__ g, uint64_t rows,
                                                                             int n4, float* __restrict__ gx) {
    const int lane = threadIdx.x & 31;
    const uint64_t step = (uint64_t)gridDim.x * LOSS_WARPS;
    for (uint64_t r = (uint64_t)blockIdx.x * LOSS_WARPS + (threadIdx.x >> 5); r < rows; r += step) {
        const float4* p = reinterpret_cast<const float4*>(x) + r * (uint64_t)n4;
        float4* q = reinterpret_cast<float4*>(gx) + r * (uint64_t)n4;
        const float c = -g[r];
        auto grad = [&](const float4& v) { return make_float4(c * sig_neg(v.x), c * sig_neg(v.y), c * sig_neg(v.z), c * sig_neg(v.w)); };
        int i = lane;
        for (; i + 96 < n4; i += 128) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = __ldcs(p + i + 32 * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) q[i + 32 * k] = grad(v[k]);
        }
        for (; i < n4; i += 32) q[i] = grad(__ldcs(p + i));
    }
}

static unsigned loss_grid(uint64_t rows, int n_sm) {
    return (unsigned)std::min<uint64_t>((rows + LOSS_WARPS - 1) / LOSS_WARPS, (uint64_t)n_sm * 8);
}

cudaError_t softplus_rows(const float* x, uint64_t rows, int n, float* out, int n_sm, cudaStream_t s) {
    softplus_rows_kernel<<<loss_grid(rows, n_sm), 32 * LOSS_WARPS, 0, s>>>(x, rows, n / 4, out);
    return cudaGetLastError();
}

cudaError_t softplus_rows_grad(const float* x, const float* g, uint64_t rows, int n, float* gx, int n_sm, cudaStream_t s) {
    softplus_rows_grad_kernel<<<loss_grid(rows, n_sm), 32 * LOSS_WARPS, 0, s>>>(x, g, rows, n / 4, gx);
    return cudaGetLastError();
}

}  // namespace ldpcb200
