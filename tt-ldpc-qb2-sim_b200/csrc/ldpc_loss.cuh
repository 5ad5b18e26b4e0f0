// Row sums of softplus(-x) and their adjoint (loss.cu): x [rows][n], n a multiple of 4, arrays 16-byte aligned.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace ldpcb200 {

cudaError_t softplus_rows(const float* x, uint64_t rows, int n, float* out, int n_sm, cudaStream_t s);
cudaError_t softplus_rows_grad(const float* x, const float* g, uint64_t rows, int n, float* gx, int n_sm, cudaStream_t s);

}  // namespace ldpcb200
