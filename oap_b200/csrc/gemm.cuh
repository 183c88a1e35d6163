// General FP64 matrix product of the operator surface (gemm.cu).
#pragma once

#include <cuda_runtime.h>

namespace oapb {

// C (M x N) = A (M x K) B (K x N), row-major split planes; a null plane of A or
// B is zero, a null plane of C is not written.
int launch_gemm(const double* are, const double* aim, const double* bre, const double* bim, double* cre, double* cim,
                int M, int N, int K, cudaStream_t s);

}  // namespace oapb
