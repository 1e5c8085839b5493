// FP64 Gram by exact splitting on the tensor cores (blas64_split.cu).
#pragma once

#include "common.cuh"

namespace igd {

// out (a x b) [+]= A W B^T; part: max_blocks (>= 1) partials of a * b integer pairs, emax: a + b ints.
int gram64_split_launch(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                        const double* w, double* out, int accumulate, longlong2* part, int max_blocks, int* emax,
                        cudaStream_t st);

}  // namespace igd
