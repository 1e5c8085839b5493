// FP64 Gram by exact splitting on the tensor cores (blas64_split.cu).
#pragma once

#include "common.cuh"

namespace igd {

// Workspace: partials of a * b integer pairs (16-byte aligned), then the a + b row exponents.
inline long long gram64_split_bytes(long long partials, int a, int b) {
  return 16 * partials * a * b + ((a + b + 1LL) & ~1LL) * (long long)sizeof(int);
}
// Partials that a workspace holds.
inline int gram64_split_room(long long bytes, int a, int b) {
  const long long rest = bytes - gram64_split_bytes(0, a, b);
  return rest < 0 ? 0 : (int)std::min<long long>(rest / (16LL * a * b), 1 << 20);
}

// out (a x b) [+]= A W B^T with room for max_blocks (>= 1) partials in the workspace.
int gram64_split_launch(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                        const double* w, double* out, int accumulate, void* workspace, int max_blocks, cudaStream_t st);

}  // namespace igd
