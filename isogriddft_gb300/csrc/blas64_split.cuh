// FP64 Gram by exact splitting on the tensor cores (blas64_split.cu).
#pragma once

#include "common.cuh"

namespace igd {

constexpr int GRAM64_TILE = 4;  // the plain kernel's output tile

// Outputs that the plain kernel forms: need of each output (0 not, else see gram_redo_kernel), and the tiles with
// such an output, each marked and listed once.
struct Gram64Marks {
  int *tiles, *listed, *list, *need;
};

// Ints behind the partials: a + b row exponents and the marks.
inline long long gram64_tiles(int a, int b) {
  return (long long)((a + GRAM64_TILE - 1) / GRAM64_TILE) * ((b + GRAM64_TILE - 1) / GRAM64_TILE);
}
inline long long gram64_split_ints(int a, int b) {
  return (a + b + 2 * gram64_tiles(a, b) + 1 + (long long)a * b + 1) & ~1LL;
}
// Workspace: partials of a * b integer pairs (16-byte aligned), then the ints.
inline long long gram64_split_bytes(long long partials, int a, int b) {
  return 16 * partials * a * b + gram64_split_ints(a, b) * (long long)sizeof(int);
}
// Partials that a workspace holds.
inline int gram64_split_room(long long bytes, int a, int b) {
  const long long rest = bytes - gram64_split_bytes(0, a, b);
  return rest < 0 ? 0 : (int)std::min<long long>(rest / (16LL * a * b), 1 << 20);
}

// out (a x b) [+]= A W B^T with room for max_blocks (>= 1) partials in the workspace.
int gram64_split_launch(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                        const double* w, double* out, int accumulate, void* workspace, int max_blocks, cudaStream_t st);

// The marked outputs again by the plain FP64 kernel (blas.cu); part: room for `partials` sums of every output, one
// per 16384 points at least.
int gram64_plain_redo(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                      const double* w, double* out, int accumulate, int sym, const Gram64Marks& marks, double* part,
                      long long partials, cudaStream_t st);

}  // namespace igd
