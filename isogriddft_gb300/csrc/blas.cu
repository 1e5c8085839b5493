// Tall-skinny block linear algebra of the eigensolver (K6 Gram, K7 rotation).
//
// Orbital blocks are row-major (k, n): each orbital is one contiguous field.
// Gram: G[i][j] = sum_p A_i[p] W[p] B_j[p]  (weighted_overlap_matrix,
// ks/eigensolver.py:246-272; _weighted_overlap_columns, ks/eigensolver_jax.py:105)
// Rotation: out_j = sum_i A_i C1[i][j] + sum_i B_i C2[i][j]  (basis @ coeffs and
// the two-part compressions of ks/eigensolver_jax.py:178-251).
// FP32 data: products and per-thread sums (at most 64 points) in FP32, block
// and cross-block accumulation in FP64; FP64 data: FP64 throughout, or on large
// grids exact products of digits with a bound on the error (blas64_split.cu).  Cross-block
// sums are deterministic (per-block partials reduced in a second kernel).
#include "blas64_split.cuh"
#include "common.cuh"
#include "gram_tc.cuh"
#include "tma.cuh"

namespace igd {
namespace {

constexpr int GTH = 256;   // threads per Gram block
constexpr long long kGramTcMinPoints = 1LL << 18;  // below this the CUDA-core kernels have less set-up
thread_local int g_gram_path = 0;                   // igd_gram_select
thread_local int g_gram_last = 0;                   // kernel of this thread's last Gram (1 tensor, 2 pipe, 3 tiled)
// FP64: the splitting kernel takes about 22 clocks a point for every 16 x 24 outputs (splitting) plus
// 8 (row exponents), the plain kernels 0.57 a point and output (FP64 pipe).  363609 points, plain /
// split: 4 x 4 111 / 57 us (launch-bound plain grid), 8 x 8 109 / 61, 12 x 12 176 / 82, 21 x 21
// 505 / 161, 34 x 34 1068 / 374; 2000003 points: 4 x 4 122 / 198, 8 x 8 357 / 227, 21 x 21 2519 / 755.
// It would pay from about a thousand points on, but its correctly rounded sums
// differ from the plain ones in the last bit, and on small grids an eigensolve of a closure that is
// not self-adjoint turns that into 1e-8 of an unconverged orbital; below the size where the FP32
// Gram changes kernels too, the plain sums and with them the recorded iterates are kept.
inline bool gram64_split_pays(long long n, int a, int b) {
  return n >= kGramTcMinPoints && 0.57 * a * b > 22.0 * ((a + 15) / 16) * ((b + 23) / 24) + 8.0;
}
constexpr int GPT = 64;    // points per thread and block column (FP32 partial sums stay short)

// FP64 to FP32 on the integer ALUs, as widen (common.cuh).
__device__ __noinline__ float narrow_slow(double x) { return (float)x; }
__device__ __forceinline__ float narrow(double x) {  // to nearest, ties to even
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), e = (hi >> 20) & 0x7ffu;
  if (e - 897u > 253u) return narrow_slow(x);
  unsigned f = (((hi & 0x7fffffffu) - 0x38000000u) << 3) | (lo >> 29);
  const unsigned rest = lo & 0x1fffffffu;
  f += rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
  return __uint_as_float(f | (hi & 0x80000000u));
}
__device__ __forceinline__ double narrow(double x, double) { return x; }
__device__ __forceinline__ float narrow(double x, float) { return narrow(x); }

// Register-tiled tall-skinny Gram.  Block (x, y): tile y of TR x TR outputs
// (rows i0.., columns j0..) over the points of column slice x; each thread
// streams its points straight from global memory (TR + TR + 1 coalesced loads,
// TR^2 FMAs per point) into TR^2 register accumulators of T, then the block
// reduces them in FP64 into part[x][a][b].  The FP64 pipe bounded the FP32 form: it
// converted w at every point of every tile, and 16 sums over 32 lanes one after the
// other took 80 additions per warp.  The lanes now halve the number of sums they
// hold at every step of the same tree (16 additions), and w is narrowed on the
// integer ALUs (35 x 35 over 870001 FP32 points 458 -> 367 us, 21 x 21 215 -> 179, over 20001 26 -> 22; FP64
// 250 thousand points and fewer 7 to 12 %; unrolled by four or eight the large FP32 cases take a fifth more,
// and tiles of 5 to 8 are slower throughout).
// gram_tile_part: one such tile and slice, into part[slice].
template <typename T, int TR>
__device__ __forceinline__ void gram_tile_part(long long n, int a, int b, const T* __restrict__ A, long long sa,
                                               const T* __restrict__ B, long long sb, const double* __restrict__ w,
                                               double* __restrict__ part, int tile, int slice, int slices) {
  const int tb = (b + TR - 1) / TR;
  const int i0 = (tile / tb) * TR, j0 = (tile % tb) * TR;
  T acc[TR][TR];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < TR; ++c) acc[r][c] = T(0);
  const T* Ar[TR];
  const T* Br[TR];
#pragma unroll
  for (int r = 0; r < TR; ++r) {
    Ar[r] = i0 + r < a ? A + (long long)(i0 + r) * sa : nullptr;
    Br[r] = j0 + r < b ? B + (long long)(j0 + r) * sb : nullptr;
  }
#pragma unroll 2
  for (long long p = slice * (long long)GTH + threadIdx.x; p < n; p += (long long)slices * GTH) {
    T av[TR], bv[TR];
    const T wp = w ? narrow(w[p], T()) : T(1);
#pragma unroll
    for (int r = 0; r < TR; ++r) {
      av[r] = Ar[r] ? Ar[r][p] : T(0);
      bv[r] = Br[r] ? Br[r][p] * wp : T(0);
    }
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
      for (int c = 0; c < TR; ++c) acc[r][c] += av[r] * bv[c];
  }
  // Sums over the lanes: step `off` pairs lanes off apart, the upper one of which goes on with the
  // second half of the values, so each pair adds every value once; lane l ends with value `at`.
  static_assert(TR * TR == 16, "four halvings");
  constexpr int WARPS = GTH / 32;
  __shared__ double scratch[WARPS][TR * TR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] = widen(acc[e / TR][e % TR]);
  int at = 0;
#pragma unroll
  for (int half = 8, off = 16; half >= 1; half /= 2, off /= 2) {
    const bool up = lane & off;
    at += up ? half : 0;
#pragma unroll
    for (int e = 0; e < half; ++e) {
      const double keep = up ? v[e + half] : v[e], send = up ? v[e] : v[e + half];
      v[e] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  if (!(lane & 1)) scratch[warp][at] = v[0];
  __syncthreads();
  if (threadIdx.x < 16) {
    const int e = threadIdx.x, r = i0 + e / TR, c = j0 + e % TR;
    static_assert(WARPS == 8, "the tree over eight warps");
    auto pair = [&](int q) { return scratch[q][e] + scratch[q + 4][e]; };
    if (r < a && c < b)
      part[(long long)slice * a * b + (long long)r * b + c] = (pair(0) + pair(2)) + (pair(1) + pair(3));
  }
}

template <typename T, int TR>
__global__ void __launch_bounds__(GTH) gram_tile_kernel(long long n, int a, int b, const T* __restrict__ A,
                                                        long long sa, const T* __restrict__ B, long long sb,
                                                        const double* __restrict__ w, double* __restrict__ part) {
  gram_tile_part<T, TR>(n, a, b, A, sa, B, sb, w, part, blockIdx.y, blockIdx.x, gridDim.x);
}

// The listed tiles of a product that another kernel has formed, again: few tiles in as many slices as fill the
// SMs, many in slices of the plain kernel's length.  The last block of a tile (its count goes up from 1) sums
// the partials and writes the outputs marked in need (2: itself; 1: likewise, or from above the diagonal of a
// symmetric product).
template <int TR>
__global__ void __launch_bounds__(GTH) gram_redo_kernel(long long n, int a, int b, const double* __restrict__ A,
                                                        long long sa, const double* __restrict__ B, long long sb,
                                                        const double* __restrict__ w, const Gram64Marks marks, int sym,
                                                        double* part, long long partials, double* out, int accumulate) {
  __shared__ int last;
  const int count = *marks.listed, tb = (b + TR - 1) / TR;
  if (count == 0) return;
  const long long fill = gridDim.x / count, least = (n + GTH * GPT - 1) / (GTH * GPT);
  const int slices = (int)min(max(min(fill, (n + 4 * GTH - 1) / (4 * GTH)), least), partials);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long item = blockIdx.x; item < (long long)count * slices; item += gridDim.x) {
    const int tile = marks.list[item / slices];
    gram_tile_part<double, TR>(n, a, b, A, sa, B, sb, w, part, tile, (int)(item % slices), slices);
    if (threadIdx.x < 32) {
      __threadfence();  // the partial, written by this warp, is visible before the count
      __syncwarp();
      if (threadIdx.x == 0) last = atomicAdd(marks.tiles + tile, 1) == slices;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      for (int e = warp; e < TR * TR; e += GTH / 32) {
        const int r = (tile / tb) * TR + e / TR, c = (tile % tb) * TR + e % TR;
        if (r >= a || c >= b) continue;
        const long long at = (long long)r * b + c, mirror = (long long)c * b + r;
        double sum = 0.0;
        for (int k = lane; k < slices; k += 32) sum += __ldcg(part + (long long)k * a * b + at);
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
        if (lane != 0) continue;
        const int kind = marks.need[at];
        if (kind == 2 || (kind == 1 && !(sym && r > c))) out[at] = accumulate ? out[at] + sum : sum;
        if (sym && r < c && marks.need[mirror] == 1) out[mirror] = accumulate ? out[mirror] + sum : sum;
      }
    }
    __syncthreads();  // `last` and the tile's scratch are used again
  }
}

// 16-byte asynchronous global->shared copy; the bytes beyond src_bytes are zero-filled.
__device__ __forceinline__ void cp16_zfill(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}

template <typename T>
struct GVec;
template <>
struct GVec<float> {
  using V = float4;
  static constexpr int W = 4;
  __device__ static float dot(const float4& x, const float4& y) { return x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w; }
};
template <>
struct GVec<double> {
  using V = double2;
  static constexpr int W = 2;
  __device__ static double dot(const double2& x, const double2& y) { return x.x * y.x + x.y * y.y; }
};

// Pipelined tall-skinny Gram: every value of A, B and w comes from global
// memory once, by 16-byte cp.async copies into a double-buffered shared chunk
// of P points (all rows; rows padded to a multiple of 4 and their stride by
// one vector against bank conflicts) while the previous chunk is summed.  Each
// group of TPT threads owns a 4 x 4 output tile and sums its share of a chunk
// with 16-byte shared loads (8 loads, 64 FMAs per 4 FP32 points); B is scaled
// by w in shared memory once per chunk.  FP32: per-thread sums of at most 32
// points, compensated (Neumaier) FP32 accumulation across chunks, FP64 tile
// reduction over the group's lanes and across blocks (per-block partials).
template <typename T>
__global__ void __launch_bounds__(GTH) gram_pipe_kernel(long long n, int a, int b, const T* __restrict__ A,
                                                        long long sa, const T* __restrict__ B, long long sb,
                                                        const double* __restrict__ w, double* __restrict__ part, int P,
                                                        int TPT) {
  using G = GVec<T>;
  using V = typename G::V;
  constexpr int VW = G::W;
  extern __shared__ __align__(16) unsigned char gsm[];
  const int ap = (a + 3) & ~3, bp = (b + 3) & ~3, PP = P + VW;
  const size_t rows = (size_t)(ap + bp) * PP;
  T* const buf0 = reinterpret_cast<T*>(gsm);
  double* const wb0 = reinterpret_cast<double*>(buf0 + 2 * rows);
  const int tb = bp / 4, ntiles = (ap / 4) * tb;
  const int tid = threadIdx.x, tile = tid / TPT, lt = tid % TPT;
  const bool act = tile < ntiles;
  const int i0 = act ? (tile / tb) * 4 : 0, j0 = act ? (tile % tb) * 4 : 0;
  const int vpr = P / VW;  // vectors per row of a chunk
  // padding rows stay zero (never copied into)
  for (int q = 0; q < 2; ++q) {
    T* As = buf0 + q * rows;
    for (int e = tid; e < (ap - a) * PP; e += GTH) As[(size_t)a * PP + e] = T(0);
    for (int e = tid; e < (bp - b) * PP; e += GTH) As[(size_t)(ap + b) * PP + e] = T(0);
  }
  const long long nchunks = (n + P - 1) / P;
  auto issue = [&](long long c, int q) {
    const long long p0 = c * P;
    T* As = buf0 + q * rows;
    T* Bs = As + (size_t)ap * PP;
    for (int e = tid; e < (a + b) * vpr; e += GTH) {
      const int row = e / vpr, v = e - row * vpr;
      const long long p = p0 + (long long)v * VW, left = n - p;
      const int bytes = left >= VW ? 16 : (left > 0 ? (int)left * (int)sizeof(T) : 0);
      if (row < a)
        cp16_zfill(As + (size_t)row * PP + v * VW, A + (long long)row * sa + (bytes ? p : 0), bytes);
      else
        cp16_zfill(Bs + (size_t)(row - a) * PP + v * VW, B + (long long)(row - a) * sb + (bytes ? p : 0), bytes);
    }
    if (w) {
      double* wq = wb0 + q * P;
      for (int e = tid; e < P / 2; e += GTH) {
        const long long p = p0 + 2 * e, left = n - p;
        const int bytes = left >= 2 ? 16 : (left > 0 ? 8 : 0);
        cp16_zfill(wq + 2 * e, w + (bytes ? p : 0), bytes);
      }
    }
  };
  T hi[4][4], lo[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) hi[r][c] = lo[r][c] = T(0);
  long long c = blockIdx.x;
  if (c < nchunks) issue(c, 0);
  cp_async_commit();
  for (int q = 0; c < nchunks; c += gridDim.x, q ^= 1) {
    if (c + gridDim.x < nchunks) issue(c + gridDim.x, q ^ 1);
    cp_async_commit();
    cp_async_wait<1>();  // chunk c has landed (the next may still be in flight)
    __syncthreads();
    T* As = buf0 + q * rows;
    T* Bs = As + (size_t)ap * PP;
    if (w) {
      const double* wq = wb0 + q * P;
      for (int e = tid; e < b * P; e += GTH) {
        const int j = e / P, x = e - j * P;
        Bs[(size_t)j * PP + x] *= T(wq[x]);
      }
      __syncthreads();
    }
    if (act) {
      const V* Av = reinterpret_cast<const V*>(As + (size_t)i0 * PP);
      const V* Bv = reinterpret_cast<const V*>(Bs + (size_t)j0 * PP);
      const int rowv = PP / VW;
      for (int g0 = lt; g0 < vpr; g0 += 8 * TPT) {
        T sacc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) sacc[r][cc] = T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int g = g0 + u * TPT;
          if (g < vpr) {
            V av[4], bv[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) av[r] = Av[r * rowv + g];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) bv[cc] = Bv[cc * rowv + g];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int cc = 0; cc < 4; ++cc) sacc[r][cc] += G::dot(av[r], bv[cc]);
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            if constexpr (sizeof(T) == 8) {
              hi[r][cc] += sacc[r][cc];
            } else {  // Neumaier: the rounding error of each addition goes to lo
              const T t = hi[r][cc] + sacc[r][cc];
              lo[r][cc] += fabsf(hi[r][cc]) >= fabsf(sacc[r][cc]) ? (hi[r][cc] - t) + sacc[r][cc]
                                                                  : (sacc[r][cc] - t) + hi[r][cc];
              hi[r][cc] = t;
            }
          }
      }
    }
    __syncthreads();  // buffer q is refilled by the next iteration's copies
  }
  cp_async_wait<0>();
  // FP64 sum over the TPT contiguous lanes of each tile group
  double v[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) v[r][cc] = (double)hi[r][cc] + (double)lo[r][cc];
  for (int off = TPT / 2; off > 0; off >>= 1)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) v[r][cc] += __shfl_down_sync(0xffffffffu, v[r][cc], off);
  if (act && lt == 0) {
    double* pb = part + (long long)blockIdx.x * a * b;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc)
        if (i0 + r < a && j0 + cc < b) pb[(long long)(i0 + r) * b + j0 + cc] = v[r][cc];
  }
}

// out[e] (+)= sum over blocks of part[k][e]: one warp per output (lanes stride
// over the blocks, then a fixed-order shuffle tree: deterministic).
__global__ void gram_reduce_kernel(int nblocks, int ab, const double* __restrict__ part, double* __restrict__ out,
                                   int accumulate) {
  const int lane = threadIdx.x & 31;
  for (int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < ab; e += (gridDim.x * blockDim.x) >> 5) {
    double s = 0.0;
    for (int k = lane; k < nblocks; k += 32) s += part[(long long)k * ab + e];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) out[e] = accumulate ? out[e] + s : s;
  }
}

constexpr int RTH = 256;
// FP32 rotations.  Two points per thread from ROT_PAIR_POINTS on: 21 rows to 20 columns take 8.4 us with
// one and 7.4 with two over 117649 points; over 40000, 5.3 with one.
constexpr long long ROT_PAIR_POINTS = 100000;
// The pipeline's batches and its lower line: 22 rows to 20 columns over 363608 points take 15.2 us there and
// 14.9 in the register kernel, 50 to 35 over 10^6 124 and 160, 19 to 12 23 and 37 (rotate_kernel).  Up to
// ROT_PIPE_COEF coefficients, rows x columns, fit beside the ring.  Up to 16 columns the ring is 96 KB, and from
// about 16 KB of coefficients on (at the padded width) a CTA is alone on its SM: slower, but still ahead of
// rotate_kernel.  2^19 points, pipeline / rotate_kernel: 341 rows to 12 columns 177 / 300 us (two CTAs), 512 to
// 12 300 / 439 (one), 256 to 13 162 / 230 (two), 470 to 13 328 / 407 (one), 384 to 16 275 / 335 (one), 1536 to 4
// 616 / 839 (one), 6144 to 1 2407 / 10155 (one).
constexpr int ROT_STAGES = 3, ROT_ROWS = 8;
constexpr long long ROT_PIPE_POINTS = 1 << 19, ROT_PIPE_COEF = 6 * 1024;

// out[j][p] (+)= sum_i A[i][p] C1[i][j] + sum_i B[i][p] C2[i][j] for j in
// [j0, j0 + RC), RC from rotate_dispatch.
template <typename T, int RC>
__global__ void __launch_bounds__(RTH) rotate_kernel(long long n, int a, const T* __restrict__ A, long long sa,
                                                     const double* __restrict__ C1, int b, const T* __restrict__ B,
                                                     long long sb, const double* __restrict__ C2, int c,
                                                     T* __restrict__ out, long long so, int accumulate) {
  extern __shared__ __align__(16) unsigned char rsm[];
  T* cs = reinterpret_cast<T*>(rsm);  // (a + b) x RC
  const int j0 = blockIdx.y * RC;
  const int nj = min(RC, c - j0);
  for (int e = threadIdx.x; e < (a + b) * RC; e += RTH) {
    const int i = e / RC, jj = e - i * RC;
    double v = 0.0;
    if (jj < nj) v = i < a ? C1[(long long)i * c + j0 + jj] : C2[(long long)(i - a) * c + j0 + jj];
    cs[e] = T(v);
  }
  __syncthreads();
  for (long long p = blockIdx.x * (long long)RTH + threadIdx.x; p < n; p += (long long)gridDim.x * RTH) {
    T acc[RC];
#pragma unroll
    for (int jj = 0; jj < RC; ++jj) acc[jj] = T(0);
    // rows in batches of 8: the batch's loads are all in flight before its FMAs
    auto rows = [&](const T* __restrict__ M, long long sm, int m, const T* coef) {
      int i = 0;
      for (; i + 8 <= m; i += 8) {
        T x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = M[(long long)(i + u) * sm + p];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const T* row = coef + (i + u) * RC;
#pragma unroll
          for (int jj = 0; jj < RC; ++jj) acc[jj] += x[u] * row[jj];
        }
      }
      for (; i < m; ++i) {
        const T x = M[(long long)i * sm + p];
        const T* row = coef + i * RC;
#pragma unroll
        for (int jj = 0; jj < RC; ++jj) acc[jj] += x * row[jj];
      }
    };
    rows(A, sa, a, cs);
    if (b) rows(B, sb, b, cs + a * RC);
#pragma unroll
    for (int jj = 0; jj < RC; ++jj)
      if (jj < nj) {
        T* o = out + (long long)(j0 + jj) * so + p;
        *o = accumulate ? *o + acc[jj] : acc[jj];
      }
  }
}

template <typename T, int RC>
int rotate_launch(long long n, int a, const T* A, long long sa, const double* C1, int b, const T* B, long long sb,
                  const double* C2, int c, T* out, long long so, int accumulate, cudaStream_t st) {
  const size_t smem = (size_t)(a + b) * RC * sizeof(T);
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(rotate_kernel<T, RC>), smem) != IGD_OK) return IGD_ERR_CUDA;
  const long long blocks = std::min<long long>((n + RTH - 1) / RTH, 152LL * 8);
  dim3 grid((unsigned)blocks, (c + RC - 1) / RC);
  rotate_kernel<T, RC><<<grid, RTH, smem, st>>>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate);
  return IGD_OK;
}

// Two FP32 FMAs on a packed pair, each rounded as fmaf: same rate as two FMAs, half the issue slots.
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long x, unsigned long long c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(x), "l"(c));
}
__device__ __forceinline__ unsigned long long dup2(float x) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ float lane_of(unsigned long long d, int odd) {
  return __uint_as_float((unsigned)(odd ? d >> 32 : d));
}

// FP32 rotation with the rows straight from memory, for rows that the pipeline
// cannot copy in 16-byte pieces and for small grids: PP points per thread, RTH
// apart, so the loads are coalesced whatever the strides and the alignment, and
// packed column pairs, up to the next multiple of four.  50 rows to 35 columns
// over 1000003 points: rotate_kernel (two tiles of 32) 317 us, this form 160; 22 to
// 20 over 363609: 26.8 and 15.8.
template <int RC, int PP>
__global__ void __launch_bounds__(RTH, RC * PP <= 20 ? 3 : 2) rotate32_kernel(long long n, int a, const float* __restrict__ A,
                                                          long long sa, const double* __restrict__ C1, int b,
                                                          const float* __restrict__ B, long long sb,
                                                          const double* __restrict__ C2, int c,
                                                          float* __restrict__ out, long long so, int accumulate) {
  constexpr int U = PP == 2 && RC >= 24 ? (RC >= 32 ? 4 : 2) : 8;  // rows whose loads are in flight together
  extern __shared__ __align__(16) unsigned char rsm[];
  float* cs = reinterpret_cast<float*>(rsm);  // (a + b) x RC
  const int j0 = blockIdx.y * RC;
  const int nj = min(RC, c - j0);
  for (int e = threadIdx.x; e < (a + b) * RC; e += RTH) {
    const int i = e / RC, jj = e - i * RC;
    double v = 0.0;
    if (jj < nj) v = i < a ? C1[(long long)i * c + j0 + jj] : C2[(long long)(i - a) * c + j0 + jj];
    cs[e] = float(v);
  }
  __syncthreads();
  for (long long p0 = blockIdx.x * (long long)(RTH * PP) + threadIdx.x; p0 < n;
       p0 += (long long)gridDim.x * (RTH * PP)) {
    unsigned long long acc[PP][RC / 2];
#pragma unroll
    for (int q = 0; q < PP; ++q)
#pragma unroll
      for (int jj = 0; jj < RC / 2; ++jj) acc[q][jj] = 0ull;
    bool in[PP];
#pragma unroll
    for (int q = 0; q < PP; ++q) in[q] = p0 + q * RTH < n;
    auto rows = [&](const float* __restrict__ M, long long sm, int m, const float* coef) {
      M += p0;
      auto row_fma = [&](const float(&x)[PP], const float* row) {
        unsigned long long xx[PP];
#pragma unroll
        for (int q = 0; q < PP; ++q) xx[q] = dup2(x[q]);
#pragma unroll
        for (int j4 = 0; j4 < RC / 4; ++j4) {
          const ulonglong2 k = reinterpret_cast<const ulonglong2*>(row)[j4];
#pragma unroll
          for (int q = 0; q < PP; ++q) {
            fma2(acc[q][2 * j4], xx[q], k.x);
            fma2(acc[q][2 * j4 + 1], xx[q], k.y);
          }
        }
      };
      int i = 0;
      for (; i + U <= m; i += U) {
        float x[U][PP];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < PP; ++q) x[u][q] = in[q] ? M[(long long)(i + u) * sm + q * RTH] : 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) row_fma(x[u], coef + (i + u) * RC);
      }
      for (; i < m; ++i) {
        float x[PP];
#pragma unroll
        for (int q = 0; q < PP; ++q) x[q] = in[q] ? M[(long long)i * sm + q * RTH] : 0.f;
        row_fma(x, coef + i * RC);
      }
    };
    rows(A, sa, a, cs);
    if (b) rows(B, sb, b, cs + a * RC);
#pragma unroll
    for (int q = 0; q < PP; ++q)
      if (in[q]) {
#pragma unroll
        for (int jj = 0; jj < RC; ++jj)
          if (jj < nj) {
            float* o = out + (long long)(j0 + jj) * so + p0 + q * RTH;
            const float v = lane_of(acc[q][jj / 2], jj & 1);
            *o = accumulate ? *o + v : v;
          }
      }
  }
}

template <int RC>
int rotate32_launch(long long n, int a, const float* A, long long sa, const double* C1, int b, const float* B,
                    long long sb, const double* C2, int c, float* out, long long so, int accumulate, cudaStream_t st) {
  const size_t smem = (size_t)(a + b) * RC * sizeof(float);
  auto go = [&](auto kern, int pp) {
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != IGD_OK) return IGD_ERR_CUDA;
    const long long blocks = std::min<long long>((n + RTH * pp - 1) / (RTH * pp), 152LL * 8);
    kern<<<dim3((unsigned)blocks, (c + RC - 1) / RC), RTH, smem, st>>>(n, a, A, sa, C1, b, B, sb, C2, c, out, so,
                                                                       accumulate);
    return IGD_OK;
  };
  if (n >= ROT_PAIR_POINTS) return go(rotate32_kernel<RC, 2>, 2);
  return go(rotate32_kernel<RC, 1>, 1);
}

// FP32 rotation through a shared-memory pipeline: the sums of rotate_kernel in
// the same order.  A CTA takes tiles of PT points and all H * CW output columns;
// a thread takes Q groups of four consecutive points and CW columns, so a
// 16-byte coefficient read serves 16 Q FMAs (one point per thread: four, and
// the shared-memory port is the bound).  Rows arrive in batches of ROT_ROWS
// through a ring of ROT_STAGES cp.async stages that runs on across tiles.
// 47 rows to 32 columns over 192^3 points: rotate_kernel 1009 us, this form 549
// (floor 329 at the memory, 285 at the FP32 pipe), with Q = 1 and CW = 16, whose
// coefficient reads weigh more, 599; with one batch of 4 rows per stage 710.
template <int Q, int CW, int H>
__global__ void __launch_bounds__(RTH, Q * CW <= 16 ? 2 : 1)
    rotate_pipe_kernel(long long n, int a, const float* __restrict__ A, long long sa, const double* __restrict__ C1,
                       int b, const float* __restrict__ B, long long sb, const double* __restrict__ C2, int c,
                       float* __restrict__ out, long long so, int accumulate) {
  constexpr int TH = RTH / H, PT = 4 * Q * TH, W = H * CW;
  extern __shared__ __align__(16) unsigned char rsm[];
  float* xs = reinterpret_cast<float*>(rsm);    // ROT_STAGES x ROT_ROWS x PT
  float* cs = xs + ROT_STAGES * ROT_ROWS * PT;  // (a + b) x W
  const int j0 = blockIdx.y * W;
  const int m = a + b, tid = threadIdx.x;
  for (int e = tid; e < m * W; e += RTH) {
    const int i = e / W, jj = e - i * W;
    double v = 0.0;
    if (j0 + jj < c) v = i < a ? C1[(long long)i * c + j0 + jj] : C2[(long long)(i - a) * c + j0 + jj];
    cs[e] = float(v);
  }
  const int batches = (m + ROT_ROWS - 1) / ROT_ROWS;
  const long long tiles = (n + PT - 1) / PT;
  const long long mine = tiles > blockIdx.x ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  // tile and batch of the next stage to fetch, stages left
  long long ft = blockIdx.x, left = mine * batches;
  int fb = 0;
  const unsigned xs0 = (unsigned)__cvta_generic_to_shared(xs);
  auto fetch = [&](int slot) {
    if (left > 0) {
      --left;
      constexpr int V = PT / 4;  // 16-byte pieces of a row; points past n read as zero
      const long long p0 = ft * PT;
      const int i0 = fb * ROT_ROWS, rows = min(ROT_ROWS, m - i0);
      const int x = (tid % V) * 4;
      const long long rest = n - p0 - x;
      const int bytes = rest >= 4 ? 16 : rest > 0 ? (int)rest * 4 : 0;
      for (int r = tid / V; r < rows; r += RTH / V) {
        const int i = i0 + r;
        const float* src = (i < a ? A + (long long)i * sa : B + (long long)(i - a) * sb) + (bytes ? p0 + x : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                         xs0 + (unsigned)((slot * ROT_ROWS + r) * PT + x) * 4u),
                     "l"(src), "r"(bytes)
                     : "memory");
      }
      if (++fb == batches) {
        fb = 0;
        ft += gridDim.x;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int k = 0; k < ROT_STAGES - 1; ++k) fetch(k);

  const int part = tid / TH, px = (tid % TH) * 4;
  int slot = 0;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    unsigned long long acc[4 * Q][CW / 2];
#pragma unroll
    for (int q = 0; q < 4 * Q; ++q)
#pragma unroll
      for (int jj = 0; jj < CW / 2; ++jj) acc[q][jj] = 0ull;
    for (int ib = 0; ib < batches; ++ib) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(ROT_STAGES - 2) : "memory");
      __syncthreads();  // the stage is visible, and every thread has left the one refilled next
      fetch(slot == 0 ? ROT_STAGES - 1 : slot - 1);
      const float* x0 = xs + slot * ROT_ROWS * PT + px;
      const float* k0 = cs + ib * ROT_ROWS * W + part * CW;
      const int rows = min(ROT_ROWS, m - ib * ROT_ROWS);
      auto row = [&](int r) {
        unsigned long long xx[4 * Q];
#pragma unroll
        for (int g = 0; g < Q; ++g) {
          const float4 x = *reinterpret_cast<const float4*>(x0 + r * PT + g * 4 * TH);
          xx[4 * g] = dup2(x.x);
          xx[4 * g + 1] = dup2(x.y);
          xx[4 * g + 2] = dup2(x.z);
          xx[4 * g + 3] = dup2(x.w);
        }
#pragma unroll
        for (int j4 = 0; j4 < CW / 4; ++j4) {
          const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(k0 + r * W + 4 * j4);
#pragma unroll
          for (int q = 0; q < 4 * Q; ++q) {
            fma2(acc[q][2 * j4], xx[q], k.x);
            fma2(acc[q][2 * j4 + 1], xx[q], k.y);
          }
        }
      };
      if (rows == ROT_ROWS) {
#pragma unroll 2  // four spill
        for (int r = 0; r < ROT_ROWS; ++r) row(r);
      } else {
        for (int r = 0; r < rows; ++r) row(r);
      }
      slot = slot == ROT_STAGES - 1 ? 0 : slot + 1;
    }
#pragma unroll
    for (int g = 0; g < Q; ++g) {
      const long long p = t * PT + g * 4 * TH + px;
#pragma unroll
      for (int jj = 0; jj < CW; ++jj) {
        const int j = j0 + part * CW + jj;
        if (j >= c) continue;
        float* o = out + (long long)j * so + p;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = lane_of(acc[4 * g + q][jj / 2], jj & 1);
        if (p + 4 <= n) {
          float4* o4 = reinterpret_cast<float4*>(o);
          if (accumulate) {
            const float4 w = *o4;
            *o4 = make_float4(w.x + v[0], w.y + v[1], w.z + v[2], w.w + v[3]);
          } else {
            *o4 = make_float4(v[0], v[1], v[2], v[3]);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (p + q < n) o[q] = accumulate ? o[q] + v[q] : v[q];
        }
      }
    }
  }
}

template <int Q, int CW, int H>
int rotate_pipe_launch(long long n, int a, const float* A, long long sa, const double* C1, int b, const float* B,
                       long long sb, const double* C2, int c, float* out, long long so, int accumulate,
                       cudaStream_t st) {
  constexpr int PT = 4 * Q * RTH / H, W = H * CW;
  const size_t smem = (size_t)ROT_STAGES * ROT_ROWS * PT * 4 + (size_t)(a + b) * W * 4;
  auto kern = rotate_pipe_kernel<Q, CW, H>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != IGD_OK) return IGD_ERR_CUDA;
  const long long blocks = std::min<long long>((n + PT - 1) / PT, (Q * CW <= 16 ? 2LL : 1LL) * device_sm_count());
  kern<<<dim3((unsigned)blocks, (c + W - 1) / W), RTH, smem, st>>>(n, a, A, sa, C1, b, B, sb, C2, c, out, so,
                                                                   accumulate);
  return IGD_OK;
}

template <typename T>
int rotate_dispatch(long long n, int a, const T* A, long long sa, const double* C1, int b, const T* B, long long sb,
                    const double* C2, int c, T* out, long long so, int accumulate, cudaStream_t st) {
  // coefficients of one column tile in shared memory, by the padded widths of the plain kernel; every
  // other form's tile is no larger
  const int rc = c <= 4 ? 4 : c <= 8 ? 8 : c <= 16 ? 16 : 32;
  if ((size_t)(a + b) * rc * sizeof(T) > 200 * 1024) return IGD_ERR_TOO_LARGE;
  if constexpr (sizeof(T) == 8) {
    // The FP64 pipe (two lanes per clock and SM) bounds this form, so no column is padded: equal
    // tiles of at most 20 columns (40 accumulator registers), the width compiled in.  21 -> 20
    // columns over 363609 points: one 32-column tile 424 us, 20 columns 269 us; 21 -> 1 with 4 columns 58
    // us, with one 19 us.
    const int tiles = (c + 19) / 20;
    switch ((c + tiles - 1) / tiles) {
#define IGD_ROT(RC) \
  case RC: return rotate_launch<T, RC>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
      IGD_ROT(1) IGD_ROT(2) IGD_ROT(3) IGD_ROT(4) IGD_ROT(5) IGD_ROT(6) IGD_ROT(7) IGD_ROT(8) IGD_ROT(9) IGD_ROT(10)
      IGD_ROT(11) IGD_ROT(12) IGD_ROT(13) IGD_ROT(14) IGD_ROT(15) IGD_ROT(16) IGD_ROT(17) IGD_ROT(18) IGD_ROT(19)
      IGD_ROT(20)
#undef IGD_ROT
    }
    return IGD_ERR_ARG;
  } else {
    const int cols = std::min(c, 64);
    auto al = [](const void* p, long long s) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && s % 4 == 0; };
    if (n >= ROT_PIPE_POINTS && (long long)(a + b) * cols <= ROT_PIPE_COEF && al(A, sa) && (b == 0 || al(B, sb)) &&
        al(out, so)) {
#define IGD_ROT(LO, Q, CW, HH) \
  if (cols > LO) return rotate_pipe_launch<Q, CW, HH>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
      IGD_ROT(48, 1, 16, 4)
      IGD_ROT(32, 1, 12, 4)
      IGD_ROT(24, 2, 8, 4)
      IGD_ROT(16, 1, 12, 2)
      IGD_ROT(12, 1, 16, 1)
      IGD_ROT(8, 1, 12, 1)
      IGD_ROT(4, 1, 8, 1)
      IGD_ROT(0, 1, 4, 1)
#undef IGD_ROT
    }
    // up to 16 columns the plain kernel's occupancy counts for more: 19 rows to 12 columns over 1000003
    // points take 37.5 us there, 46 with packed pairs
    if (c <= 4) return rotate_launch<T, 4>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
    if (c <= 8) return rotate_launch<T, 8>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
    if (c <= 16) return rotate_launch<T, 16>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
    const int tiles = (c + 31) / 32;
    switch (((c + tiles - 1) / tiles + 3) / 4) {
#define IGD_ROT(Q) \
  case Q: return rotate32_launch<4 * Q>(n, a, A, sa, C1, b, B, sb, C2, c, out, so, accumulate, st);
      IGD_ROT(5) IGD_ROT(6) IGD_ROT(7) IGD_ROT(8)
#undef IGD_ROT
    }
    return IGD_ERR_ARG;
  }
}

// Blocks (and per-block partials) of a Gram: one column slice of GTH x GPT
// points per block for the register-tiled kernel, a persistent grid of up to
// 608 blocks (4 per SM) for the pipelined one.
inline int gram_tiled_blocks(long long n) {
  const long long per = (long long)GTH * GPT;
  return (int)std::max<long long>(1, std::min<long long>((n + per - 1) / per, 4096));
}
inline int gram_pipe_blocks(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 608)); }
inline int gram_blocks(long long n) { return std::max(gram_tiled_blocks(n), gram_pipe_blocks(n)); }

// Chunk length P (points, a power of two) and threads per output tile TPT of
// gram_pipe_kernel, with its shared-memory bytes; false when it does not apply
// (more than 64 x 64 outputs, unaligned rows, or no chunk fits 96 KB).
template <typename T>
bool gram_pipe_plan(int a, int b, const void* A, long long sa, const void* B, long long sb, const double* w, int* P,
                    int* TPT, size_t* smem) {
  constexpr int VW = 16 / (int)sizeof(T);
  auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (!al(A) || !al(B) || (w && !al(w)) || sa % VW != 0 || sb % VW != 0) return false;
  const int ap = (a + 3) & ~3, bp = (b + 3) & ~3, ntiles = (ap / 4) * (bp / 4);
  if (ntiles > GTH) return false;
  auto bytes = [&](int p) { return 2 * ((size_t)(ap + bp) * (p + VW) * sizeof(T) + (size_t)p * sizeof(double)); };
  int p = 256;
  while (p > 32 && bytes(p) > 96 * 1024) p >>= 1;
  if (bytes(p) > 96 * 1024) return false;
  int tpt = 32;
  while (tpt > 1 && (tpt * ntiles > GTH || p / VW < tpt)) tpt >>= 1;
  *P = p;
  *TPT = tpt;
  *smem = bytes(p);
  return true;
}

template <typename T>
int gram_pipe_launch(long long n, int a, int b, const T* A, long long sa, const T* B, long long sb, const double* w,
                     double* part, int nb, cudaStream_t st) {
  int P = 0, TPT = 0;
  size_t smem = 0;
  if (!gram_pipe_plan<T>(a, b, A, sa, B, sb, w, &P, &TPT, &smem)) return -1;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gram_pipe_kernel<T>), smem) != IGD_OK) return IGD_ERR_CUDA;
  gram_pipe_kernel<T><<<nb, GTH, smem, st>>>(n, a, b, A, sa, B, sb, w, part, P, TPT);
  return IGD_OK;
}

// Damped Jacobi sweep for (T + sigma) t = r on k columns:
// first: t = dinv r; else t += omega dinv (r - tt - sigma t), tt = T t.
template <typename T>
__global__ void jacobi_kernel(long long n, int k, const T* __restrict__ r, long long sr, T* __restrict__ t,
                              long long st, const T* __restrict__ tt, long long stt, const T* __restrict__ dinv,
                              T sigma, T omega, int first) {
  const int c = blockIdx.y;  // one column per grid row: no division per element
  const T* rc = r + c * sr;
  T* tc = t + c * st;
  const T* ttc = first ? nullptr : tt + c * stt;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const T rv = rc[p], di = dinv[p];
    if (first)
      tc[p] = di * rv;
    else
      tc[p] += omega * di * (rv - ttc[p] - sigma * tc[p]);
  }
}

}  // namespace

int gram64_plain_redo(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                      const double* w, double* out, int accumulate, int sym, const Gram64Marks& marks, double* part,
                      long long partials, cudaStream_t st) {
  gram_redo_kernel<GRAM64_TILE><<<2 * device_sm_count(), GTH, 0, st>>>(n, a, b, A, sa, B, sb, w, marks, sym, part,
                                                                       partials, out, accumulate);
  return launch_status();
}
}  // namespace igd

using namespace igd;

// Residual preconditioner step (see jacobi_kernel); dinv = 1 / (diag(T) + sigma).
extern "C" int igd_precond_jacobi(int dtype, long long n, int k, const void* r, long long sr, void* t, long long st,
                                  const void* tt, long long stt, const void* dinv, double sigma, double omega,
                                  int first, void* stream) {
  if (n <= 0 || k <= 0 || k > 65535 || !r || !t || !dinv || (!first && !tt)) return IGD_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  const dim3 blocks((unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152LL * 16 / k + 1)),
                    (unsigned)k);
  if (dtype == IGD_F32)
    jacobi_kernel<float><<<blocks, 256, 0, s>>>(n, k, static_cast<const float*>(r), sr, static_cast<float*>(t), st,
                                                static_cast<const float*>(tt), stt, static_cast<const float*>(dinv),
                                                (float)sigma, (float)omega, first);
  else if (dtype == IGD_F64)
    jacobi_kernel<double><<<blocks, 256, 0, s>>>(n, k, static_cast<const double*>(r), sr, static_cast<double*>(t), st,
                                                 static_cast<const double*>(tt), stt,
                                                 static_cast<const double*>(dinv), sigma, omega, first);
  else
    return IGD_ERR_DTYPE;
  return launch_status();
}

// Gram kernel choice for the calling host thread (tests): 0 automatic, 1 the
// tcgen05 kernel where it applies, 2 the pipelined CUDA-core kernel, 3 the
// register-tiled kernel, 4 the FP64 splitting kernel (FP64 data).
extern "C" int igd_gram_select(int path) {
  if (path < 0 || path > 4) return IGD_ERR_ARG;
  g_gram_path = path;
  return IGD_OK;
}

// Per-block partials of the plain kernels and the FP32 tensor-core one; the workspace that every call needs.
static long long gram_plain_bytes(long long n, int a, int b) {
  return (long long)gram_blocks(n) * a * b * (long long)sizeof(double);
}

// Kernel used by the calling thread's last igd_block_gram (0 before any call).
extern "C" int igd_gram_last_path(void) { return g_gram_last; }

extern "C" long long igd_block_gram_workspace_bytes(long long n, int a, int b) {
  if (n <= 0 || a <= 0 || b <= 0) return -1;
  return gram_plain_bytes(n, a, b) + gram64_split_bytes(1, a, b);
}

// out (a x b, FP64, row-major) [+]= A W B^T for row-major blocks A (a x n, row
// stride sa) and B (b x n, stride sb); w (n doubles) may be NULL.
extern "C" int igd_block_gram(int dtype, long long n, int a, const void* A, long long sa, int b, const void* B,
                              long long sb, const double* w, double* out, int accumulate, void* workspace,
                              long long workspace_bytes, void* stream) {
  if (n <= 0 || a <= 0 || b <= 0 || !A || !B || !out || !workspace) return IGD_ERR_ARG;
  if (workspace_bytes < gram_plain_bytes(n, a, b)) return IGD_ERR_ARG;
  if (dtype != IGD_F32 && dtype != IGD_F64) return IGD_ERR_DTYPE;
  cudaStream_t st = as_stream(stream);
  int nb = gram_pipe_blocks(n);
  double* part = static_cast<double*>(workspace);
  const int path = g_gram_path;
  // FP32: the tcgen05 3xTF32 kernel (outputs up to 64 x 64, 16-byte rows) on large grids
  if (dtype == IGD_F32 && (path == 1 || (path == 0 && n >= kGramTcMinPoints))) {
    const int r = gram_tc_launch(n, a, b, static_cast<const float*>(A), sa, static_cast<const float*>(B), sb, w, part,
                                 gram_blocks(n), device_error_word(), st);
    if (r > 0) {
      g_gram_last = 1;
      const int ab = a * b;
      gram_reduce_kernel<<<std::min((ab * 32 + 255) / 256, 1024), 256, 0, st>>>(r, ab, part, out, accumulate);
      return launch_status();
    }
    if (r != -1) return r;
  }
  // FP64: exact splitting, in a workspace that is aligned for its pairs of integers and holds at least one
  // partial; as many CTAs as there is room for (the plain kernels' partials alone: 304, two to an SM)
  if (dtype == IGD_F64 && (path == 4 || (path == 0 && gram64_split_pays(n, a, b))) &&
      (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0) {
    const int room = gram64_split_room(workspace_bytes, a, b);
    if (room >= 1) {
      g_gram_last = 4;
      return gram64_split_launch(n, a, static_cast<const double*>(A), sa, b, static_cast<const double*>(B), sb, w, out,
                                 accumulate, workspace, room, st);
    }
  }
  // the pipelined kernel when rows are 16-byte aligned and outputs <= 64 x 64, else the register-tiled one
  const int e = path == 3 ? -1
                : dtype == IGD_F32 ? gram_pipe_launch<float>(n, a, b, static_cast<const float*>(A), sa,
                                                             static_cast<const float*>(B), sb, w, part, nb, st)
                                   : gram_pipe_launch<double>(n, a, b, static_cast<const double*>(A), sa,
                                                              static_cast<const double*>(B), sb, w, part, nb, st);
  if (e > 0) return e;
  if (e < 0) nb = gram_tiled_blocks(n);
  g_gram_last = e == 0 ? 2 : 3;
  if (e == 0) {
    // launched
  } else if (dtype == IGD_F32) {
    constexpr int TR = 4;
    dim3 grid(nb, ((a + TR - 1) / TR) * ((b + TR - 1) / TR));
    gram_tile_kernel<float, TR><<<grid, GTH, 0, st>>>(n, a, b, static_cast<const float*>(A), sa,
                                                      static_cast<const float*>(B), sb, w, part);
  } else {
    constexpr int TR = 4;
    dim3 grid(nb, ((a + TR - 1) / TR) * ((b + TR - 1) / TR));
    gram_tile_kernel<double, TR><<<grid, GTH, 0, st>>>(n, a, b, static_cast<const double*>(A), sa,
                                                       static_cast<const double*>(B), sb, w, part);
  }
  const int ab = a * b;
  gram_reduce_kernel<<<std::min((ab * 32 + 255) / 256, 1024), 256, 0, st>>>(nb, ab, part, out, accumulate);
  return launch_status();
}

// out (c x n, row stride so) [+]= A^T C1 + B^T C2 with FP64 coefficient matrices
// C1 (a x c) and C2 (b x c) on the device (B / C2 may be absent with b = 0).
// out must not alias A or B.
extern "C" int igd_block_rotate(int dtype, long long n, int a, const void* A, long long sa, const double* C1, int b,
                                const void* B, long long sb, const double* C2, int c, void* out, long long so,
                                int accumulate, void* stream) {
  if (n <= 0 || a < 0 || b < 0 || a + b == 0 || c <= 0 || !out || (a && (!A || !C1)) || (b && (!B || !C2)))
    return IGD_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  int e;
  if (dtype == IGD_F32)
    e = rotate_dispatch<float>(n, a, static_cast<const float*>(A), sa, C1, b, static_cast<const float*>(B), sb, C2, c,
                               static_cast<float*>(out), so, accumulate, st);
  else if (dtype == IGD_F64)
    e = rotate_dispatch<double>(n, a, static_cast<const double*>(A), sa, C1, b, static_cast<const double*>(B), sb, C2,
                                c, static_cast<double*>(out), so, accumulate, st);
  else
    return IGD_ERR_DTYPE;
  if (e != IGD_OK) return e;
  return launch_status();
}

// Stream-ordered host-to-device copy of small coefficient matrices from pinned
// staging memory (one runtime call, none of a framework's dispatch).
extern "C" int igd_copy_h2d(void* dst, const void* src, long long bytes, void* stream) {
  if (!dst || !src || bytes < 0) return IGD_ERR_ARG;
  if (bytes == 0) return IGD_OK;
  return cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyHostToDevice, as_stream(stream)) == cudaSuccess
             ? IGD_OK
             : IGD_ERR_CUDA;
}
