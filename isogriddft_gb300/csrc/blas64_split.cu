// FP64 Gram products (K6) by exact splitting on the tensor cores.
//
// Reference: weighted_overlap_matrix (ks/eigensolver.py:246-272).
//
// GB300's FP64 pipe runs two lanes per clock and SM, so an FP64 Gram of 21 x 21 outputs costs 220
// clocks of it per point.  Here every FP64 value becomes a fixed-point number of 63 bits relative to
// the largest exponent of its row, and that seven balanced digits of nine bits, digits in
// [-256, 255], which FP16 holds exactly (Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 95
// (2012): error-free splitting into slices whose products accumulate without rounding).  The
// products of two digits are integers of at most 2^16; an FP32 accumulator takes 256 of them
// without rounding, so the sums of all digit pairs of one weight (28 pairs in seven levels; lower
// ones are below 2^-58 of the largest product) are exact integers over a window of 32 points,
// collected as int32 and turned into FP64 once per output.  Splitting is integer work (about 35
// instructions a value) and bounds the kernel: integer pipe 48 % and issue 47 % active with two CTAs of
// four warps on an SM.  The products go through mma.sync m16n8k16 (FP16 in, FP32 out), whose fragments are
// the splitting's own registers (the tensor pipe is 30 % active: operands staged for tcgen05 would only add
// traffic).
//
// What is lost are bits below 2^-61 of the row's largest value: nothing of the values within 2^-9 of
// it, everything of those below 2^-61.  Against the sum of |a w b|, on which the plain kernels' rounding
// depends, that is little where the rows overlap and all of it where they are localised in different
// places.  So the kernel bounds its own error.  The leading digit d of a value is nearest to it in units
// of 2^-7 of the row's power of two M, and only values of d = 0 lose bits.  In units of 2^-14 Ma Mb, over
// n points and C CTAs:
//   sum |a w b|  >=  0.249 T,              T = sum |da| |db|
//   truncation   <=  2^-54 (Z + 1.01 n),   Z = sum of |db| where da = 0 and of |da| where db = 0
//   digit pairs left out, and roundings of the last level's sums, at most 2^-54 (1.9 n + 256 C).
// Two more products per step sum G = 2 T - Z, and G >= n / 5 + 18 C holds the error below 66 * 2^-53
// sum |a w b|: the plain kernels' own bound is that of the 78 to 110 roundings of a sum.  Outputs of a smaller
// G are summed again by the plain kernel, tile by tile, in the same call, but for those so small that the
// plain kernel would round them to subnormal numbers.  On the blocks of an eigensolve the errors are half
// of the plain kernels' (root mean square 0.15 and 0.28 of 2^-53 sum |a w b|).
//
// Measured, 363609 points, plain kernel / this one: 21 x 21 505 / 161 us (153 without the guard), 34 x 34
// 1068 / 374 us; 25 us more with one tile summed again, 661 and 1446 us with all of them (rows localised at
// opposite ends).  Against 113-bit sums over 64^3 points of Gaussians, Slater and p functions, noise, spikes and
// constants, the largest error of the outputs it keeps is 1.2 * 2^-53 sum |a w b|, that of the plain
// kernels 1.1 to 60 (tests/test_gram_fp64_split_gpu.py, tests/test_gram_fp64_guard_gpu.py).
#include <algorithm>

#include <cuda_fp16.h>

#include "blas64_split.cuh"

namespace igd {
namespace {

constexpr int SL = 7;                                    // digits (slices) per value, levels of their products
constexpr long long BIAS = 256LL * (((1LL << 62) - 1 + (1LL << 62)) / 511);  // sum of 256 * 512^k, k < 7
static_assert(BIAS == 256LL * (1 + 512LL + 512LL * 512 + 512LL * 512 * 512 + 512LL * 512 * 512 * 512 +
                               512LL * 512 * 512 * 512 * 512 + 512LL * 512 * 512 * 512 * 512 * 512),
              "one balanced offset per digit");

__device__ __forceinline__ int biased_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// x * 2^(61 - (emax - 1022)) truncated to an integer, plus the digit offsets; |x| < 2^(emax - 1022),
// emax >= 1.
__device__ __forceinline__ unsigned long long fixed63(double x, int emax) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  const unsigned long long mant = ((unsigned long long)((hi & 0xfffff) | (e ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(x);
  const int d = min(emax - max(e, 1), 63);  // subnormals have the exponent of the smallest normal
  const long long m = (long long)((mant << 8) >> d), s = (long long)(hi >> 31);
  return (unsigned long long)(((m ^ s) - s) + BIAS);
}

// Digits of two values, most significant first, as packed FP16 pairs (x0 in the low half).
__device__ __forceinline__ void digits2(unsigned long long t0, unsigned long long t1, uint32_t (&d)[SL]) {
  const unsigned l0 = (unsigned)t0, h0 = (unsigned)(t0 >> 32), l1 = (unsigned)t1, h1 = (unsigned)(t1 >> 32);
  const __half2 off = __half2half2(__float2half(-1280.f));
  auto pack = [&](unsigned a, unsigned b16) {  // 1024 + digit + 256, then exact subtraction
    const unsigned v = (a & 0x1ffu) | (b16 & 0x1ff0000u) | 0x64006400u;
    const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&v), off);
    return *reinterpret_cast<const uint32_t*>(&r);
  };
  d[6] = pack(l0, l1 << 16);
  d[5] = pack(l0 >> 9, l1 << 7);
  d[4] = pack(l0 >> 18, l1 >> 2);
  d[3] = pack(__funnelshift_r(l0, h0, 27), __funnelshift_r(l1, h1, 11));
  d[2] = pack(h0 >> 4, h1 << 12);
  d[1] = pack(h0 >> 13, h1 << 3);
  d[0] = pack(h0 >> 22, h1 >> 6);
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
      "%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Seven level sums (weights 512^-l) as two integers of units 512^-2 and 512^-6.
__device__ __forceinline__ longlong2 halves(const int (&s)[SL]) {
  return make_longlong2(((long long)s[0] << 18) + ((long long)s[1] << 9) + (long long)s[2],
                        ((long long)s[3] << 27) + ((long long)s[4] << 18) + ((long long)s[5] << 9) + (long long)s[6]);
}
// The sum (lo in units of 512^-6, rounded to 512^-5 here: its floor showed as a bias of 2^-55) and G as a
// pair: all of the sum but its low 27 bits, and those with G above them.
__device__ __forceinline__ longlong2 pack(long long hi, long long lo, long long guard) {
  constexpr long long LOW = (1LL << 27) - 1;
  lo = (lo + 256) >> 9;
  return make_longlong2(hi + (lo >> 27), (lo & LOW) | (long long)((unsigned long long)guard << 27));
}
// (hi 2^27 + lo) 2^shift, rounded once.
__device__ __forceinline__ double join(long long hi, long long lo, int shift) {
  const double h = (double)hi;
  const long long rest = hi - (long long)h;  // what the conversion rounded off
  return scalbn(fma(h, 134217728.0, fma((double)rest, 134217728.0, (double)lo)), shift);
}

// ------------------------------------------------------------------------------------- Gram
// Largest biased exponent of every row of A and of w B (bounded by the factors' exponents);
// rows of A first.  2047 marks a row with an infinity or a NaN.  A thread keeps the exponents of w
// at its eight points while it runs over the rows (U loads in flight, five instructions a value).
constexpr int EU = 8, ETH = 128, ER = 6;  // points per thread, threads, rows per CTA
__global__ void __launch_bounds__(ETH) row_exponent_kernel(long long n, int a, const double* __restrict__ A,
                                                           long long sa, int b, const double* __restrict__ B,
                                                           long long sb, const double* __restrict__ w,
                                                           int* __restrict__ emax) {
  __shared__ int top[ER];
  const int first = blockIdx.y * ER, past = min(a + b, first + ER);
  if (threadIdx.x < ER) top[threadIdx.x] = 0;
  __syncthreads();
  const long long p0 = (long long)blockIdx.x * (ETH * EU) + threadIdx.x;
  const bool whole = (long long)(blockIdx.x + 1) * (ETH * EU) <= n;
  int off[EU], ew[EU];
#pragma unroll
  for (int u = 0; u < EU; ++u) {
    off[u] = whole || p0 + ETH * u < n ? ETH * u : 0;  // threads past the end repeat a point
    const long long p = min(p0 + off[u], n - 1);
    off[u] = (int)(p - p0);
    ew[u] = w ? max(biased_exponent(__ldg(w + p)), 1) - 1022 : 1;
  }
  const bool wbad = [&] {
    bool f = false;
#pragma unroll
    for (int u = 0; u < EU; ++u) f |= ew[u] == 0x7ff - 1022;
    return f;
  }();
#pragma unroll 3
  for (int r = first; r < past; ++r) {
    const double* const x = (r < a ? A + (long long)r * sa : B + (long long)(r - a) * sb) + p0;
    int m = 0;
    double v[EU];
#pragma unroll
    for (int u = 0; u < EU; ++u) v[u] = __ldg(x + off[u]);
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int e = biased_exponent(v[u]);
      // |w| < 2^(ew - 1022), |b| < 2^(eb - 1022): the product's biased exponent is at most ew + eb - 1022
      m = max(m, r < a || !w ? e : (e == 0x7ff ? e : max(e, 1) + ew[u]));
    }
    if (r >= a && w && wbad) m = 0x7ff;
    m = __reduce_max_sync(0xffffffffu, min(m, 0x7ff));
    if ((threadIdx.x & 31) == 0) atomicMax(top + (r - first), m);
  }
  __syncthreads();
  if (threadIdx.x < past - first && top[threadIdx.x] > 0) atomicMax(emax + first + threadIdx.x, top[threadIdx.x]);
}

__device__ __forceinline__ uint32_t half2_bits(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// Of two packed digits: the magnitudes, and ones where they are zero.
__device__ __forceinline__ __half2 magnitude2(uint32_t d) { return __habs2(*reinterpret_cast<const __half2*>(&d)); }
__device__ __forceinline__ __half2 zeros2(uint32_t d) {
  return __heq2(magnitude2(d), __half2half2(__float2half(0.f)));
}

constexpr int GW = 4, GNT = 3;             // warps per CTA; 8-column tiles per warp
constexpr int GROWS = 16 + 8 * GNT + 1;    // staged rows of a warp: A, B, w
constexpr int GPITCH = 36;                 // doubles per staged row of 32 points (conflict-free fragment loads)
constexpr size_t GSMEM = (size_t)GW * 2 * GROWS * GPITCH * sizeof(double);

// One warp: 16 rows of A (blockIdx.y) by 24 columns of B (blockIdx.z) over windows of 32 points,
// the next window's values on their way by cp.async (8-byte copies: any alignment) while this one
// is split and multiplied.  Fragment k indices are points in an order that keeps a thread's
// loads on four neighbouring points.
__global__ void __launch_bounds__(32 * GW, 2)
    gram64_kernel(long long n, int a, const double* __restrict__ A, long long sa, int b, const double* __restrict__ B,
                  long long sb, const double* __restrict__ w, const int* __restrict__ emax, int sym,
                  longlong2* __restrict__ part) {
  const int i0 = blockIdx.y * 16, j0 = blockIdx.z * 8 * GNT;
  if (sym && j0 + 8 * GNT <= i0) return;  // below the diagonal: mirrored by the reduction
  extern __shared__ __align__(16) double gsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  double* const st0 = gsm + (size_t)warp * 2 * GROWS * GPITCH;
  const int na = min(16, a - i0), nb = min(8 * GNT, b - j0);
  for (int e = lane; e < 2 * GROWS * GPITCH; e += 32) st0[e] = 0.0;  // rows past the operands stay zero
  __syncwarp();
  auto copy = [&](long long p0, int q) {
    double* const d = st0 + q * GROWS * GPITCH + lane;
    const long long p = p0 + lane;
    const bool in = p < n;
    const long long pc = in ? p : 0;
    for (int r = 0; r < na; ++r) cp_async_zfill<8>(d + r * GPITCH, A + (long long)(i0 + r) * sa + pc, in);
    for (int r = 0; r < nb; ++r) cp_async_zfill<8>(d + (16 + r) * GPITCH, B + (long long)(j0 + r) * sb + pc, in);
    if (w) cp_async_zfill<8>(d + (GROWS - 1) * GPITCH, w + pc, in);
  };
  const int r0 = i0 + g, r1 = i0 + g + 8;
  const int ea0 = r0 < a ? max(emax[r0], 1) : 1, ea1 = r1 < a ? max(emax[r1], 1) : 1;
  int eb[GNT];
#pragma unroll
  for (int q = 0; q < GNT; ++q) {
    const int j = j0 + 8 * q + g;
    eb[q] = j < b ? max(emax[a + j], 1) : 1;
  }
  int s[GNT][4][SL];
#pragma unroll
  for (int q = 0; q < GNT; ++q)
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int l = 0; l < SL; ++l) s[q][c][l] = 0;
  int sg[GNT][4];  // G: at most 2^20 a window
#pragma unroll
  for (int q = 0; q < GNT; ++q)
#pragma unroll
    for (int c = 0; c < 4; ++c) sg[q][c] = 0;
  const long long step = (long long)gridDim.x * GW * 32;
  long long p0 = ((long long)blockIdx.x * GW + warp) * 32;
  if (p0 < n) copy(p0, 0);
  cp_async_commit();
  for (int buf = 0; p0 < n; p0 += step, buf ^= 1) {
    if (p0 + step < n) copy(p0 + step, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncwarp();
    const double* const sd = st0 + buf * GROWS * GPITCH + t;
    uint32_t fa[2][4][SL], ga[2][4], za[2][4];  // A fragments of both 16-point halves; 2 |da|, and -1 where da = 0
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double *x0 = sd + g * GPITCH + 16 * h, *x1 = x0 + 8 * GPITCH;
      digits2(fixed63(x0[0], ea0), fixed63(x0[4], ea0), fa[h][0]);
      digits2(fixed63(x1[0], ea1), fixed63(x1[4], ea1), fa[h][1]);
      digits2(fixed63(x0[8], ea0), fixed63(x0[12], ea0), fa[h][2]);
      digits2(fixed63(x1[8], ea1), fixed63(x1[12], ea1), fa[h][3]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const __half2 v = magnitude2(fa[h][k][0]);
        ga[h][k] = half2_bits(__hadd2(v, v));
        za[h][k] = half2_bits(__hneg2(zeros2(fa[h][k][0])));
      }
    }
#pragma unroll
    for (int q = 0; q < GNT; ++q) {
      if (j0 + 8 * q >= b) break;  // uniform
      float acc[SL][4], accg[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int l = 0; l < SL; ++l)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[l][c] = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double *xb = sd + (16 + 8 * q + g) * GPITCH + 16 * h, *xw = sd + (GROWS - 1) * GPITCH + 16 * h;
        double x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = w ? xb[4 * k] * xw[4 * k] : xb[4 * k];
        uint32_t b0[SL], b1[SL];
        digits2(fixed63(x[0], eb[q]), fixed63(x[1], eb[q]), b0);
        digits2(fixed63(x[2], eb[q]), fixed63(x[3], eb[q]), b1);
        const __half2 m0 = magnitude2(b0[0]), m1 = magnitude2(b1[0]), less = __half2half2(__float2half(-0.5f));
        mma16816(accg, ga[h][0], ga[h][1], ga[h][2], ga[h][3], half2_bits(__hfma2(zeros2(b0[0]), less, m0)),
                 half2_bits(__hfma2(zeros2(b1[0]), less, m1)));
        mma16816(accg, za[h][0], za[h][1], za[h][2], za[h][3], half2_bits(m0), half2_bits(m1));
        // consecutive products go to different levels (independent accumulators)
#pragma unroll
        for (int i = 0; i < SL; ++i)
#pragma unroll
          for (int j = 0; j < SL - i; ++j)
            mma16816(acc[i + j], fa[h][0][i], fa[h][1][i], fa[h][2][i], fa[h][3][i], b0[j], b1[j]);
        // the next level, scaled into the last one (2^-9 of a unit is exact in FP16; the accumulator may round
        // below one unit here)
        const __half2 sc = __half2half2(__float2half(1.f / 512.f));
#pragma unroll
        for (int j = 1; j < SL; ++j) {
          const __half2 v0 = __hmul2(*reinterpret_cast<const __half2*>(&b0[j]), sc);
          const __half2 v1 = __hmul2(*reinterpret_cast<const __half2*>(&b1[j]), sc);
          mma16816(acc[SL - 1], fa[h][0][SL - j], fa[h][1][SL - j], fa[h][2][SL - j], fa[h][3][SL - j],
                   *reinterpret_cast<const uint32_t*>(&v0), *reinterpret_cast<const uint32_t*>(&v1));
        }
      }
#pragma unroll
      for (int l = 0; l < SL; ++l)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[q][c][l] += __float2int_rn(acc[l][c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) sg[q][c] += __float2int_rn(accg[c]);
    }
    __syncwarp();  // this buffer is refilled by the next window's copies
  }
  // integer sums of the warps of this CTA, one partial per CTA, in which the last level is rounded
  longlong2 (*const red)[16][8 * GNT] = reinterpret_cast<longlong2 (*)[16][8 * GNT]>(gsm);
  int (*const redg)[16][8 * GNT] = reinterpret_cast<int (*)[16][8 * GNT]>(red + GW);
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll
  for (int q = 0; q < GNT; ++q)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      red[warp][g + (c >= 2 ? 8 : 0)][8 * q + 2 * t + (c & 1)] = halves(s[q][c]);
      redg[warp][g + (c >= 2 ? 8 : 0)][8 * q + 2 * t + (c & 1)] = sg[q][c];
    }
  __syncthreads();
  longlong2* const pb = part + (long long)blockIdx.x * a * b;
  for (int e = threadIdx.x; e < 16 * 8 * GNT; e += 32 * GW) {
    const int i = e / (8 * GNT), j = e - i * (8 * GNT);
    if (i0 + i < a && j0 + j < b) {
      long long hi = 0, lo = 0, gg = 0;
#pragma unroll
      for (int q = 0; q < GW; ++q) {
        hi += red[q][i][j].x;
        lo += red[q][i][j].y;
        gg += redg[q][i][j];
      }
      pb[(long long)(i0 + i) * b + j0 + j] = pack(hi, lo, gg);
    }
  }
}

// out[i][j] (+)= sum over CTAs, one warp per output; a symmetric product takes its lower triangle
// from the upper.  Marked for the plain kernel, and not written: outputs whose row or column holds an
// infinity or a NaN (or may overflow, in the mirrored product too; need = 2), and those of G below `least`
// (need = 1) whose products the plain kernel does not round to subnormal numbers: its unit is 2^-1074 there
// at every product, and this kernel's bound, 2^-68 Ma Mb (131 n + 256 C), is less up to Ma Mb = 2^-1016
// (rows of zeros are among these).
__global__ void gram64_reduce_kernel(int nblocks, int a, int b, const int* __restrict__ emax, int sym, long long least,
                                     const longlong2* __restrict__ part, double* __restrict__ out, int accumulate,
                                     const Gram64Marks marks) {
  const int lane = threadIdx.x & 31, tb = (b + GRAM64_TILE - 1) / GRAM64_TILE;
  const long long ab = (long long)a * b;
  for (long long e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < ab; e += (gridDim.x * blockDim.x) >> 5) {
    const int i = (int)(e / b), j = (int)(e - (long long)i * b);
    const int ei0 = emax[i], ej0 = emax[a + j];
    int kind = 0;
    double v = 0.0;
    const bool turn = sym && i > j;
    if (ei0 >= 0x7ff || ej0 >= 0x7ff || (sym && (emax[j] >= 0x7ff || emax[a + i] >= 0x7ff))) {
      kind = 2;
    } else {
      const long long at = turn ? (long long)j * b + i : e;
      long long hi = 0, lo = 0, guard = 0;
      for (int k = lane; k < nblocks; k += 32) {
        const longlong2 x = part[(long long)k * ab + at];
        hi += x.x;
        lo += x.y & ((1LL << 27) - 1);
        guard += x.y >> 27;
      }
      for (int off = 16; off > 0; off >>= 1) {
        hi += __shfl_xor_sync(0xffffffffu, hi, off);
        lo += __shfl_xor_sync(0xffffffffu, lo, off);
        guard += __shfl_xor_sync(0xffffffffu, guard, off);
      }
      // a value of row r is its integer times 2^(emax - 1022 - 61); units 512^(12 - 5)
      const int ei = max(turn ? emax[j] : ei0, 1), ej = max(turn ? emax[a + i] : ej0, 1);
      v = join(hi, lo, ei + ej - 2166 + 63);
      if (guard < least && ei + ej > 2 * 1022 - 1016) kind = 1;
    }
    if (lane == 0) {
      marks.need[e] = kind;
      if (kind) {
        const int r = kind == 1 && turn ? j : i, c = kind == 1 && turn ? i : j;
        const int tile = (r / GRAM64_TILE) * tb + c / GRAM64_TILE;
        if (atomicExch(marks.tiles + tile, 1) == 0) marks.list[atomicAdd(marks.listed, 1)] = tile;
      } else {
        out[e] = accumulate ? out[e] + v : v;
      }
    }
  }
}

}  // namespace

// At most 120 windows per warp (an int32 level sum takes 127 windows of at most 2^24): more than max_blocks CTAs
// can take go in pieces, each with its own row exponents, added up in the output.  9.5 million points:
// three pieces.
int gram64_split_launch(long long n, int a, const double* A, long long sa, int b, const double* B, long long sb,
                        const double* w, double* out, int accumulate, void* workspace, int max_blocks, cudaStream_t st) {
  constexpr long long MOST = 120, WINDOW = 32 * GW;
  longlong2* const part = static_cast<longlong2*>(workspace);
  const long long ntiles = gram64_tiles(a, b);
  int* const emax = reinterpret_cast<int*>(part + (long long)max_blocks * a * b);
  int* const tiles = emax + a + b;
  const Gram64Marks marks{tiles, tiles + ntiles, tiles + ntiles + 1, tiles + 2 * ntiles + 1};
  const int sms = device_sm_count();
  const int ty = (a + 15) / 16, tz = (b + 8 * GNT - 1) / (8 * GNT);
  const int sym = A == B && sa == sb && a == b;
  const long long windows = (n + WINDOW - 1) / WINDOW, pieces = (windows + MOST * max_blocks - 1) / (MOST * max_blocks);
  const long long step = (windows + pieces - 1) / pieces * WINDOW;  // points of a piece
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gram64_kernel), GSMEM) != IGD_OK) return IGD_ERR_CUDA;
  for (long long p0 = 0; p0 < n; p0 += step) {
    const long long m = std::min(step, n - p0), mw = (m + WINDOW - 1) / WINDOW;
    const double *pa = A + p0, *pb = B + p0, *pw = w ? w + p0 : nullptr;
    const long long want = std::min<long long>(mw, std::max<long long>(1, 2LL * sms / ((long long)ty * tz)));
    const int grid = (int)std::min<long long>(std::max(want, (mw + MOST - 1) / MOST), max_blocks);
    if (cudaMemsetAsync(emax, 0, sizeof(int) * (a + b + ntiles + 1), st) != cudaSuccess) return IGD_ERR_CUDA;
    row_exponent_kernel<<<dim3((unsigned)((m + ETH * EU - 1) / (ETH * EU)), (a + b + ER - 1) / ER), ETH, 0, st>>>(
        m, a, pa, sa, b, pb, sb, pw, emax);
    gram64_kernel<<<dim3((unsigned)grid, ty, tz), 32 * GW, GSMEM, st>>>(m, a, pa, sa, b, pb, sb, pw, emax, sym, part);
    gram64_reduce_kernel<<<(int)std::min<long long>(((long long)a * b + 7) / 8, 1024), 256, 0, st>>>(
        grid, a, b, emax, sym, (mw * WINDOW + 4) / 5 + 18LL * grid, part, out, accumulate || p0 > 0, marks);
    const int r = gram64_plain_redo(m, a, pa, sa, b, pb, sb, pw, out, accumulate || p0 > 0, sym, marks,
                                    static_cast<double*>(workspace), 2LL * max_blocks, st);
    if (r != IGD_OK) return r;
  }
  return launch_status();
}

}  // namespace igd
