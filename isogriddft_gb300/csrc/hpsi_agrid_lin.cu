// Linear-tile A-grid H.Psi stencils (K1 for FP64 and for FP32 rows the TMA kernels cannot take).
//
// Same arithmetic as hpsi_agrid.cu (flux form of ops/kinetic.py:212-358 with ghost-value
// closures, plus v_eff psi of ks/eigensolver.py:753-756), for rows of up to 256 points and any
// alignment.
//
// A tile is a run of whole rows of the (y, z) plane.  Whole rows are contiguous in memory, so
// the tile's points are numbered linearly and thread t owns points t, t + NT, ...: every lane
// works whatever the row length (a lane-per-z tile of 32 wastes 16 % of its lanes on rows of
// 81 points), global accesses coalesce without any alignment rule, and a thread's points stay
// the same along the whole x march.  In shared memory each row has one ghost cell on either
// side, so the z faces need no branches in the main loop: the cells hold zeros (trial fix) or
// are extrapolated once per plane by a few threads (production closure).  psi planes stream
// through a ring by element-wise cp.async; F^y and F^z go through shared memory (double
// buffered by step parity), F^x stays in registers, and the output of plane s-1 is formed in
// step s, so the trial fix needs one barrier per plane and the production closure two.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace igd {
namespace {

struct LinArgs {
  int nx, ny, nz, nb;
  long long ostride, n;
  int tiles, groups, total;  // total = tiles * groups * nx march steps
  unsigned rnz;               // ceil(2^32 / nz): e / nz = umulhi(e, rnz) for the tile's point numbers (below 2^13)
  // Krylov mode (one orbital): faces written as zero, acc[0] += sum out * y (y = dot_y, or the
  // input when dot_y is null), acc[1] += sum out * out (only when dot_y is null); nothing runs
  // while *skip != 0
  const void* dot_y;
  double* dot_acc;
  const int* skip;
};

template <typename T>
__device__ __forceinline__ T lin_ext3(T a, T b, T c) { return T(3) * a - T(3) * b + c; }

// Every CTA marches an equal contiguous share of the (unit, plane) list, a unit being a row tile
// and an orbital group (the groups of a tile next to each other: they share its geometry in L2).
// A share never starts on plane 1 or 2 of a unit: the production closure's lower-face output
// needs the march through plane 2 in one segment.
__device__ __forceinline__ int lin_bound(int b, const LinArgs& a) {
  const int w = (int)((long long)b * a.total / gridDim.x), x = w % a.nx;
  return x == 1 || x == 2 ? w - x : w;
}

// One segment: rows [j0, j0 + oy), planes [x0, x1), orbitals from o0, and the planes sb .. se
// that the march covers (one plane more on either side for F^x; the last segment starts early
// enough for F^x(nx-3), which the last face's ghost needs); psi planes up to `last` are read.
struct LinSeg {
  int j0, oy, x0, x1, o0, sb, se, last;
};
__device__ __forceinline__ LinSeg lin_seg(const LinArgs& a, int pos, int end, int NB) {
  LinSeg t;
  const int unit = pos / a.nx, tile = unit / a.groups;
  t.j0 = tile * a.ny / a.tiles;
  t.oy = (tile + 1) * a.ny / a.tiles - t.j0;
  t.x0 = pos - unit * a.nx;
  t.x1 = min(a.nx, t.x0 + (end - pos));
  t.o0 = (unit - tile * a.groups) * NB;
  t.sb = t.x0 == 0 ? 0 : min(t.x0 - 1, a.nx - 3);
  t.se = t.x1 == a.nx ? a.nx - 1 : t.x1;
  t.last = min(a.nx - 1, t.se + 1);
  return t;
}

// Production closure: ghost cells of one psi plane (rows of P = nz + 2 cells, first row j0 - 2)
// beyond the z faces and on the rows beyond the y faces.  V: the values of one cell.
template <typename V, int NT>
__device__ __forceinline__ void fill_psi(V* d, int ny, int nz, int j0, int oy) {
  const int P = nz + 2, tid = threadIdx.x ^ (NT / 2);  // from the middle warp on
  for (int e = tid; e < 2 * (oy + 2); e += NT) {
    const int yy = 1 + (e >> 1), j = j0 - 2 + yy;
    if (j < 0 || j >= ny) continue;
    V* const c = d + yy * P;
    if (e & 1)
      c[nz + 1] = lin_ext3(c[nz], c[nz - 1], c[nz - 2]);
    else
      c[0] = lin_ext3(c[1], c[2], c[3]);
  }
  if (j0 <= 1)
    for (int z = tid; z < nz; z += NT) {
      V* const c = d + (1 - j0) * P + 1 + z;
      c[0] = lin_ext3(c[P], c[2 * P], c[3 * P]);
    }
  if (j0 + oy >= ny - 1)
    for (int z = NT - 1 - tid; z < nz; z += NT) {
      V* const c = d + (ny - j0 + 2) * P + 1 + z;
      c[0] = lin_ext3(c[-P], c[-2 * P], c[-3 * P]);
    }
}

// The same for the fluxes of one plane (first row j0 - 1): F^z beyond the z faces, F^y on the
// rows beyond the y faces.
template <typename V, int NT>
__device__ __forceinline__ void fill_flux(V* fy, V* fz, int ny, int nz, int j0, int oy) {
  const int P = nz + 2, tid = NT - 1 - threadIdx.x;  // from the last warp down: it owns the fewest points
  for (int e = tid; e < 2 * oy; e += NT) {
    V* const c = fz + (1 + (e >> 1)) * P;
    if (e & 1)
      c[nz + 1] = lin_ext3(c[nz], c[nz - 1], c[nz - 2]);
    else
      c[0] = lin_ext3(c[1], c[2], c[3]);
  }
  if (j0 == 0)
    for (int z = tid; z < nz; z += NT) {
      V* const c = fy + 1 + z;
      c[0] = lin_ext3(c[P], c[2 * P], c[3 * P]);
    }
  if (j0 + oy == ny)
    for (int z = NT - 1 - tid; z < nz; z += NT) {
      V* const c = fy + (oy + 1) * P + 1 + z;
      c[0] = lin_ext3(c[-P], c[-2 * P], c[-3 * P]);
    }
}

// ------------------------------------------------------------------------------- FP64
// GB300 runs two FP64 lanes per clock and SM (0.58 T FMA/s measured), so this form is bound by
// its FP64 instruction count: 20 per point and orbital (gradients 3, fluxes 9, divergence 5,
// scaling and v psi 3).  Hence the rows above and below the tile compute F^y only (6) and the
// planes just outside a segment F^x only (6), and the tile's own rows are numbered before the
// halo rows, so that warps do one or the other.  psi(s-1), psi(s) and psi(s+1) are read from a
// 5-slot ring (shared-memory bandwidth is idle here); the registers hold the plane's geometry,
// loaded ahead of the barrier that opens its step.
constexpr int L64_NT = 256, L64_PPT = 4, L64_RING = 5, L64_MINB = 2;
constexpr int L64_LD = L64_PPT + 4, L64_PH = 2;  // copies and halo points per thread (rows of at most NT points)

__host__ __device__ inline size_t lin64_cells(int oy, int nz) {
  return (size_t)(nz + 2) * (L64_RING * (oy + 4) + 4 * (oy + 2));
}

__device__ __noinline__ double mul64(double x, double y) { return x * y; }

// x * kscale for kscale = +-2^kexp by integer arithmetic on x's exponent (exact, and off the
// FP64 pipe); zeros, subnormals and values near the ends of the exponent range are multiplied,
// in a call, because a predicated-off FP64 instruction takes its slot all the same.
__device__ __forceinline__ double mul_pow2(double x, double kscale, int kexp, unsigned sign) {
  const int hi = __double2hiint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  if (e - 64u > 1900u) return mul64(x, kscale);
  return __hiloint2double((hi + (kexp << 20)) ^ (int)sign, __double2loint(x));
}

template <bool PROD, bool KRY, bool HASV>
__global__ void __launch_bounds__(L64_NT, L64_MINB)
    hpsi_lin64_kernel(const double* __restrict__ coeffs, const double* __restrict__ veff,
                      const double* __restrict__ psi, double* __restrict__ out, const LinArgs a, double kscale,
                      int kexp, unsigned ksign) {
  constexpr int NT = L64_NT, PPT = L64_PPT, RING = L64_RING, LD = L64_LD, PH = L64_PH;
  if constexpr (KRY) {
    if (a.skip && *a.skip) return;  // the Krylov solve has stopped: uniform for the whole launch
  }
  extern __shared__ __align__(16) double sm64[];
  const int tid = threadIdx.x, nx = a.nx, ny = a.ny, nz = a.nz, P = nz + 2;
  const long long plane = (long long)ny * nz, n = a.n;
  double d0 = 0.0, d1 = 0.0;
  const int end = lin_bound(blockIdx.x + 1, a);
  for (int pos = lin_bound(blockIdx.x, a); pos < end;) {
    const LinSeg t = lin_seg(a, pos, end, 1);
    pos += t.x1 - t.x0;
    const int j0 = t.j0, oy = t.oy;
    const int psz = (oy + 4) * P, fsz = (oy + 2) * P;
    double* const fbuf = sm64 + RING * psz;
    // ghost cells read as zero (trial fix); the production closure writes every ghost it reads
    if (!PROD)
      for (int e = tid; e < RING * psz + 4 * fsz; e += NT) sm64[e] = 0.0;

    const int jlo = max(j0 - 2, 0), jhi = min(j0 + oy + 1, ny - 1);
    const int cnt = (jhi - jlo + 1) * nz;
    int dst[LD];
#pragma unroll
    for (int l = 0; l < LD; ++l) {
      const int e = tid + l * NT, r = __umulhi(e, a.rnz);
      dst[l] = (jlo - (j0 - 2)) * P + 1 + e + 2 * r;
    }
    const double* const pin = psi + (long long)t.o0 * a.ostride + (long long)jlo * nz;
    double* const pout = out + (long long)t.o0 * a.ostride;
    auto load_plane = [&](int p, double* d) {
      const double* const s = pin + (long long)p * plane;
#pragma unroll
      for (int l = 0; l < LD; ++l)
        if (tid + l * NT < cnt) cp_async_zfill<8>(d + dst[l], s + (unsigned)(tid + l * NT), true);
    };

    // own points tid + i * NT (rows R = 1 .. oy of the flux tile): cell ci in a flux buffer, ci + P
    // in a psi slot, column col; threads past the last point repeat it and store nothing
    const int own = oy * nz, mine = (own - tid + NT - 1) / NT;  // number of this thread's points
    int ci[PPT];
    unsigned col[PPT];
    unsigned face = 0;  // bit i: point i lies on a y or z face
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      const int q = min(tid + i * NT, own - 1), r = __umulhi(q, a.rnz), z = q - r * nz;
      ci[i] = (r + 1) * P + 1 + z;
      col[i] = (unsigned)(j0 * nz + q);
      if (j0 + r == 0 || j0 + r == ny - 1 || z == 0 || z == nz - 1) face |= 1u << i;
    }
    // halo points, dealt from the last thread down (the threads with fewer own points): cells of
    // rows 0 and oy + 1, or -1
    int hc[PH], hcol[PH];
#pragma unroll
    for (int h = 0; h < PH; ++h) {
      const int e = NT - 1 - tid + h * NT, up = e >= nz, z = e - up * nz;
      const int R = up ? oy + 1 : 0, j = j0 - 1 + R;
      hc[h] = e < 2 * nz && j >= 0 && j < ny ? R * P + 1 + z : -1;
      hcol[h] = hc[h] < 0 ? 0 : j * nz + z;
    }

    if (!PROD) __syncthreads();  // the zero fill precedes the copies
    auto slot = [&](int k) { return sm64 + (k >= RING ? k - RING : k) * psz; };  // slot of plane p: (p - sb + 1) mod RING
    for (int p = max(t.sb - 1, 0); p <= t.sb + 1; ++p) load_plane(p, slot(p - t.sb + 1));
    cp_async_commit();
    if (t.sb + 2 <= t.last) load_plane(t.sb + 2, slot(3));
    cp_async_commit();
    if constexpr (PROD) {
      cp_async_wait<0>();
      __syncthreads();
      fill_psi<double, NT>(slot(1), ny, nz, j0, oy);
      if (t.sb == 0) {  // psi(-1) = 3 psi(0) - 3 psi(1) + psi(2) at the own and halo points
        double* const g = slot(0);
        const double *p0 = slot(1), *p1 = slot(2), *p2 = slot(3);
        for (int e = tid; e < (oy + 2) * nz; e += NT) {
          const int c = P + 1 + e + 2 * __umulhi(e, a.rnz);
          g[c] = lin_ext3(p0[c], p1[c], p2[c]);
        }
      }
    }
    double fx[PPT], f1[PPT], f2[PPT];  // F^x(s), F^x(s-1), F^x(s-2) at the own points
#pragma unroll
    for (int i = 0; i < PPT; ++i) fx[i] = f1[i] = f2[i] = 0.0;

    // output of plane op at point i: df = F^x(op + 1) - F^x(op - 1), ps = psi(op)
    auto emit = [&](int i, int op, double df, double ps, double ij, double v) {
      const long long go = (long long)op * plane;
      const double* const fy = fbuf + (2 * (op & 1)) * fsz + ci[i];
      const double* const fz = fy + fsz;
      double val = mul_pow2(ij, kscale, kexp, ksign) * (df + (fy[P] - fy[-P]) + (fz[1] - fz[-1]));
      if constexpr (HASV) val += v * ps;
      if constexpr (KRY) {
        // faces of a Krylov vector stay zero; the dots then cover interior points only
        if (((face >> i) & 1u) || op == 0 || op == nx - 1) val = 0.0;
        if (a.dot_y) {
          d0 += val * __ldg(static_cast<const double*>(a.dot_y) + go + col[i]);
        } else {
          d0 += val * ps;
          d1 += val * val;
        }
      }
      (pout + go)[col[i]] = val;
    };

    int k = 1;  // slot index of plane s
    for (int s = t.sb; s <= t.se; ++s) {
      const int op = s - 1;
      const bool mid = s >= t.x0 && s < t.x1;  // plane s is an output plane: its F^y and F^z are needed
      const bool outp = op >= t.x0 && op < t.x1;
      const double* const cs = coeffs + (long long)s * plane;
      double axx[PPT], ayy[PPT], azz[PPT], axy[PPT], axz[PPT], ayz[PPT];
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        axx[i] = __ldg(cs + col[i]);
        ayy[i] = __ldg(cs + n + col[i]);
        azz[i] = __ldg(cs + 2 * n + col[i]);
        axy[i] = __ldg(cs + 3 * n + col[i]);
        axz[i] = __ldg(cs + 4 * n + col[i]);
        ayz[i] = __ldg(cs + 5 * n + col[i]);
      }
      cp_async_wait<1>();
      __syncthreads();  // plane s+1 has landed, plane s's ghosts and the fluxes of plane s-1 are complete
      double *const prv = slot(k + RING - 1), *const cur = slot(k), *const nxt = slot(k + 1);
      if (s + 3 <= t.last) load_plane(s + 3, slot(k + 3));  // into the slot of plane s-2
      cp_async_commit();
      if (s + 1 == nx) {
        // psi(nx) at the own and halo points: 3 psi(nx-1) - 3 psi(nx-2) + psi(nx-3), or zero
        const double* const pr2 = slot(k + RING - 2);
        for (int e = tid; e < (oy + 2) * nz; e += NT) {
          const int c = P + 1 + e + 2 * __umulhi(e, a.rnz);
          nxt[c] = PROD ? lin_ext3(cur[c], prv[c], pr2[c]) : 0.0;
        }
        __syncthreads();
      }
      if (PROD && outp) fill_flux<double, NT>(fbuf + 2 * (op & 1) * fsz, fbuf + (2 * (op & 1) + 1) * fsz, ny, nz, j0, oy);
      double* const fy = fbuf + 2 * (s & 1) * fsz;
      double* const fz = fy + fsz;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        if (i >= mine) continue;
        const int c = ci[i] + P;
        const double gx = nxt[c] - prv[c], gy = cur[c + P] - cur[c - P], gz = cur[c + 1] - cur[c - 1];
        fx[i] = axx[i] * gx + axy[i] * gy + axz[i] * gz;
        if (mid) {
          fy[ci[i]] = axy[i] * gx + ayy[i] * gy + ayz[i] * gz;
          fz[ci[i]] = axz[i] * gx + ayz[i] * gy + azz[i] * gz;
        }
      }
      if (mid) {
#pragma unroll
        for (int h = 0; h < PH; ++h) {
          if (hc[h] < 0) continue;
          const int c = hc[h] + P;
          const double* const g = cs + hcol[h];
          fy[hc[h]] = __ldg(g + 3 * n) * (nxt[c] - prv[c]) + __ldg(g + n) * (cur[c + P] - cur[c - P]) +
                      __ldg(g + 5 * n) * (cur[c + 1] - cur[c - 1]);
        }
      }
      if (outp) {
        const double* const co = coeffs + 6 * n + (long long)op * plane;
        const double* const vo = veff + (long long)op * plane;
        double ij[PPT], v[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
          ij[i] = __ldg(co + col[i]);
          v[i] = HASV ? __ldg(vo + col[i]) : 0.0;
        }
        if (PROD) __syncthreads();  // the flux ghosts of plane s-1 are complete
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (i < mine) emit(i, op, fx[i] - f2[i], prv[ci[i] + P], ij[i], v[i]);
      }
      if (PROD && s + 1 <= t.last) fill_psi<double, NT>(nxt, ny, nz, j0, oy);
      if (PROD && !KRY && s == 2 && t.x0 == 0) {
        // F^x ghost below the lower face, 3 F(0) - 3 F(1) + F(2): plane 0 was written without it
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (i < mine)
            pout[col[i]] = fma(-kscale * __ldg(coeffs + 6 * n + col[i]), lin_ext3(f2[i], f1[i], fx[i]), pout[col[i]]);
      }
      if (s < nx - 1)
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
          f2[i] = f1[i];
          f1[i] = fx[i];
        }
      k = k + 1 == RING ? 0 : k + 1;
    }

    // ---- plane nx-1: fx, f1, f2 hold F^x(nx-1), F^x(nx-2), F^x(nx-3)
    if (t.x1 == nx) {
      __syncthreads();
      if constexpr (PROD) {
        fill_flux<double, NT>(fbuf + 2 * ((nx - 1) & 1) * fsz, fbuf + (2 * ((nx - 1) & 1) + 1) * fsz, ny, nz, j0, oy);
        __syncthreads();
      }
      const double* const cur = slot(k + RING - 1);
      const long long go = (long long)(nx - 1) * plane;
#pragma unroll
      for (int i = 0; i < PPT; ++i)
        if (i < mine)
          emit(i, nx - 1, (PROD ? lin_ext3(fx[i], f1[i], f2[i]) : 0.0) - f1[i], cur[ci[i] + P],
               __ldg(coeffs + 6 * n + go + col[i]), HASV ? __ldg(veff + go + col[i]) : 0.0);
    }
    __syncthreads();  // the next segment reuses the buffers
  }
  if constexpr (KRY) {
    double v2[2] = {d0, d1};
    block_atomic_add<2, NT>(a.dot_acc, v2);
  }
}

// ------------------------------------------------------------------------------- FP32
// Bound by shared-memory wavefronts and instruction issue, so a cell holds the values of all NB
// orbitals: one 16-byte shared load brings a neighbour of four orbitals, its address is formed
// once, and the arithmetic runs on the packed FP32x2 pipe across orbital pairs.  psi planes come
// by plain coalesced loads (one per orbital and point) held in registers for one step and then
// stored as whole cells.
constexpr int L32_NT = 512, L32_RING = 4;

template <int NB>
__host__ __device__ inline size_t lin32_cells(int oy, int nz) {
  return (size_t)(nz + 2) * (L32_RING * (oy + 4) + 4 * (oy + 2));
}

template <int NB>
struct alignas(4 * NB) Cell {
  float v[NB];
};
template <int NB>
__device__ __forceinline__ Cell<NB> cfma(float s, Cell<NB> b, Cell<NB> c) {
  Cell<NB> r;
  if constexpr (NB == 1) {
    r.v[0] = fmaf(s, b.v[0], c.v[0]);
  } else {
#pragma unroll
    for (int o = 0; o < NB; o += 2) {
      const float2 q = __ffma2_rn(make_float2(s, s), make_float2(b.v[o], b.v[o + 1]), make_float2(c.v[o], c.v[o + 1]));
      r.v[o] = q.x;
      r.v[o + 1] = q.y;
    }
  }
  return r;
}
template <int NB>
__device__ __forceinline__ Cell<NB> cmul(float s, Cell<NB> b) {
  Cell<NB> r;
  if constexpr (NB == 1) {
    r.v[0] = s * b.v[0];
  } else {
#pragma unroll
    for (int o = 0; o < NB; o += 2) {
      const float2 q = __fmul2_rn(make_float2(s, s), make_float2(b.v[o], b.v[o + 1]));
      r.v[o] = q.x;
      r.v[o + 1] = q.y;
    }
  }
  return r;
}
template <int NB>
__device__ __forceinline__ Cell<NB> csub(Cell<NB> a, Cell<NB> b) { return cfma(-1.f, b, a); }  // a - b, one rounding
template <int NB>
__device__ __forceinline__ Cell<NB> cadd(Cell<NB> a, Cell<NB> b) { return cfma(1.f, b, a); }
// 3 a - 3 b + c in the rounding order of the scalar kernels: fma(3, a, -3 b) + c
template <int NB>
__device__ __forceinline__ Cell<NB> lin_ext3(Cell<NB> a, Cell<NB> b, Cell<NB> c) {
  return cadd(cfma(3.f, a, cmul(-3.f, b)), c);
}
// a1 g1 + a2 g2 + a3 g3 in the rounding order of the scalar kernels: fma(a3, g3, fma(a1, g1, a2 g2))
template <int NB>
__device__ __forceinline__ Cell<NB> cflux(float a1, Cell<NB> g1, float a2, Cell<NB> g2, float a3, Cell<NB> g3) {
  return cfma(a3, g3, cfma(a1, g1, cmul(a2, g2)));
}

// DOT: products and per-thread sums of the Krylov dots.
template <int NB, int PPT, bool PROD, bool KRY, typename DOT = float>
__global__ void __launch_bounds__(L32_NT, 1)
    hpsi_lin32_kernel(const float* __restrict__ coeffs, const float* __restrict__ veff, const float* __restrict__ psi,
                      float* __restrict__ out, const LinArgs a, float kscale, float vscale) {
  static_assert(!KRY || NB == 1, "the Krylov mode serves one orbital");
  constexpr int NT = L32_NT, RING = L32_RING;
  constexpr int LD = (3 * PPT + 1) / 2;  // psi cells copied per thread and plane: (oy + 4) nz <= 1.5 NT PPT (oy >= 2)
  using C = Cell<NB>;
  if constexpr (KRY) {
    if (a.skip && *a.skip) return;  // the Krylov solve has stopped: uniform for the whole launch
  }
  extern __shared__ __align__(16) float sm32[];
  const int tid = threadIdx.x, nx = a.nx, ny = a.ny, nz = a.nz, P = nz + 2;
  // every global access is a 64-bit base plus a 32-bit byte offset (checked on the host)
  const unsigned plane4 = 4u * (unsigned)(ny * nz), n4 = 4u * (unsigned)a.n;
  const auto ld = [](const float* b, unsigned off) {
    return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(b) + off));
  };
  const auto at = [](float* b, unsigned off) -> float& { return *reinterpret_cast<float*>(reinterpret_cast<char*>(b) + off); };
  C zero;
#pragma unroll
  for (int o = 0; o < NB; ++o) zero.v[o] = 0.f;
  DOT d0 = 0, d1 = 0;  // Krylov dots: a few dozen terms per thread, FP64 across threads
  const auto dot = [](float x) -> DOT {
    if constexpr (sizeof(DOT) == 8)
      return widen(x);
    else
      return x;
  };
  const int end = lin_bound(blockIdx.x + 1, a);
  for (int pos = lin_bound(blockIdx.x, a); pos < end;) {
    const LinSeg t = lin_seg(a, pos, end, NB);
    pos += t.x1 - t.x0;
    const int j0 = t.j0, oy = t.oy, nv = min(NB, a.nb - t.o0);
    const int psz = (oy + 4) * P, fsz = (oy + 2) * P;
    C* const ring = reinterpret_cast<C*>(sm32);
    C* const fbuf = ring + RING * psz;
    // ghost cells read as zero (trial fix); the production closure writes every ghost it reads
    if (!PROD)
      for (int e = tid; e < RING * psz + 4 * fsz; e += NT) ring[e] = zero;

    const int jlo = max(j0 - 2, 0), jhi = min(j0 + oy + 1, ny - 1);
    const int cnt = (jhi - jlo + 1) * nz;
    int dst[LD];
#pragma unroll
    for (int l = 0; l < LD; ++l) {
      const int e = tid + l * NT;
      dst[l] = e < cnt ? (jlo - (j0 - 2)) * P + 1 + e + 2 * (int)__umulhi(e, a.rnz) : -1;
    }
    const float* pin[NB];  // orbitals past nv repeat the last one and are not stored
    float* pout[NB];
#pragma unroll
    for (int o = 0; o < NB; ++o) {
      pin[o] = psi + (long long)(t.o0 + min(o, nv - 1)) * a.ostride;
      pout[o] = out + (long long)(t.o0 + min(o, nv - 1)) * a.ostride;
    }
    C stage[LD];
    auto fetch = [&](int p) {
      const unsigned off = (unsigned)p * plane4 + 4u * (unsigned)(jlo * nz + tid);
#pragma unroll
      for (int l = 0; l < LD; ++l)
        if (dst[l] >= 0)
#pragma unroll
          for (int o = 0; o < NB; ++o) stage[l].v[o] = ld(pin[o], off + 4u * l * NT);
    };
    auto put = [&](C* d) {
#pragma unroll
      for (int l = 0; l < LD; ++l)
        if (dst[l] >= 0) d[dst[l]] = stage[l];
    };

    // own points tid + i * NT of the flux tile (row R = 0 .. oy + 1, j = j0 - 1 + R):
    // cell ci in a flux buffer, ci + P in a psi plane
    int ci[PPT];
    unsigned col[PPT];
    bool real[PPT], emit[PPT], face[PPT];
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      const int q = tid + i * NT, R = __umulhi(q, a.rnz), z = q - R * nz, j = j0 - 1 + R;
      const bool in = q < (oy + 2) * nz;
      real[i] = in && j >= 0 && j < ny;
      ci[i] = in ? R * P + 1 + z : 1;
      emit[i] = real[i] && R >= 1 && R <= oy;
      face[i] = j == 0 || j == ny - 1 || z == 0 || z == nz - 1;
      col[i] = real[i] ? 4u * (unsigned)(j * nz + z) : 0u;
    }

    if (!PROD) __syncthreads();  // the zero fill precedes the copies
    auto slot = [&](int k) { return ring + (k & (RING - 1)) * psz; };  // slot of plane p: (p - sb + 1) mod RING
    for (int p = max(t.sb - 1, 0); p <= t.sb + 1; ++p) {
      fetch(p);
      put(slot(p - t.sb + 1));
    }
    if (t.sb + 2 <= t.last) fetch(t.sb + 2);
    if constexpr (PROD) {
      __syncthreads();
      fill_psi<C, NT>(slot(1), ny, nz, j0, oy);
      if (t.sb == 0)  // psi(-1) = 3 psi(0) - 3 psi(1) + psi(2)
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (real[i]) {
            C p2;
#pragma unroll
            for (int o = 0; o < NB; ++o)
              p2.v[o] = ld(pin[o], 2u * plane4 + col[i]);
            slot(0)[ci[i] + P] = lin_ext3(slot(1)[ci[i] + P], slot(2)[ci[i] + P], p2);
          }
    }
    C fx[PPT], f1[PPT], f2[PPT];  // F^x(s), F^x(s-1), F^x(s-2) at the own points
#pragma unroll
    for (int i = 0; i < PPT; ++i) fx[i] = f1[i] = f2[i] = zero;

    // outputs of plane op at point i: df = F^x(op + 1) - F^x(op - 1), ps = psi(op)
    auto store = [&](int i, int op, C df, C ps, float kij, float vv) {
      const C* const fy = fbuf + 2 * (op & 1) * fsz + ci[i];
      const C* const fz = fy + fsz;
      C val = cmul(kij, cadd(cadd(df, csub(fy[P], fy[-P])), csub(fz[1], fz[-1])));
      if (veff) val = cfma(vv, ps, val);
      const unsigned go = (unsigned)op * plane4 + col[i];
      if constexpr (KRY) {
        // faces of a Krylov vector stay zero; the dots then cover interior points only
        if (face[i] || op == 0 || op == nx - 1) val = zero;
        if (a.dot_y) {
          d0 = fma(dot(val.v[0]), dot(ld(static_cast<const float*>(a.dot_y), go)), d0);
        } else {
          const DOT v0 = dot(val.v[0]);
          d0 = fma(v0, dot(ps.v[0]), d0);
          d1 = fma(v0, v0, d1);
        }
      }
#pragma unroll
      for (int o = 0; o < NB; ++o)
        if (o < nv) at(pout[o], go) = val.v[o];
    };
    auto scale_k = [&](int i, int op) { return kscale * ld(coeffs, 6u * n4 + (unsigned)op * plane4 + col[i]); };
    auto scale_v = [&](int i, int op) { return veff ? vscale * ld(veff, (unsigned)op * plane4 + col[i]) : 0.f; };

    int k = 1;  // slot index of plane s
    for (int s = t.sb; s <= t.se; ++s) {
      const int op = s - 1;
      const bool outp = op >= t.x0 && op < t.x1;
      // geometry of plane s and the scales of plane s-1, in flight across the barrier
      float axx[PPT], ayy[PPT], azz[PPT], axy[PPT], axz[PPT], ayz[PPT], kij[PPT], vv[PPT];
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const unsigned g = (unsigned)s * plane4 + col[i];
        axx[i] = ld(coeffs, g);
        ayy[i] = ld(coeffs, g + n4);
        azz[i] = ld(coeffs, g + 2u * n4);
        axy[i] = ld(coeffs, g + 3u * n4);
        axz[i] = ld(coeffs, g + 4u * n4);
        ayz[i] = ld(coeffs, g + 5u * n4);
        kij[i] = scale_k(i, max(op, 0));
        vv[i] = scale_v(i, max(op, 0));
      }
      __syncthreads();  // plane s+1 is stored, plane s's ghosts and the fluxes of plane s-1 are complete
      C *const prv = slot(k + RING - 1), *const cur = slot(k), *const nxt = slot(k + 1);
      if (s + 1 == nx) {
        // psi(nx) = 3 psi(nx-1) - 3 psi(nx-2) + psi(nx-3), or zero; plane nx-3 is still in its slot
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (real[i]) {
            const int c = ci[i] + P;
            nxt[c] = PROD ? lin_ext3(cur[c], prv[c], slot(k + 2)[c]) : zero;
          }
      }
      if (PROD && outp) fill_flux<C, NT>(fbuf + 2 * (op & 1) * fsz, fbuf + (2 * (op & 1) + 1) * fsz, ny, nz, j0, oy);
      C* const fy = fbuf + 2 * (s & 1) * fsz;
      C* const fz = fy + fsz;
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int c = ci[i] + P;
        const C gx = csub(nxt[c], prv[c]);
        const C gy = csub(cur[c + P], cur[c - P]);
        const C gz = csub(cur[c + 1], cur[c - 1]);
        fx[i] = cflux(axx[i], gx, axy[i], gy, axz[i], gz);
        if (real[i]) {
          fy[ci[i]] = cflux(axy[i], gx, ayy[i], gy, ayz[i], gz);
          fz[ci[i]] = cflux(axz[i], gx, ayz[i], gy, azz[i], gz);
        }
      }
      if (s + 2 <= t.last) put(slot(k + 2));  // plane s+2 into the slot of plane s-2
      if (s + 3 <= t.last) fetch(s + 3);
      if (PROD && outp) __syncthreads();  // the flux ghosts of plane s-1 are complete
      if (PROD && s + 1 <= t.last) fill_psi<C, NT>(nxt, ny, nz, j0, oy);
      if (outp)
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (emit[i]) store(i, op, csub(fx[i], f2[i]), prv[ci[i] + P], kij[i], vv[i]);
      if (PROD && !KRY && s == 2 && t.x0 == 0) {
        // F^x ghost below the lower face, 3 F(0) - 3 F(1) + F(2): plane 0 was written without it
#pragma unroll
        for (int i = 0; i < PPT; ++i)
          if (emit[i]) {
            const float k0 = -scale_k(i, 0);
            const C g = lin_ext3(f2[i], f1[i], fx[i]);
#pragma unroll
            for (int o = 0; o < NB; ++o)
              if (o < nv) at(pout[o], col[i]) = fmaf(k0, g.v[o], at(pout[o], col[i]));
          }
      }
      if (s < nx - 1)
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
          f2[i] = f1[i];
          f1[i] = fx[i];
        }
      ++k;
    }

    // ---- plane nx-1: fx, f1, f2 hold F^x(nx-1), F^x(nx-2), F^x(nx-3)
    if (t.x1 == nx) {
      __syncthreads();
      if constexpr (PROD) {
        fill_flux<C, NT>(fbuf + 2 * ((nx - 1) & 1) * fsz, fbuf + (2 * ((nx - 1) & 1) + 1) * fsz, ny, nz, j0, oy);
        __syncthreads();
      }
      const C* const cur = slot(k + RING - 1);
#pragma unroll
      for (int i = 0; i < PPT; ++i)
        if (emit[i])
          // the scalar kernels form this ghost as fma(-3, F(nx-2), 3 F(nx-1)) + F(nx-3)
          store(i, nx - 1, csub(PROD ? cadd(cfma(-3.f, f1[i], cmul(3.f, fx[i])), f2[i]) : zero, f1[i]),
                cur[ci[i] + P], scale_k(i, nx - 1), scale_v(i, nx - 1));
    }
    __syncthreads();  // the next segment reuses the buffers
  }
  if constexpr (KRY) {
    double v2[2] = {(double)d0, (double)d1};
    block_atomic_add<2, NT>(a.dot_acc, v2);
  }
}

// ------------------------------------------------------------------------------- host side
struct LinPlan {
  int oymax, tiles;
  long long ctas;
};

// Row tiles and CTAs: the choice whose estimated time is lowest.  A tile's rows share their halo
// rows, a share's planes two extra planes and the first loads; both are cheapest when long, while
// the shares have to fill the SMs.  What decides on small grids is the largest share: with as many
// CTAs per unit as divide the grid, no share crosses a unit (which would march the extra planes and
// load the first ones twice).  Costs in SM clocks: `full` per own point (all NB orbitals), `halo` per
// halo point (its loads included), `edge` per own point of an extra plane; a march step and, `start`
// times, a segment's first loads add `step` clocks of latency, and a CTA alone on its SM runs `lone`
// times longer.  Fitted to 400 timed plans of 24 FP64 and 20 FP32 cases (grids of 17 thousand to 1.3
// million points, 1 to 20 orbitals), whose picks are then within 4 % (FP64) and 6 % (FP32) of the
// fastest but for 15 % on 25x27x29.  FP64, production closure, with shares cut regardless of the units
// (two CTAs per SM) / as here: 67x67x81 36.9 / 30.5 us, 57x73x61 30.7 / 21.7, 96x96x96 68.0 / 50.5,
// 48x80x150 69.7 / 40.5, eight orbitals on 45x51x47 61.5 / 49.1, 20 on 25x27x29 50.7 / 31.5, 20 on
// 67x67x81 317 either way; FP32, one orbital on 57x73x61 10.4 / 9.4, eight on 45x51x47 14.0 / 11.8.
struct LinCost {
  int oycap, maxres, values;  // tallest tile, CTAs per SM, shared values per cell
  size_t value_bytes;
  double full, halo, edge, step, start, lone;
};

template <typename CELLS>
LinPlan lin_search(int nx, int ny, int nz, int groups, CELLS cells, const LinCost& c) {
  const int sms = device_sm_count();
  LinPlan best{0, 0, 0};
  double tbest = 0.0;
  for (int tiles = c.oycap >= 2 ? (ny + c.oycap - 1) / c.oycap : ny; ny / tiles >= 2; ++tiles) {
    const int oy = (ny + tiles - 1) / tiles;  // tallest tile
    const int res = (int)std::min<size_t>(c.maxres, 227 * 1024 / (cells(oy, nz) * c.values * c.value_bytes + 1024));
    if (res < 1) continue;
    const long long units = (long long)tiles * groups, total = units * nx;
    if (total > 0x3fffffff) break;
    const double pl = (c.full * ny / tiles + 2 * c.halo) * nz, ed = c.edge * oy * nz;
    auto consider = [&](long long ctas) {
      if (ctas < 1 || ctas > total) return;
      long long share = (total + ctas - 1) / ctas;  // planes of the largest share
      double segs = 2.0 + (double)(share / nx);
      if (ctas % units == 0) {
        segs = 1.0;
        share = (nx + ctas / units - 1) / (ctas / units);
      } else if (units % ctas == 0) {
        segs = (double)(units / ctas);
      }
      const long long per_sm = (ctas + sms - 1) / sms;
      const double t = (per_sm == 1 ? c.lone : (double)per_sm) * (share * pl + segs * 2 * ed) +
                       (share + c.start * segs) * c.step;
      if (best.tiles == 0 || t < tbest) {
        tbest = t;
        best = LinPlan{oy, tiles, ctas};
      }
    };
    for (int r = res; r >= 1; --r) {
      const long long cap = (long long)sms * r;
      consider(std::min(cap, total));
      for (int least = 2; least <= 4; ++least) consider(std::min(cap, (total + least - 1) / least));
      if (units <= cap)
        consider(cap / units * units);
      else
        consider(units / ((units + cap - 1) / cap));
    }
  }
  return best;
}

// The search takes a few microseconds of host time: the last plans of each host thread are kept
// (they depend on the sizes alone).
template <typename CELLS>
LinPlan lin_plan(int nx, int ny, int nz, int groups, CELLS cells, const LinCost& c) {
  struct Entry {
    int nx, ny, nz, groups, values, cap;
    size_t bytes;
    LinPlan plan;
  };
  constexpr int N = 8;
  static thread_local Entry kept[N] = {};
  static thread_local int next = 0;
  for (const Entry& e : kept)
    if (e.nx == nx && e.ny == ny && e.nz == nz && e.groups == groups && e.values == c.values && e.cap == c.oycap &&
        e.bytes == c.value_bytes)
      return e.plan;
  const LinPlan p = lin_search(nx, ny, nz, groups, cells, c);
  kept[next] = Entry{nx, ny, nz, groups, c.values, c.oycap, c.value_bytes, p};
  next = (next + 1) % N;
  return p;
}

LinArgs lin_args(const LinPlan& p, int nx, int ny, int nz, int nb, long long ostride, int groups, const void* dot_y,
                 double* dot_acc, const int* skip) {
  LinArgs a;
  a.nx = nx; a.ny = ny; a.nz = nz; a.nb = nb;
  a.n = (long long)nx * ny * nz;
  a.ostride = nb > 1 ? ostride : a.n;
  a.tiles = p.tiles; a.groups = groups;
  a.total = (int)((long long)p.tiles * groups * nx);
  a.rnz = (unsigned)(((1ULL << 32) + nz - 1) / nz);
  a.dot_y = dot_y;
  a.dot_acc = dot_acc;
  a.skip = skip;
  return a;
}

template <bool PROD, bool KRY, bool HASV>
int lin64_launch(const double* coeffs, const double* veff, const double* psi, double* out, int nx, int ny, int nz,
                 int nb, long long ostride, double kscale, cudaStream_t st, const double* dot_y = nullptr,
                 double* dot_acc = nullptr, const int* skip = nullptr) {
  int kexp = 0;
  if (std::fabs(std::frexp(kscale, &kexp)) != 0.5) return -1;  // powers of two only
  --kexp;
  if (kexp < -32 || kexp > 32) return -1;
  const LinPlan p = lin_plan(nx, ny, nz, nb, lin64_cells,
                             LinCost{std::min(ny, L64_NT * L64_PPT / nz), L64_MINB, 1, sizeof(double), 10.5, 28.6, 13.5,
                                     1600.0, 3.3, 1.16});
  if (p.tiles == 0) return -1;
  const size_t smem = lin64_cells(p.oymax, nz) * sizeof(double);
  auto kern = hpsi_lin64_kernel<PROD, KRY, HASV>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != IGD_OK) return IGD_ERR_CUDA;
  const LinArgs a = lin_args(p, nx, ny, nz, nb, ostride, nb, dot_y, dot_acc, skip);
  kern<<<(unsigned)p.ctas, L64_NT, smem, st>>>(coeffs, veff, psi, out, a, kscale, kexp, kscale < 0 ? 0x80000000u : 0u);
  return launch_status();
}

template <bool PROD>
int lin64_v(const double* c, const double* v, const double* p, double* o, int nx, int ny, int nz, int nb,
            long long ostride, double kscale, double vscale, cudaStream_t st) {
  if (!v) return lin64_launch<PROD, false, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, st);
  if (vscale != 1.0) return -1;
  return lin64_launch<PROD, false, true>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, st);
}

template <int NB, int PPT, bool PROD, bool KRY, typename DOT = float>
int lin32_launch(const float* coeffs, const float* veff, const float* psi, float* out, int nx, int ny, int nz, int nb,
                 long long ostride, double kscale, double vscale, cudaStream_t st, const float* dot_y = nullptr,
                 double* dot_acc = nullptr, const int* skip = nullptr) {
  const int groups = (nb + NB - 1) / NB;
  const double pt = 0.6 + 0.7 * NB;
  const LinPlan p = lin_plan(nx, ny, nz, groups, lin32_cells<NB>,
                             LinCost{std::min(ny, L32_NT * PPT / nz - 2), 1, NB, sizeof(float), pt, 1.8 * pt, 0.85 * pt,
                                     1250.0, 4.5, 1.0});
  if (p.tiles == 0) return -1;
  const size_t smem = lin32_cells<NB>(p.oymax, nz) * sizeof(float) * NB;
  auto kern = hpsi_lin32_kernel<NB, PPT, PROD, KRY, DOT>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != IGD_OK) return IGD_ERR_CUDA;
  const LinArgs a = lin_args(p, nx, ny, nz, nb, ostride, groups, dot_y, dot_acc, skip);
  kern<<<(unsigned)p.ctas, L32_NT, smem, st>>>(coeffs, veff, psi, out, a, (float)kscale, (float)vscale);
  return launch_status();
}

// Rows of at most 256 points: a tile holds at least three output rows with their halo, and the
// copies and halo points per thread cover it.  The seven FP32 coefficient fields are addressed
// with 32-bit byte offsets.
bool lin_ok(int nx, int ny, int nz) {
  return nz <= 256 && (long long)ny * nz < (1LL << 28) && 28LL * nx * ny * nz < (1LL << 32);
}

template <bool PROD>
int lin32_nb(const float* c, const float* v, const float* p, float* o, int nx, int ny, int nz, int nb, long long ostride,
             double kscale, double vscale, cudaStream_t st) {
  // two points per thread hold two rows and their halo up to 204 points a row (oycap 3: every
  // ny >= 3 splits into tiles of two rows or more); longer rows take three, for two orbitals
  if (nz > L32_NT * 2 / 5) {
    if (nb >= 2) return lin32_launch<2, 3, PROD, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
    return lin32_launch<1, 3, PROD, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
  }
  if (nb >= 3) return lin32_launch<4, 2, PROD, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
  if (nb == 2) return lin32_launch<2, 2, PROD, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
  return lin32_launch<1, 2, PROD, false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
}

}  // namespace

int hpsi_agrid_lin_launch(int dtype, int closure, int nx, int ny, int nz, const void* coeffs, const void* veff,
                          const void* psi, void* out, int nb, long long ostride, double kscale, double vscale,
                          cudaStream_t st) {
  if (!lin_ok(nx, ny, nz)) return -1;
  const bool prod = closure == IGD_CLOSURE_PRODUCTION;
  if (dtype == IGD_F32) {
    const float *c = static_cast<const float*>(coeffs), *v = static_cast<const float*>(veff),
                *p = static_cast<const float*>(psi);
    float* o = static_cast<float*>(out);
    return prod ? lin32_nb<true>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st)
                : lin32_nb<false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
  }
  if (dtype == IGD_F64) {
    const double *c = static_cast<const double*>(coeffs), *v = static_cast<const double*>(veff),
                 *p = static_cast<const double*>(psi);
    double* o = static_cast<double*>(out);
    return prod ? lin64_v<true>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st)
                : lin64_v<false>(c, v, p, o, nx, ny, nz, nb, ostride, kscale, vscale, st);
  }
  return -1;
}

// lin_ok's rows split into tiles of two rows or more for every ny >= 3, so an applicable grid always has a plan.
bool hpsi_agrid_lin_krylov_applies(int nx, int ny, int nz) { return lin_ok(nx, ny, nz); }

int hpsi_agrid_lin_krylov(int dtype, int nx, int ny, int nz, const void* coeffs, const void* psi, void* out,
                          double kscale, const void* dot_y, double* dot_acc, const int* skip, bool dots64,
                          cudaStream_t st) {
  if (!lin_ok(nx, ny, nz) || !dot_acc) return -1;
  const long long n = (long long)nx * ny * nz;
  if (dtype == IGD_F64)
    return lin64_launch<true, true, false>(static_cast<const double*>(coeffs), nullptr, static_cast<const double*>(psi),
                                           static_cast<double*>(out), nx, ny, nz, 1, n, kscale, st,
                                           static_cast<const double*>(dot_y), dot_acc, skip);
  const float *c = static_cast<const float*>(coeffs), *p = static_cast<const float*>(psi),
              *y = static_cast<const float*>(dot_y);
  float* o = static_cast<float*>(out);
  const auto run = [&](auto dot) {
    using D = decltype(dot);
    if (nz > L32_NT * 2 / 5)
      return lin32_launch<1, 3, true, true, D>(c, nullptr, p, o, nx, ny, nz, 1, n, kscale, 0.0, st, y, dot_acc, skip);
    return lin32_launch<1, 2, true, true, D>(c, nullptr, p, o, nx, ny, nz, 1, n, kscale, 0.0, st, y, dot_acc, skip);
  };
  return dots64 ? run(0.0) : run(0.f);
}

}  // namespace igd
