// Pointwise LSDA exchange-correlation (K9) and spin-density build (K10).
//
// LSDA: the reference evaluates "lda,vwn" through PySCF/libxc
// (xc/lsda.py:70-121): Slater exchange plus the VWN5 correlation fit of
// Vosko, Wilk and Nusair (Can. J. Phys. 58, 1200 (1980)) with its spin
// interpolation; PW92 (Perdew and Wang, PRB 45, 13244 (1992)) is offered as
// an option.  Written from those published forms: per channel
//   G(x) = A [ln(x^2/X) + 2b/Q atan(Q/(2x+b))
//             - b x0/X(x0) (ln((x-x0)^2/X) + 2(b+2x0)/Q atan(Q/(2x+b)))],
// x = sqrt(rs), X = x^2 + b x + c, Q = sqrt(4c - b^2);
// eps_c = eps_P + alpha f(z)(1-z^4)/f''(0) + (eps_F - eps_P) f(z) z^4 and
// v_s = eps - rs/3 d eps/d rs +- (1 -+ z) d eps/dz.  Density validation and
// clipping follow xc/lsda.py:57-67; points below 1e-15 total density give 0.
//
// Density: rho_s = sum_i occ_i |psi_i|^2 (scf/driver.py:663-676), its integral
// and renormalisation (:679-690) and the weighted residual (:693-702).
#include "common.cuh"
#include "lsda_tables.cuh"

namespace igd {
namespace {

constexpr int XB = 256;
inline int xblocks(long long n) { return (int)std::min<long long>((n + XB - 1) / XB, 152LL * 8); }

template <typename M>
struct VwnChan {
  M A, b, c, x0;
};

template <typename M>
__device__ __forceinline__ void vwn_channel(M x, const VwnChan<M>& p, M& g, M& dgdx) {
  const M X = x * x + p.b * x + p.c;
  const M X0 = p.x0 * p.x0 + p.b * p.x0 + p.c;
  const M Q = sqrt(M(4) * p.c - p.b * p.b);
  const M t = M(2) * x + p.b;
  const M at = atan(Q / t);
  const M k = p.b * p.x0 / X0;
  g = p.A * (log(x * x / X) + (M(2) * p.b / Q) * at -
             k * (log((x - p.x0) * (x - p.x0) / X) + (M(2) * (p.b + M(2) * p.x0) / Q) * at));
  const M den = t * t + Q * Q;
  dgdx = p.A * (M(2) / x - t / X - M(4) * p.b / den -
                k * (M(2) / (x - p.x0) - t / X - M(4) * (p.b + M(2) * p.x0) / den));
}

template <typename M>
struct PwChan {
  M A, a1, b1, b2, b3, b4;
};

template <typename M>
__device__ __forceinline__ void pw_channel(M rs, const PwChan<M>& p, M& g, M& dgdrs) {
  const M s = sqrt(rs);
  const M qd = M(2) * p.A * (p.b1 * s + p.b2 * rs + p.b3 * rs * s + p.b4 * rs * rs);
  const M dqd = M(2) * p.A * (M(0.5) * p.b1 / s + p.b2 + M(1.5) * p.b3 * s + M(2) * p.b4 * rs);
  const M lg = log1p(M(1) / qd);
  g = -M(2) * p.A * (M(1) + p.a1 * rs) * lg;
  dgdrs = -M(2) * p.A * p.a1 * lg + M(2) * p.A * (M(1) + p.a1 * rs) * dqd / (qd * qd + qd);
}

// Energy per particle and potentials at one point (rho = ru64 + rd64 >= 1e-15) by the closed forms in M.
template <typename M, int FUNC>
__device__ __forceinline__ void lsda_point(double ru64, double rd64, double rho64, M& e, M& vu, M& vd) {
  const M pi = M(3.14159265358979323846);
  const M fpp = M(4) / (M(9) * (cbrt(M(2)) - M(1)));
  const M fden = M(2) * cbrt(M(2)) - M(2);
  const M cx = cbrt(M(6) / pi);
  const M u = M(ru64), d = M(rd64), r = M(rho64);
  const M cu = cbrt(u), cd = cbrt(d);
  const M ex = -M(0.75) * cx * (u * cu + d * cd);
  const M vxu = -cx * cu, vxd = -cx * cd;
  M z = (u - d) / r;
  z = z > M(1) ? M(1) : (z < M(-1) ? M(-1) : z);
  const M rs = cbrt(M(3) / (M(4) * pi * r));
  M gp, dgp, gf, dgf, ga, dga;
  if (FUNC == 0) {
    const M x = sqrt(rs);
    const VwnChan<M> P{M(0.0310907), M(3.72744), M(12.9352), M(-0.10498)};
    const VwnChan<M> F{M(0.01554535), M(7.06042), M(18.0578), M(-0.32500)};
    const VwnChan<M> Al{M(-1) / (M(6) * pi * pi), M(1.13107), M(13.0045), M(-0.0047584)};
    vwn_channel(x, P, gp, dgp);
    vwn_channel(x, F, gf, dgf);
    vwn_channel(x, Al, ga, dga);
    const M to_rs = M(1) / (M(2) * x);
    dgp *= to_rs;
    dgf *= to_rs;
    dga *= to_rs;
  } else {
    const PwChan<M> P{M(0.031091), M(0.21370), M(7.5957), M(3.5876), M(1.6382), M(0.49294)};
    const PwChan<M> F{M(0.015545), M(0.20548), M(14.1189), M(6.1977), M(3.3662), M(0.62517)};
    const PwChan<M> Al{M(0.016887), M(0.11125), M(10.357), M(3.6231), M(0.88026), M(0.49671)};
    pw_channel(rs, P, gp, dgp);
    pw_channel(rs, F, gf, dgf);
    pw_channel(rs, Al, ga, dga);
    ga = -ga;
    dga = -dga;
  }
  // 1 +- z from the spin densities directly (no cancellation when one spin is tiny)
  const M opz = M(2) * u / r, omz = M(2) * d / r;
  const M a = cbrt(opz), b = cbrt(omz);
  const M f = (opz * a + omz * b - M(2)) / fden;
  const M df = (M(4) / M(3)) * (a - b) / fden;
  const M z3 = z * z * z, z4 = z3 * z;
  const M ec = gp + ga * f * (M(1) - z4) / fpp + (gf - gp) * f * z4;
  const M decrs = dgp + dga * f * (M(1) - z4) / fpp + (dgf - dgp) * f * z4;
  const M decz = ga * (df * (M(1) - z4) - M(4) * z3 * f) / fpp + (gf - gp) * (df * z4 + M(4) * z3 * f);
  const M base = ec - rs / M(3) * decrs;
  e = ex / r + ec;
  vu = vxu + base + omz * decz;
  vd = vxd + base - opz * decz;
}

// FP32 math; I/O in T; energy reduction in FP64.
template <typename T, typename M, int FUNC>
__global__ void lsda_kernel(long long n, const T* __restrict__ ru_in, const T* __restrict__ rd_in, T* __restrict__ eps,
                            T* __restrict__ vu, T* __restrict__ vd, T* __restrict__ edens,
                            const double* __restrict__ w, double* energy, int* flags) {
  double e_acc = 0.0;
  int fl = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double ru64 = (double)ru_in[i], rd64 = (double)rd_in[i];
    if (!isfinite(ru64) || !isfinite(rd64)) fl |= 1;
    if (ru64 < -1.0e-14 || rd64 < -1.0e-14) fl |= 2;
    ru64 = fmax(ru64, 0.0);
    rd64 = fmax(rd64, 0.0);
    const double rho64 = ru64 + rd64;
    M e_out = M(0), vu_out = M(0), vd_out = M(0);
    if (rho64 >= 1.0e-15) {
      lsda_point<M, FUNC>(ru64, rd64, rho64, e_out, vu_out, vd_out);
    }
    if (eps) eps[i] = T(e_out);
    if (vu) vu[i] = T(vu_out);
    if (vd) vd[i] = T(vd_out);
    const double ed = rho64 * (double)e_out;
    if (edens) edens[i] = T(ed);
    if (w) e_acc += ed * w[i];
  }
  if (energy) {
    double a[1] = {e_acc};
    block_atomic_add<1, XB>(energy, a);
  }
  if (fl) atomicOr(flags, fl);
}

// ---- FP64 math.
// GB300's FP64 pipe runs two lanes per clock and SM, so this kernel's time is its FP64 instruction
// count: the closed forms take about 750 a point (6 logs, 3 arctangents, 5 cube roots, 30
// divisions), this form about 160.  The three correlation channels come from piecewise
// polynomials in x = sqrt(rs) (lsda_tables.cuh), their rs-derivatives from the channels' rational
// forms (VWN: rs dG/drs = A (c (x - x0) - b x0 x) / ((x - x0) X)), and every root and reciprocal
// from an FP32 seed and one series step of third or fourth order; comparisons, exponent scaling
// and conversions run on the integer pipe.  128^3 points: 2.67 ms with the closed forms, 0.62 ms.
// Errors against 45-digit values stay at the level of the closed forms (a few 1e-16).

// Leading 24 bits of a positive double inside the FP32 exponent range, and back.
__device__ __forceinline__ float trunc_f32(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  return __int_as_float((int)__funnelshift_l((unsigned)lo, (unsigned)hi, 3) & 0x7fffff | (((hi >> 20) - 896) << 23));
}
__device__ __forceinline__ double widen_f32(float x) {
  const int b = __float_as_int(x);
  return __hiloint2double((b >> 3) + (896 << 20), b << 29);
}
__device__ __forceinline__ float ex2_f32(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1 / d for positive d in the FP32 exponent range
__device__ __forceinline__ double rcp64(double d) {
  const double y = widen_f32(__frcp_rn(trunc_f32(d)));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);  // y (1 + e + e^2), e below 2^-22
}
// Cube root of a double >= 0; subnormals (below every density that matters) in a call, because a
// predicated-off FP64 instruction takes its slot on the pipe all the same.
__device__ __noinline__ double cbrt_call(double u) { return cbrt(u); }
__device__ __forceinline__ double cbrt64(double u) {
  const int hi = __double2hiint(u);
  if (hi < 0x00100000) return __double_as_longlong(u) == 0 ? 0.0 : cbrt_call(u);
  const int k = (int)((unsigned)((hi >> 20) + 2049) / 3u) - 1024;  // floor(exponent / 3)
  const double m = __hiloint2double(hi - 3 * (k << 20), __double2loint(u));  // [1, 8)
  const double w = widen_f32(ex2_f32(__log2f(trunc_f32(m)) * (-1.f / 3.f)));  // about m^(-1/3)
  const double e = fma(-m, w * w * w, 1.0);
  const double v = fma(w, e * fma(e, 2.0 / 9.0, 1.0 / 3.0), w);  // m^(-1/3): the series of (1 - e)^(-1/3)
  const double v2 = v * v, c = m * v2;
  const double r = fma(fma(-(c * c), c, m), v2 * (1.0 / 3.0), c);  // one Newton step on the residual m - c^3
  return __hiloint2double(__double2hiint(r) + (k << 20), __double2loint(r));
}

constexpr int LSDA_ROW = 3 * LSDA_COEFS + 2;  // doubles per interval in shared memory (the pad spreads the banks)

// One channel's energy polynomial at s.
__device__ __forceinline__ double lsda_poly(const double* __restrict__ c, double s) {
  const double2* const q = reinterpret_cast<const double2*>(c);
  double2 t = q[LSDA_COEFS / 2 - 1];
  double p = fma(t.y, s, t.x);
#pragma unroll
  for (int k = LSDA_COEFS / 2 - 2; k >= 0; --k) {
    t = q[k];
    p = fma(fma(p, s, t.y), s, t.x);
  }
  return p;
}
// rs dG/drs / 3 of a VWN channel
__device__ __forceinline__ double vwn_slope(double x, double A, double b, double c, double x0) {
  const double num = fma(A / 3.0 * (c - b * x0), x, -(A / 3.0 * c * x0));
  return num * rcp64((x - x0) * fma(x, x + b, c));
}
// rs dG/drs / 3 of a PW92 channel with energy g = -2 A (1 + a1 rs) log1p(1 / q)
__device__ __forceinline__ double pw_slope(double x, double rs, double g, double A, double a1, double b1, double b2,
                                           double b3, double b4) {
  const double q = 2 * A * x * fma(x, fma(x, fma(x, b4, b3), b2), b1);
  const double rdq = A * x * fma(x, fma(x, fma(x, 4 * b4, 3 * b3), 2 * b2), b1);  // rs dq/drs
  const double l = fma(a1, rs, 1.0);
  return (1.0 / 3.0) * fma(a1 * rs * rcp64(l), g, 2 * A * l * rdq * rcp64(fma(q, q, q)));
}

// The closed forms, for densities above the tables (called for the same reason).
template <int FUNC>
__device__ __noinline__ void lsda_point64(double ru, double rd, double3* out) {
  double e = 0.0, vu = 0.0, vd = 0.0;
  if (ru + rd >= 1.0e-15) lsda_point<double, FUNC>(ru, rd, ru + rd, e, vu, vd);
  *out = make_double3(e, vu, vd);
}

template <typename T, int FUNC>
__global__ void __launch_bounds__(XB, 3) lsda64_kernel(long long n, const T* __restrict__ ru_in,
                                                    const T* __restrict__ rd_in, T* __restrict__ eps,
                                                    T* __restrict__ vu, T* __restrict__ vd, T* __restrict__ edens,
                                                    const double* __restrict__ w, double* energy, int* flags) {
  __shared__ __align__(16) double tab[LSDA_INTERVALS * LSDA_ROW];
  for (int i = threadIdx.x; i < LSDA_INTERVALS * LSDA_COEFS * 3; i += XB) {
    const int row = i / (3 * LSDA_COEFS), q = i - row * (3 * LSDA_COEFS), k = q / 3, ch = q - 3 * k;
    tab[row * LSDA_ROW + ch * LSDA_COEFS + k] = (&lsda_table[FUNC][0][0][0])[i];
  }
  __syncthreads();
  const double pi = 3.14159265358979323846, cb2 = 1.25992104989487316477;  // 2^(1/3)
  const double cx = 1.24070098179880017333;                                // (6 / pi)^(1/3)
  const double kx = 0.78762331789974325053;                                // (3 / (4 pi))^(1/6)
  const double fpp = 4.0 / (9.0 * (cb2 - 1.0)), fden = 2.0 * cb2 - 2.0;
  double e_acc = 0.0;
  int fl = 0;
  for (long long i = blockIdx.x * (long long)XB + threadIdx.x; i < n; i += (long long)gridDim.x * XB) {
    double u = (double)ru_in[i], d = (double)rd_in[i];
    const long long ub = __double_as_longlong(u), db = __double_as_longlong(d);
    constexpr long long INF = 0x7ff0000000000000LL, SIGN = (long long)(1ull << 63);
    const long long tol = 0x3d06849b86a12b9bLL;  // 1e-14
    const bool bad = (ub & ~SIGN) >= INF || (db & ~SIGN) >= INF;
    if (bad) fl |= 1;
    if ((ub < 0 && (ub & ~SIGN) > tol && (ub & ~SIGN) <= INF) || (db < 0 && (db & ~SIGN) > tol && (db & ~SIGN) <= INF))
      fl |= 2;
    if (ub < 0 && (ub & ~SIGN) <= INF) u = 0.0;  // fmax(u, 0); a NaN goes through as fmax gives 0 below
    if (db < 0 && (db & ~SIGN) <= INF) d = 0.0;
    if ((ub & ~SIGN) > INF) u = 0.0;
    if ((db & ~SIGN) > INF) d = 0.0;
    const double r = u + d;
    const long long rb = __double_as_longlong(r);
    double e_out, vu_out, vd_out;
    // the tables cover 1e-15 <= r < 2^15
    const bool tail = rb < 0x3cd203af9ee75616LL;  // r < 1e-15
    if (rb >= 0x40e0000000000000LL) {
      double3 o;
      lsda_point64<FUNC>(u, d, &o);
      e_out = o.x;
      vu_out = o.y;
      vd_out = o.z;
    } else {
      const double rr = tail ? 1.0e-15 : r;
      // y = r^(-1/6): the series of (1 - e)^(-1/6) about the FP32 seed
      const double y0 = widen_f32(ex2_f32(__log2f(trunc_f32(rr)) * (-1.f / 6.f)));
      const double y3 = y0 * y0 * y0, ey = fma(-rr, y3 * y3, 1.0);
      const double y = fma(y0, ey * fma(ey, fma(ey, 91.0 / 1296.0, 7.0 / 72.0), 1.0 / 6.0), y0);
      const double x = kx * y, inv = rcp64(rr);
      // interval of x and the position in it, from the bits of x
      const int xh = __double2hiint(x), xl = __double2loint(x);
      const int row = min(max((xh >> 17) - ((1023 + LSDA_LOW) << 3), 0), LSDA_INTERVALS - 1);
      const double s =
          __hiloint2double(0x3ff00000 | ((int)__funnelshift_l((unsigned)xl, (unsigned)xh, 3) & 0xfffff), xl << 3) - 1.5;
      const double* const c = tab + row * LSDA_ROW;
      const double gp = lsda_poly(c, s), gf = lsda_poly(c + LSDA_COEFS, s), ga = lsda_poly(c + 2 * LSDA_COEFS, s);
      double hp, hf, ha;  // rs dG/drs / 3
      if (FUNC == 0) {
        hp = vwn_slope(x, 0.0310907, 3.72744, 12.9352, -0.10498);
        hf = vwn_slope(x, 0.01554535, 7.06042, 18.0578, -0.32500);
        ha = vwn_slope(x, -1.0 / (6.0 * pi * pi), 1.13107, 13.0045, -0.0047584);
      } else {
        const double rs = x * x;
        hp = pw_slope(x, rs, gp, 0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294);
        hf = pw_slope(x, rs, gf, 0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517);
        ha = -pw_slope(x, rs, -ga, 0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671);
      }
      const double cu = cbrt64(u), cd = cbrt64(d);
      const double inv2 = inv + inv, opz = u * inv2, omz = d * inv2, z = (u - d) * inv;
      const double ky2 = cb2 * (y * y), ca = cu * ky2, cbz = cd * ky2;  // cube roots of 1 +- z
      const double f = fma(opz, ca, fma(omz, cbz, -2.0)) * (1.0 / fden), df = (ca - cbz) * (4.0 / (3.0 * fden));
      const double z2 = z * z, z4 = z2 * z2, q4 = fma(-1.0 / fpp, z4, 1.0 / fpp);  // (1 - z^4) / f''(0)
      const double fa = f * q4, fz = f * z4, z3f = z2 * z * f, dg = gf - gp;
      const double ec = fma(ga, fa, fma(dg, fz, gp));
      const double slope = fma(ha, fa, fma(hf - hp, fz, hp));
      const double decz = fma(ga, fma(z3f, -4.0 / fpp, df * q4), dg * fma(z3f, 4.0, df * z4));
      const double base = ec - slope;
      const double exr = fma(u, cu, d * cd) * (-0.75 * cx);
      e_out = fma(exr, inv, ec);
      vu_out = fma(omz, decz, fma(-cx, cu, base));
      vd_out = fma(-opz, decz, fma(-cx, cd, base));
      if (tail) e_out = vu_out = vd_out = 0.0;
    }
    if (eps) eps[i] = T(e_out);
    if (vu) vu[i] = T(vu_out);
    if (vd) vd[i] = T(vd_out);
    const double ed = r * e_out;
    if (edens) edens[i] = T(ed);
    if (w) e_acc = fma(ed, w[i], e_acc);
  }
  if (energy) {
    double a[1] = {e_acc};
    block_atomic_add<1, XB>(energy, a);
  }
  if (fl) atomicOr(flags, fl);
}

constexpr int DENS_MAXNB = IGD_DENSITY_VALUES;  // occupations held in shared memory

// Where a density kernel's occupations come from: device memory, or (p null) the launch's own arguments.
struct Occupations {
  const double* p;
  double v[DENS_MAXNB];
  __device__ __forceinline__ double at(int o) const { return p ? p[o] : v[o]; }
};

// rho = sum_i occ_i psi_i^2 (FP64 out); *integral += sum rho W.  Up to DENS_MAXNB occupations are
// converted to the orbital type once per block (SHARED): converted at every point they kept the FP64
// pipe busy.  16 FP32 orbitals over 127^3 points: 75.9 us, now 32.9 (memory floor 24).
template <typename T, bool SHARED>
__global__ void density_kernel(long long n, int nb, long long stride, const T* __restrict__ psi,
                               const __grid_constant__ Occupations occ, const double* __restrict__ w,
                               double* __restrict__ rho, double* integral, int accumulate) {
  __shared__ T so[SHARED ? DENS_MAXNB : 1];
  if constexpr (SHARED) {
    for (int o = threadIdx.x; o < nb; o += blockDim.x) so[o] = T(occ.at(o));
    __syncthreads();
  }
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    // sum over orbitals in the orbital type (FP32 orbitals: FP32 squares and sum,
    // GB300's FP64 pipe would bound the kernel), stored and integrated in FP64
    T t = T(0);
#pragma unroll 8
    for (int o = 0; o < nb; ++o) {
      const T p = psi[(long long)o * stride + i];
      t += (SHARED ? so[o] : T(occ.p[o])) * p * p;
    }
    const double r = (accumulate ? rho[i] : 0.0) + (double)t;
    rho[i] = r;
    if (w) acc += r * w[i];
  }
  if (integral) {
    double a[1] = {acc};
    block_atomic_add<1, XB>(integral, a);
  }
}

// 16-byte form for FP32 orbitals (4 consecutive points per thread; n and the
// orbital stride multiples of 4, 16-byte aligned data): occupations converted
// to FP32 once per block into shared memory (a per-point FP64 conversion would
// bound the kernel on GB300's FP64 pipe), FP32 squares and sum over orbitals,
// FP64 density and integral.  The orbital loop is unrolled by 16 to have enough loads in
// flight: 16 orbitals over 128^3 points 43.6 us with 4, 40.5 with 8, 36.0 with 16 (memory floor 25).
__global__ void density_v4_kernel(long long n4, int nb, long long stride, const float* __restrict__ psi,
                                  const __grid_constant__ Occupations occ, const double* __restrict__ w,
                                  double* __restrict__ rho, double* integral, int accumulate) {
  __shared__ float so[DENS_MAXNB];
  for (int o = threadIdx.x; o < nb; o += blockDim.x) so[o] = (float)occ.at(o);
  __syncthreads();
  double acc = 0.0;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* pq = psi + 4 * q;
#pragma unroll 16
    for (int o = 0; o < nb; ++o) {
      const float4 p = __ldg(reinterpret_cast<const float4*>(pq + (long long)o * stride));
      const float c = so[o];
      t.x = fmaf(c * p.x, p.x, t.x);
      t.y = fmaf(c * p.y, p.y, t.y);
      t.z = fmaf(c * p.z, p.z, t.z);
      t.w = fmaf(c * p.w, p.w, t.w);
    }
    double2* r2 = reinterpret_cast<double2*>(rho + 4 * q);
    double2 a = make_double2((double)t.x, (double)t.y), b = make_double2((double)t.z, (double)t.w);
    if (accumulate) {
      const double2 ra = r2[0], rb = r2[1];
      a.x += ra.x;
      a.y += ra.y;
      b.x += rb.x;
      b.y += rb.y;
    }
    r2[0] = a;
    r2[1] = b;
    if (w) {
      const double2 wa = __ldg(reinterpret_cast<const double2*>(w + 4 * q)),
                    wb = __ldg(reinterpret_cast<const double2*>(w + 4 * q + 2));
      acc += a.x * wa.x + a.y * wa.y + b.x * wb.x + b.y * wb.y;
    }
  }
  if (integral) {
    double v[1] = {acc};
    block_atomic_add<1, XB>(integral, v);
  }
}

// rho *= target / integral (integral read on the device; no host sync).  128^3 points: 11.2 us with a
// division per thread, now 7.2.
template <bool PAIRS>
__global__ void renorm_kernel(long long n, double* __restrict__ rho, const double* integral, double target,
                              int* flags) {
  // one division per block: per thread the divisions took longer than the pass over memory
  __shared__ double factor;
  __shared__ int go;
  if (threadIdx.x == 0) {
    const double s = *integral;
    factor = target / s;
    if (!(s > 0.0) && blockIdx.x == 0) atomicOr(flags, 4);
    go = s > 0.0;
  }
  __syncthreads();
  if (!go) return;
  const double f = factor;
  const long long at = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  if constexpr (PAIRS) {  // n counts pairs
    double2* const r2 = reinterpret_cast<double2*>(rho);
    for (long long i = at; i < n; i += step) {
      const double2 v = r2[i];
      r2[i] = make_double2(v.x * f, v.y * f);
    }
  } else {
    for (long long i = at; i < n; i += step) rho[i] *= f;
  }
}

// sum ((up_o - up_i)^2 + (dn_o - dn_i)^2) W
__global__ void residual2_kernel(long long n, const double* __restrict__ ui, const double* __restrict__ di,
                                 const double* __restrict__ uo, const double* __restrict__ dout,
                                 const double* __restrict__ w, double* out) {
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double a = uo[i] - ui[i], b = dout[i] - di[i];
    acc += (a * a + b * b) * w[i];
  }
  double a[1] = {acc};
  block_atomic_add<1, XB>(out, a);
}

__global__ void zero1(double* p) { *p = 0.0; }

}  // namespace
}  // namespace igd

using namespace igd;

// LSDA on n points.  dtype = I/O type, math = IGD_F64 or IGD_F32 arithmetic,
// functional 0 = Slater + VWN5 ("lda,vwn"), 1 = Slater + PW92.  Any output may be
// NULL.  energy (device double) = sum rho eps W when w and energy are given
// (zeroed first).  flags (device int) |= 1 non-finite input, 2 negative below
// -1e-14 (the caller raises).
extern "C" int igd_lsda(int dtype, int math, int functional, long long n, const void* rho_up, const void* rho_down,
                        void* eps, void* v_up, void* v_down, void* energy_density, const double* w, double* energy,
                        int* flags, void* stream) {
  if (n <= 0 || !rho_up || !rho_down || !flags || functional < 0 || functional > 1) return IGD_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  if (energy) zero1<<<1, 1, 0, st>>>(energy);
  const int g = xblocks(n);
#define IGD_LSDA_LAUNCH(T, M, F)                                                                                   \
  lsda_kernel<T, M, F><<<g, XB, 0, st>>>(n, static_cast<const T*>(rho_up), static_cast<const T*>(rho_down),        \
                                         static_cast<T*>(eps), static_cast<T*>(v_up), static_cast<T*>(v_down),     \
                                         static_cast<T*>(energy_density), w, energy, flags)
  const int g64 = (int)std::min<long long>((n + XB - 1) / XB, (long long)device_sm_count() * 3);
#define IGD_LSDA64_LAUNCH(T, F)                                                                                   \
  lsda64_kernel<T, F><<<g64, XB, 0, st>>>(n, static_cast<const T*>(rho_up), static_cast<const T*>(rho_down),      \
                                          static_cast<T*>(eps), static_cast<T*>(v_up), static_cast<T*>(v_down),   \
                                          static_cast<T*>(energy_density), w, energy, flags)
  if (dtype == IGD_F64 && math == IGD_F64) {
    if (functional == 0) IGD_LSDA64_LAUNCH(double, 0); else IGD_LSDA64_LAUNCH(double, 1);
  } else if (dtype == IGD_F64 && math == IGD_F32) {
    if (functional == 0) IGD_LSDA_LAUNCH(double, float, 0); else IGD_LSDA_LAUNCH(double, float, 1);
  } else if (dtype == IGD_F32 && math == IGD_F32) {
    if (functional == 0) IGD_LSDA_LAUNCH(float, float, 0); else IGD_LSDA_LAUNCH(float, float, 1);
  } else if (dtype == IGD_F32 && math == IGD_F64) {
    if (functional == 0) IGD_LSDA64_LAUNCH(float, 0); else IGD_LSDA64_LAUNCH(float, 1);
  } else {
    return IGD_ERR_DTYPE;
  }
#undef IGD_LSDA_LAUNCH
#undef IGD_LSDA64_LAUNCH
  return launch_status();
}

static int density_launch(int dtype, long long n, int nb, long long stride, const void* psi, const Occupations& occupations,
                          const double* w, double* rho, double* integral, int accumulate, cudaStream_t st) {
  if (integral) zero1<<<1, 1, 0, st>>>(integral);
  auto plain = [&](auto zero) {
    using T = decltype(zero);
    auto kern = nb <= DENS_MAXNB ? density_kernel<T, true> : density_kernel<T, false>;
    kern<<<xblocks(n), XB, 0, st>>>(n, nb, stride, static_cast<const T*>(psi), occupations, w, rho, integral,
                                    accumulate);
  };
  if (dtype == IGD_F64)
    plain(0.0);
  else if (dtype == IGD_F32 && n % 4 == 0 && stride % 4 == 0 && nb <= DENS_MAXNB &&
           ((reinterpret_cast<uintptr_t>(psi) | reinterpret_cast<uintptr_t>(rho) | reinterpret_cast<uintptr_t>(w)) &
            15u) == 0)
    density_v4_kernel<<<xblocks(n / 4), XB, 0, st>>>(n / 4, nb, stride, static_cast<const float*>(psi), occupations,
                                                     w, rho, integral, accumulate);
  else if (dtype == IGD_F32)
    plain(0.f);
  else
    return IGD_ERR_DTYPE;
  return launch_status();
}

// rho (FP64, n) = [rho +] sum_i occupations[i] psi_i^2 over nb orbitals of `dtype`
// separated by stride elements; occupations: nb device doubles.  integral (device,
// may be NULL) = sum rho W (zeroed first).
extern "C" int igd_density(int dtype, long long n, int nb, long long stride, const void* psi, const double* occupations,
                           const double* w, double* rho, double* integral, int accumulate, void* stream) {
  if (n <= 0 || nb < 0 || !rho || (nb > 0 && (!psi || !occupations))) return IGD_ERR_ARG;
  Occupations occ{};
  occ.p = nb ? occupations : nullptr;
  return density_launch(dtype, n, nb, stride, psi, occ, w, rho, integral, accumulate, as_stream(stream));
}

// The same with the occupations (at most IGD_DENSITY_VALUES host doubles) in the launch's arguments.
extern "C" int igd_density_values(int dtype, long long n, int nb, long long stride, const void* psi,
                                  const double* occupations, const double* w, double* rho, double* integral,
                                  int accumulate, void* stream) {
  if (n <= 0 || nb < 0 || nb > DENS_MAXNB || !rho || (nb > 0 && (!psi || !occupations))) return IGD_ERR_ARG;
  Occupations occ{};
  for (int o = 0; o < nb; ++o) occ.v[o] = occupations[o];
  return density_launch(dtype, n, nb, stride, psi, occ, w, rho, integral, accumulate, as_stream(stream));
}

// rho *= target / *integral on the device (flags |= 4 when the integral is not positive).
extern "C" int igd_density_renormalize(long long n, double* rho, const double* integral, double target, int* flags,
                                       void* stream) {
  if (n <= 0 || !rho || !integral || !flags) return IGD_ERR_ARG;
  if (n % 2 == 0 && (reinterpret_cast<uintptr_t>(rho) & 15u) == 0)
    renorm_kernel<true><<<xblocks(n / 2), XB, 0, as_stream(stream)>>>(n / 2, rho, integral, target, flags);
  else
    renorm_kernel<false><<<xblocks(n), XB, 0, as_stream(stream)>>>(n, rho, integral, target, flags);
  return launch_status();
}

// *out = sum ((up_out - up_in)^2 + (dn_out - dn_in)^2) W (square of _density_residual).
extern "C" int igd_density_residual2(long long n, const double* up_in, const double* dn_in, const double* up_out,
                                     const double* dn_out, const double* w, double* out, void* stream) {
  if (n <= 0 || !up_in || !dn_in || !up_out || !dn_out || !w || !out) return IGD_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  zero1<<<1, 1, 0, st>>>(out);
  residual2_kernel<<<xblocks(n), XB, 0, st>>>(n, up_in, dn_in, up_out, dn_out, w, out);
  return launch_status();
}
