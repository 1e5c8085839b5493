"""Writes isogriddft_gb300/csrc/lsda_tables.cuh: the correlation energies of the LSDA channels as
piecewise polynomials (needs mpmath; a few seconds).

    python tests/golden/make_lsda_tables.py

Per functional (VWN5: Vosko, Wilk and Nusair, Can. J. Phys. 58, 1200 (1980); PW92: Perdew and Wang,
PRB 45, 13244 (1992)) and channel (paramagnetic, ferromagnetic, spin stiffness) the energy is a
function of x = sqrt(rs).  Each octave of x from 2^-3 to 2^8 is cut into eight equal intervals, and on
each the Chebyshev interpolant of degree 11 (relative error below 4e-17, printed) is expanded in
powers of s in [-1/2, 1/2], the position in the interval.  Constants are the doubles of the kernel's
own formulas, so both describe the same function.
"""

import os

import mpmath as mp

mp.mp.dps = 45
LOW, HIGH, PER, DEG = -3, 8, 8, 11
OUT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "..", "isogriddft_gb300", "csrc",
                   "lsda_tables.cuh")


def vwn(A, b, c, x0):
    A, b, c, x0 = (mp.mpf(v) for v in (A, b, c, x0))
    X0, Q = x0 * x0 + b * x0 + c, mp.sqrt(4 * c - b * b)

    def g(x):
        X, at = x * x + b * x + c, mp.atan(Q / (2 * x + b))
        return A * (mp.log(x * x / X) + 2 * b / Q * at
                    - b * x0 / X0 * (mp.log((x - x0) ** 2 / X) + 2 * (b + 2 * x0) / Q * at))

    return g


def pw(A, a1, b1, b2, b3, b4, sign=1):
    A, a1, b1, b2, b3, b4 = (mp.mpf(v) for v in (A, a1, b1, b2, b3, b4))

    def g(x):
        rs = x * x
        q = 2 * A * (b1 * x + b2 * rs + b3 * rs * x + b4 * rs * rs)
        return -sign * 2 * A * (1 + a1 * rs) * mp.log1p(1 / q)

    return g


def channels():
    import math

    return {
        "VWN": [vwn(0.0310907, 3.72744, 12.9352, -0.10498), vwn(0.01554535, 7.06042, 18.0578, -0.32500),
                vwn(-1.0 / (6.0 * math.pi * math.pi), 1.13107, 13.0045, -0.0047584)],
        "PW": [pw(0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294),
               pw(0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517),
               pw(0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671, sign=-1)],
    }


def powers(f, lo, hi):
    """Coefficients in s (x = mid + (hi - lo) s) of the Chebyshev interpolant of degree DEG."""

    n, mid, half = DEG + 1, (lo + hi) / 2, (hi - lo) / 2
    th = [mp.pi * (k + mp.mpf(1) / 2) / n for k in range(n)]
    fv = [f(mid + half * mp.cos(t)) for t in th]
    c = [(2 if j else 1) * sum(v * mp.cos(j * t) for v, t in zip(fv, th)) / n for j in range(n)]
    a, b = [mp.mpf(1)], [mp.mpf(0), mp.mpf(1)]  # T_0, T_1 in powers of t
    out = [mp.mpf(0)] * n
    for j in range(n):
        for i, v in enumerate(a):
            out[i] += c[j] * v
        nxt = [mp.mpf(0)] + [2 * v for v in b]
        for i, v in enumerate(a):
            nxt[i] -= v
        a, b = b, nxt
    return [v * 2 ** i for i, v in enumerate(out)], abs(c[-1] / c[0])  # t = 2 s


def main():
    lines = [
        "// Piecewise polynomials of the LSDA correlation channels in x = sqrt(rs): eight intervals per",
        "// octave from 2^%d to 2^%d, coefficients of s^0 .. s^%d (s in [-1/2, 1/2] across the interval) for the" % (LOW, HIGH, DEG),
        "// paramagnetic, ferromagnetic and spin-stiffness channel.  Written by tests/golden/make_lsda_tables.py",
        "// from the published forms in 45-digit arithmetic.",
        "#pragma once",
        "",
        "namespace igd {",
        "constexpr int LSDA_LOW = %d, LSDA_PER = %d, LSDA_INTERVALS = %d, LSDA_COEFS = %d;" % (LOW, PER, (HIGH - LOW) * PER, DEG + 1),
        "// [functional][interval][power][channel]",
        "__device__ const double lsda_table[2][LSDA_INTERVALS][LSDA_COEFS][3] = {",
    ]
    for name, fs in channels().items():
        worst = mp.mpf(0)
        lines.append("{ // " + name)
        for e in range(LOW, HIGH):
            for i in range(PER):
                lo, hi = mp.mpf(2) ** e * (1 + mp.mpf(i) / PER), mp.mpf(2) ** e * (1 + mp.mpf(i + 1) / PER)
                cs = []
                for f in fs:
                    p, w = powers(f, lo, hi)
                    cs.append(p)
                    worst = max(worst, w)
                lines.append("{" + ",\n ".join("{%s}" % ",".join(repr(float(p[k])) for p in cs) for k in range(DEG + 1)) + "},")
        lines.append("},")
        print(name, "last Chebyshev coefficient over the first, at most", mp.nstr(worst, 3))
    lines += ["};", "}  // namespace igd", ""]
    with open(OUT, "w") as f:
        f.write("\n".join(lines))


if __name__ == "__main__":
    main()
