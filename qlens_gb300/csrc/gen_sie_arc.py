"""Generate sie_arc_table.h: the two functions of a core-free isothermal ellipsoid's
deflection,

    A(s) = atan(sqrt(s)) / sqrt(s),    B(s) = asinh(sqrt(s)) / sqrt(s),

as polynomials on every sixteenth of an octave of s from 2^-20 to 2^12.  Both are
analytic for s > -1, so on an interval [a, 17a/16] their Chebyshev coefficients
fall by at least 33 + sqrt(33^2 - 1) = 66 a degree: degree 8 truncates at about
4e-17 relative.  The coefficients are those of the Chebyshev interpolant in
60-digit arithmetic, in powers of t in [-1/2, 1/2], whose terms fall by 33 a
degree: 6 to 8 are below 1e-9 of the value and are held in FP32 (6e-17 of it).
"""
import mpmath as mp
import numpy as np

mp.mp.dps = 60
E0, E1, PER, DEG, ND = -20, 12, 16, 8, 6


def A(s):
    return mp.atan(mp.sqrt(s)) / mp.sqrt(s)


def B(s):
    return mp.asinh(mp.sqrt(s)) / mp.sqrt(s)


def monomials(f, a, h):
    """Coefficients in t of f(a + h (t + 1/2))."""
    n = DEG + 1
    th = [mp.pi * (2 * i + 1) / (2 * n) for i in range(n)]
    v = [f(a + h * (1 + mp.cos(x)) / 2) for x in th]
    cheb = [mp.mpf(2) / n * sum(v[i] * mp.cos(k * th[i]) for i in range(n)) for k in range(n)]
    cheb[0] /= 2
    T = [[mp.mpf(1)], [mp.mpf(0), mp.mpf(2)]]             # T_k(2 t) in powers of t
    for k in range(2, n):
        p = [mp.mpf(0)] + [4 * c for c in T[-1]]
        for i, c in enumerate(T[-2]):
            p[i] -= c
        T.append(p)
    return [sum(cheb[k] * T[k][i] for k in range(i, n)) for i in range(n)]


def main(out):
    with open(out, "w") as f:
        f.write("// Generated by gen_sie_arc.py; do not edit.\n"
                "// A(s) = atan(sqrt s) / sqrt s, then B(s) = asinh(sqrt s) / sqrt s, in powers of t\n"
                "// in [-1/2, 1/2] on each sixteenth of an octave of s from 2^%d to 2^%d: terms 0-5,\n"
                "// and 6-8 in FP32.\n#pragma once\n\n" % (E0, E1))
        n = (E1 - E0) * PER
        f.write("#define QLP_SIE_E0 (%d)\n#define QLP_SIE_N %d\n" % (E0, n))
        rows = []
        for g in (A, B):
            for e in range(E0, E1):
                for j in range(PER):
                    h = mp.mpf(2) ** e / PER
                    rows.append([float(x) for x in monomials(g, (PER + j) * h, h)])
        f.write("\n#define QLP_SIE_C_INIT { \\\n")
        f.write(" \\\n".join("    " + ", ".join("%.*g" % (18 - k, x) for k, x in enumerate(r[:ND])) + "," for r in rows))
        f.write(" \\\n}\n\n#define QLP_SIE_F_INIT { \\\n")
        lo = [[float(np.float32(x)) for x in r[ND:]] + [0.0] for r in rows]
        f.write(" \\\n".join("    " + ", ".join("%.9gf" % x if "e" in "%.9g" % x or "." in "%.9g" % x else "%.1ff" % x
                                                for x in r) + "," for r in lo))
        f.write(" \\\n}\n")


if __name__ == "__main__":
    import os
    main(os.path.join(os.path.dirname(os.path.abspath(__file__)), "sie_arc_table.h"))
