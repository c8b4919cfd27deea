"""Generate nfw_kappa_table.h: the NFW convergence K(s) = kappa / ks,

    K(s) = 2 (1 - F) / (s - 1),  F = atan(sqrt(s-1)) / sqrt(s-1)  (s > 1),
                                 F = atanh(sqrt(1-s)) / sqrt(1-s) (s < 1),

as polynomials on every sixteenth of an octave of s = (xi / rs)^2 from 2^-20 to
2^18.  K is analytic for s > 0 (s = 1 is removable, 0 the only singularity), so
on an interval [a, 17a/16] its Chebyshev coefficients fall by 33 + sqrt(33^2 - 1)
= 66 a degree: degree 8 truncates at about 4e-17 relative.  The coefficients are
those of the Chebyshev interpolant in 60-digit arithmetic, in powers of t in
[-1/2, 1/2], whose terms fall by 33 a degree: 6 to 8 are below 1e-9 of the value
and are held in FP32 (6e-17 of the value).
"""
import mpmath as mp
import numpy as np

mp.mp.dps = 60
E0, E1, PER, DEG, ND = -20, 18, 16, 8, 6


def K(s):
    s = mp.mpf(s)
    d = s - 1
    if abs(d) < mp.mpf(10) ** -12:
        return mp.mpf(2) / 3 - mp.mpf(2) * d / 5          # never hit by a Chebyshev node
    F = mp.atan(mp.sqrt(d)) / mp.sqrt(d) if d > 0 else mp.atanh(mp.sqrt(-d)) / mp.sqrt(-d)
    return 2 * (1 - F) / d


def monomials(a, h):
    """Coefficients in t of K(a + h (t + 1/2))."""
    n = DEG + 1
    th = [mp.pi * (2 * i + 1) / (2 * n) for i in range(n)]
    f = [K(a + h * (1 + mp.cos(x)) / 2) for x in th]
    cheb = [mp.mpf(2) / n * sum(f[i] * mp.cos(k * th[i]) for i in range(n)) for k in range(n)]
    cheb[0] /= 2
    T = [[mp.mpf(1)], [mp.mpf(0), mp.mpf(2)]]             # T_k(2 t) in powers of t
    for k in range(2, n):
        p = [mp.mpf(0)] + [4 * c for c in T[-1]]
        for i, c in enumerate(T[-2]):
            p[i] -= c
        T.append(p)
    return [sum(cheb[k] * T[k][i] for k in range(i, n)) for i in range(n)]


def main(out):
    hi, lo = [], []
    for e in range(E0, E1):
        for j in range(PER):
            h = mp.mpf(2) ** e / PER
            c = monomials((PER + j) * h, h)
            hi.append([float(x) for x in c[:ND]])
            lo.append([float(np.float32(float(x))) for x in c[ND:]] + [0.0])
    with open(out, "w") as f:
        f.write("// Generated by gen_nfw_kappa.py; do not edit.\n"
                "// K(s) = kappa / ks of the NFW profile in powers of t in [-1/2, 1/2] on each\n"
                "// sixteenth of an octave of s from 2^%d to 2^%d: terms 0-5, and 6-8 in FP32.\n#pragma once\n\n"
                % (E0, E1))
        f.write("#define QLP_NFWK_E0 (%d)\n#define QLP_NFWK_N %d\n\n#define QLP_NFWK_C_INIT { \\\n" % (E0, len(hi)))
        f.write(" \\\n".join("    " + ", ".join("%.*g" % (18 - k, x) for k, x in enumerate(r)) + "," for r in hi))
        f.write(" \\\n}\n\n#define QLP_NFWK_F_INIT { \\\n")
        f.write(" \\\n".join("    " + ", ".join("%.9gf" % x if "e" in "%.9g" % x or "." in "%.9g" % x else "%.1ff" % x
                                                for x in r) + "," for r in lo))
        f.write(" \\\n}\n")


if __name__ == "__main__":
    import os
    main(os.path.join(os.path.dirname(os.path.abspath(__file__)), "nfw_kappa_table.h"))
