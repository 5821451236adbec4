"""Generates o3g_gauss_poly.h: piecewise polynomials for the FP32 Gaussian core.

The library's Gaussian core (no counterpart in the reference) is, with q = d^2 / sigma^2
and rho = sqrt(q),

    r3  = G(q) / sigma^3,   G(q) = [erf(rho / sqrt 2) - sqrt(2/pi) rho exp(-q/2)] / rho^3,
    bbb = D(q) / sigma^5,   D(q) = 2 G'(q),

and G(q) = q^(-3/2) (the singular kernel) to float precision beyond q = 48.  On [0, 48] the
FP32 kernels evaluate G from the polynomials written here instead of erf/exp, and the
gradient's factor -bbb/3 from the same polynomial's derivative: one polynomial of degree DEG
per interval [2 j, 2 j + 2) in

    tau = fma(u, -1.5, 1.5),   u = q - 2 j   (exact),

so that dG/dtau = G'(q) / -1.5 = -D(q) / 3 is the number the kernels need, and one table
of DEG + 1 floats per interval serves both.  24 intervals: a warp's lanes read coefficient k
of their own intervals from 24 consecutive floats, which lie in different shared-memory
banks whatever mix of intervals the lanes hold.  The fit is a least-squares fit of the
relative errors of G and of D together.  G and D are computed here in double: the Taylor
series for q < 1 (30 terms) and the closed form above.  The reported errors are those of
the float32 evaluation (Horner's rule for G and its derivative) at float q.

Run from this directory:  python gauss_poly_gen.py   (rewrites o3g_gauss_poly.h and
o3g_gauss_poly_ds.h and prints the worst relative error of each evaluation).
"""
import os

import numpy as np
from numpy.polynomial import chebyshev as C
from scipy.special import erf

# the accurate mode's intervals: [j, j + 1) for j = 0..47
EDGES = [float(j) for j in range(49)]
# the FP32 table: interval j covers [2 j, 2 j + 2)
N32 = 24
DEG = 7
CONST = np.sqrt(2.0 / np.pi)


def _coef(n):
    v = 1.0 / (2 * n + 1)
    for k in range(1, n):
        v /= 2 * k
    return v if n % 2 == 1 else -v


def gauss_G(q):
    q = np.asarray(q, dtype=np.float64)
    out = np.empty_like(q)
    s = q < 1.0
    g = np.zeros_like(q[s])
    for n in range(30, 0, -1):
        g = g * q[s] + _coef(n)
    out[s] = CONST * g
    ql = q[~s]
    rho = np.sqrt(ql)
    out[~s] = (erf(rho / np.sqrt(2.0)) - CONST * rho * np.exp(-0.5 * ql)) / rho ** 3
    return out


def gauss_D(q):
    q = np.asarray(q, dtype=np.float64)
    out = np.empty_like(q)
    s = q < 1.0
    gp = np.zeros_like(q[s])
    for n in range(30, 1, -1):
        gp = gp * q[s] + (n - 1) * _coef(n)
    out[s] = 2.0 * CONST * gp
    ql = q[~s]
    out[~s] = (CONST * np.exp(-0.5 * ql) - 3.0 * gauss_G(ql)) / ql
    return out


def gauss_D3(q):
    return -gauss_D(q) / 3.0


def _fma32(a, b, c):
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(np.float32)


def eval32(row, lo, q):
    """G and -D/3 as the kernels evaluate them: float32, fused multiply-adds; row is c[DEG]..c[0]."""
    q = np.asarray(q, np.float32)
    u = (q.astype(np.float64) - lo).astype(np.float32)
    t = _fma32(u, np.float32(-1.5), np.float32(1.5))
    c = [np.float32(v) for v in row]
    d = np.full_like(t, c[0])
    g = _fma32(np.full_like(t, c[0]), t, c[1])
    for k in range(2, len(c)):
        d = _fma32(d, t, g)
        g = _fma32(g, t, c[k])
    return g, d


def fit():
    table, worst = [], [0.0, 0.0]
    x = np.cos(np.pi * (np.arange(400) + 0.5) / 400)       # Chebyshev nodes
    for j in range(N32):
        lo = 2.0 * j
        q = lo + 1.0 + x
        t = -1.5 * x
        V = np.vander(t, DEG + 1, increasing=True)
        dV = np.zeros_like(V)
        dV[:, 1:] = V[:, :-1] * np.arange(1, DEG + 1)
        # the unknowns in the Chebyshev basis of x, for conditioning
        M = np.linalg.lstsq(V, C.chebvander(x, DEG), rcond=None)[0]
        G, D3 = gauss_G(q), gauss_D3(q)
        A = np.vstack([V / G[:, None], dV / D3[:, None]])
        c = M @ np.linalg.lstsq(A @ M, np.ones(2 * x.size), rcond=None)[0]
        row = [np.float32(v) for v in c[::-1]]
        qq = np.linspace(lo, lo + 2.0, 40001).astype(np.float32)
        g, d = eval32(row, lo, qq)
        q64 = qq.astype(np.float64)
        worst[0] = max(worst[0], float(np.max(np.abs(g / gauss_G(q64) - 1.0))))
        worst[1] = max(worst[1], float(np.max(np.abs(d / gauss_D3(q64) - 1.0))))
        table.append(row)
    return table, worst


def write(table, worst, path):
    lines = []
    for e in range(DEG + 1):
        vals = ", ".join("%.9ef" % np.float32(row[e]) for row in table)
        lines.append("    // c%d\n    %s," % (DEG - e, vals))
    body = "\n".join(lines)
    txt = f"""// o3g_gauss_poly.h -- GENERATED by gauss_poly_gen.py (do not edit): piecewise polynomials of
// the FP32 Gaussian core on q in [0, 48]: G(q) (r3 = G / sigma^3), degree {DEG} in
// tau = fma(q - 2 j, -1.5, 1.5) on interval j = [2 j, 2 j + 2); dG/dtau = -G'(q) 2/3 is the
// gradient's -bbb/3 = (dG/dtau) / sigma^5.  Evaluated in float32 with fused multiply-adds
// at a float q, G stays within {worst[0]:.2e} and dG/dtau within {worst[1]:.2e} relative of the
// double-precision functions.
#pragma once

namespace o3g {{

constexpr int kGaussPolyDeg = {DEG};
constexpr int kGaussPolyN = {len(table)};        // intervals; interval j covers [2 j, 2 j + 2)
// coefficient c_k of interval j at kGaussPoly[({DEG} - k) * kGaussPolyN + j]
__device__ const __align__(16) float kGaussPoly[{DEG + 1} * {len(table)}] = {{
{body}
}};

}}  // namespace o3g
"""
    with open(path, "w") as f:
        f.write(txt)


# ---- the accurate (double-single) evaluation: o3g_gauss_poly_ds.h ----------------------
# Degree DEG_DS in t = 2 q - (2 j + 1) on interval j.  The kernel runs Horner's rule in float
# for the coefficients of degree >= 3 (together at most 0.14 % of |G| or |D| on every
# interval, so their float rounding stays near 1e-10 relative) and in double-single
# arithmetic for degrees 2, 1, 0, whose coefficients are stored as (hi, lo) float pairs.
DEG_DS = 8
NDS = 3          # low-order coefficients kept as (hi, lo) pairs
STRIDE_DS = 2 * (DEG_DS + 1 - NDS) + 4 * NDS


def _split(v):
    hi = np.float32(v)
    return hi, np.float32(v - np.float64(hi))


def fit_ds():
    table, worst = [], 0.0
    for lo, hi in zip(EDGES[:-1], EDGES[1:]):
        s, o = 2.0 / (hi - lo), -(hi + lo) / (hi - lo)
        q = np.linspace(lo, hi, 40001)
        t = q * s + o
        row = []
        polys = []
        for F in (gauss_G, gauss_D3):
            y = F(q)
            polys.append(C.cheb2poly(C.chebfit(t, y, DEG_DS)))
            # the kernel's evaluation: float tail, then (hi, lo) steps (double stands in for
            # double-single arithmetic, which carries about 44 bits)
            qq = np.linspace(lo - 1e-4 * (hi - lo), hi + 1e-4 * (hi - lo), 4001)
            qq = qq[qq >= 0]
            tt = qq * s + o
            tf = tt.astype(np.float32)
            p = polys[-1]
            acc = np.full_like(tf, np.float32(p[DEG_DS]))
            for k in range(DEG_DS - 1, NDS - 1, -1):
                acc = (acc.astype(np.float64) * tf + np.float64(np.float32(p[k]))).astype(np.float32)
            v = acc.astype(np.float64)
            for k in range(NDS - 1, -1, -1):
                h, l = _split(p[k])
                v = v * tt + (np.float64(h) + np.float64(l))
            yy = F(qq)
            worst = max(worst, float(np.max(np.abs(v - yy) / np.abs(yy))))
        for k in range(DEG_DS, NDS - 1, -1):
            row += [np.float32(polys[0][k]), np.float32(polys[1][k])]
        for k in range(NDS - 1, -1, -1):
            gh, gl = _split(polys[0][k])
            dh, dl = _split(polys[1][k])
            row += [gh, gl, dh, dl]
        assert len(row) == STRIDE_DS
        table.append(row)
    return table, worst


def write_ds(table, worst, path):
    names = ["%s%d" % (f, k) for k in range(DEG_DS, NDS - 1, -1) for f in ("G", "D")] + \
            ["%s%d%s" % (f, k, h) for k in range(NDS - 1, -1, -1) for f in ("G", "D") for h in ("hi", "lo")]
    lines = []
    for k in range(STRIDE_DS):
        vals = ", ".join("%.9ef" % np.float32(row[k]) for row in table)
        lines.append("    // %s\n    %s," % (names[k], vals))
    body = "\n".join(lines)
    txt = f"""// o3g_gauss_poly_ds.h -- GENERATED by gauss_poly_gen.py (do not edit): piecewise polynomials
// of the Gaussian core for the accurate (double-single) precision mode: G(q) and
// D(q) = -(2/3) G'(q), degree {DEG_DS} in t = 2 q - (2 j + 1) on interval j.
// Coefficients of degree >= {NDS} are floats (Horner in float); degrees
// {NDS - 1}..0 are (hi, lo) float pairs (Horner in double-single).  Evaluated that way from an
// exact q the result stays within {worst:.2e} relative of the double-precision functions
// (D, which is rounded to float, needs the pairs of degrees 1 and 0 only).
#pragma once

namespace o3g {{

constexpr int kGaussDsN = {len(table)};        // intervals; interval j covers [j, j + 1)
constexpr int kGaussDsDeg = {DEG_DS};
constexpr int kGaussDsPairs = {NDS};
constexpr int kGaussDsStride = {STRIDE_DS};   // (G[k], D[k]) for k = {DEG_DS}..{NDS}, then (G[k] hi, lo, D[k] hi, lo) for k = {NDS - 1}..0
// entry e of interval j at kGaussPolyDs[e * kGaussDsN + j]
__device__ const __align__(16) float kGaussPolyDs[{STRIDE_DS} * {len(table)}] = {{
{body}
}};

}}  // namespace o3g
"""
    with open(path, "w") as f:
        f.write(txt)


if __name__ == "__main__":
    here = os.path.dirname(os.path.abspath(__file__))
    tab, w = fit()
    out = os.path.join(here, "o3g_gauss_poly.h")
    write(tab, w, out)
    print("wrote %s; worst float32 relative errors %.3e (G) %.3e (derivative)" % (out, w[0], w[1]))
    tab, w = fit_ds()
    out = os.path.join(here, "o3g_gauss_poly_ds.h")
    write_ds(tab, w, out)
    print("wrote %s; worst relative error %.3e" % (out, w))
