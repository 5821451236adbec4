// o3g_ds.cuh -- the accurate precision mode (O3G_PREC_ACCURATE) of the particle pair
// kernels: double-single ("float-float") arithmetic on FP32 instructions.
//
// A value is carried as hi + lo (two floats, |lo| about ulp(hi)/2 or less), about 44
// significant bits.  Per pair the mode forms, in double-single:
//   * the separation d = t - s (exact: a two-sum of the float coordinates);
//   * d^2 and the core parameter sigma^2 = sr^2 + tr^2 from exact products (fma);
//   * the core factor r3 (RM: (d^2 + sigma^2)^(-3/2); Gaussian: G(q) / sigma^3 from the
//     double-single polynomials of o3g_gauss_poly_ds.h; beyond q = 48 and in far tiles the
//     singular d^(-3): powers of the reciprocal square root from the hardware estimate and
//     its residual in double-single);
//   * the cross product d x s (s, the strength, is a float);
// and adds each velocity term r3 (d x s) unrounded into a double-single running sum (a
// two-sum into the partial, the errors into a second float), folded every 16 sources into
// the (hi, lo) accumulators by a two-sum (exact in any order; COMPENSATED's Fast2Sum is
// not when the running sum is smaller than the partial).  The outputs are floats, so what
// remains of the velocity error is their final rounding.  Gradient terms use the double-
// single core rounded to float and the float separation, as in COMPENSATED.  Every operation is an explicitly rounded
// intrinsic (__fadd_rn, __fmul_rn, __fmaf_rn), so the compiler neither contracts nor
// reorders the error-free transformations.
//
// What bounds it is the FMA pipe.  Intermediate values stay unnormalised where the next operation
// takes them so (a low part of up to 2^-20 of the high one), one renormalisation per sum of
// squares and per q.  RM takes 176 operations a pair and 230 cycles per pair and warp scheduler (32,768
// particles of a Gaussian cloud), Gaussian 231; renormalising every result took 1.2 and 1.3 times as long.
//
// Error-free transformations: two-sum (Knuth), fast two-sum (Dekker, |a| >= |b|), and the
// product error fma(a, b, -a b) -- the standard float-float toolkit (Dekker 1971; Hida, Li
// and Bailey 2001).
#pragma once

#include "o3g_common.cuh"
#include "o3g_gauss_poly_ds.h"

namespace o3g {

struct dsf {
  float h, l;
};

__device__ __forceinline__ dsf ds_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}
// |a| >= |b| (or a == 0)
__device__ __forceinline__ dsf ds_fast(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ dsf ds_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}
// the square of d = d.h + d.l (d.l^2, below 2^-48 relative, dropped), unnormalised
__device__ __forceinline__ dsf ds_sq(dsf d) {
  const float p = __fmul_rn(d.h, d.h);
  return {p, __fmaf_rn(__fadd_rn(d.h, d.h), d.l, __fmaf_rn(d.h, d.h, -p))};
}
// x y, unnormalised: the low part of either may be up to 2^-20 of its high one (the product of the
// low parts is dropped)
__device__ __forceinline__ dsf ds_mul(dsf x, dsf y) {
  const float p = __fmul_rn(x.h, y.h);
  return {p, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.h, y.h, -p)))};
}
// Powers of x^(-1/2) from the hardware estimate y and its residual r = 1 - x y^2 (from exact
// products; below 2^-21): x^(-3/2) = y^3 (1 + 3/2 r + 15/8 r^2) and x^(-1) = y^2 (1 + r + r^2),
// unnormalised, the next terms below 2^-62.  Renormalising the root, its square and its cube took
// twice the operations.
struct dsrs {
  dsf r3, r2;
};
__device__ __forceinline__ dsrs ds_rsqrt32(dsf x) {
  const float y = rsq_hw(x.h);
  const dsf y2 = ds_prod(y, y);
  float r = __fmaf_rn(-x.h, y2.h, 1.0f);
  r = __fmaf_rn(-x.h, y2.l, r);
  r = __fmaf_rn(-x.l, y2.h, r);
  dsrs o;
  o.r2 = {y2.h, __fmaf_rn(y2.h, __fmaf_rn(r, r, r), y2.l)};
  const float c = __fmul_rn(y2.h, y);
  const float q = __fmul_rn(r, __fmaf_rn(1.875f, r, 1.5f));
  o.r3 = {c, __fmaf_rn(c, q, __fmaf_rn(y2.l, y, __fmaf_rn(y2.h, y, -c)))};
  return o;
}
// p u - q v (p, q double-single, u, v float), unnormalised: the sum hi + lo is the value
// to about 2^-46 of |p u| + |q v|
__device__ __forceinline__ dsf ds_cross(dsf p, float u, dsf q, float v) {
  dsf a = ds_prod(p.h, u);
  a.l = __fmaf_rn(p.l, u, a.l);
  dsf b = ds_prod(q.h, v);
  b.l = __fmaf_rn(q.l, v, b.l);
  const dsf s = ds_two_sum(a.h, -b.h);
  return {s.h, __fadd_rn(s.l, __fsub_rn(a.l, b.l))};
}
__device__ __forceinline__ float ds_round(dsf x) { return __fadd_rn(x.h, x.l); }
// acc + acc_lo += x * c without rounding the product: its high part goes into acc by a
// two-sum, the rounding errors (of the product and of that sum) into acc_lo
__device__ __forceinline__ void ds_accum(float& acc, float& acc_lo, dsf x, dsf c) {
  const float th = __fmul_rn(x.h, c.h);
  float tl = __fmaf_rn(x.h, c.h, -th);
  tl = __fmaf_rn(x.h, c.l, tl);
  tl = __fmaf_rn(x.l, c.h, tl);
  const dsf sm = ds_two_sum(acc, th);
  acc = sm.h;
  acc_lo = __fadd_rn(acc_lo, __fadd_rn(sm.l, tl));
}

// c + g t, all double-single and unnormalised, the low parts about an ulp of c or t
__device__ __forceinline__ dsf ds_horner(dsf g, dsf t, float ch, float cl) {
  const dsf p = ds_mul(g, t);
  const dsf s = ds_two_sum(ch, p.h);
  return {s.h, __fadd_rn(s.l, __fadd_rn(p.l, cl))};
}
// G(q) (and D(q) = -(2/3) G'(q) when GRAD) of the Gaussian core for q in [0, 48], q double-single:
// Horner's rule in float for the degrees >= kGaussDsPairs, then in double-single (D, which is
// rounded to float, in double-single for the last two steps only)
template <bool GRAD>
__device__ __forceinline__ void gauss_poly_ds(dsf q, dsf& G, dsf& D) {
  constexpr int N = kGaussDsN;
  const float* tb = kGaussPolyDs;
  // interval j covers [j, j + 1), t = 2 q - (2 j + 1); 2 q.h - (2 j + 1) and its error (0 but for j = 0) by a
  // fast two-sum
  const float fj = fminf(floorf(q.h), (float)(N - 1));
  const int j = (int)fj;
  const float o = __fmaf_rn(-2.0f, fj, -1.0f);
  dsf t = ds_fast(o, __fadd_rn(q.h, q.h));
  t.l = __fmaf_rn(2.0f, q.l, t.l);
  constexpr int NF = kGaussDsDeg + 1 - kGaussDsPairs;      // float coefficients per function
  static_assert(kGaussDsPairs == 3, "degrees 2 to 0");
  float g = __ldg(tb + j), d = GRAD ? __ldg(tb + N + j) : 0.f;
#pragma unroll
  for (int k = 1; k < NF; ++k) {
    g = __fmaf_rn(g, t.h, __ldg(tb + 2 * k * N + j));
    if (GRAD) d = __fmaf_rn(d, t.h, __ldg(tb + (2 * k + 1) * N + j));
  }
  dsf gg{g, 0.f}, dd{d, 0.f};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int e = 2 * NF + 4 * k;
    gg = ds_horner(gg, t, __ldg(tb + e * N + j), __ldg(tb + (e + 1) * N + j));
    if (GRAD) {
      if (k == 0) dd.h = __fmaf_rn(d, t.h, __ldg(tb + (e + 2) * N + j));
      else        dd = ds_horner(dd, t, __ldg(tb + (e + 2) * N + j), __ldg(tb + (e + 3) * N + j));
    }
  }
  G = gg;
  D = dd;
}

// Core factor in double-single for CORE_SING, CORE_RM and CORE_GAUSS: r3 (unnormalised) and b3 =
// -bbb/3 (rounded to float, when GRAD), from the separation and the radii sr, tr (tr = 0 for
// singular targets).  The sums of squares are chains of two-sums with one renormalisation.
template <int C, bool GRAD>
__device__ __forceinline__ void core_ds(dsf dx, dsf dy, dsf dz, float sr, float tr, dsf& r3, float& b3) {
  const dsf px = ds_sq(dx), py = ds_sq(dy), pz = ds_sq(dz);
  const dsf s1 = ds_two_sum(px.h, py.h);
  const dsf s2 = ds_two_sum(s1.h, pz.h);
  const float l2 = __fadd_rn(__fadd_rn(__fadd_rn(px.l, py.l), pz.l), __fadd_rn(s1.l, s2.l));
  dsf a = s2, g{0.f, 0.f};
  if (C != CORE_SING) {
    // sigma^2 = sr^2 + tr^2
    const dsf qs = ds_prod(sr, sr), qt = ds_prod(tr, tr);
    g = ds_two_sum(qs.h, qt.h);
    g.l = __fadd_rn(g.l, __fadd_rn(qs.l, qt.l));
  }
  if (C == CORE_RM) {
    // CoreFunc.h:66-71: r2 = d^2 + sr^2 + tr^2, r3 = r2^-1.5, bbb = -3 r3 / r2 (b3 = r3 / r2)
    a = ds_two_sum(s2.h, g.h);
    a = ds_fast(a.h, __fadd_rn(__fadd_rn(a.l, l2), g.l));
  } else {
    a = ds_fast(s2.h, l2);
  }
  // Gaussian: the singular kernel beyond q = 48 (the correction is below 3e-10 there)
  if (C == CORE_GAUSS && !(a.h > 48.0f * g.h)) {
    g = ds_fast(g.h, g.l);
    const dsrs rg = ds_rsqrt32(g);
    dsf q = ds_mul(a, rg.r2), G, D;
    q = ds_fast(q.h, q.l);
    gauss_poly_ds<GRAD>(q, G, D);
    r3 = ds_mul(G, rg.r3);
    if (GRAD) b3 = __fmul_rn(__fmul_rn(ds_round(D), ds_round(rg.r3)), ds_round(rg.r2));
    return;
  }
  const dsrs rs = ds_rsqrt32(a);
  r3 = rs.r3;
  if (GRAD) b3 = __fmul_rn(ds_round(rs.r3), ds_round(rs.r2));
}

}  // namespace o3g
