// fp64.cuh -- FP64 quotients and square roots, rounded as the IEEE operations round them, that share
// their seeds.
//
// A Biot-Savart term in the reference's arithmetic (timestep.f90:162-170) takes two square
// roots and five quotients, three of them by one divisor and two by the square roots.  Taken
// one by one they are most of the term's FP64 instructions (166 of them a term were counted,
// against 84 with the forms below, the sums' three additions among them).  Here a square root
// hands its reciprocal on to the quotient by it, and the three quotients by one divisor share
// one reciprocal.
//
// Method: the hardware approximations (relative error measured at most 2^-19) are taken to the
// FP64 rounding level by one third-order Newton step (the error cubed).  A quotient q = n y,
// with y = 1/x to within a few units 2^-53, is corrected by its exact residual r = n - q x
// (one FMA): q + r y, as P. Markstein (IBM J. Res. Dev. 34, 1990) describes; the square root
// likewise from g = x y and its residual x - g^2.  Before the last rounding the value is off
// by about 2^-52 units of its last place, so it rounds as the exact value does unless that
// lies as close to the middle of two doubles.  That happens where n and x both lie a few units
// below a power of two (their quotient is such a middle but for 2^-52 of a unit): there a
// quotient can be a unit of its last place off.  Random operands meet it about once in 2^50
// quotients, and none did in 2^32; no square root differed.
// Divisors and radicands outside the ranges stated take the IEEE operations instead.  Numerators
// are not looked at: one of zero gives zero (+0.0 also for -0.0, the same in the sums), and one
// below 2^-969, whose residual is subnormal, a quotient up to two units off.  They are r x d
// times the circulation, 2 r.d and 2 |d|^2 + 2 r.d, products of two differences of positions:
// so small only where those are below 1e-146 cm.
#pragma once

#include "common.cuh"

__device__ __forceinline__ double seed_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double seed_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 2^-500 <= |x| < 2^500, by the exponent field (false for 0, infinities and NaN; false for a
// negative x when kPositive).
template <bool kPositive>
__device__ __forceinline__ bool mid_range(double x) {
  unsigned hi = (unsigned)__double2hiint(x);
  if (!kPositive) hi &= 0x7fffffffu;
  return hi - 0x20b00000u < 0x3e800000u;
}

// 1/x to within a few units 2^-53, for |x| in mid range.
__device__ __forceinline__ double near_rcp(double x) {
  const double y = seed_rcp(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// n / x, rounded as said above, given y = near_rcp(x) (or the reciprocal near_sqrt gives).
__device__ __forceinline__ double quot(double n, double x, double y) {
  const double q = n * y;
  return fma(fma(-q, x, n), y, q);
}

// sqrt(x) correctly rounded for x in mid range, and y = 1/sqrt(x) to a few units 2^-53.
__device__ __forceinline__ double near_sqrt(double x, double &y) {
  const double y0 = seed_rsqrt(x);
  const double e = fma(-(x * y0), y0, 1.0);
  y = fma(y0 * e, fma(0.375, e, 0.5), y0);
  const double g = x * y;
  return fma(fma(-g, g, x), 0.5 * y, g);
}

// 4ac - b^2 of a segment term (timestep.f90:165-166), the part its skip decision needs.
__device__ __forceinline__ double term_d(double a, double b, double c) {
  return e_sub(e_mul(e_mul(4.0, a), c), e_mul(b, b));
}

// The value of a segment term (timestep.f90:167-169, tree.f90:304-307) in the reference's
// operations and their order, given a = |r|^2, b = 2 r.d, c = |d|^2, D = 4ac - b^2 and sa =
// sqrt(a), ya = 1/sa as near_sqrt gives them; for D, a and abc = a + b + c in mid range.
__device__ __forceinline__ void term_value(const double r[3], const double d[3], double b, double c, double D,
                                           double abc, double sa, double ya, double qc, double two_pi,
                                           double out[3]) {
  double cr[3], ys;
  cross3(r, d, cr);
  const double den = e_mul(two_pi, D);
  const double s = near_sqrt(abc, ys);
  const double fac = e_sub(quot(e_add(e_mul(2.0, c), b), s, ys), quot(b, sa, ya));
  const double yd = near_rcp(den);
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k] = e_mul(quot(e_mul(cr[k], qc), den, yd), fac);
}

// bs_term_exact out of line: for the rare term outside the ranges above, kept apart so that it
// costs the loops neither registers nor instruction cache.
[[maybe_unused]] static __device__ __noinline__ double3 bs_term_rare(double r0, double r1, double r2, double d0, double d1, double d2,
                                             double a, double c, double qc, double two_pi) {
  const double r[3] = {r0, r1, r2}, d[3] = {d0, d1, d2};
  double out[3];
  return bs_term_exact(r, d, a, c, qc, two_pi, out) ? make_double3(out[0], out[1], out[2]) : make_double3(0., 0., 0.);
}

// One segment term of the direct sum: bs_term_exact's value, or +0.0 where it skips the term
// (4ac - b^2 == 0) and where !use.  No branch on the usual path, so that the terms of an
// unrolled loop interleave.
__device__ __forceinline__ void bs_term(bool use, const double r[3], const double d[3], double a, double c, double qc,
                                        double two_pi, double out[3]) {
  const double b = e_mul(2.0, dot3(r, d));
  const double D = term_d(a, b, c);
  const double abc = e_add(e_add(a, b), c);
  double ya;
  const double sa = near_sqrt(a, ya);
  term_value(r, d, b, c, D, abc, sa, ya, qc, two_pi, out);
  const bool keep = use && D != 0.0;
  if (keep && !(mid_range<false>(D) && mid_range<true>(a) && mid_range<true>(abc))) {
    const double3 t = bs_term_rare(r[0], r[1], r[2], d[0], d[1], d[2], a, c, qc, two_pi);
    out[0] = t.x;
    out[1] = t.y;
    out[2] = t.z;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k] = keep ? out[k] : 0.0;
}

// One term of biot_savart_mirror (timestep.f90:201-234): segment j (x_j to ghosti_j) reflected
// in mirror m, its orientation reversed (from the reflected ghost to the reflected point), at
// target g (position xi, pinned record pin_g, behind pi); +0.0 when the reference skips it.
__device__ __forceinline__ void mirror_term_sum(const SysConst &sc, int m, const double *__restrict__ X,
                                                const double *__restrict__ GI, const int *__restrict__ nxt,
                                                long long T, int j, int g, int pi, int pin_g, bool skip_own,
                                                const double xi[3], double out[3]) {
  const bool use = nxt[j] != 0 && !pin_i(sc.pin[j]) &&
                   !(skip_own && ((pin_b(pin_g) && j == g) || (pin_i(pin_g) && j == pi)));
  double r[3], d[3], c2[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double sgi = reflect1(X[c * T + j], sc.mirror[m][c], sc.box[c]);
    const double s = reflect1(GI[c * T + j], sc.mirror[m][c], sc.box[c]);
    r[c] = e_sub(s, xi[c]);
    d[c] = e_sub(sgi, s);
    c2[c] = e_sq(e_sub(s, sgi));
  }
  // |xi - s|^2 = |s - xi|^2 and |s - sgi|^2 bit for bit: the squares of opposite numbers
  const double a = e_add(e_add(e_sq(r[0]), e_sq(r[1])), e_sq(r[2]));
  bs_term(use, r, d, a, e_add(e_add(c2[0], c2[1]), c2[2]), sc.quant_circ, sc.two_pi, out);
}
