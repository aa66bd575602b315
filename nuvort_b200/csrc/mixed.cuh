// mixed.cuh -- shared pieces of the mixed-precision non-local sum.
//
// Far field in FP32 with the cancellation-free form of the segment formula.  For a
// segment from A to B = A + d seen from x, with r = A - x and e = r + d = B - x, the
// reference's term (timestep.f90:162-169)
//   Gamma/(2 pi) (r x d)/(4ac - b^2) ((2c+b)/sqrt(a+b+c) - b/sqrt(a))
// (a = |r|^2, b = 2 r.d, c = |d|^2) equals
//   Gamma/(4 pi) (r x d) (|r| + |e|) / (|r| |e| (|r| |e| + r.e)),
// which subtracts nothing when the target is far from the segment (r.e ~ +|r||e|), so FP32
// keeps ~1e-7 relative accuracy where the original form loses digits to 4ac - b^2 and to
// the bracket.  The near field (leaves or segments closer than near_radius) and the terms
// FP32 would evaluate badly run in FP64: the reference's own arithmetic decides whether a term
// is skipped (4ac - b^2 against its threshold), and its value comes from the same
// cancellation-free form in FP64 (term64_stable), equal to the reference's to ~1e-15.
#pragma once

#include "common.cuh"

// The denominator |r||e| + r.e cancels when the segment subtends nearly 180 degrees at the
// target (r.e ~ -|r||e|).  Since (|r||e| + r.e)(|r||e| - r.e) = |r x e|^2 = |r x d|^2, it is
// taken as |r x d|^2 / (|r||e| - r.e) when r.e < 0, which subtracts nothing either.
//
// Conditioning guards of the FP32 segment term: a far term is evaluated in FP64 when
//   |r||e| + r.e < angle |r||e|         (the segment subtends more than ~154 degrees at the
//                                        target for angle 0.1: the target is close to a long
//                                        segment, where r x circ keeps only ~1e-6 of its
//                                        digits in FP32 and the term is large),
//   |r x circ|^2 < line |circ|^2 min(|r|^2, |e|^2)   (the target lies near the segment's line),
//   |e|^2 < end max(|r|^2, |circ|^2)    (the target lies near the far end: e = r + circ loses
//                                        digits).
struct Fp32Guards {
  float angle = 0.1f, line = 1e-3f, end = 1e-2f;
};

// FP64 reciprocal and reciprocal square root by Newton's iteration (y <- y + y(1 - x y) and
// y <- y + y(1 - x y^2)/2), each started from the FP32 hardware approximation (relative error
// ~1e-7) and iterated twice: the error squares at every step, so two steps reach the FP64
// rounding level.  Arguments outside the FP32 exponent range take the IEEE operation.
__device__ __forceinline__ double rcp64(double x) {
  const double ax = fabs(x);
  if (!(ax > 1e-30 && ax < 1e30)) return 1.0 / x;
  double y = (double)__fdividef(1.f, (float)x);
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}
__device__ __forceinline__ double rsqrt64(double x) {
  if (!(x > 1e-30 && x < 1e30)) return 1.0 / sqrt(x);
  double y = (double)rsqrtf((float)x);
  double e = fma(-x * y, y, 1.0);
  y = fma(0.5 * y, e, y);
  e = fma(-x * y, y, 1.0);
  return fma(0.5 * y, e, y);
}

// One segment term in FP64 from the cancellation-free form above:
//   gq (r x d)(1/|r| + 1/|e|) / (|r||e| + r.e),  e = r + d, gq = Gamma/(4 pi),
// given rr = |r|^2.  Agrees with the reference's expression (timestep.f90:162-169) to a few
// FP64 roundings; the caller takes the reference's decision whether to skip the term.
__device__ __forceinline__ void term64_stable(const double r[3], const double d[3], double rr, double gq,
                                              double out[3]) {
  const double e[3] = {r[0] + d[0], r[1] + d[1], r[2] + d[2]};
  const double ee = e[0] * e[0] + e[1] * e[1] + e[2] * e[2];
  const double re = r[0] * e[0] + r[1] * e[1] + r[2] * e[2];
  const double cr[3] = {r[1] * d[2] - r[2] * d[1], r[2] * d[0] - r[0] * d[2], r[0] * d[1] - r[1] * d[0]};
  const double ia = rsqrt64(rr), ib = rsqrt64(ee);
  const double pp = (rr * ia) * (ee * ib);
  double f;
  if (re >= 0.0) {
    f = gq * (ia + ib) * rcp64(pp + re);
  } else {
    const double cr2 = cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2];
    f = gq * (ia + ib) * (pp - re) * rcp64(cr2);
  }
  out[0] = f * cr[0];
  out[1] = f * cr[1];
  out[2] = f * cr[2];
}

// ---- two FP32 values in one 64-bit register (packed FADD, FMUL, FFMA of sm_100) --------------
// The packed instructions do two operations at the FP32 pipe's rate for one issue slot; each
// half is rounded as the scalar operation rounds it.
struct f32x2 {
  unsigned long long v;
};
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float lo2(f32x2 x) {
  return __uint_as_float((unsigned)x.v);
}
__device__ __forceinline__ float hi2(f32x2 x) {
  return __uint_as_float((unsigned)(x.v >> 32));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// Hardware 1/sqrt and 1/x without the scaling that denormal operands would need: the callers'
// operands are squared distances and their products, far inside the normal range, or belong
// to a term whose FP32 value is not used.
__device__ __forceinline__ float rsqrt_fast(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_fast(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The FP32 segment records of the direct sum, two segments side by side: 24 floats a pair,
// {xh yh}{zh xl}{yl zl}{dx dy}{dz far}{-dx -dy}, each name the pair's two values; far is the
// squared distance beyond which a target takes the segment's term without any guard
// (far_ratio |d|^2, and at least the near radius).  System slot k (from 1) is half (k-1) & 1
// of the pair at seg32_at(base, k).
__host__ __device__ __forceinline__ long long seg32_at(long long base, int k) {
  return 12 * (base + 1) + 24 * (long long)((k - 1) >> 1);
}

// Terms beyond far_ratio |d|^2 are taken without the angle and end guards: there, beyond 4|d|,
// the segment subtends less than 30 degrees, r.e > 0 and |e| > 3/4 |r|, so that neither acts.
// (The line guard does: r x d cancels for a target near the line however far it is.)  Guards
// that a caller widened past these bounds apply to every term.
inline float far_ratio(const Fp32Guards &g) { return g.angle <= 1.9f && g.end <= 0.5f ? 16.f : 3e38f; }

// What a lane holds of its target for the packed terms, and a pair of segments (or accepted
// tree nodes) as a 24-float record q (see seg32_at): r from the target, its square, the term's
// parts.
struct LaneTarget {
  f32x2 h[3], l[3];  // minus the target (direct sum: image shift - target), FP32 high and low
};
struct PairVec {
  f32x2 rx, ry, rz, a;
};
__device__ __forceinline__ PairVec pair_vec(const ulonglong2 *q, const LaneTarget &t) {
  const ulonglong2 v0 = q[0], v1 = q[1], v2 = q[2];
  PairVec r;
  r.rx = add2(add2({v0.x}, t.h[0]), add2({v1.y}, t.l[0]));
  r.ry = add2(add2({v0.y}, t.h[1]), add2({v2.x}, t.l[1]));
  r.rz = add2(add2({v1.x}, t.h[2]), add2({v2.y}, t.l[2]));
  r.a = fma2(r.rx, r.rx, fma2(r.ry, r.ry, mul2(r.rz, r.rz)));
  return r;
}
struct PairSeg {
  f32x2 dx, dy, dz, ndx, ndy, far;  // d, -dx, -dy, the far bound (direct sum)
};
__device__ __forceinline__ PairSeg pair_seg(const ulonglong2 *q) {
  const ulonglong2 v3 = q[3], v4 = q[4], v5 = q[5];
  return {{v3.x}, {v3.y}, {v4.x}, {v5.x}, {v5.y}, {v4.y}};
}
struct PairGeo {
  f32x2 cx, cy, cz;      // r x d
  f32x2 ee, re, pp, num; // |e|^2, r.e, |r||e|, 1/|r| + 1/|e| with e = r + d
};
__device__ __forceinline__ PairGeo pair_geo(const PairVec &r, const PairSeg &d) {
  const f32x2 kMinus = pack2(-1.f, -1.f);
  PairGeo g;
  const f32x2 ex = add2(r.rx, d.dx), ey = add2(r.ry, d.dy), ez = add2(r.rz, d.dz);
  g.ee = fma2(ex, ex, fma2(ey, ey, mul2(ez, ez)));
  g.re = fma2(r.rx, ex, fma2(r.ry, ey, mul2(r.rz, ez)));
  g.cx = fma2(r.ry, d.dz, mul2(r.rz, d.ndy));
  g.cy = fma2(r.rz, d.dx, mul2(mul2(r.rx, kMinus), d.dz));
  g.cz = fma2(r.rx, d.dy, mul2(r.ry, d.ndx));
  const f32x2 ia = pack2(rsqrt_fast(lo2(r.a)), rsqrt_fast(hi2(r.a)));
  const f32x2 ib = pack2(rsqrt_fast(lo2(g.ee)), rsqrt_fast(hi2(g.ee)));
  g.pp = mul2(mul2(r.a, ia), mul2(g.ee, ib));
  g.num = add2(ia, ib);
  return g;
}
__device__ __forceinline__ f32x2 square2(f32x2 x, f32x2 y, f32x2 z) {
  return fma2(x, x, fma2(y, y, mul2(z, z)));
}

// One node as the mixed walk reads it: 64 bytes, four 16-byte loads.
struct __align__(16) WalkNode {
  float4 a;  // centre (FP32 high part), accept threshold t1^2 rounded to FP32
  float4 b;  // centre (FP32 low part: centre - high part), |circ|^2 in FP32
  float4 c;  // circulation in FP32, unused
  int4 d;    // pcount, first child, number of children, first member's infront (a leaf's: prv of it)
};

struct MixedNodes {  // per tree node, built after the FP64 node sums
  double4 *C = nullptr;  // cent.xyz, accept threshold t1^2 (dist^2 > t1^2 opens nothing)
  double2 *G = nullptr;  // geo^2, t0^2 for the dist <= geo branch (theta0 > 2/sqrt(3) only)
  WalkNode *W = nullptr;
};

// Kahan-compensated FP32 accumulation of one tile's partial sum into (s, comp).
__device__ __forceinline__ void kahan_add(float &s, float &comp, float v) {
  const float y = v - comp;
  const float t = s + y;
  comp = (t - s) - y;
  s = t;
}
