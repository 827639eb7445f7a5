// tri_test.cuh -- what the FP64 point-in-triangle tests of the rasteriser
// (rasterizer.cu) and the lift (lift.cu) share: a float pre-test that keeps
// clear misses off the FP64 pipe, a division by a denominator whose reciprocal
// is known, and the sign of a quotient without the division.  GB300 issues an
// FP64 warp instruction every 16 cycles, whatever its active lanes, so both
// kernels first look for a candidate in floats and then test it with all lanes
// together.
#pragma once

#include <cuda_runtime.h>

namespace cvtgb {

// Squared edge lengths up to which a weight's products stay finite (below 2^1000), so
// that no numerator is NaN: what quot_negative and below_zero need, and what lets a box
// bound where a test passes.  Longer triangles take the plain test everywhere.
constexpr double kMaxLen2 = 0x1p499;

__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// RN(num / den), y = RN(1 / den): Markstein's theorem (IBM J. Res. Dev. 34, 1990):
// with y correctly rounded and q within an ulp of the quotient, q + (num - den q) y
// in two fused steps is the correctly rounded quotient.  The first step makes q
// from num y (within 1.5 ulp) faithful, the second rounds it.  Exponents within 400
// of 1 keep every remainder exact and normal; other operands (zeros among them)
// take the division.  Five FP64 instructions.
__device__ __forceinline__ double div_by(double num, double den, double y) {
  const unsigned en = (unsigned)(exp_field(num) - 623), ed = (unsigned)(exp_field(den) - 623);
  if (en > 800u || ed > 800u) return __ddiv_rn(num, den);
  double q = __dmul_rn(num, y);
  q = __fma_rn(__fma_rn(-den, q, num), y, q);
  return __fma_rn(__fma_rn(-den, q, num), y, q);
}

// RN(num / den) < 0 for den > 0, decided from the exponents: num negative and the
// quotient too large to round to -0 (false: divide to know).
__device__ __forceinline__ bool quot_negative(double num, double den) {
  const int en = exp_field(num);
  return __double2hiint(num) < 0 && en > 0 && en + 1000 > exp_field(den);
}

// x < 0 (x not NaN) on the integer pipe
__device__ __forceinline__ bool below_zero(double x) {
  return __double_as_longlong(x) < 0 && (__double_as_longlong(x) << 1) != 0;
}

// A float pre-test that rejects a point clearly outside a triangle before the
// FP64 test, for triangles with conditioning kappa = d00 d11 / denom <= 2^20 (sgn =
// 0: no pre-test).  In scaled units (pixels, grid cells), r = q - P1, edge
// functions E0 = v0 x r, E1 = (v1 - v0) x (r - v0), E2 = (-v1) x (r - v1), all >= 0
// inside a counter-clockwise triangle (sgn folds the orientation).  With M at
// least the largest coordinate magnitude (so |r| <= 1.5 M) and L the longest edge,
// the float error of each E_k is below L (2^-21 M + 2^-19 L) (rounded coordinates and
// edge vectors, three roundings in the products); so sgn E_k < -t with t = L (2^-20 M
// + 2^-16 L) means E_k < -2^-17 L^2 exactly: the point lies more than 2^-17 L outside the
// triangle.  The FP64 test passes only within D < 2^-48 kappa (D + L), 2^-28 (D + L) at
// most, so the reference's test fails too.  Where the two axes' scales differ by up
// to 4, distances and lengths change by at most 4 against each other: still far
// beyond the FP64 error.
struct TriPre {
  float p1x, p1y, v0x, v0y, v1x, v1y, t, sgn;
};

__device__ __forceinline__ bool pre_outside(const TriPre &q, float px, float py) {
  const float rx = px - q.p1x, ry = py - q.p1y;
  const float e0 = q.v0x * ry - q.v0y * rx;
  const float e1 = (q.v1x - q.v0x) * (ry - q.v0y) - (q.v1y - q.v0y) * (rx - q.v0x);
  const float e2 = q.v1y * (rx - q.v1x) - q.v1x * (ry - q.v1y);
  return fminf(q.sgn * e0, fminf(q.sgn * e1, q.sgn * e2)) < -q.t;
}

// (x1, y1): P1 relative to the grid's origin; n: the largest coordinate of a
// query in scaled units.
__device__ __forceinline__ TriPre make_pre(double x1, double y1, double v0x, double v0y, double v1x,
                                           double v1y, double sx, double sy, float n, double cond) {
  TriPre q{0, 0, 0, 0, 0, 0, 0, 0};
  if (!(cond <= 1048576.0)) return q;
  const double cr = v0x * v1y - v0y * v1x;
  if (!(cr != 0.0) || !isfinite(cr)) return q;
  const float p1x = (float)(x1 * sx), p1y = (float)(y1 * sy);
  const float ax = (float)(v0x * sx), ay = (float)(v0y * sy);
  const float bx = (float)(v1x * sx), by = (float)(v1y * sy);
  // (a few roundings: covered by the factor on the threshold)
  const float l0 = sqrtf(ax * ax + ay * ay), l2 = sqrtf(bx * bx + by * by);
  const float l1 = sqrtf((bx - ax) * (bx - ax) + (by - ay) * (by - ay));
  const float L = fmaxf(l0, fmaxf(l1, l2));
  const float M = fmaxf(n, fmaxf(fabsf(p1x), fabsf(p1y)) + 4.f * L);
  if (!(L >= 1e-9f && M <= 1e9f)) return q;  // keep the floats away from over/underflow
  q.p1x = p1x, q.p1y = p1y;
  q.v0x = ax, q.v0y = ay, q.v1x = bx, q.v1y = by;
  q.t = L * (0x1p-20f * M + 0x1p-16f * L) * 1.0625f;
  q.sgn = cr > 0 ? 1.f : -1.f;
  return q;
}

}  // namespace cvtgb
