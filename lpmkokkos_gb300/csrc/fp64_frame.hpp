// fp64_frame.hpp -- how the FP64 pair kernels (pair_fp64.cu) see a point: its defect from the unit
// sphere and the FP32 digits of its coordinates.  Device code.
#pragma once

#include "engine.hpp"

namespace lpm {

// q below which, or negative, a pair is evaluated in the reference's operations (q = 2 (1 - x.y + eps^2);
// on the sphere the pair's distance is below 2^-6): a source and its own target, points that fall on
// a source, pairs about the cone x.y = 1 of a point outside the sphere.
constexpr double kNearQ = 0x1p-12;
// Sources and targets farther than this from the unit sphere (| 1 - |x|^2 |), or not finite, are
// evaluated in the reference's operations in all their pairs.  q = |y - x|^2 + (1 - |x|^2) + (1 - |y|^2)
// + 2 eps^2 cancels where the points lie outside: |y - x|^2, known to 2^-48 of itself, is then at most q
// and twice this limit, so the error is 2^-52, as that of 1 - x.y in FP64.
constexpr double kMaxDefect = 1.0 / 32.0;

// 1 - |x|^2, exact to a rounding of the result for |x| near 1: the squares and their sum keep their
// rounding errors (fused multiply-add; Knuth's two-sum).
__device__ __forceinline__ double defectOf(double x, double y, double z) {
  const double p0 = __dmul_rn(x, x), p1 = __dmul_rn(y, y), p2 = __dmul_rn(z, z);
  double lo = fma(x, x, -p0) + fma(y, y, -p1) + fma(z, z, -p2);
  const double s1 = __dadd_rn(p0, p1);
  const double z1 = __dsub_rn(s1, p0);
  lo += __dsub_rn(p0, __dsub_rn(s1, z1)) + __dsub_rn(p1, z1);
  const double s2 = __dadd_rn(s1, p2);
  const double z2 = __dsub_rn(s2, s1);
  lo += __dsub_rn(s1, __dsub_rn(s2, z2)) + __dsub_rn(p2, z2);
  return __dsub_rn(1.0, s2) - lo;
}

// A point's defect, NaN where it is not near the sphere, which makes every q with it NaN.
__device__ __forceinline__ double sphereDefect(double x, double y, double z) {
  const double d = defectOf(x, y, z);
  return fabs(d) <= kMaxDefect ? d : __longlong_as_double(0x7ff8000000000000ll);
}

// x = a + b + c: a a multiple of 2^-21, b of 2^-45, |b| <= 2^-22, c the rest rounded to FP32
// (exact for |x| >= 2^-23).  |x| <= 2: differences of digits are exact in FP32.
__device__ __forceinline__ void splitDigits(double x, float& a, float& b, float& c) {
  const double ad = rint(x * 0x1p21) * 0x1p-21;
  const double r = x - ad;
  const double bd = rint(r * 0x1p45) * 0x1p-45;
  a = __double2float_rn(ad);
  b = __double2float_rn(bd);
  c = __double2float_rn(r - bd);
}

// Exponents that sources' weights are stored with, and that of no weight.  FP32 would lose weights above 2^128,
// and digits of those below 2^-70.
constexpr int kMinWeightExp = -1000, kMaxWeightExp = 1022, kNoWeightExp = -4000;
__device__ __forceinline__ double powerOf2(int e) { return __hiloint2double((1023 + e) << 20, 0); }  // |e| <= 1022

// v = h + l: h a multiple of 2^-28 where |v| <= 2^-4, else v rounded to FP32.
__device__ __forceinline__ void splitDefect(double v, float& h, float& l) {
  const double hd = fabs(v) <= 0.0625 ? rint(v * 0x1p28) * 0x1p-28 : (double)__double2float_rn(v);
  h = __double2float_rn(hd);
  l = __double2float_rn(v - hd);
}

}  // namespace lpm
