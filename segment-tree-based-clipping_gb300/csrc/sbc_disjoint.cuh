// sbc_disjoint.cuh -- a float test that spares most candidate edge pairs the
// FP64 classifier (GB300's FP64 rate is a small fraction of its float rate).
#pragma once

#include "sbc_internal.cuh"

namespace sbc {
namespace {

// A vertex as float pairs: hi = x rounded to float, lo = (x - hi) rounded to
// float, so hi + lo is within 2^-48 |x| of the double, and lo has x - hi's
// sign.  By integer operations (GB300 converts doubles at its FP64 rate)
// except near the ends of float's range.
__device__ __forceinline__ float2 float_parts(double x) {
  const long long u = __double_as_longlong(x);
  const int e = (int)(u >> 52) & 0x7ff;
  const unsigned sign = (unsigned)(u >> 32) & 0x80000000u;
  if (e >= 960 && e < 1150) {
    const long long m = (u & 0xfffffffffffffll) | 0x10000000000000ll;
    const int h = (int)((m + (1ll << 28)) >> 29);  // 24 bits, halves up
    const int rest = (int)(m - ((long long)h << 29));
    const float lo = __fmul_rn(__int2float_rn(rest), __int_as_float((e - 948) << 23));
    return make_float2(__uint_as_float(sign | (unsigned)(((e - 896) << 23) + (h - 0x800000))),
                       __uint_as_float(__float_as_uint(lo) ^ sign));
  }
  const float hi = __double2float_rn(x);
  const double rest = dsub(x, (double)hi);
  float lo = __double2float_rn(rest);
  if (lo == 0.f && rest != 0.0) lo = rest > 0.0 ? 1.4e-45f : -1.4e-45f;
  return make_float2(hi, lo);
}
__device__ __forceinline__ float4 float_pair(double x, double y) {
  const float2 a = float_parts(x), b = float_parts(y);
  return make_float4(a.x, b.x, a.y, b.y);
}

// hi + lo rounded to a float below (above) it
__device__ __forceinline__ float parts_below(float hi, float lo) {
  if (!(lo < 0.f)) return hi;
  const int u = __float_as_int(hi);
  return hi == 0.f ? __int_as_float(0x80000001) : __int_as_float(u > 0 ? u - 1 : u + 1);
}
__device__ __forceinline__ float parts_above(float hi, float lo) { return -parts_below(-hi, -lo); }
// the box of the edge between two vertices: low x and y, high x and y
__device__ __forceinline__ float4 float_box(const float4& a, const float4& b) {
  return make_float4(fminf(parts_below(a.x, a.z), parts_below(b.x, b.z)),
                     fminf(parts_below(a.y, a.w), parts_below(b.y, b.w)),
                     fmaxf(parts_above(a.x, a.z), parts_above(b.x, b.z)),
                     fmaxf(parts_above(a.y, a.w), parts_above(b.y, b.w)));
}

__device__ __forceinline__ float vdx(const float4& a, const float4& b) {
  return __fadd_rn(__fsub_rn(a.x, b.x), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float vdy(const float4& a, const float4& b) {
  return __fadd_rn(__fsub_rn(a.y, b.y), __fsub_rn(a.w, b.w));
}
__device__ __forceinline__ float fcross(float ax, float ay, float bx, float by) {
  return __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
}

// True only when lineSegmentIntersection2 (seg_isect) certainly returns 0
// for P = (p1, p2), Q = (q1, q2), decided in float from vertex hi/lo pairs.
//
// With a = q1 - p1, b = q2 - p1, w = p2 - p1 the four areas seg_isect uses
// are AP1 = a x b, AQ1 = w x a, AQ2 = w x b and AP2 = AP1 + AQ1 - AQ2.
//  * If AP1 and AP2 have the same strict sign, |AP1| > 2e-9 and
//    |AP1| > 2e-9 |AP2|, then alpha = AP1 / (AP1 - AP2) is > 1 or
//    < -EPSILON, and the collinear branch (|AP1| < EPSILON) is excluded:
//    the type is 0.
//  * If AQ1 and AQ2 have the same strict sign, |AQ1| > 2e-9 |AQ2| and
//    |AP1| > 2e-9, then beta is > 1 or < -EPSILON in the general branch and
//    the collinear branch is excluded again: the type is 0.
// Segments that do not meet satisfy one of the two unless they are within
// the float error of touching.  Each float area carries the bound
// 32 u m^2 + 64 u^2 m M (u = 2^-24, m = largest difference component,
// M = coordinate magnitude), at least 2.6 times the worst case of the
// difference and product rounding; the FP64 areas of seg_isect differ from
// the exact ones by about 1e-15 m^2, far inside it.
__device__ __forceinline__ bool certainly_disjoint(const float4& p1, const float4& p2,
                                                   const float4& q1, const float4& q2) {
  const float ax = vdx(q1, p1), ay = vdy(q1, p1);
  const float bx = vdx(q2, p1), by = vdy(q2, p1);
  const float wx = vdx(p2, p1), wy = vdy(p2, p1);
  const float AP1 = fcross(ax, ay, bx, by);
  const float AQ1 = fcross(wx, wy, ax, ay);
  const float AQ2 = fcross(wx, wy, bx, by);
  const float AP2 = __fsub_rn(__fadd_rn(AP1, AQ1), AQ2);
  const float m = fmaxf(fmaxf(fmaxf(fabsf(ax), fabsf(ay)), fmaxf(fabsf(bx), fabsf(by))),
                        fmaxf(fabsf(wx), fabsf(wy)));
  const float M = __fadd_rn(fmaxf(fabsf(p1.x), fabsf(p1.y)), __fmul_rn(2.f, m));
  const float u = 5.9604645e-8f;  // 2^-24
  const float Bx = __fadd_rn(__fmul_rn(__fmul_rn(32.f * u, m), m),
                             __fadd_rn(__fmul_rn(__fmul_rn(64.f * u * u, m), M), 1e-30f));
  const float B2 = __fadd_rn(__fmul_rn(3.f, Bx),
                             __fmul_rn(4.f * u, __fadd_rn(__fadd_rn(fabsf(AP1), fabsf(AQ1)), fabsf(AQ2))));
  const float L1 = __fsub_rn(fabsf(AP1), Bx);
  if (!(L1 > 2e-9f)) return false;  // also keeps the collinear branch out
  const bool sameP = (AP1 > Bx && AP2 > B2) || (AP1 < -Bx && AP2 < -B2);
  if (sameP && L1 > __fmul_rn(2e-9f, __fadd_rn(fabsf(AP2), B2))) return true;
  const bool sameQ = (AQ1 > Bx && AQ2 > Bx) || (AQ1 < -Bx && AQ2 < -Bx);
  const float LQ1 = __fsub_rn(fabsf(AQ1), Bx);
  return sameQ && LQ1 > __fmul_rn(2e-9f, __fadd_rn(fabsf(AQ2), Bx));
}

}  // namespace
}  // namespace sbc
