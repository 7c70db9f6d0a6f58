// Fixed-point slicing of the mixed path's kinetic contractions, shared by the
// tensor-core kernels (bsl_kinetic_tc.cu) and the small-grid kernel
// (bsl_small.cu): both must cut the same slices.
#pragma once

#include "bsl_device.cuh"

namespace bsl {
namespace {

constexpr int kVS = 4;  // slices of v
constexpr int kTS = 4;  // slices of T

// exponent e with max|x| 2^-e in [0.5, 1]; 0 for an all-zero plane
__device__ __forceinline__ int plane_exponent(float maxabs) {
  if (!(maxabs > 0.f)) return 0;
  return max(-100, ilogbf(maxabs) + 1);
}

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((min(max(e, -126), 127) + 127) << 23); }

// Four 9-bit slices of a double-float value already scaled to |y| < 256 (hi and
// lo multiplied by the same power of two): y = a1 + 2^-9 a2 + 2^-18 a3 +
// 2^-27 a4 + O(2^-28), each a an integer in [-256, 256].  Every step is exact
// except the last rounding.
__device__ __forceinline__ void slice4(float yh, float yl, float (&a)[kVS]) {
  a[0] = rintf(yh);
  float r = __fmul_rn(__fadd_rn(__fsub_rn(yh, a[0]), yl), 512.f);
  a[1] = rintf(r);
  r = __fmul_rn(__fsub_rn(r, a[1]), 512.f);
  a[2] = rintf(r);
  r = __fmul_rn(__fsub_rn(r, a[2]), 512.f);
  a[3] = rintf(r);
}

// The class sums c0 .. c3 as a double-float pair times `scale` (a power of
// two).  The classes are exact integers below 2^24: the head is c0 + 2^-9 c1
// with its rounding error, the tail collects that error and the two smaller
// classes (its own rounding is ~2^-33 of the head); the pair is left
// unnormalised (|lo| may slightly exceed half an ulp of hi), which the
// double-float additions accept.
__device__ __forceinline__ float2 combine_classes(float c0, float c1, float c2, float c3, float scale) {
  float h, e;
  two_sum(c0, __fmul_rn(c1, 0x1p-9f), h, e);
  const float l = __fmaf_rn(c3, 0x1p-27f, __fmaf_rn(c2, 0x1p-18f, e));
  return make_float2(__fmul_rn(h, scale), __fmul_rn(l, scale));
}

}  // namespace
}  // namespace bsl
