// Double-single (float-float) arithmetic for the FP32-pipe kernels that must
// deliver FP64-level accuracy.
//
// A value is the unevaluated sum h + l of two floats (~48-bit significand).
// Error-free transformations: Knuth's TwoSum, Dekker's FastTwoSum and the
// FMA-based TwoProd; the double-word algorithms follow the analysis of
// Joldes, Muller and Popescu (ACM TOMS 44(4), 2017).  Files using these
// functions are compiled with --fmad=false (every intended FMA is an
// explicit fmaf, no product is fused into a later addition) and -ftz=true.
#pragma once

#include <cuda_runtime.h>

namespace ommp {
namespace gpu {

struct dsf {
  float h, l;
};

// s + e = a + b exactly (Knuth)
__device__ __forceinline__ dsf two_sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  float e = (a - (s - bb)) + (b - bb);
  return {s, e};
}
// s + e = a + b exactly when |a| >= |b| or a = 0 (Dekker)
__device__ __forceinline__ dsf fast_two_sum(float a, float b) {
  float s = a + b;
  float e = b - (s - a);
  return {s, e};
}
// t - s of two coordinates split on a common grid (launch_split): the two
// leading differences are exact and |th - sh| is 0 or at least |tm - sm|, so
// the fast sum is exact too
__device__ __forceinline__ dsf ds_delta(float th, float tm, float tl, float sh, float sm, float sl) {
  const float dh = th - sh, dm = tm - sm;
  const float h = dh + dm;
  return {h, (dm - (h - dh)) + (tl - sl)};
}
// 1/sqrt(a): FP32 estimate refined by one FP32 Newton step to y, then
// y (1 + e / 2 + 3 e^2 / 8), e = 1 - a y^2 formed in double-single
__device__ __forceinline__ dsf ds_rsqrt(dsf a) {
  const float y0 = rsqrtf(a.h);
  const float y = fmaf(0.5f * y0, fmaf(-(a.h * y0), y0, 1.f), y0);
  const float p = y * y;
  const float th = a.h * p;
  const float tl = fmaf(a.l, p, fmaf(a.h, fmaf(y, y, -p), fmaf(a.h, p, -th)));
  const float e = (1.0f - th) - tl;  // 1 - th is exact: th is within 2^-21 of 1
  return fast_two_sum(y, (y * e) * fmaf(0.375f, e, 0.5f));
}
__device__ __forceinline__ dsf to_ds(double v) {
  float h = (float)v;
  return {h, (float)(v - (double)h)};
}

__device__ __forceinline__ dsf ds_add(dsf x, dsf y) {
  const dsf s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, s.l + (x.l + y.l));
}

// operators for generic formulas: products and sums keep their low part as it
// comes (a few ulp of the high part, so that the neglected product of two low
// parts stays near 2^-45), accumulation renormalises
__device__ __forceinline__ dsf operator*(dsf x, dsf y) {
  const float p = x.h * y.h;
  return {p, fmaf(x.l, y.h, fmaf(x.h, y.l, fmaf(x.h, y.h, -p)))};
}
__device__ __forceinline__ dsf operator*(dsf x, float y) {
  const float p = x.h * y;
  return {p, fmaf(x.l, y, fmaf(x.h, y, -p))};
}
__device__ __forceinline__ dsf operator*(float y, dsf x) { return x * y; }
__device__ __forceinline__ dsf operator-(dsf x) { return {-x.h, -x.l}; }
__device__ __forceinline__ dsf operator+(dsf x, dsf y) {
  const dsf s = two_sum(x.h, y.h);
  return {s.h, s.l + (x.l + y.l)};
}
__device__ __forceinline__ dsf operator-(dsf x, dsf y) { return x + (-y); }
__device__ __forceinline__ dsf &operator+=(dsf &x, dsf y) { return x = ds_add(x, y); }
__device__ __forceinline__ dsf &operator-=(dsf &x, dsf y) { return x = ds_add(x, -y); }

}  // namespace gpu
}  // namespace ommp
