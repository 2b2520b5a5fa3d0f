// Pair arithmetic in double-single for the kernels of FP64 accuracy on the FP32
// pipes (tmu_sym.cu, fmm_near.cu, m2d.cu, grad_sym.cu).
//
// Tensors of a pair are written with the unit-length vector n = d y, y the FP32
// reciprocal distance; for the dipole field
//   E = 3 r^-5 (mu.d) d - r^-3 mu = K (mu.n) n - k3 mu.
// Coordinates come split on a grid into three floats (launch_split), so
// differences are exact; |n|^2 is within 2^-22 of 1 and its deviation eps is
// collected exactly by adding the squares to 2; the damped inverse powers
// follow from powers of y by first- and second-order factors in eps:
// r^-m = y^m (1 - eps)^(-m/2).
// Files using these functions are compiled with --fmad=false -ftz=true.
#pragma once

#include "ds_math.cuh"
#include "kernels.h"
#include "pair_math.cuh"

namespace ommp {
namespace gpu {
namespace {

// 2^e of the scaling of a product's dipoles from the largest high word of
// |x| (0 when all are zero: no scaling)
__device__ __forceinline__ int dsp_exponent(unsigned emax) {
  const int e = (int)(emax >> 20);
  return e == 0 ? 0 : e - 1023 + 12;
}
__device__ __forceinline__ double pow2(int e) {  // |e| <= 1022
  return __hiloint2double((1023 + e) << 20, 0);
}
// v 2^-e without leaving the range of a double's exponent
__device__ __forceinline__ double scale_down(double v, int e) {
  const int h = e / 2;
  return v * pow2(-h) * pow2(-(e - h));
}
__device__ __forceinline__ double scale_up(double v, int e) {
  const int h = e / 2;
  return v * pow2(h) * pow2(e - h);
}

// difference of two sites, its FP32 square and reciprocal length
struct DspDelta {
  dsf x, y, z;
  float r2, ri;
};
__device__ __forceinline__ DspDelta dsp_delta(const float (&t)[9], const float (&s)[9]) {
  DspDelta d;
  d.x = ds_delta(t[0], t[3], t[6], s[0], s[3], s[6]);
  d.y = ds_delta(t[1], t[4], t[7], s[1], s[4], s[7]);
  d.z = ds_delta(t[2], t[5], t[8], s[2], s[5], s[8]);
  d.r2 = fmaf(d.x.h, d.x.h, fmaf(d.y.h, d.y.h, d.z.h * d.z.h));
  const float y0 = rsqrtf(d.r2);
  d.ri = fmaf(0.5f * y0, fmaf(-(d.r2 * y0), y0, 1.f), y0);
  return d;
}

// Whether the pair is left to FP64: close, or its damping reaches the leading
// float.  AMOEBA damping differs from 1 by a polynomial in x = a u^3 times
// exp(-x); beyond xmin it is small enough to be formed in FP32 and subtracted
// from the low parts (x > 0 then: the exponent; sites without a Thole factor
// give a NaN and are not damped).  Wang-AL pairs are masked up to
// kSymNear2Wang (their damping range is shorter).
template <bool AMOEBA>
__device__ __forceinline__ bool dsp_masked(float r2, float2 wat, float2 was, float xmin, float &x) {
  x = 0.f;
  if (!AMOEBA) return !(r2 >= kSymNear2Wang) || maybe_damped_wang(r2, wat, was);
  const float u2 = r2 * wat.x * was.x;
  const float x2 = fminf(wat.y, was.y) * (u2 * u2 * u2);
  if (!(r2 >= kSymNear2) || x2 < xmin * xmin * 1.0002f) return true;
  if (x2 < 2601.f) x = x2 * rsqrtf(x2);
  return false;
}

// n = d y and eps = 1 - |n|^2
// (EXTRA: as the sum of two floats; eps alone is within about 2^-47)
struct DspUnit {
  dsf x, y, z;
  float ri, eps, epsl;
};
template <bool EXTRA = false>
__device__ __forceinline__ DspUnit dsp_unit(const DspDelta &d, float y) {
  DspUnit n;
  n.ri = y;
  n.x.h = d.x.h * y;
  n.y.h = d.y.h * y;
  n.z.h = d.z.h * y;
  n.x.l = fmaf(d.x.l, y, fmaf(d.x.h, y, -n.x.h));
  n.y.l = fmaf(d.y.l, y, fmaf(d.y.h, y, -n.y.h));
  n.z.l = fmaf(d.z.l, y, fmaf(d.z.h, y, -n.z.h));
  // the squares added to 2 in exact fast sums
  const float px = n.x.h * n.x.h, py = n.y.h * n.y.h, pz = n.z.h * n.z.h;
  const float qx = fmaf(n.x.h + n.x.h, n.x.l, fmaf(n.x.h, n.x.h, -px));
  const float qy = fmaf(n.y.h + n.y.h, n.y.l, fmaf(n.y.h, n.y.h, -py));
  const float qz = fmaf(n.z.h + n.z.h, n.z.l, fmaf(n.z.h, n.z.h, -pz));
  const float s1 = 2.f + px, s2 = s1 + py, s3 = s2 + pz;
  const float rx = px - (s1 - 2.f), ry = py - (s2 - s1), rz = pz - (s3 - s2);
  if (EXTRA) {
    const dsf a = two_sum(rx, ry), b = two_sum(a.h, rz), c = two_sum(3.f - s3, -b.h);
    const dsf e = two_sum(c.h, c.l - ((a.l + b.l) + ((qx + qy) + qz)));
    n.eps = e.h;
    n.epsl = e.l;
  } else {
    n.eps = (3.f - s3) - (((qx + qy) + qz) + ((rx + ry) + rz));
    n.epsl = 0.f;
  }
  return n;
}
// (1 - eps)^(-m/2) - 1
template <int M>
__device__ __forceinline__ float dsp_power(float eps) {
  return eps * fmaf(0.125f * M * (M + 2), eps, 0.5f * M);
}
// (h + l) (1 - eps)^(-m/2) with both parts of eps, renormalised
template <int M>
__device__ __forceinline__ dsf dsp_scaled(float h, float l, const DspUnit &n) {
  const float wh = 0.5f * M * n.eps;
  const float wl = fmaf(0.125f * M * (M + 2) * n.eps, n.eps, fmaf(0.5f * M, n.epsl, fmaf(0.5f * M, n.eps, -wh)));
  const float u = h * wh;
  const dsf s = fast_two_sum(h, u);
  return {s.h, s.l + (l + fmaf(h, wl, fmaf(h, wh, -u)))};
}
// c * (h + l) * (1 + w), c exact in FP32
__device__ __forceinline__ dsf dsp_coef(float c, float h, float l, float w) {
  const float p = c * h;
  return {p, fmaf(p, w, fmaf(c, l, fmaf(c, h, -p)))};
}

// a b, the low part not renormalised
__device__ __forceinline__ dsf dsp_mul(dsf a, dsf b) {
  const float p = a.h * b.h;
  return {p, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -p)))};
}
// acc += a b, the low part collected (renormalised by the caller)
__device__ __forceinline__ void dsp_acc(float &ah, float &al, dsf a, dsf b) {
  const dsf p = dsp_mul(a, b);
  const dsf s = two_sum(ah, p.h);
  ah = s.h;
  al += s.l + p.l;
}
__device__ __forceinline__ void dsp_acc(dsf &acc, dsf a, dsf b) { dsp_acc(acc.h, acc.l, a, b); }
// a.b, the low part not renormalised
__device__ __forceinline__ dsf dsp_dot(dsf a0, dsf a1, dsf a2, dsf b0, dsf b1, dsf b2) {
  const dsf p = dsp_mul(a0, b0), q = dsp_mul(a1, b1), r = dsp_mul(a2, b2);
  const dsf u1 = two_sum(p.h, q.h);
  const dsf u2 = two_sum(u1.h, r.h);
  return {u2.h, ((p.l + q.l) + r.l) + (u1.l + u2.l)};
}
__device__ __forceinline__ dsf dsp_norm(dsf a) { return fast_two_sum(a.h, a.l); }

// The dipole field of one pair, E = K (mu.n) n - k3 mu.
struct DsPair {
  DspUnit n;
  dsf k;  // -k3
  dsf K;  // 3 r^-5 / y^2
};

// MASKED: pairs left to FP64 and the site itself give nothing here (masked is
// set).  1 - (1 + x) exp(-x) differs from 1 by less than 2^-24 for x > 20
// (from about 6.6 bohr of the damping range's 9 in water).
template <bool MASKED, bool AMOEBA>
__device__ __forceinline__ DsPair dsp_geometry(const float (&t)[9], const float (&s)[9], float2 wat, float2 was,
                                               bool &masked) {
  const DspDelta d = dsp_delta(t, s);
  float y = d.ri, x = 0.f;
  if (MASKED) {
    masked = dsp_masked<AMOEBA>(d.r2, wat, was, 20.f, x);
    if (masked) y = 0.f;
  }
  DsPair g;
  g.n = dsp_unit(d, y);
  const float w3 = dsp_power<3>(g.n.eps), w5 = dsp_power<5>(g.n.eps);
  const float y2 = y * y, y2l = fmaf(y, y, -y2);
  const float Y = y2 * y, Yl = fmaf(y2l, y, fmaf(y2, y, -Y));
  g.k = {-Y, -fmaf(Y, w3, Yl)};
  g.K = dsp_coef(3.f, Y, Yl, w5);
  if (MASKED && AMOEBA && x > 0.f) {
    const float e = __expf(-x);
    g.k.l = fmaf(-g.k.h, e, g.k.l);
    g.K.l = fmaf(-g.K.h, fmaf(x, e, e), g.K.l);
  }
  return g;
}

__device__ __forceinline__ void dsp_column(const DsPair &g, const float (&mh)[3], const float (&ml)[3], float (&ah)[3],
                                           float (&al)[3]) {
  const dsf mx{mh[0], ml[0]}, my{mh[1], ml[1]}, mz{mh[2], ml[2]};
  const dsf f = dsp_mul(g.K, dsp_dot(mx, my, mz, g.n.x, g.n.y, g.n.z));
  dsp_acc(ah[0], al[0], f, g.n.x);
  dsp_acc(ah[0], al[0], g.k, mx);
  dsp_acc(ah[1], al[1], f, g.n.y);
  dsp_acc(ah[1], al[1], g.k, my);
  dsp_acc(ah[2], al[2], f, g.n.z);
  dsp_acc(ah[2], al[2], g.k, mz);
}

}  // namespace
}  // namespace gpu
}  // namespace ommp
