// Pair arithmetic in double-single for the kernels of FP64 accuracy on the FP32
// pipes (tmu_sym.cu, fmm_near.cu): the dipole field of a pair in the
// unit-length form
//   E = 3 r^-5 (mu.d) d - r^-3 mu = K (mu.n) n - k3 mu,   n = d y,
// y the FP32 reciprocal distance.  Coordinates come split on a grid into three
// floats (split_coordinates), so differences are exact; |n|^2 is within 2^-22
// of 1 and its deviation eps is collected exactly by adding the squares to 2;
// r^-3 and 3 r^-5 follow from y^3 by a first- and second-order factor in eps.
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

// The dipole field of one pair: E = K (mu.n) n - k3 mu.
struct DsPair {
  float xh, xl, yh, yl, zh, zl;  // n = d y
  float kh, kl;                  // -k3
  float Kh, Kl;                  // 3 r^-5 / y^2
};

__device__ __forceinline__ void dsp_diff(float th, float tm, float tl, float sh, float sm, float sl, float &h,
                                         float &l) {
  // grid splits: the two leading differences are exact and |th - sh| is 0 or
  // at least |tm - sm|, so the fast sum is exact too
  const float dh = th - sh, dm = tm - sm;
  h = dh + dm;
  l = (dm - (h - dh)) + (tl - sl);
}

// MASKED: pairs left to FP64 and the site itself give nothing here (masked is
// set): the close ones and those whose damping reaches the leading float.
// AMOEBA damping 1 - (1 + x) exp(-x) with x = a u^3 > 20 (from about 6.6 bohr
// of 9 in water) differs from 1 by less than 2^-24, so an FP32 exponential in
// the low parts is enough.  The radii keep the double-single share of the
// product's error below that of the FP64 kernel this one replaced.
template <bool MASKED, bool AMOEBA>
__device__ __forceinline__ DsPair dsp_geometry(const float (&t)[9], const float (&s)[9], float2 wat, float2 was,
                                                bool &masked) {
  float dx, dy, dz, ex, ey, ez;
  dsp_diff(t[0], t[3], t[6], s[0], s[3], s[6], dx, ex);
  dsp_diff(t[1], t[4], t[7], s[1], s[4], s[7], dy, ey);
  dsp_diff(t[2], t[5], t[8], s[2], s[5], s[8], dz, ez);
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float y0 = rsqrtf(r2);
  float y = fmaf(0.5f * y0, fmaf(-(r2 * y0), y0, 1.f), y0);
  float damp3 = 0.f, damp5 = 0.f;
  if (MASKED) {
    if (AMOEBA) {
      const float u2 = r2 * wat.x * was.x;
      const float x2 = fminf(wat.y, was.y) * (u2 * u2 * u2);
      masked = !(r2 >= kSymNear2) || !(x2 >= 400.1f);
      if (!masked) {
        const float x = x2 * rsqrtf(x2);
        damp3 = __expf(-x);
        damp5 = fmaf(x, damp3, damp3);
      }
    } else {
      masked = !(r2 >= kSymNear2Wang) || maybe_damped_wang(r2, wat, was);
    }
    if (masked) y = 0.f;
  }
  DsPair g;
  g.xh = dx * y;
  g.yh = dy * y;
  g.zh = dz * y;
  g.xl = fmaf(ex, y, fmaf(dx, y, -g.xh));
  g.yl = fmaf(ey, y, fmaf(dy, y, -g.yh));
  g.zl = fmaf(ez, y, fmaf(dz, y, -g.zh));
  // eps = 1 - |n|^2: the squares added to 2 in exact fast sums
  const float px = g.xh * g.xh, py = g.yh * g.yh, pz = g.zh * g.zh;
  const float qx = fmaf(g.xh + g.xh, g.xl, fmaf(g.xh, g.xh, -px));
  const float qy = fmaf(g.yh + g.yh, g.yl, fmaf(g.yh, g.yh, -py));
  const float qz = fmaf(g.zh + g.zh, g.zl, fmaf(g.zh, g.zh, -pz));
  const float s1 = 2.f + px, s2 = s1 + py, s3 = s2 + pz;
  const float rx = px - (s1 - 2.f), ry = py - (s2 - s1), rz = pz - (s3 - s2);
  const float eps = (3.f - s3) - (((qx + qy) + qz) + ((rx + ry) + rz));
  // r^-3 = y^3 (1 - eps)^(-3/2), 3 r^-5 d d = 3 y^3 (1 - eps)^(-5/2) n n
  const float w3 = eps * fmaf(1.875f, eps, 1.5f);
  const float w5 = eps * fmaf(4.375f, eps, 2.5f);
  const float y2 = y * y, y2l = fmaf(y, y, -y2);
  const float Y = y2 * y, Yl = fmaf(y2l, y, fmaf(y2, y, -Y));
  g.kh = -Y;
  g.kl = -fmaf(Y, w3, Yl);
  g.Kh = 3.f * Y;
  g.Kl = fmaf(g.Kh, w5, fmaf(3.f, Yl, fmaf(3.f, Y, -g.Kh)));
  if (MASKED && AMOEBA) {
    g.kl = fmaf(-g.kh, damp3, g.kl);
    g.Kl = fmaf(-g.Kh, damp5, g.Kl);
  }
  return g;
}

__device__ __forceinline__ void dsp_acc(float &ah, float &al, float xh, float xl, float yh, float yl) {
  const float p = xh * yh;
  const float q = fmaf(xl, yh, fmaf(xh, yl, fmaf(xh, yh, -p)));
  const dsf s = two_sum(ah, p);
  ah = s.h;
  al += s.l + q;
}

__device__ __forceinline__ void dsp_column(const DsPair &g, const float (&mh)[3], const float (&ml)[3],
                                           float (&ah)[3], float (&al)[3]) {
  const float q0 = mh[0] * g.xh, q1 = mh[1] * g.yh, q2 = mh[2] * g.zh;
  const float f0 = fmaf(ml[0], g.xh, fmaf(mh[0], g.xl, fmaf(mh[0], g.xh, -q0)));
  const float f1 = fmaf(ml[1], g.yh, fmaf(mh[1], g.yl, fmaf(mh[1], g.yh, -q1)));
  const float f2 = fmaf(ml[2], g.zh, fmaf(mh[2], g.zl, fmaf(mh[2], g.zh, -q2)));
  const dsf u1 = two_sum(q0, q1);
  const dsf u2 = two_sum(u1.h, q2);
  const float t = ((f0 + f1) + f2) + (u1.l + u2.l);
  const float fh = g.Kh * u2.h;
  const float fl = fmaf(g.Kl, u2.h, fmaf(g.Kh, t, fmaf(g.Kh, u2.h, -fh)));
  dsp_acc(ah[0], al[0], fh, fl, g.xh, g.xl);
  dsp_acc(ah[0], al[0], g.kh, g.kl, mh[0], ml[0]);
  dsp_acc(ah[1], al[1], fh, fl, g.yh, g.yl);
  dsp_acc(ah[1], al[1], g.kh, g.kl, mh[1], ml[1]);
  dsp_acc(ah[2], al[2], fh, fl, g.zh, g.zl);
  dsp_acc(ah[2], al[2], g.kh, g.kl, mh[2], ml[2]);
}

}  // namespace
}  // namespace gpu
}  // namespace ommp
