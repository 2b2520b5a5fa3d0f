// Pair formulas of the static-static interaction (fixedelec.cu in FP64, m2m.cu
// in double-single): undamped potential, field, field gradient and contracted
// field Hessian of a multipole, as templates over the scalar type T and the
// weight type W (a scalar, or gradmath::One).  Constants are written as floats:
// all are exact in single precision.
#pragma once

#include "grad_math.cuh"

namespace ommp {
namespace gpu {
namespace {

// accumulators of one target: energy pass V (+ E, G); gradient pass E, G, h
template <bool AMOEBA, bool GRAD>
struct M2mNV {
  static constexpr int N = GRAD ? (AMOEBA ? 12 : 3) : (AMOEBA ? 10 : 1);
};

// potential, field and (AMOEBA) field gradient of the multipole q at
// d = target - source with undamped r^-1 .. r^-9
template <bool AMOEBA, typename T, typename W>
__device__ __forceinline__ void m2m_pair(const T *q, T dx, T dy, T dz, T rinv, W w, T *acc) {
  const T ir2 = rinv * rinv, k3 = rinv * ir2, k5 = k3 * ir2;
  if (!AMOEBA) {
    acc[0] += w * (q[0] * rinv);
    return;
  }
  const T k7 = k5 * ir2, k9 = k7 * ir2;
  const T md = q[1] * dx + q[2] * dy + q[3] * dz;
  const T tx = q[4] * dx + q[5] * dy + q[7] * dz;
  const T ty = q[5] * dx + q[6] * dy + q[8] * dz;
  const T tz = q[7] * dx + q[8] * dy + q[9] * dz;
  const T s = tx * dx + ty * dy + tz * dz;
  acc[0] += w * (q[0] * rinv + md * k3 + 3.0f * s * k5);
  const T c = q[0] * k3 + 3.0f * md * k5 + 15.0f * s * k7;
  acc[1] += w * (c * dx - q[1] * k3 - 6.0f * k5 * tx);
  acc[2] += w * (c * dy - q[2] * k3 - 6.0f * k5 * ty);
  acc[3] += w * (c * dz - q[3] * k3 - 6.0f * k5 * tz);
  gradmath::multipole_grad<true>(q, dx, dy, dz, k3, k5, k7, k9, w, acc + 4);
}

// field E, field gradient G and (AMOEBA) h_a = sum_bc Qt_bc H_bca of the
// multipole q at d = target - source (undamped), added with weight w;
// Qt (xx, xy, yy, xz, yz, zz) and trq are the target's quadrupole and trace.
// Field Hessians of a charge, dipole and quadrupole contracted with Qt
// (u = Qt d, sg = d.Qt.d; source t = Qs d, s = d.Qs.d):
//   charge      q (15 k7 sg d - 3 k5 (2 u + trq d))
//   dipole      gradmath::dipole_hess_q
//   quadrupole  945 k11 s sg d - 105 k9 (s (2 u + trq d) + 2 sg t + 4 (t.u) d)
//               + 30 k7 (2 Qs u + (Qs:Qt) d + 2 Qt t + trq t)
template <bool AMOEBA, typename T, typename W>
__device__ __forceinline__ void m2m_pair_grad(const T *q, T dx, T dy, T dz, T rinv, W w, const T *Qt, T trq, T *acc) {
  const T ir2 = rinv * rinv, k3 = rinv * ir2;
  if (!AMOEBA) {
    const T c = q[0] * k3;
    acc[0] += w * (c * dx);
    acc[1] += w * (c * dy);
    acc[2] += w * (c * dz);
    return;
  }
  const T k5 = k3 * ir2, k7 = k5 * ir2, k9 = k7 * ir2, k11 = k9 * ir2;
  const T md = q[1] * dx + q[2] * dy + q[3] * dz;
  const T tx = q[4] * dx + q[5] * dy + q[7] * dz;
  const T ty = q[5] * dx + q[6] * dy + q[8] * dz;
  const T tz = q[7] * dx + q[8] * dy + q[9] * dz;
  const T s = tx * dx + ty * dy + tz * dz;
  const T c = q[0] * k3 + 3.0f * md * k5 + 15.0f * s * k7;
  acc[0] += w * (c * dx - q[1] * k3 - 6.0f * k5 * tx);
  acc[1] += w * (c * dy - q[2] * k3 - 6.0f * k5 * ty);
  acc[2] += w * (c * dz - q[3] * k3 - 6.0f * k5 * tz);
  gradmath::multipole_grad<true>(q, dx, dy, dz, k3, k5, k7, k9, w, acc + 3);
  // h: target quadrupole against the source's field Hessian
  const T ux = Qt[0] * dx + Qt[1] * dy + Qt[3] * dz;
  const T uy = Qt[1] * dx + Qt[2] * dy + Qt[4] * dz;
  const T uz = Qt[3] * dx + Qt[4] * dy + Qt[5] * dz;
  const T sg = ux * dx + uy * dy + uz * dz;
  const T tu = tx * ux + ty * uy + tz * uz;
  const T qq = q[4] * Qt[0] + q[6] * Qt[2] + q[9] * Qt[5] + 2.0f * (q[5] * Qt[1] + q[7] * Qt[3] + q[8] * Qt[4]);
  // Qs u and Qt t
  const T px = q[4] * ux + q[5] * uy + q[7] * uz;
  const T py = q[5] * ux + q[6] * uy + q[8] * uz;
  const T pz = q[7] * ux + q[8] * uy + q[9] * uz;
  const T ox = Qt[0] * tx + Qt[1] * ty + Qt[3] * tz;
  const T oy = Qt[1] * tx + Qt[2] * ty + Qt[4] * tz;
  const T oz = Qt[3] * tx + Qt[4] * ty + Qt[5] * tz;
  const T cd = 15.0f * k7 * q[0] * sg - 3.0f * k5 * q[0] * trq + 945.0f * k11 * s * sg -
                    105.0f * k9 * (s * trq + 4.0f * tu) + 30.0f * k7 * qq;
  const T cu = -6.0f * k5 * q[0] - 210.0f * k9 * s;
  const T ct = -210.0f * k9 * sg + 30.0f * k7 * trq;
  const T cp = 60.0f * k7;
  T h[3];
  h[0] = cd * dx + cu * ux + ct * tx + cp * (px + ox);
  h[1] = cd * dy + cu * uy + ct * ty + cp * (py + oy);
  h[2] = cd * dz + cu * uz + ct * tz + cp * (pz + oz);
  gradmath::dipole_hess_q(&q[1], md, dx, dy, dz, Qt, trq, k5, k7, k9, gradmath::One{}, h);
  acc[9] += w * h[0];
  acc[10] += w * h[1];
  acc[11] += w * h[2];
}

template <bool AMOEBA, bool GRAD, typename T, typename W>
__device__ __forceinline__ void m2m_any(const T *q, T dx, T dy, T dz, T rinv, W w, const T *Qt, T trq, T *acc) {
  if (GRAD)
    m2m_pair_grad<AMOEBA>(q, dx, dy, dz, rinv, w, Qt, trq, acc);
  else
    m2m_pair<AMOEBA>(q, dx, dy, dz, rinv, w, acc);
}

}  // namespace
}  // namespace gpu
}  // namespace ommp
