// Pair pass of the polarization-energy gradient (polelec_geomgrad,
// src/mod_geomgrad.F90:113-277): per static site the unscaled force and, for
// AMOEBA, the torque on its static multipole, from one evaluation of every
// unordered pair.
//
// With U = q V + m.grad V + Q:grad grad V the energy of the static multipole
// (q, m, Q) of one site in the potential V of the mean dipole p = (D + P) / 2
// of another, and the dipole-dipole energy (D P' + P D') / 2 = p p' - d d'
// (d = (D - P) / 2; zero for water), a pair's energy is
//   U(t; p_s) + U(s; p_t) + p_t p_s - d_t d_s,
// its gradient acts on the two sites with opposite signs, and the rotation of
// the frames needs only the torque of U, tau = -m x E + 2 vec(Q G).  The two
// ordered passes that formed the field gradients of either dipole set, the
// field, its gradient and its contracted Hessian at every site took 2 x 2,703
// FP32 operations per pair in double-single, or 2 x 207 on the FP64 pipe; the
// pair form takes about 2,080 (ncu).  p_t p_s is covered by adding p / 2 to m.
//
// Notation (n the unit vector from s to t, a = p.n, b = m.n, T = Q n,
// s = n.T, R = Q p'; K = y^3, G = 3 y^3, F = 3 y^4, C = 15 y^4, F5 = 3 y^5,
// H = 15 y^5, D = 105 y^5 with the damping factors of r^-3 (K), r^-5 (G, F,
// F5), r^-7 (C, H) and r^-9 (D)):
//   force on t = n [a_s (-G q_t + C b_t - D s_t) + a_t (G q_s + C b_s + D s_s)
//                   - F (m_t.p_s + m_s.p_t) + 2 H (T_t.p_s - T_s.p_t)]
//              + p_s (K q_t - F b_t + H s_t) - p_t (K q_s + F b_s + H s_s)
//              + a_s (2 H T_t - F m_t) - a_t (2 H T_s + F m_s) + 2 F5 (R_s - R_t)
//   torque on t = [a_s (2 C T_t - G m_t) - 2 F R_t] x n + [K m_t - 2 F T_t] x p_s
//   torque on s = [2 F R_s - a_t (G m_s + 2 C T_s)] x n + [K m_s + 2 F T_s] x p_t
// (R_t = Q_t p_s, R_s = Q_s p_t; the torques with m alone), and for
// quadrupoles that are not traceless the terms of trace_force.  The formulas are
// written once for double and for double-single numbers.
//
// Schedule, near pairs and accumulation are those of the symmetric T.mu
// (tmu_sym.cu): half-shell slots of 128-site tiles, a 32-step rotation per
// 32 x 32 sub-tile pair, close and strongly damped pairs (x < 28: the r^-9
// damping reaches farther) queued for FP64, fixed-point sums.  Sub-tile pairs
// without a polarizable site are skipped.  The dipoles are scaled by a power
// of two as in the products, and so is the other factor of every term, the
// static multipoles and unscaled dipoles, unless it is near one: with
// charges of 1e-8 and dipoles of 1e-5 the terms of the fixed-point sums would
// else lose 1e-11 of their value, with dipoles of 1e-8 8e-9.
//
// Products and sums keep their low parts unrenormalised, the accumulators are
// renormalised per pair: renormalising every product cost 7 % for errors of
// 7.5e-15.
//
// 30,000 sites: 76 -> 35 ms in the mixed modes, 330 ms in FP64 before; 90,000:
// 668 -> 311 ms (2.95 s in FP64).  Error against 64 bits 0.95e-14 to 1.2e-14
// (before 2.7e-14 in FP64, 3e-14 to 6e-14 in double-single).  255 registers
// without spills at 2 CTAs per SM: bound by FP32 issue at 8 warps (71 % of the
// issue slots, 2,076 operations per pair; at 6,000 sites 54 %, a quarter of the
// stalls the fetch of the 2,600-instruction step, which far and near
// sub-tiles' warps pass through at different places).
//
// Built with --fmad=false -ftz=true: every FMA is explicit.
#include <algorithm>

#include "ds_pair.cuh"
#include "grad_math.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int TILE = 128, SUB = 32;
constexpr float FAR = 1.0e6f;

struct GradSymJob {
  DevSites s;
  const double *p, *d;    // [m][3] scaled mean dipole and half difference
  const int *any;         // [0] some d is not zero, [1] some quadrupole has a trace
  const double *q;        // [m][10 or 1] scaled static multipoles
  const int *eu;          // 2^eu takes a scaled dipole to their scale
  const unsigned *polar;  // [ceil(m / 32)] sites of the sub-tile that are polarizable
  unsigned long long *lo, *hi, *bad;
  int ntile, K, chunk, nchunk, quarters, items;
  float r2near;
  int *err;
};

// --- numbers: double, or a double-single pair ------------------------------------
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ dsf mul(dsf a, dsf b) { return dsp_mul(a, b); }
__device__ __forceinline__ void mad(double &c, double a, double b) { c = fma(a, b, c); }
__device__ __forceinline__ void mad(dsf &c, dsf a, dsf b) { dsp_acc(c, a, b); }
__device__ __forceinline__ double neg(double a) { return -a; }
__device__ __forceinline__ dsf neg(dsf a) { return {-a.h, -a.l}; }
__device__ __forceinline__ double twice(double a) { return a + a; }
__device__ __forceinline__ dsf twice(dsf a) { return {a.h + a.h, a.l + a.l}; }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ dsf sub(dsf a, dsf b) {
  const dsf s = two_sum(a.h, -b.h);
  return {s.h, s.l + (a.l - b.l)};
}
__device__ __forceinline__ double dot(const double *a, const double *b) {
  return fma(a[0], b[0], fma(a[1], b[1], a[2] * b[2]));
}
__device__ __forceinline__ dsf dot(const dsf *a, const dsf *b) {
  return dsp_dot(a[0], a[1], a[2], b[0], b[1], b[2]);
}
// Q v, Q = xx, xy, yy, xz, yz, zz
template <typename T>
__device__ __forceinline__ void apply(const T *Q, const T *v, T *o) {
  const T r0[3] = {Q[0], Q[1], Q[3]}, r1[3] = {Q[1], Q[2], Q[4]}, r2[3] = {Q[3], Q[4], Q[5]};
  o[0] = dot(r0, v);
  o[1] = dot(r1, v);
  o[2] = dot(r2, v);
}
// o += u x v
template <typename T>
__device__ __forceinline__ void add_cross(const T *u, const T *v, T *o) {
  mad(o[0], u[1], v[2]);
  mad(o[0], neg(u[2]), v[1]);
  mad(o[1], u[2], v[0]);
  mad(o[1], neg(u[0]), v[2]);
  mad(o[2], u[0], v[1]);
  mad(o[2], neg(u[1]), v[0]);
}

// static multipole and dipole of a site: q, m + p / 2, m, Q, trace of Q, p
template <typename T, bool AMOEBA>
struct Site {
  T q, mp[3], m[3], Q[6], tr, p[3];
};
template <typename T>
struct Site<T, false> {
  T q, p[3];
};

template <typename T>
struct Powers {
  T K, G, F, C, F5, H, D;
};

// force on t (added to f), torques on t and s (added)
template <typename T>
__device__ __forceinline__ void pair_force(const Site<T, true> &t, const Site<T, true> &s, const T *n,
                                           const Powers<T> &k, T *f, T *tau_t, T *tau_s) {
  T Tt[3], Ts[3];
  apply(t.Q, n, Tt);
  apply(s.Q, n, Ts);
  const T as = dot(s.p, n), at = dot(t.p, n), bt = dot(t.mp, n), bs = dot(s.mp, n);
  const T st = dot(Tt, n), ss = dot(Ts, n);
  const T nF = neg(k.F), H2 = twice(k.H);
  // n
  T x1 = mul(neg(k.G), t.q), x2 = mul(k.G, s.q);
  mad(x1, k.C, bt);
  mad(x1, neg(k.D), st);
  mad(x2, k.C, bs);
  mad(x2, k.D, ss);
  T X = mul(as, x1);
  mad(X, at, x2);
  mad(X, nF, dot(t.mp, s.p));
  mad(X, nF, dot(s.mp, t.p));
  mad(X, H2, dot(Tt, s.p));
  mad(X, neg(H2), dot(Ts, t.p));
  // p_s, p_t
  T ws = mul(k.K, t.q), wt = mul(neg(k.K), s.q);
  mad(ws, nF, bt);
  mad(ws, k.H, st);
  mad(wt, nF, bs);
  mad(wt, neg(k.H), ss);
  T Rt[3], Rs[3];
  apply(t.Q, s.p, Rt);
  apply(s.Q, t.p, Rs);
  const T F52 = twice(k.F5), F2 = twice(k.F), C2 = twice(k.C);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T u = mul(H2, Tt[c]), v = mul(neg(H2), Ts[c]);
    mad(u, nF, t.mp[c]);
    mad(v, nF, s.mp[c]);
    mad(f[c], X, n[c]);
    mad(f[c], ws, s.p[c]);
    mad(f[c], wt, t.p[c]);
    mad(f[c], as, u);
    mad(f[c], at, v);
    mad(f[c], F52, sub(Rs[c], Rt[c]));
  }
  T u[3], w[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T v = mul(C2, Tt[c]);
    mad(v, neg(k.G), t.m[c]);
    u[c] = mul(as, v);
    mad(u[c], neg(F2), Rt[c]);
    w[c] = mul(k.K, t.m[c]);
    mad(w[c], neg(F2), Tt[c]);
  }
  add_cross(u, n, tau_t);
  add_cross(w, s.p, tau_t);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T v = mul(C2, Ts[c]);
    mad(v, k.G, s.m[c]);
    u[c] = mul(neg(at), v);
    mad(u[c], F2, Rs[c]);
    w[c] = mul(k.K, s.m[c]);
    mad(w[c], F2, Ts[c]);
  }
  add_cross(u, n, tau_s);
  add_cross(w, t.p, tau_s);
}

// The trace of the quadrupole of a site in the field of the dipole p of the
// other: the reference keeps it in the Hessian contraction (the force on the
// static site) and drops it in the field of the quadrupole, so it acts on one
// side only.  n and p.n change sign together: the same form for either site.
template <typename T>
__device__ __forceinline__ void trace_force(T tr, const T *p, const T *n, const Powers<T> &k, T *f) {
  const T x = mul(mul(k.H, tr), dot(p, n)), w = mul(neg(k.F5), tr);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    mad(f[c], x, n[c]);
    mad(f[c], w, p[c]);
  }
}

// charges and dipoles only; p2 the unscaled dipole of t (the dipole-dipole
// energy takes one scaled factor, as the others)
template <typename T>
__device__ __forceinline__ void pair_force(const Site<T, false> &t, const T *p2, const Site<T, false> &s, const T *n,
                                           const Powers<T> &k, T *f) {
  const T as = dot(s.p, n), at = dot(t.p, n), a2 = dot(p2, n);
  T X = mul(mul(neg(k.G), t.q), as);
  mad(X, mul(k.G, s.q), at);
  mad(X, neg(k.F), dot(p2, s.p));
  mad(X, mul(k.C, a2), as);
  T ws = mul(k.K, t.q);
  mad(ws, neg(k.F), a2);
  const T wt = mul(neg(k.K), s.q), w2 = mul(neg(k.F), as);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    mad(f[c], X, n[c]);
    mad(f[c], ws, s.p[c]);
    mad(f[c], wt, t.p[c]);
    mad(f[c], w2, p2[c]);
  }
}

// the dipole-dipole gradient of (dt, ds), subtracted from f
template <typename T>
__device__ __forceinline__ void delta_force(const T *dt, const T *ds, const T *n, const Powers<T> &k, T *f) {
  const T at = dot(dt, n), as = dot(ds, n);
  T X = mul(k.F, dot(dt, ds));
  mad(X, mul(neg(k.C), at), as);
  const T ws = mul(k.F, at), wt = mul(k.F, as);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    mad(f[c], X, n[c]);
    mad(f[c], ws, ds[c]);
    mad(f[c], wt, dt[c]);
  }
}

// FP64 value v of the staged record: which of the floats h, l of a site hold it
// (see stage): q, m + p / 2 (3), m (3), Q (6), tr, p (3), d (3)
template <bool AMOEBA>
struct Rec {
  static constexpr int NV = AMOEBA ? 20 : 4;  // values in double-single
  static constexpr int R = (9 + 2 * NV + 3) / 4;
};

template <bool AMOEBA>
__device__ __forceinline__ void site_values(const GradSymJob &jb, int i, int eu, double *v) {
  const double *q = jb.q + (size_t)i * (AMOEBA ? 10 : 1), *p = jb.p + 3 * (size_t)i;
  v[0] = q[0];
  if (!AMOEBA) {
    for (int c = 0; c < 3; ++c) v[1 + c] = p[c];
    return;
  }
  for (int c = 0; c < 3; ++c) {
    v[1 + c] = fma(0.5, scale_up(p[c], eu), q[1 + c]);
    v[4 + c] = q[1 + c];
    v[14 + c] = p[c];
    v[17 + c] = jb.d[3 * (size_t)i + c];
  }
  for (int c = 0; c < 6; ++c) v[7 + c] = q[4 + c];
  v[13] = (q[4] + q[6]) + q[9];
}

template <typename T>
__device__ __forceinline__ void fill(Site<T, true> &s, const T *v) {
  s.q = v[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) s.mp[c] = v[1 + c], s.m[c] = v[4 + c], s.p[c] = v[14 + c];
#pragma unroll
  for (int c = 0; c < 6; ++c) s.Q[c] = v[7 + c];
  s.tr = v[13];
}
template <typename T>
__device__ __forceinline__ void fill(Site<T, false> &s, const T *v) {
  s.q = v[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) s.p[c] = v[1 + c];
}

template <bool AMOEBA>
struct GradSmem {
  static constexpr int NO = AMOEBA ? 6 : 3;  // outputs of a site: force, torque
  float4 rec[Rec<AMOEBA>::R][TILE];
  double accj[4][NO][TILE];
  float2 wa[TILE];
  unsigned short queue[4][SUB * SUB];
};

__device__ __forceinline__ void fixed_add_to(const GradSymJob &jb, size_t o, double v) {
  fixed_add_int(jb.lo + o, jb.hi + o, v, jb.bad);
}

// the queued pairs in FP64, one per lane
template <bool AMOEBA>
__device__ __noinline__ void grad_queued(const GradSymJob &jb, const unsigned short *queue, int count, int lane,
                                         int i0, int j0, int eu, bool delta, bool trace) {
  constexpr int NO = GradSmem<AMOEBA>::NO;
  const DevSites &s = jb.s;
  for (int e = lane; e < count; e += 32) {
    const int q = queue[e], i = i0 + (q >> 5), j = j0 + (q & 31);
    if (i >= s.m || j >= s.m || i == j) continue;
    const bool pi_pol = (jb.polar[i / 32] >> (i % 32)) & 1u, pj_pol = (jb.polar[j / 32] >> (j % 32)) & 1u;
    if (!pi_pol && !pj_pol) continue;
    const Pos64 pi = s.mm_pos[i], pj = s.mm_pos[j];
    const double d[3] = {pi.x - pj.x, pi.y - pj.y, pi.z - pj.z};
    const double r2 = fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]));
    if (coincident(r2)) {
      atomicOr(jb.err, 1);
      continue;
    }
    const double y = rinv_f64(r2, r2_f32(r2));
    double k3, k5, k7, k9;
    gradmath::damped_k<AMOEBA>(r2, y, pi.w * pj.w, AMOEBA ? fmin(s.mm_a[i], s.mm_a[j]) : 0.0, s.damp_thr, true, k3, k5,
                               k7, k9);
    const double r = r2 * y;
    const double n[3] = {d[0] * y, d[1] * y, d[2] * y};
    Powers<double> k;
    k.K = k3;
    k.F5 = 3.0 * k5;
    k.F = k.F5 * r;
    k.G = k.F * r;
    k.H = 15.0 * k7 * r2;
    k.C = k.H * r;
    k.D = 105.0 * k9 * r2 * r2;
    constexpr int NV = Rec<AMOEBA>::NV;
    double vi[NV], vj[NV];
    site_values<AMOEBA>(jb, i, eu, vi);
    site_values<AMOEBA>(jb, j, eu, vj);
    double f[3] = {0.0, 0.0, 0.0}, gi[3] = {0.0, 0.0, 0.0}, gj[3] = {0.0, 0.0, 0.0}, tt[3] = {0.0, 0.0, 0.0}, ts[3] = {0.0, 0.0, 0.0};
    Site<double, AMOEBA> a, b;
    fill(a, vi);
    fill(b, vj);
    if constexpr (AMOEBA) {
      pair_force(a, b, n, k, f, tt, ts);
      if (trace) {
        trace_force(a.tr, b.p, n, k, gi);
        trace_force(b.tr, a.p, n, k, gj);
      }
      if (delta) {
        const double du[3] = {scale_up(vi[17], eu), scale_up(vi[18], eu), scale_up(vi[19], eu)};
        delta_force(du, vj + 17, n, k, f);
      }
    } else {
      const double pu[3] = {scale_up(vi[1], eu), scale_up(vi[2], eu), scale_up(vi[3], eu)};
      pair_force(a, pu, b, n, k, f);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      fixed_add_to(jb, (size_t)i * NO + c, f[c] + gi[c]);
      fixed_add_to(jb, (size_t)j * NO + c, gj[c] - f[c]);
      if (AMOEBA) {
        fixed_add_to(jb, (size_t)i * NO + 3 + c, tt[c]);
        fixed_add_to(jb, (size_t)j * NO + 3 + c, ts[c]);
      }
    }
  }
}

__device__ __forceinline__ float box_gap2(const float4 &alo, const float4 &ahi, const float4 &blo, const float4 &bhi) {
  const float gx = fmaxf(0.f, fmaxf(blo.x - ahi.x, alo.x - bhi.x));
  const float gy = fmaxf(0.f, fmaxf(blo.y - ahi.y, alo.y - bhi.y));
  const float gz = fmaxf(0.f, fmaxf(blo.z - ahi.z, alo.z - bhi.z));
  return fmaf(gx, gx, fmaf(gy, gy, gz * gz));
}

template <bool AMOEBA>
__global__ void __launch_bounds__(TILE, AMOEBA ? 2 : 4) k_grad_sym(const __grid_constant__ GradSymJob jb,
                                                                   unsigned *__restrict__ next) {
  constexpr int NO = GradSmem<AMOEBA>::NO, NV = Rec<AMOEBA>::NV, R = Rec<AMOEBA>::R;
  extern __shared__ float4 dyn[];
  GradSmem<AMOEBA> &sm = *reinterpret_cast<GradSmem<AMOEBA> *>(dyn);
  __shared__ int s_item;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const DevSites &s = jb.s;
  const int m = s.m, nsub = (m + SUB - 1) / SUB;
  const int eu = *jb.eu;
  const bool delta = AMOEBA && jb.any[0] != 0, trace = AMOEBA && jb.any[1] != 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_item = (int)atomicAdd(next, 1u);
    __syncthreads();
    const int item = s_item;
    if (item >= jb.items) break;
    const int q = item % jb.quarters, unit = item / jb.quarters;
    const int js0 = q * (4 / jb.quarters), js1 = js0 + 4 / jb.quarters;
    const int I = unit / jb.nchunk;
    const int ti = I * TILE + tid;
    const bool vi = ti < m;
    float tg[9];
    dsf tv[NV];
    {
      const float4 h = vi ? s.mm_split[ti] : make_float4(FAR, FAR, FAR, 0.f);
      const float4 c = vi ? s.mm_split[(size_t)m + ti] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 l = vi ? s.mm_split[2 * (size_t)m + ti] : make_float4(0.f, 0.f, 0.f, 0.f);
      tg[0] = h.x, tg[1] = h.y, tg[2] = h.z, tg[3] = c.x, tg[4] = c.y, tg[5] = c.z, tg[6] = l.x, tg[7] = l.y,
      tg[8] = l.z;
      double v[NV];
      if (vi) site_values<AMOEBA>(jb, ti, eu, v);
#pragma unroll
      for (int c2 = 0; c2 < NV; ++c2) {
        // the difference dipoles (and, without multipoles, the second copy of
        // the dipole) enter the target's side unscaled
        const double w = !vi ? 0.0 : (AMOEBA && c2 >= 17) ? scale_up(v[c2], eu) : v[c2];
        tv[c2] = to_ds(w);
      }
    }
    dsf p2[3];
    if (!AMOEBA)
#pragma unroll
      for (int c = 0; c < 3; ++c) p2[c] = to_ds(vi ? scale_up(jb.p[3 * (size_t)ti + c], eu) : 0.0);
    const float2 wai = vi ? s.mm_wa32[ti] : make_float2(0.f, 0.f);
    double sumi[NO];
#pragma unroll
    for (int c = 0; c < NO; ++c) sumi[c] = 0.0;
    const int k0 = (unit - I * jb.nchunk) * jb.chunk;
    const int k1 = min(jb.K + 1, k0 + jb.chunk);
    for (int k = k0; k < k1; ++k) {
      int J = I + k;
      if (J >= jb.ntile) J -= jb.ntile;
      if (k > 0 && 2 * k == jb.ntile && I >= jb.ntile / 2) continue;  // the other tile of the pair owns it
      const bool diag = k == 0;
      const bool near_slot = !(box_gap2(s.mm_tile_box32[2 * I], s.mm_tile_box32[2 * I + 1], s.mm_tile_box32[2 * J],
                                        s.mm_tile_box32[2 * J + 1]) > jb.r2near);
      __syncthreads();
      if (warp >= js0 && warp < js1) {
        const int sj = J * TILE + tid;
        const bool v = sj < m;
        const float4 h = v ? s.mm_split[sj] : make_float4(-FAR, -FAR, -FAR, 0.f);
        const float4 c = v ? s.mm_split[(size_t)m + sj] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 l = v ? s.mm_split[2 * (size_t)m + sj] : make_float4(0.f, 0.f, 0.f, 0.f);
        float f[4 * R] = {h.x, h.y, h.z, c.x, c.y, c.z, l.x, l.y, l.z};
        double w[NV];
        if (v) site_values<AMOEBA>(jb, sj, eu, w);
#pragma unroll
        for (int c2 = 0; c2 < NV; ++c2) {
          const dsf d = to_ds(v ? w[c2] : 0.0);
          f[9 + 2 * c2] = d.h;
          f[10 + 2 * c2] = d.l;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) sm.rec[r][tid] = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
        sm.wa[tid] = v ? s.mm_wa32[sj] : make_float2(0.f, 0.f);
      }
      __syncthreads();
      const int si = 4 * I + warp;
      for (int js = js0; js < js1; ++js) {
        const int sj = 4 * J + js;
        const bool skip = si >= nsub || sj >= nsub || (diag && js < warp) || (jb.polar[si] | jb.polar[sj]) == 0u;
        if (skip) {
#pragma unroll
          for (int c = 0; c < NO; ++c) sm.accj[warp][c][js * SUB + lane] = 0.0;
          continue;
        }
        const bool self = diag && js == warp;
        const bool near =
            near_slot && (self || !(box_gap2(s.mm_sub_box32[2 * si], s.mm_sub_box32[2 * si + 1],
                                             s.mm_sub_box32[2 * sj], s.mm_sub_box32[2 * sj + 1]) > jb.r2near));
        int queued = 0;
        dsf ai[NO], aj[NO];
#pragma unroll
        for (int c = 0; c < NO; ++c) ai[c] = aj[c] = dsf{0.f, 0.f};
#pragma unroll 1
        for (int t = 0; t < SUB; ++t) {
          const int jl = js * SUB + ((lane + t) & 31);
          float f[4 * R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 v = sm.rec[r][jl];
            f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
          }
          float sc[9];
#pragma unroll
          for (int c = 0; c < 9; ++c) sc[c] = f[c];
          const DspDelta d = dsp_delta(tg, sc);
          float y = d.ri, x = 0.f;
          if (near) {
            bool masked = dsp_masked<AMOEBA>(d.r2, wai, sm.wa[jl], 28.f, x);
            // a sub-tile with itself meets every pair twice: formed once
            const bool second = self && ((lane + t) & 31) <= lane;
            if (masked || second) y = 0.f;
            masked = masked && !second;
            const unsigned mask = __ballot_sync(0xffffffffu, masked);
            if (masked)
              sm.queue[warp][queued + __popc(mask & ((1u << lane) - 1u))] = (unsigned short)(lane * 32 + ((lane + t) & 31));
            queued += __popc(mask);
          }
          const DspUnit u = dsp_unit(d, y);
          const dsf n[3] = {u.x, u.y, u.z};
          const float w3 = dsp_power<3>(u.eps), w5 = dsp_power<5>(u.eps), w7 = dsp_power<7>(u.eps),
                      w9 = dsp_power<9>(u.eps);
          const float y2 = y * y, y2l = fmaf(y, y, -y2);
          const float y3 = y2 * y, y3l = fmaf(y2l, y, fmaf(y2, y, -y3));
          const float y4 = y3 * y, y4l = fmaf(y3l, y, fmaf(y3, y, -y4));
          const float y5 = y4 * y, y5l = fmaf(y4l, y, fmaf(y4, y, -y5));
          Powers<dsf> k;
          k.K = {y3, fmaf(y3, w3, y3l)};
          k.G = dsp_coef(3.f, y3, y3l, w5);
          k.F = dsp_coef(3.f, y4, y4l, w5);
          k.C = dsp_coef(15.f, y4, y4l, w7);
          if (AMOEBA) {
            k.F5 = dsp_coef(3.f, y5, y5l, w5);
            k.H = dsp_coef(15.f, y5, y5l, w7);
            k.D = dsp_coef(105.f, y5, y5l, w9);
          }
          if (AMOEBA && x > 0.f) {  // weak damping, within the low parts
            const float e3 = __expf(-x), e5 = fmaf(x, e3, e3), x2 = x * x;
            const float e7 = fmaf(0.6f * x2, e3, e5), e9 = fmaf(fmaf(9.f / 35.f, x, 18.f / 35.f) * x2, e3, e5);
            k.K.l = fmaf(-k.K.h, e3, k.K.l);
            k.G.l = fmaf(-k.G.h, e5, k.G.l);
            k.F.l = fmaf(-k.F.h, e5, k.F.l);
            k.F5.l = fmaf(-k.F5.h, e5, k.F5.l);
            k.C.l = fmaf(-k.C.h, e7, k.C.l);
            k.H.l = fmaf(-k.H.h, e7, k.H.l);
            k.D.l = fmaf(-k.D.h, e9, k.D.l);
          }
          dsf sv[NV];
#pragma unroll
          for (int c = 0; c < NV; ++c) sv[c] = dsf{f[9 + 2 * c], f[10 + 2 * c]};
          Site<dsf, AMOEBA> st, ss;
          fill(st, tv);
          fill(ss, sv);
          dsf g[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
          if constexpr (AMOEBA) {
            pair_force(st, ss, n, k, g, ai + 3, aj + 3);
            if (trace) {
              trace_force(st.tr, ss.p, n, k, ai);
              trace_force(ss.tr, st.p, n, k, aj);
            }
            if (delta) delta_force(tv + 17, sv + 17, n, k, g);
          } else {
            pair_force(st, p2, ss, n, k, g);
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const dsf p = two_sum(ai[c].h, g[c].h), r = two_sum(aj[c].h, -g[c].h);
            ai[c] = {p.h, ai[c].l + (p.l + g[c].l)};
            aj[c] = {r.h, aj[c].l + (r.l - g[c].l)};
          }
#pragma unroll
          for (int c = 0; c < NO; ++c) {
            ai[c] = dsp_norm(ai[c]);
            aj[c] = dsp_norm(aj[c]);
            aj[c].h = __shfl_sync(0xffffffffu, aj[c].h, (lane + 1) & 31);
            aj[c].l = __shfl_sync(0xffffffffu, aj[c].l, (lane + 1) & 31);
          }
        }
        if (near) {
          __syncwarp();
          grad_queued<AMOEBA>(jb, sm.queue[warp], queued, lane, I * TILE + warp * SUB, J * TILE + js * SUB, eu, delta,
                              trace);
          __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          sumi[c] += (double)ai[c].h + (double)ai[c].l;
          sm.accj[warp][c][js * SUB + lane] = (double)aj[c].h + (double)aj[c].l;
        }
      }
      __syncthreads();
      const int sj = J * TILE + tid;
      if (warp >= js0 && warp < js1 && sj < m) {
#pragma unroll
        for (int c = 0; c < NO; ++c)
          fixed_add_to(jb, (size_t)sj * NO + c,
                       ((sm.accj[0][c][tid] + sm.accj[1][c][tid]) + sm.accj[2][c][tid]) + sm.accj[3][c][tid]);
      }
    }
    if (vi) {
#pragma unroll
      for (int c = 0; c < NO; ++c) fixed_add_to(jb, (size_t)ti * NO + c, sumi[c]);
    }
  }
}

// scaled mean dipoles and half differences in static-site order, whether any
// difference is not zero and whether any quadrupole has a trace beyond
// rounding; the static multipoles scaled by 2^-es, es from their exponent and
// that of the dipoles, and eu = ex - es
__global__ void k_grad_dipoles(int m, int n, int nset, const int *__restrict__ mm_polar, const double *__restrict__ ipd,
                               const unsigned *__restrict__ word, double *__restrict__ p, double *__restrict__ d,
                               const double *__restrict__ q, int q_e, double *__restrict__ qs, int *any, int *eu) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int j = mm_polar[i], ex = dsp_exponent(*word);
  const int es = scaling_exponent(max(q_e, *word >> 20 ? (int)(*word >> 20) - 1023 : kNoExponent));
  if (i == 0) *eu = ex - es;
  const int ld = nset == 2 ? 10 : 1;
  for (int c = 0; c < ld; ++c) qs[(size_t)i * ld + c] = scale_down(q[(size_t)i * ld + c], es);
  bool diff = false;
  for (int c = 0; c < 3; ++c) {
    const double a = j >= 0 ? scale_down(ipd[3 * (size_t)j + c], ex) : 0.0;
    const double b = nset == 2 ? (j >= 0 ? scale_down(ipd[3 * ((size_t)n + j) + c], ex) : 0.0) : a;
    p[3 * (size_t)i + c] = 0.5 * (a + b);
    d[3 * (size_t)i + c] = 0.5 * (a - b);
    diff = diff || a != b;
  }
  if (diff) any[0] = 1;
  if (nset == 2) {
    const double *Q = q + (size_t)i * 10 + 4;
    const double diag = fmax(fmax(fabs(Q[0]), fabs(Q[2])), fabs(Q[5]));
    if (fabs((Q[0] + Q[2]) + Q[5]) > 2e-15 * diag) any[1] = 1;
  }
}

template <bool AMOEBA>
int resident() {
  static const int r = [] {
    int v = 0;
    cudaFuncSetAttribute(k_grad_sym<AMOEBA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(GradSmem<AMOEBA>));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_grad_sym<AMOEBA>, TILE, sizeof(GradSmem<AMOEBA>));
    return v < 1 ? 1 : v;
  }();
  return r;
}

}  // namespace

// the buffer of launch_grad_sym: fixed-point words (lo, hi) of the outputs,
// flag, counter and scale of the dipoles, two flags, scale of the multipoles,
// dipoles and differences, scaled multipoles
size_t grad_sym_doubles(const DevSites &s) {
  const size_t no = s.amoeba ? 6 : 3;
  return (2 * no + 6 + (s.amoeba ? 10 : 1)) * (size_t)s.m + 4;
}

void launch_grad_sym(const DevSites &s, const double *ipd, const int *mm_polar, const unsigned *polar, double *buf,
                     int *err, cudaStream_t st) {
  if (s.m == 0 || s.n == 0) return;
  const size_t no = s.amoeba ? 6 : 3, nset = s.amoeba ? 2 : 1;
  GradSymJob j{};
  j.s = s;
  j.lo = reinterpret_cast<unsigned long long *>(buf);
  j.hi = j.lo + no * s.m;
  j.bad = j.hi + no * s.m;
  unsigned *next = reinterpret_cast<unsigned *>(j.bad + 1), *word = next + 1;
  int *any = reinterpret_cast<int *>(j.bad + 2);
  double *p = reinterpret_cast<double *>(j.bad + 4);
  j.p = p;
  j.d = p + 3 * (size_t)s.m;
  j.any = any;
  double *q = p + 6 * (size_t)s.m;
  j.q = q;
  int *eu = reinterpret_cast<int *>(j.bad + 3);
  j.eu = eu;
  j.polar = polar;
  j.err = err;
  j.r2near = near_range2(s, s.m2d_r2max32);
  j.ntile = (s.m + TILE - 1) / TILE;
  j.K = j.ntile / 2;
  const int ctas = (s.amoeba ? resident<true>() : resident<false>()) * sm_count();
  const long long units = (long long)j.ntile * (j.K + 1);
  // about 16 items per CTA; with fewer than 8 slots per CTA quarters of a slot
  j.chunk = (int)std::max(1LL, std::min(units / (16LL * ctas), (long long)j.K + 1));
  j.nchunk = (j.K + j.chunk) / j.chunk;
  j.quarters = units < 8LL * ctas ? 4 : 1;
  j.items = j.ntile * j.nchunk * j.quarters;
  cudaMemsetAsync(buf, 0, (2 * no * s.m + 4) * sizeof(double), st);
  launch_max_word(nset * 3 * (size_t)s.n, ipd, word, st, true);
  add_launch_count(2);
  k_grad_dipoles<<<(s.m + 255) / 256, 256, 0, st>>>(s.m, s.n, (int)nset, mm_polar, ipd, word, p,
                                                    p + 3 * (size_t)s.m, s.mm_q, s.q_e, q, any, eu);
  const int grid = std::min(ctas, j.items);
  if (s.amoeba)
    k_grad_sym<true><<<grid, TILE, sizeof(GradSmem<true>), st>>>(j, next);
  else
    k_grad_sym<false><<<grid, TILE, sizeof(GradSmem<false>), st>>>(j, next);
}

}  // namespace gpu
}  // namespace ommp
