// Geometric gradient of the polarization energy on the GPU
// (polelec_geomgrad, src/mod_geomgrad.F90:113-277).
//
// The reference builds, with the converged induced dipoles, the field
// gradient of the static multipoles and of the induced dipoles at the
// polarizable sites (Egrd_M2D, Egrd_D2D) and the field, field gradient and
// Hessian of the induced dipoles at the static sites (E/Egrd/EHes_D2M), then
// contracts them with the multipoles and adds the torque of the frame
// rotation.  Here every unordered pair of sites is evaluated once:
//   k_grad_sym     (grad_sym.cu) per static site the unscaled force and the
//                  torque on its static multipole
//   k_grad_finish  per site: the scaled pairs corrected by (s - 1) times their
//                  term (M2D p/d scales, D2D u scales, and for D2M the M2D
//                  lists read the other way), the gradient assembled, and the
//                  forces of the frame rotation evaluated (grad_math.cuh:
//                  frame_pullback)
//   k_grad_gather  the frame terms added to the atoms they act on through a
//                  fixed reverse list (deterministic; no atomics)
// AMOEBA uses both dipole sets: E/Egrd/EHes_D2M average the P dipoles with
// the d scales and the D dipoles with the p scales; Wang-AL has one set and
// only the charge terms.
#include <algorithm>
#include <cstdio>
#include <limits>
#include <vector>

#include "engine.h"
#include "ds_pair.cuh"
#include "grad_math.cuh"

namespace ommp {

// device data of the gradient (built on the first call; topology only, the
// positions and lab-frame multipoles are the system's)
struct GradState {
  int mm = 0;
  double *q0 = nullptr;        // [mm][10] local-frame multipoles (AMOEBA)
  int4 *frame = nullptr;       // frame kind, z, x, y atoms (self when absent)
  int *mm_polar = nullptr;     // [mm] polarizable index or -1
  int *t_ri = nullptr, *t_src = nullptr;  // M2D lists read by static site
  double *t_sP = nullptr, *t_sD = nullptr;
  int *r_ri = nullptr, *r_src = nullptr;  // frame atom -> (site, slot) entries
  unsigned *polar = nullptr;   // [ceil(mm / 32)] polarizable sites
  double *sums = nullptr;      // fixed-point sums and dipoles of the pair pass
  double *base = nullptr;      // [mm][3]
  double *rot = nullptr;       // [mm][4][3]
  double *grad = nullptr;      // [mm][3]
};

void free_grad_state(GradState *g) {
  if (!g) return;
  void *bufs[] = {g->q0, g->frame, g->mm_polar, g->t_ri, g->t_src, g->t_sP, g->t_sD, g->r_ri, g->r_src,
                  g->polar, g->sums, g->base, g->rot, g->grad};
  for (void *b : bufs)
    if (b) cudaFree(b);
  delete g;
}

namespace gpu {
namespace {

constexpr int GTPB = 128;

struct GradArgs {
  int mm, n;
  const Pos64 *mm_pos;
  const double *mm_a, *mm_q;
  const int *mm_polar, *polar_mm;
  const double *ipd;  // [n_ipd][n][3]
  const int *m2d_ri, *m2d_src;
  const double *m2d_sP, *m2d_sD;
  const int *d2d_ri, *d2d_src;
  const double *d2d_s;
  const int *t_ri, *t_src;
  const double *t_sP, *t_sD;
  const double *q0;
  const int4 *frame;
  const int *r_ri, *r_src;
  double *base, *rot, *grad;
  // the pair pass's fixed-point sums [mm][6 or 3], flag and scales
  const unsigned long long *lo, *hi, *bad;
  double thr;
  int *err;
};

// exact damped factors of the pair (target t, source i) for the list passes
template <bool AMOEBA>
__device__ __forceinline__ bool pair_k(const GradArgs &g, const Pos64 &pt, double at, int i, double *d, double *k) {
  const Pos64 ps = g.mm_pos[i];
  d[0] = pt.x - ps.x;
  d[1] = pt.y - ps.y;
  d[2] = pt.z - ps.z;
  const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
  if (r2 < 4.9e-28) return false;
  const double rinv = 1.0 / sqrt(r2);
  gradmath::damped_k<AMOEBA>(r2, rinv, pt.w * ps.w, fmin(at, AMOEBA ? g.mm_a[i] : 0.0), g.thr, true, k[0], k[1],
                             k[2], k[3]);
  return true;
}

template <bool AMOEBA>
__global__ void k_grad_finish(GradArgs g) {
  constexpr int LD = AMOEBA ? 10 : 1;
  constexpr int NO = AMOEBA ? 6 : 3;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.mm) return;
  double sums[NO];
  const int ex = dsp_exponent(reinterpret_cast<const unsigned *>(g.bad + 1)[1]);
  const int es = ex - *reinterpret_cast<const int *>(g.bad + 3);
  for (int c = 0; c < NO; ++c) {
    const size_t o = (size_t)t * NO + c;
    const double v = scale_up(scale_up(fixed_value(g.lo[o], g.hi[o]), ex), es);
    sums[c] = *g.bad ? __longlong_as_double(0x7ff8000000000000ll) : v;
  }
  // corrections of the scaled pairs
  double hd[6] = {0, 0, 0, 0, 0, 0}, hp[6] = {0, 0, 0, 0, 0, 0}, e[3] = {0, 0, 0}, h[3] = {0, 0, 0};
  const Pos64 pt = g.mm_pos[t];
  const double at = AMOEBA ? g.mm_a[t] : 0.0;
  const double *q = &g.mm_q[(size_t)t * LD];
  double Qt[6] = {0, 0, 0, 0, 0, 0};
  if (AMOEBA)
    for (int c = 0; c < 6; ++c) Qt[c] = q[4 + c];
  const double trq = Qt[0] + Qt[2] + Qt[5];
  double gm[6] = {0, 0, 0, 0, 0, 0};  // field gradient of the mean dipole
  const double *ipdP = g.ipd + (AMOEBA ? (size_t)3 * g.n : 0);
  int bad = 0;
  double dP[6] = {0, 0, 0, 0, 0, 0}, dD[6] = {0, 0, 0, 0, 0, 0};
  const int j = g.mm_polar[t];
  if (j >= 0) {
    // static multipoles, p / d scales
    for (int kk = g.m2d_ri[j]; kk < g.m2d_ri[j + 1]; ++kk) {
      const int i = g.m2d_src[kk];
      double d[3], k[4];
      if (!pair_k<AMOEBA>(g, pt, at, i, d, k)) {
        bad = 1;
        continue;
      }
      double gg[6] = {0, 0, 0, 0, 0, 0};
      gradmath::multipole_grad<AMOEBA>(&g.mm_q[(size_t)i * LD], d[0], d[1], d[2], k[0], k[1], k[2], k[3], 1.0, gg);
      const double cp = g.m2d_sP[kk] - 1.0, cd = AMOEBA ? g.m2d_sD[kk] - 1.0 : 0.0;
      for (int c = 0; c < 6; ++c) {
        dP[c] += cp * gg[c];
        dD[c] += cd * gg[c];
      }
    }
    // induced dipoles, u scales
    for (int kk = g.d2d_ri[j]; kk < g.d2d_ri[j + 1]; ++kk) {
      const int p = g.d2d_src[kk];
      double d[3], k[4];
      if (!pair_k<AMOEBA>(g, pt, at, g.polar_mm[p], d, k)) {
        bad = 1;
        continue;
      }
      const double c = g.d2d_s[kk] - 1.0;
      const double *mD = &g.ipd[3 * (size_t)p];
      gradmath::dipole_grad(mD, gradmath::dot3(mD, d), d[0], d[1], d[2], k[1], k[2], c, hd);
      if (AMOEBA) {
        const double *mP = &ipdP[3 * (size_t)p];
        gradmath::dipole_grad(mP, gradmath::dot3(mP, d), d[0], d[1], d[2], k[1], k[2], c, hp);
      }
    }
  }
  // induced dipoles at the static site: the M2D lists read by static site
  for (int kk = g.t_ri[t]; kk < g.t_ri[t + 1]; ++kk) {
    const int p = g.t_src[kk];
    double d[3], k[4];
    if (!pair_k<AMOEBA>(g, pt, at, g.polar_mm[p], d, k)) {
      bad = 1;
      continue;
    }
    const double *mD = &g.ipd[3 * (size_t)p], *mP = &ipdP[3 * (size_t)p];
    const double cp = g.t_sP[kk] - 1.0, cd = AMOEBA ? g.t_sD[kk] - 1.0 : 0.0;
    double mc[3];
    for (int c = 0; c < 3; ++c) mc[c] = AMOEBA ? 0.5 * (cp * mD[c] + cd * mP[c]) : cp * mD[c];
    const double md = gradmath::dot3(mc, d);
    gradmath::dipole_field(mc, md, d[0], d[1], d[2], k[0], k[1], 1.0, e);
    if (AMOEBA) {
      gradmath::dipole_grad(mc, md, d[0], d[1], d[2], k[1], k[2], 1.0, gm);
      gradmath::dipole_hess_q(mc, md, d[0], d[1], d[2], Qt, trq, k[1], k[2], k[3], 1.0, h);
    }
  }
  if (bad) atomicOr(g.err, 1);
  // assembly (src/mod_geomgrad.F90:132-271)
  double b[3];
  for (int c = 0; c < 3; ++c) b[c] = sums[c] - q[0] * e[c];
  if (AMOEBA) {
    double x[3];
    gradmath::sym_apply(gm, &q[1], x);
    for (int c = 0; c < 3; ++c) b[c] += x[c] - h[c];
  }
  if (j >= 0) {
    const double *mD = &g.ipd[3 * (size_t)j];
    if (AMOEBA) {
      const double *mP = &ipdP[3 * (size_t)j];
      double GP[6], GD[6], x[3], y[3];
      for (int c = 0; c < 6; ++c) {
        GP[c] = dP[c] + hp[c];
        GD[c] = dD[c] + hd[c];
      }
      gradmath::sym_apply(GP, mD, x);
      gradmath::sym_apply(GD, mP, y);
      for (int c = 0; c < 3; ++c) b[c] += 0.5 * (x[c] + y[c]);
    } else {
      double GM[6], x[3];
      for (int c = 0; c < 6; ++c) GM[c] = dP[c] + hd[c];
      gradmath::sym_apply(GM, mD, x);
      for (int c = 0; c < 3; ++c) b[c] += x[c];
    }
  }
  for (int c = 0; c < 3; ++c) g.base[3 * (size_t)t + c] = b[c];
  if (AMOEBA) {
    // torque of the frame rotation of the site's dipole and quadrupole
    const int4 f = g.frame[t];
    double out[4][3];
    const Pos64 pz = g.mm_pos[f.y], px = g.mm_pos[f.z], py = g.mm_pos[f.w];
    const double c0[3] = {pt.x, pt.y, pt.z}, cz[3] = {pz.x, pz.y, pz.z}, cx[3] = {px.x, px.y, px.z},
                 cy[3] = {py.x, py.y, py.z};
    if (!gradmath::frame_pullback(f.x, c0, cz, cx, cy, &g.q0[(size_t)t * 10], e, gm, out, sums + 3)) atomicOr(g.err, 2);
    double *r = &g.rot[12 * (size_t)t];
    for (int w = 0; w < 4; ++w)
      for (int c = 0; c < 3; ++c) r[3 * w + c] = out[w][c];
  }
}

// frame terms of every site for a given field E [mm][3] and field gradient
// G [mm][6] (rotation_geomgrad): rot [mm][4][3], error bit 2 on a degenerate frame
__global__ void k_rot_terms(int mm, const Pos64 *__restrict__ pos, const int4 *__restrict__ frame,
                            const double *__restrict__ q0, const double *__restrict__ E, const double *__restrict__ G,
                            double *__restrict__ rot, int *err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= mm) return;
  const int4 f = frame[t];
  const Pos64 pt = pos[t], pz = pos[f.y], px = pos[f.z], py = pos[f.w];
  const double c0[3] = {pt.x, pt.y, pt.z}, cz[3] = {pz.x, pz.y, pz.z}, cx[3] = {px.x, px.y, px.z},
               cy[3] = {py.x, py.y, py.z};
  double out[4][3];
  if (!gradmath::frame_pullback(f.x, c0, cz, cx, cy, &q0[(size_t)t * 10], &E[3 * (size_t)t], &G[6 * (size_t)t], out))
    atomicOr(err, 2);
  double *r = &rot[12 * (size_t)t];
  for (int w = 0; w < 4; ++w)
    for (int c = 0; c < 3; ++c) r[3 * w + c] = out[w][c];
}

__global__ void k_grad_gather(int mm, bool amoeba, const double *__restrict__ base, const double *__restrict__ rot,
                              const int *__restrict__ r_ri, const int *__restrict__ r_src, double *__restrict__ grad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= mm) return;
  double s[3] = {base[3 * (size_t)t], base[3 * (size_t)t + 1], base[3 * (size_t)t + 2]};
  if (amoeba)
    for (int k = r_ri[t]; k < r_ri[t + 1]; ++k) {
      const double *r = &rot[3 * (size_t)r_src[k]];
      for (int c = 0; c < 3; ++c) s[c] += r[c];
    }
  for (int c = 0; c < 3; ++c) grad[3 * (size_t)t + c] = s[c];
}

}  // namespace
}  // namespace gpu

// device lists and buffers of the gradient (topology only): built once
int System::ensure_grad_state() {
  if (grad_) return kOk;
  const int mm = d_.m, n = d_.n;
  const bool amoeba = m_.amoeba;
  int st;
  GradState *gs = new GradState();
  gs->mm = mm;
  // M2D lists read by static site, and the frame reverse list
  std::vector<int> t_ri(mm + 1, 0), t_src(m2d_pairs_.src.size());
  std::vector<double> t_sP(t_src.size()), t_sD(t_src.size());
  for (size_t k = 0; k < m2d_pairs_.src.size(); ++k) t_ri[m2d_pairs_.src[k] + 1]++;
  for (int i = 0; i < mm; ++i) t_ri[i + 1] += t_ri[i];
  {
    std::vector<int> fill(t_ri.begin(), t_ri.end() - 1);
    for (int j = 0; j < n; ++j)
      for (int k = m2d_pairs_.ri[j]; k < m2d_pairs_.ri[j + 1]; ++k) {
        const int i = m2d_pairs_.src[k], at = fill[i]++;
        t_src[at] = j;
        t_sP[at] = m2d_pairs_.sP[k];
        t_sD[at] = amoeba ? m2d_pairs_.sD[k] : 1.0;
      }
  }
  std::vector<int4> fr(mm);
  std::vector<int> r_ri(mm + 1, 0), r_src;
  for (int i = 0; i < mm; ++i) {
    const int fk = amoeba ? m_.frame[i] : 0;
    fr[i] = make_int4(fk, m_.iz[i] >= 0 ? m_.iz[i] : i, m_.ix[i] >= 0 ? m_.ix[i] : i, m_.iy[i] >= 0 ? m_.iy[i] : i);
  }
  {
    std::vector<std::vector<int>> rev(mm);
    for (int i = 0; i < mm; ++i) {
      if (fr[i].x == 0) continue;
      const int atoms[4] = {i, fr[i].y, fr[i].z, fr[i].w};
      for (int w = 0; w < 4; ++w) rev[atoms[w]].push_back(4 * i + w);
    }
    for (int i = 0; i < mm; ++i) {
      r_ri[i + 1] = r_ri[i] + (int)rev[i].size();
      r_src.insert(r_src.end(), rev[i].begin(), rev[i].end());
    }
  }
  auto alloc = [&](auto *&p, size_t cnt) {
    return cudaMalloc((void **)&p, std::max<size_t>(cnt, 1) * sizeof(*p)) == cudaSuccess ? 0 : 1;
  };
  int bad = alloc(gs->q0, amoeba ? 10 * (size_t)mm : 1) | alloc(gs->frame, mm) | alloc(gs->mm_polar, mm) |
            alloc(gs->t_ri, mm + 1) | alloc(gs->t_src, t_src.size()) | alloc(gs->t_sP, t_src.size()) |
            alloc(gs->t_sD, t_src.size()) | alloc(gs->r_ri, mm + 1) | alloc(gs->r_src, r_src.size()) |
            alloc(gs->polar, (mm + 31) / 32) | alloc(gs->sums, gpu::grad_sym_doubles(d_)) |
            alloc(gs->base, 3 * (size_t)mm) | alloc(gs->rot, 12 * (size_t)mm) | alloc(gs->grad, 3 * (size_t)mm);
  if (bad) {
    cudaGetLastError();
    free_grad_state(gs);
    set_last_error("out of device memory for the polarization gradient");
    return kErrMemory;
  }
  auto up = [&](void *dst, const void *src, size_t bytes) {
    if (bytes) cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st_);
  };
  if (amoeba) up(gs->q0, m_.q0.data(), 10 * (size_t)mm * sizeof(double));
  up(gs->frame, fr.data(), mm * sizeof(int4));
  up(gs->mm_polar, m_.mm_polar.data(), mm * sizeof(int));
  std::vector<unsigned> polar((mm + 31) / 32, 0u);
  for (int i = 0; i < mm; ++i)
    if (m_.mm_polar[i] >= 0) polar[i / 32] |= 1u << (i % 32);
  up(gs->polar, polar.data(), polar.size() * sizeof(unsigned));
  up(gs->t_ri, t_ri.data(), t_ri.size() * sizeof(int));
  up(gs->t_src, t_src.data(), t_src.size() * sizeof(int));
  up(gs->t_sP, t_sP.data(), t_sP.size() * sizeof(double));
  up(gs->t_sD, t_sD.data(), t_sD.size() * sizeof(double));
  up(gs->r_ri, r_ri.data(), r_ri.size() * sizeof(int));
  up(gs->r_src, r_src.data(), r_src.size() * sizeof(int));
  st = check(cudaStreamSynchronize(st_), "gradient setup");  // host vectors die here
  if (st) {
    free_grad_state(gs);
    return st;
  }
  grad_ = gs;
  return kOk;
}

int System::polelec_geomgrad(double *grad_h) {
  const int mm = d_.m, n = d_.n;
  std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
  if (n == 0) return kOk;
  int st;
  if (!ipd_done_) {
    st = ensure_m2d();
    if (st) return st;
    st = polarization(e_m2d_, kSolverNone, kMatvNone, nullptr);
    if (st) return st;
  }
  const bool amoeba = m_.amoeba;
  st = ensure_grad_state();
  if (st) return st;
  GradState &gs = *grad_;
  gpu::GradArgs a{};
  a.mm = mm;
  a.n = n;
  a.mm_pos = d_.mm_pos;
  a.mm_a = d_.mm_a;
  a.mm_q = d_.mm_q;
  a.mm_polar = gs.mm_polar;
  a.polar_mm = d_.polar_mm;
  a.ipd = ipd_;
  a.m2d_ri = d_.m2d_ri;
  a.m2d_src = d_.m2d_src;
  a.m2d_sP = d_.m2d_sP;
  a.m2d_sD = d_.m2d_sD;
  a.d2d_ri = d_.d2d_ri;
  a.d2d_src = d_.d2d_src;
  a.d2d_s = d_.d2d_s;
  a.t_ri = gs.t_ri;
  a.t_src = gs.t_src;
  a.t_sP = gs.t_sP;
  a.t_sD = gs.t_sD;
  a.q0 = gs.q0;
  a.frame = gs.frame;
  a.r_ri = gs.r_ri;
  a.r_src = gs.r_src;
  a.lo = reinterpret_cast<const unsigned long long *>(gs.sums);
  a.hi = a.lo + (size_t)(amoeba ? 6 : 3) * mm;
  a.bad = a.hi + (size_t)(amoeba ? 6 : 3) * mm;
  a.base = gs.base;
  a.rot = gs.rot;
  a.grad = gs.grad;
  a.thr = d_.damp_thr;
  a.err = flag_;
  cudaMemsetAsync(flag_, 0, sizeof(int), st_);
  const int tb = (mm + gpu::GTPB - 1) / gpu::GTPB;
  KEv ev{};
  if (ktime_on_) ev = kt_begin(3, 1);
  gpu::launch_grad_sym(d_, ipd_, gs.mm_polar, gs.polar, gs.sums, flag_, st_);
  if (ktime_on_) kt_end(ev);
  if (amoeba)
    gpu::k_grad_finish<true><<<tb, gpu::GTPB, 0, st_>>>(a);
  else
    gpu::k_grad_finish<false><<<tb, gpu::GTPB, 0, st_>>>(a);
  gpu::k_grad_gather<<<(mm + 255) / 256, 256, 0, st_>>>(mm, amoeba, gs.base, gs.rot, gs.r_ri, gs.r_src, gs.grad);
  gpu::add_launch_count(2);
  int flag = 0;
  cudaMemcpyAsync(grad_h, gs.grad, 3 * (size_t)mm * sizeof(double), cudaMemcpyDeviceToHost, st_);
  cudaMemcpyAsync(&flag, flag_, sizeof(int), cudaMemcpyDeviceToHost, st_);
  st = check(cudaStreamSynchronize(st_), "polarization gradient");
  if (st) return st;
  if (flag & 1) {
    std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
    set_last_error(
        "Requesting Coulomb kernel for two atoms placed in the same point, this could be an internal bug or "
        "a problem in your input file, please check.");
    return kErrNumeric;
  }
  if (flag & 2) {
    std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
    set_last_error("Ill defined rotation axis (either u or v vectors have 0 norm.");
    return kErrInput;
  }
  return kOk;
}

// gradient = base [mm][3] + the frame forces of the static multipoles in E
// [mm][3] and field gradient G [mm][6] (device arrays), copied to grad_h
int System::frame_forces(const double *E, const double *G, const double *base, double *grad_h) {
  const int mm = d_.m;
  int st = ensure_grad_state();
  if (st) return st;
  GradState &gs = *grad_;
  const bool amoeba = m_.amoeba;
  cudaMemsetAsync(flag_, 0, sizeof(int), st_);
  if (amoeba) gpu::k_rot_terms<<<(mm + 127) / 128, 128, 0, st_>>>(mm, d_.mm_pos, gs.frame, gs.q0, E, G, gs.rot, flag_);
  gpu::k_grad_gather<<<(mm + 255) / 256, 256, 0, st_>>>(mm, amoeba, base, gs.rot, gs.r_ri, gs.r_src, gs.grad);
  gpu::add_launch_count(amoeba ? 2 : 1);
  int flag = 0;
  cudaMemcpyAsync(grad_h, gs.grad, 3 * (size_t)mm * sizeof(double), cudaMemcpyDeviceToHost, st_);
  cudaMemcpyAsync(&flag, flag_, sizeof(int), cudaMemcpyDeviceToHost, st_);
  st = check(cudaStreamSynchronize(st_), "frame forces");
  if (st) return st;
  if (flag & 2) {
    std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
    set_last_error("Ill defined rotation axis (either u or v vectors have 0 norm.");
    return kErrInput;
  }
  return kOk;
}

int System::rotation_geomgrad(const double *E_h, const double *G_h, double *grad_h) {
  const int mm = d_.m;
  std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
  if (mm == 0 || !m_.amoeba) return kOk;  // point charges have no frame
  int st = ensure_grad_state();
  if (st) return st;
  GradState &gs = *grad_;
  // E, G staged in the pair pass's buffer (18 mm doubles for AMOEBA), zero base
  double *E = gs.sums, *G = gs.sums + 3 * (size_t)mm;
  cudaMemcpyAsync(E, E_h, 3 * (size_t)mm * sizeof(double), cudaMemcpyHostToDevice, st_);
  cudaMemcpyAsync(G, G_h, 6 * (size_t)mm * sizeof(double), cudaMemcpyHostToDevice, st_);
  cudaMemsetAsync(gs.base, 0, 3 * (size_t)mm * sizeof(double), st_);
  return frame_forces(E, G, gs.base, grad_h);
}

}  // namespace ommp
