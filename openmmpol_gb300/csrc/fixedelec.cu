// Interaction energy of the static multipoles, ommp_get_fixedelec_energy
// (energy_MM_MM, src/mod_electrostatics.F90:899-941, on elec_prop_M2M's
// direct path :1678-1952 with the m-scaled pair list list_S_S :597-648).
//
//   k_m2m          (m2m.cu) per static target, unscaled sums over every other
//                  static site of the potential, field and field gradient of
//                  its multipoles (undamped: the static-static interaction has
//                  no Thole damping), split over source ranges
//   k_m2m_finish   partials summed in a fixed order, the m-scaled pairs
//                  corrected by (s - 1) times their terms, and the site's
//                  energy term q V - mu.E + Q:G (the off-diagonal quadrupole
//                  components counted twice)
// The energy is half the sum of the site terms, added on the host in site
// order (deterministic).  Computed once per geometry.
//
// Gradient, ommp_fixedelec_geomgrad (fixedelec_geomgrad,
// src/mod_geomgrad.F90:17-111, on elec_prop_M2M with field gradients and
// Hessians): the same two kernels with the GRAD flag accumulate per static
// target the field E, the field gradient G and h_a = sum_bc Q_bc H_bca, the
// field Hessian H of all other static multipoles contracted with the
// target's own quadrupole Q (the reference's q/mu/quad_elec_prop Hessians,
// :1097-1405, as closed tensor expressions).  The finish writes E, G and
// the site term -q E + mu.G - h; the frame forces of the rotated multipoles
// in E and G (rotation_geomgrad) are added by the polarization gradient's
// frame kernels.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ds_pair.cuh"
#include "engine.h"
#include "grad_math.cuh"
#include "m2m_math.cuh"

namespace ommp {

namespace gpu {
namespace {

struct M2mArgs {
  int mm, nsplit;
  int ex;  // the multipoles are scaled by 2^-ex
  const Pos64 *pos;
  const double *q;
  const int *ri, *src;
  const double *sc;
  double *partial;  // [nsplit][NV][mm]
  double *site;     // [mm] energy terms
  double *E, *G;    // [mm][3], [mm][6] field and field gradient (gradient pass)
  double *base;     // [mm][3] site gradient terms (gradient pass)
};

// Multipoles far from one, scaled by a power of two for the passes: products of
// two quadrupoles and r^-11 would leave the range of the FP32 pair pass (3e-10 of
// the gradient at 1e-12, 1e-3 at 1e-18).  The finishing pass scales back.  (Scaling
// in the pair kernel cost it 4 % at 30,000 sites for every system.)
__global__ void k_m2m_scale(int total, const double *__restrict__ q, int ex, double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) out[i] = scale_down(q[i], ex);
}

template <bool AMOEBA, bool GRAD>
__global__ void k_m2m_finish(M2mArgs a) {
  constexpr int LD = AMOEBA ? 10 : 1;
  constexpr int NV = M2mNV<AMOEBA, GRAD>::N;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.mm) return;
  double Qt[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (GRAD && AMOEBA)
    for (int c = 0; c < 6; ++c) Qt[c] = a.q[(size_t)t * LD + 4 + c];
  const double trq = Qt[0] + Qt[2] + Qt[5];
  double acc[NV];
  for (int c = 0; c < NV; ++c) {
    double s = 0.0;
    for (int p = 0; p < a.nsplit; ++p) s += a.partial[((size_t)p * NV + c) * a.mm + t];
    acc[c] = s;
  }
  const Pos64 pt = a.pos[t];
  for (int k = a.ri[t]; k < a.ri[t + 1]; ++k) {
    const int i = a.src[k];
    const Pos64 ps = a.pos[i];
    const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 < 4.9e-28) continue;  // flagged by the pair pass
    m2m_any<AMOEBA, GRAD>(&a.q[(size_t)i * LD], dx, dy, dz, 1.0 / sqrt(r2), a.sc[k] - 1.0, Qt, trq, acc);
  }
  const double *q = &a.q[(size_t)t * LD];
  auto back = [&](double v) { return scale_up(v, a.ex); };
  if (GRAD) {
    double g[3];
    for (int c = 0; c < 3; ++c) {
      a.E[3 * (size_t)t + c] = back(acc[c]);
      g[c] = -q[0] * acc[c];
    }
    if (AMOEBA) {
      double mg[3];
      gradmath::sym_apply(acc + 3, q + 1, mg);
      for (int c = 0; c < 6; ++c) a.G[6 * (size_t)t + c] = back(acc[3 + c]);
      for (int c = 0; c < 3; ++c) g[c] += mg[c] - acc[9 + c];
    }
    for (int c = 0; c < 3; ++c) a.base[3 * (size_t)t + c] = back(back(g[c]));
    return;
  }
  double e = q[0] * acc[0];
  if (AMOEBA) {
    e -= q[1] * acc[1] + q[2] * acc[2] + q[3] * acc[3];
    const double *g = acc + (GRAD ? 3 : 4);
    e += q[4] * g[0] + q[6] * g[2] + q[9] * g[5] + 2.0 * (q[5] * g[1] + q[7] * g[3] + q[8] * g[4]);
  }
  a.site[t] = back(back(e));
}

}  // namespace
}  // namespace gpu

namespace {

// list_S_S: pairs within four bonds whose m-scale is not 1, by target
void build_ss(const HostModel &m, int mm, std::vector<int> &ri, std::vector<int> &src, std::vector<double> &sc) {
  ri.assign(mm + 1, 0);
  src.clear();
  sc.clear();
  for (int i = 0; i < mm; ++i) {
    for (int l = 0; l < 4; ++l)
      for (int k = m.conn[l].ri[i]; k < m.conn[l].ri[i + 1]; ++k) {
        const double s = m.mscale[l];
        if (std::fabs(s - 1.0) > kEpsRp) {
          src.push_back(m.conn[l].ci[k]);
          sc.push_back(s);
        }
      }
    ri[i + 1] = (int)src.size();
  }
}

}  // namespace

// The pair and finish passes of the energy (grad false) or of the gradient
// (grad true: E, G and the site terms into e_out, g_out, base_out, in the kept
// buffer).
int System::m2m_launch(bool grad, double **site_out, double **e_out, double **g_out,
                       double **base_out) {
  const int mm = d_.m;
  const bool amoeba = m_.amoeba;
  const int nv = grad ? (amoeba ? 12 : 3) : (amoeba ? 10 : 1);
  std::vector<int> ri, src;
  std::vector<double> sc;
  build_ss(m_, mm, ri, src, sc);
  const int nsplit = gpu::m2m_pick_split(d_, grad, gpu::sm_count());
  const size_t out = grad ? 12 * (size_t)mm : (size_t)mm;  // E, G, base | site
  const int ex = gpu::scaling_exponent(d_.q_e);
  const size_t scaled = ex ? (size_t)d_.ld * mm : 0;
  const size_t need = (size_t)nsplit * nv * mm + out + ri.size() + 2 * src.size() + 1 + scaled;
  if (need > fe_cap_) {  // kept for the next geometry
    if (fe_buf_) cudaFree(fe_buf_);
    fe_buf_ = nullptr;
    fe_cap_ = 0;
    if (cudaMalloc((void **)&fe_buf_, need * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      fe_buf_ = nullptr;
      set_last_error("out of device memory for the static multipole field");
      return kErrMemory;
    }
    fe_cap_ = need;
  }
  double *buf = fe_buf_;
  gpu::M2mArgs a{};
  a.mm = mm;
  a.nsplit = nsplit;
  a.pos = d_.mm_pos;
  a.q = d_.mm_q;
  a.partial = buf;
  double *o = buf + (size_t)nsplit * nv * mm;
  if (grad) {
    a.E = o;
    a.G = o + 3 * (size_t)mm;
    a.base = o + 9 * (size_t)mm;
  } else {
    a.site = o;
  }
  double *sc_d = o + out;
  int *ri_d = reinterpret_cast<int *>(sc_d + std::max<size_t>(sc.size(), 1));
  int *src_d = ri_d + ri.size();
  a.ri = ri_d;
  a.src = src_d;
  a.sc = sc_d;
  gpu::DevSites d = d_;
  if (scaled) {
    double *q = fe_buf_ + need - scaled;
    gpu::k_m2m_scale<<<(unsigned)((scaled + 255) / 256), 256, 0, st_>>>((int)scaled, d_.mm_q, ex, q);
    gpu::add_launch_count(1);
    d.mm_q = q;
    a.q = q;
    a.ex = ex;
  }
  cudaMemcpyAsync(sc_d, sc.data(), sc.size() * sizeof(double), cudaMemcpyHostToDevice, st_);
  cudaMemcpyAsync(ri_d, ri.data(), ri.size() * sizeof(int), cudaMemcpyHostToDevice, st_);
  cudaMemcpyAsync(src_d, src.data(), src.size() * sizeof(int), cudaMemcpyHostToDevice, st_);
  cudaMemsetAsync(flag_, 0, sizeof(int), st_);
  const int fb = (mm + 127) / 128;
  gpu::launch_m2m(d, grad, buf, nsplit, flag_, st_);
  a.nsplit = gpu::launch_sum_splits((size_t)nv * mm, nsplit, buf, st_);
  if (amoeba && grad)
    gpu::k_m2m_finish<true, true><<<fb, 128, 0, st_>>>(a);
  else if (amoeba)
    gpu::k_m2m_finish<true, false><<<fb, 128, 0, st_>>>(a);
  else if (grad)
    gpu::k_m2m_finish<false, true><<<fb, 128, 0, st_>>>(a);
  else
    gpu::k_m2m_finish<false, false><<<fb, 128, 0, st_>>>(a);
  gpu::add_launch_count(1);
  // host vectors above die at return: wait for their copies
  int flag = 0;
  cudaMemcpyAsync(&flag, flag_, sizeof(int), cudaMemcpyDeviceToHost, st_);
  int st = check(cudaStreamSynchronize(st_), "static multipole field");
  if (st) return st;
  if (flag) {
    set_last_error(
        "Requesting Coulomb kernel for two atoms placed in the same point, this could be an internal bug or "
        "a problem in your input file, please check.");
    return kErrNumeric;
  }
  if (site_out) *site_out = a.site;
  if (e_out) *e_out = a.E;
  if (g_out) *g_out = a.G;
  if (base_out) *base_out = a.base;
  return kOk;
}

int System::fixedelec_energy(double &energy) {
  energy = 0.0;
  const int mm = d_.m;
  if (mm == 0) return kOk;
  if (fixedelec_done_) {
    energy = fixedelec_;
    return kOk;
  }
  double *site_d = nullptr;
  int st = m2m_launch(false, &site_d, nullptr, nullptr, nullptr);
  if (st) return st;
  std::vector<double> site(mm);
  cudaMemcpyAsync(site.data(), site_d, mm * sizeof(double), cudaMemcpyDeviceToHost, st_);
  st = check(cudaStreamSynchronize(st_), "static multipole energy");
  if (st) return st;
  double e = 0.0;
  for (int t = 0; t < mm; ++t) e += site[t];
  fixedelec_ = 0.5 * e;
  fixedelec_done_ = true;
  energy = fixedelec_;
  return kOk;
}

int System::fixedelec_geomgrad(double *grad_h) {
  const int mm = d_.m;
  std::fill(grad_h, grad_h + 3 * (size_t)mm, 0.0);
  if (mm == 0) return kOk;
  if (fixedelec_grad_done_) {
    std::copy(fixedelec_grad_.begin(), fixedelec_grad_.end(), grad_h);
    return kOk;
  }
  double *E = nullptr, *G = nullptr, *base = nullptr;
  int st = m2m_launch(true, nullptr, &E, &G, &base);
  if (st) return st;
  st = frame_forces(E, G, base, grad_h);  // synchronises the stream
  if (st) return st;
  fixedelec_grad_.assign(grad_h, grad_h + 3 * (size_t)mm);
  fixedelec_grad_done_ = true;
  return kOk;
}

}  // namespace ommp
