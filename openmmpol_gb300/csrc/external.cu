// Potential and field of the system at arbitrary points (QM coupling).
//
// potential_M2E / potential_D2E / field_M2E / field_D2E of the reference
// (src/mod_electrostatics.F90:3067-3336) behind ommp_{potential,field}_
// {mmpol,mm,pol}2ext (src/mod_interface.F90:250-330): every static site's
// multipoles (charge, dipole, quadrupole for AMOEBA; charge for Wang-AL) and
// every induced dipole act on every point, with the undamped Coulomb kernel
// and no screening.  The induced dipoles seen from outside are the D set for
// the potential and (P + D) / 2 for the field (AMOEBA), the single set
// otherwise.  The results are ADDED into the caller's array, as the
// reference's routines do.
//
// The sums were FP64-bound: at 20,001 points and 9,000 sites 12.8 ms for the
// static multipoles and 6.3 ms for the induced dipoles.  They run in
// double-single on the FP32 pipes (ds_pair.cuh; about 350 FP32 operations per
// point and AMOEBA site), static and induced dipole of a site added first so
// that one pass serves both.  Points and sites are split on one grid per call,
// which covers the sites and the points within kGridReach of the first one;
// points beyond (or not finite) take FP64 for all their sources and leave the
// resolution to the others (so do all points of a system as wide as that).  One thread owns a point, sources stream through shared memory in tiles of
// 128; pairs closer than 5 bohr go to a list of the point's own and are formed
// in FP64 by its thread.  The source range is split over blockIdx.y (quarters
// of a tile: a few QM nuclei alone fill the GPU) and the partials are summed in
// a fixed order: deterministic.
//
// Built with --fmad=false -ftz=true: every FMA of a pair is explicit.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ds_pair.cuh"
#include "engine.h"
#include "log.h"

namespace ommp {
namespace gpu {
namespace {

constexpr int NT = 128;
constexpr int NLIST = 24;       // listed sources per point before they are formed
constexpr float CLOSE2 = 25.f;  // bohr^2

// values of a source: q, dipole (3), with QUAD the quadrupole (6)
template <bool QUAD>
struct ExtRec {
  static constexpr int NV = QUAD ? 10 : 4;
  static constexpr int R = (9 + 2 * NV + 3) / 4;
};

// x - c as three floats on the grid g1, g1 2^-23 (launch_split)
__device__ __forceinline__ void split3(double v, double g1, float *o) {
  const double g2 = g1 * 1.1920928955078125e-7;
  const double h = rint(v / g1) * g1, m = rint((v - h) / g2) * g2;
  o[0] = (float)h;
  o[3] = (float)m;
  o[6] = (float)((v - h) - m);
}

struct ExtArgs {
  int n, m;            // points, sources
  const double *cext;
  const Pos64 *pos;    // sources
  const double *q;     // [m][ld] multipoles, or null (induced dipoles alone)
  int ld;
  const int *polar;    // [m] polarizable index of a source or -1; null: the source itself
  const double *mu, *mu2;  // induced dipoles added (null: none) and a second set averaged with them
  double c[3], g1, reach;  // the grid: origin, step, width
  const unsigned *word;  // scale of the dipoles, or null
  double *val;         // [m][NV] FP64 values
  float4 *rec;         // [R][m]
};

template <bool QUAD>
__global__ void k_ext_sources(ExtArgs a) {
  constexpr int NV = ExtRec<QUAD>::NV, R = ExtRec<QUAD>::R;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.m) return;
  double v[NV];
  for (int c = 0; c < NV; ++c) v[c] = a.q && c < a.ld ? a.q[(size_t)i * a.ld + c] : 0.0;
  const int p = a.mu ? (a.polar ? a.polar[i] : i) : -1;
  if (p >= 0) {
    const int ex = a.word ? dsp_exponent(*a.word) : 0;
    for (int c = 0; c < 3; ++c) {
      const double d = a.mu[3 * (size_t)p + c];
      v[1 + c] += scale_down(a.mu2 ? 0.5 * (a.mu2[3 * (size_t)p + c] + d) : d, ex);
    }
  }
  const Pos64 x = a.pos[i];
  float f[4 * R] = {};
  split3(x.x - a.c[0], a.g1, f);
  split3(x.y - a.c[1], a.g1, f + 1);
  split3(x.z - a.c[2], a.g1, f + 2);
  for (int c = 0; c < NV; ++c) {
    a.val[(size_t)i * NV + c] = v[c];
    const dsf d = to_ds(v[c]);
    f[9 + 2 * c] = d.h;
    f[10 + 2 * c] = d.l;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) a.rec[(size_t)r * a.m + i] = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
}

// partial[split][n][C] (C = 1 potential, 3 field)
template <bool FIELD, bool QUAD>
__global__ void __launch_bounds__(NT, 4) k_ext(const __grid_constant__ ExtArgs a, double *__restrict__ partial,
                                               int per_split, int *bad_flag) {
  constexpr int NV = ExtRec<QUAD>::NV, R = ExtRec<QUAD>::R, C = FIELD ? 3 : 1;
  __shared__ float4 s_rec[R][NT];
  __shared__ int s_list[NLIST][NT];
  const int j = blockIdx.x * NT + threadIdx.x;
  const bool valid = j < a.n;
  const int tj = valid ? j : a.n - 1;
  const double px = a.cext[3 * (size_t)tj], py = a.cext[3 * (size_t)tj + 1], pz = a.cext[3 * (size_t)tj + 2];
  float tg[9];
  const bool outside = !(fmax(fabs(px - a.c[0]), fmax(fabs(py - a.c[1]), fabs(pz - a.c[2]))) <= a.reach) ||
                       isnan(px) || isnan(py) || isnan(pz);
  split3(outside ? 0.0 : px - a.c[0], a.g1, tg);
  split3(outside ? 0.0 : py - a.c[1], a.g1, tg + 1);
  split3(outside ? 0.0 : pz - a.c[2], a.g1, tg + 2);
  double sum[C];
#pragma unroll
  for (int c = 0; c < C; ++c) sum[c] = 0.0;
  int listed = 0, bad = 0;
  // the listed pairs in FP64
  auto form = [&]() {
    for (int e = 0; e < listed; ++e) {
      const int i = s_list[e][threadIdx.x];
      const Pos64 ps = a.pos[i];
      const double dx = px - ps.x, dy = py - ps.y, dz = pz - ps.z;
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      if (r2 < 4.930380657631324e-28) {  // |r| < 100 eps: the reference stops here
        bad = 1;
        continue;
      }
      const double *q = a.val + (size_t)i * NV;
      const double k1 = rinv_f64(r2, r2_f32(r2)), ir2 = k1 * k1, k3 = k1 * ir2, k5 = k3 * ir2;
      const double md = fma(q[1], dx, fma(q[2], dy, q[3] * dz));
      double tx = 0.0, ty = 0.0, tz = 0.0, s = 0.0;
      if (QUAD) {
        tx = fma(q[4], dx, fma(q[5], dy, q[7 % NV] * dz));
        ty = fma(q[5 % NV], dx, fma(q[6 % NV], dy, q[8 % NV] * dz));
        tz = fma(q[7 % NV], dx, fma(q[8 % NV], dy, q[9 % NV] * dz));
        s = fma(tx, dx, fma(ty, dy, tz * dz));
      }
      if (!FIELD) {
        sum[0] += fma(q[0], k1, fma(md, k3, 3.0 * s * k5));
      } else {
        const double c = fma(q[0], k3, fma(3.0 * md, k5, 15.0 * s * (k5 * ir2)));
        const double k6 = 6.0 * k5;
        sum[0] += fma(c, dx, -fma(q[1], k3, k6 * tx));
        sum[C > 1 ? 1 : 0] += fma(c, dy, -fma(q[2], k3, k6 * ty));
        sum[C > 2 ? 2 : 0] += fma(c, dz, -fma(q[3], k3, k6 * tz));
      }
    }
    listed = 0;
  };
  const int s0 = blockIdx.y * per_split, s1 = min(a.m, s0 + per_split);
  for (int t0 = s0; t0 < s1; t0 += NT) {
    const int cnt = min(NT, s1 - t0);
    __syncthreads();
    if (threadIdx.x < cnt)
#pragma unroll
      for (int r = 0; r < R; ++r) s_rec[r][threadIdx.x] = a.rec[(size_t)r * a.m + t0 + threadIdx.x];
    __syncthreads();
    dsf acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = dsf{0.f, 0.f};
#pragma unroll 1
    for (int k = 0; k < cnt; ++k) {
      float f[4 * R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 v = s_rec[r][k];
        f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
      }
      float sc[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) sc[c] = f[c];
      const DspDelta d = dsp_delta(tg, sc);
      float y = d.ri;
      if (outside || !(d.r2 >= CLOSE2)) {
        y = 0.f;
        if (listed == NLIST) form();
        s_list[listed++][threadIdx.x] = t0 + k;
      }
      auto q = [&](int c) { return dsf{f[9 + 2 * c], f[10 + 2 * c]}; };
      // the charges cancel between sites: their factor is kept to 2^-48
      const DspUnit n = dsp_unit<true>(d, y);
      const float w3 = dsp_power<3>(n.eps), w5 = dsp_power<5>(n.eps);
      const float y2 = y * y, y2l = fmaf(y, y, -y2);
      const float y3 = y2 * y, y3l = fmaf(y2l, y, fmaf(y2, y, -y3));
      const dsf m = dsp_dot(q(1), q(2), q(3), n.x, n.y, n.z);
      dsf t[3], nqn{0.f, 0.f};
      if (QUAD) {
        t[0] = dsp_norm(dsp_dot(q(4), q(5), q(7), n.x, n.y, n.z));
        t[1] = dsp_norm(dsp_dot(q(5), q(6), q(8), n.x, n.y, n.z));
        t[2] = dsp_norm(dsp_dot(q(7), q(8), q(9), n.x, n.y, n.z));
        nqn = dsp_dot(t[0], t[1], t[2], n.x, n.y, n.z);
      }
      if (!FIELD) {
        const dsf V = dsp_scaled<1>(y, 0.f, n);
        dsp_acc(acc[0], V, q(0));
        dsp_acc(acc[0], dsf{y2, fmaf(y2, w3, y2l)}, m);
        if (QUAD) dsp_acc(acc[0], dsp_coef(3.f, y3, y3l, w5), nqn);
      } else {
        const dsf K = {-y3, -fmaf(y3, w3, y3l)};
        dsf c = dsp_mul(dsp_scaled<3>(y2, y2l, n), q(0));
        dsp_acc(c, dsp_coef(3.f, y3, y3l, w5), m);
        if (QUAD) {
          const float y4 = y3 * y, y4l = fmaf(y3l, y, fmaf(y3, y, -y4));
          dsp_acc(c, dsp_coef(15.f, y4, y4l, dsp_power<7>(n.eps)), nqn);
          const dsf H = dsp_coef(-6.f, y4, y4l, w5);
#pragma unroll
          for (int u = 0; u < C; ++u) dsp_acc(acc[u], H, t[u]);
        }
        c = dsp_norm(c);
        const dsf nn[3] = {n.x, n.y, n.z};
#pragma unroll
        for (int u = 0; u < C; ++u) {
          dsp_acc(acc[u], c, nn[u]);
          dsp_acc(acc[u], K, q(1 + u));
        }
      }
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = dsp_norm(acc[c]);
      if (!FIELD && (k & 3) == 3) {
        // the potential is a small remainder of the charges' partial sums:
        // they go into the FP64 sum every four sources (error of a Wang-AL
        // system's potential 1.0e-14 with whole tiles)
        sum[0] += (double)acc[0].h + (double)acc[0].l;
        acc[0] = dsf{0.f, 0.f};
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) sum[c] += (double)acc[c].h + (double)acc[c].l;
  }
  form();
  if (!valid) return;
  if (bad) atomicOr(bad_flag, 1);
#pragma unroll
  for (int c = 0; c < C; ++c) partial[((size_t)blockIdx.y * a.n + j) * C + c] = sum[c];
}

// out[j][c] = sum over the nsplit partial blocks, in order, scaled back
__global__ void k_ext_sum(size_t total, int nsplit, const double *__restrict__ partial, const unsigned *word,
                          double *__restrict__ out) {
  const int ex = word ? dsp_exponent(*word) : 0;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int p = 0; p < nsplit; ++p) s += partial[(size_t)p * total + k];
    out[k] = scale_up(s, ex);
  }
}

int blocks_for_ext(size_t n) {
  size_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 2432) b = 2432;
  return (int)b;
}

// about four waves of CTAs, at least 32 sources per split
int ext_split(int n, int m, int sms) {
  const int blocks = (n + NT - 1) / NT;
  return std::max(1, std::min((m + 31) / 32, (16 * sms + blocks - 1) / blocks));
}

template <bool QUAD>
void launch_ext(bool field, const ExtArgs &a, double *partial, int nsplit, int *bad, cudaStream_t st) {
  const int per = ((a.m + nsplit - 1) / nsplit + 31) / 32 * 32;
  const dim3 grid((a.n + NT - 1) / NT, nsplit);
  add_launch_count(2);
  k_ext_sources<QUAD><<<(a.m + 127) / 128, 128, 0, st>>>(a);
  if (field)
    k_ext<true, QUAD><<<grid, NT, 0, st>>>(a, partial, per, bad);
  else
    k_ext<false, QUAD><<<grid, NT, 0, st>>>(a, partial, per, bad);
}

}  // namespace
}  // namespace gpu

int System::ext_props(int which, bool field, int n, const double *cext_h, double *out_h) {
  if (which < 0 || which > 2 || n < 0) {
    set_last_error("external points: 'which' must be 0 (all), 1 (static) or 2 (induced), n >= 0");
    return kErrBadArg;
  }
  const bool do_mm = which != 2 && d_.m > 0, do_pol = which != 1 && d_.n > 0;
  if (do_pol && !ipd_done_) {
    set_last_error(field ? "IPD should be computed before computing D2E field."
                         : "IPD should be computed before D2E potential.");
    return kErrInput;
  }
  if (n == 0 || (!do_mm && !do_pol)) return kOk;
  const int C = field ? 3 : 1;
  // sources: the static sites (with the induced dipoles of the polarizable
  // ones), or the polarizable sites alone
  const int m = do_mm ? d_.m : d_.n;
  const bool quad = do_mm && m_.amoeba;
  const int nsplit = gpu::ext_split(n, m, gpu::sm_count());
  const size_t nval = quad ? gpu::ExtRec<true>::NV : gpu::ExtRec<false>::NV;
  const size_t nrec = quad ? gpu::ExtRec<true>::R : gpu::ExtRec<false>::R;
  const size_t need = 3 * (size_t)n + (size_t)(nsplit + 1) * n * C + (size_t)m * (nval + 2 * nrec) +
                      ((size_t)m + 1) / 2 + 4;
  if (need > ext_cap_) {
    if (ext_buf_) cudaFree(ext_buf_);
    ext_buf_ = nullptr;
    ext_cap_ = 0;
    if (cudaMalloc((void **)&ext_buf_, need * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      set_last_error("out of device memory for the external points");
      return kErrMemory;
    }
    ext_cap_ = need;
  }
  // the source records first: 16-byte aligned
  gpu::ExtArgs a{};
  a.rec = reinterpret_cast<float4 *>(ext_buf_);
  a.val = ext_buf_ + 2 * nrec * m;
  double *cext = a.val + nval * m;
  double *partial = cext + 3 * (size_t)n;
  double *out = partial + (size_t)nsplit * n * C;
  unsigned *word = reinterpret_cast<unsigned *>(out + (size_t)n * C);
  int *polar = reinterpret_cast<int *>(word + 2);
  a.n = n, a.m = m;
  a.cext = cext;
  a.pos = do_mm ? d_.mm_pos : d_.pol_pos;
  a.q = do_mm ? d_.mm_q : nullptr;
  a.ld = d_.ld;
  if (do_pol) {
    // the D set for the potential, the mean of both for the field (AMOEBA)
    a.mu = ipd_;
    a.mu2 = field && m_.amoeba ? ipd_ + 3 * (size_t)d_.n : nullptr;
    if (do_mm) {
      a.polar = polar;
      cudaMemcpyAsync(polar, m_.mm_polar.data(), (size_t)m * sizeof(int), cudaMemcpyHostToDevice, st_);
    }
  }
  // one grid for the points and the sites: about the first site, rounded to
  // whole bohr (an exact shift), as wide as the farthest site or point within
  // kGridReach
  double big = 1.0;
  for (int c = 0; c < 3; ++c) a.c[c] = std::nearbyint(m_.cmm[c]);
  for (int i = 0; i < d_.m; ++i)
    for (int c = 0; c < 3; ++c) {
      const double v = std::fabs(m_.cmm[3 * (size_t)i + c] - a.c[c]);
      if (v > big && std::isfinite(v)) big = v;
    }
  const double reach = std::max(big, gpu::kGridReach);
  for (size_t k = 0; k < 3 * (size_t)n; ++k) {
    const double v = std::fabs(cext_h[k] - a.c[k % 3]);
    if (v > big && v <= reach) big = v;
  }
  int e = 0;
  std::frexp(big, &e);
  a.g1 = std::ldexp(1.0, e - 23);
  a.reach = big > gpu::kGridReach ? -1.0 : big;
  cudaMemcpyAsync(cext, cext_h, 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice, st_);
  cudaMemsetAsync(flag_, 0, sizeof(int), st_);
  if (!do_mm) {
    a.word = word;
    gpu::launch_max_word((a.mu2 ? 2 : 1) * 3 * (size_t)d_.n, ipd_, word, st_);
  }
  if (quad)
    gpu::launch_ext<true>(field, a, partial, nsplit, flag_, st_);
  else
    gpu::launch_ext<false>(field, a, partial, nsplit, flag_, st_);
  const int left = gpu::launch_sum_splits((size_t)n * C, nsplit, partial, st_);
  gpu::k_ext_sum<<<gpu::blocks_for_ext((size_t)n * C), 256, 0, st_>>>((size_t)n * C, left, partial, a.word, out);
  gpu::add_launch_count(1);
  std::vector<double> h((size_t)n * C);
  int flag = 0;
  cudaMemcpyAsync(h.data(), out, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st_);
  cudaMemcpyAsync(&flag, flag_, sizeof(int), cudaMemcpyDeviceToHost, st_);
  int st = check(cudaStreamSynchronize(st_), "external points");
  if (st) return st;
  if (flag) {
    set_last_error(
        "Requesting Coulomb kernel for two atoms placed in the same point, this could be an internal bug or "
        "a problem in your input file, please check.");
    return kErrNumeric;
  }
  for (size_t k = 0; k < h.size(); ++k) out_h[k] += h[k];
  return kOk;
}

}  // namespace ommp
