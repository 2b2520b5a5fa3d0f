// All-pairs sums of the static-static interaction (elec_prop_M2M,
// src/mod_electrostatics.F90:1678-1952): per static target the potential,
// field and field gradient of every other static multipole (energy), or the
// field, field gradient and contracted field Hessian (gradient), unscaled.
//
// The sums were FP64-bound (6.6 and 13.7 ms at 6,000 sites).  They run in
// double-single on the FP32 pipes with the formulas of m2m_math.cuh and exact
// coordinate differences; pairs closer than 5 bohr (the excluded ones among
// them are the largest terms and have to cancel) go to a list of the target's
// own and are formed in FP64 by its thread.  Per tile the double-single sums
// are added to FP64 ones; partial [split][component][site].  6,000 sites:
// 1.09 and 2.27 ms (1.52 and 3.36 with every product and sum renormalised, for
// gradient errors of 2e-14 instead of 3.4e-14; 1.7e-13 in FP64 before).  80 % of
// the FP32 issue slots.
//
// Built with --fmad=false -ftz=true like the other double-single kernels.
#include <algorithm>

#include "ds_math.cuh"
#include "kernels.h"
#include "m2m_math.cuh"
#include "pair_math.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int NT = 128;
constexpr int NLIST = 16;       // listed sources per target before they are formed
constexpr float CLOSE2 = 25.f;  // bohr^2

template <bool AMOEBA, bool GRAD>
__device__ __noinline__ void m2m_close(const DevSites &s, int t, int i, double *sum, int &bad) {
  constexpr int LD = AMOEBA ? 10 : 1;
  const Pos64 pt = s.mm_pos[t], ps = s.mm_pos[i];
  const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  if (coincident(r2)) {
    bad = 1;
    return;
  }
  double q[LD], Q[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < LD; ++c) q[c] = s.mm_q[(size_t)i * LD + c];
  if (AMOEBA)
    for (int c = 0; c < 6; ++c) Q[c] = s.mm_q[(size_t)t * LD + 4 + c];
  m2m_any<AMOEBA, GRAD>(q, dx, dy, dz, rinv_f64(r2, r2_f32(r2)), 1.0, Q, Q[0] + Q[2] + Q[5], sum);
}

template <bool AMOEBA, bool GRAD>
__global__ void __launch_bounds__(NT) k_m2m(const __grid_constant__ DevSites s, double *__restrict__ partial,
                                            int per_split, int *err) {
  constexpr int LD = AMOEBA ? 10 : 1;
  constexpr int NV = M2mNV<AMOEBA, GRAD>::N;
  __shared__ float4 s_ph[NT], s_pm[NT], s_pl[NT];
  __shared__ float s_qh[NT * LD], s_ql[NT * LD];
  __shared__ int s_list[NLIST][NT];
  const int t = blockIdx.x * NT + threadIdx.x;
  const bool valid = t < s.m;
  const int tc = valid ? t : s.m - 1;
  const float4 th = s.mm_split[tc], td = s.mm_split[(size_t)s.m + tc], tl = s.mm_split[2 * (size_t)s.m + tc];
  dsf Q[6], trq{0.f, 0.f};
  if (GRAD && AMOEBA) {
#pragma unroll
    for (int c = 0; c < 6; ++c) Q[c] = to_ds(s.mm_q[(size_t)tc * LD + 4 + c]);
    trq = Q[0] + Q[2] + Q[5];
  }
  double sum[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) sum[c] = 0.0;
  int bad = 0, listed = 0;
  auto form = [&]() {
    for (int q = 0; q < listed; ++q) m2m_close<AMOEBA, GRAD>(s, tc, s_list[q][threadIdx.x], sum, bad);
    listed = 0;
  };
  const int s0 = blockIdx.y * per_split, s1 = min(s.m, s0 + per_split);
  for (int t0 = s0; t0 < s1; t0 += NT) {
    __syncthreads();
    const int i = t0 + threadIdx.x;
    if (i < s1) {
      s_ph[threadIdx.x] = s.mm_split[i];
      s_pm[threadIdx.x] = s.mm_split[(size_t)s.m + i];
      s_pl[threadIdx.x] = s.mm_split[2 * (size_t)s.m + i];
#pragma unroll
      for (int c = 0; c < LD; ++c) {
        const dsf q = to_ds(s.mm_q[(size_t)i * LD + c]);
        s_qh[threadIdx.x * LD + c] = q.h;
        s_ql[threadIdx.x * LD + c] = q.l;
      }
    }
    __syncthreads();
    const int cnt = min(NT, s1 - t0);
    dsf acc[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) acc[c] = dsf{0.f, 0.f};
#pragma unroll 1
    for (int k = 0; k < cnt; ++k) {
      const float4 ph = s_ph[k], pm = s_pm[k], pl = s_pl[k];
      const dsf dx = ds_delta(th.x, td.x, tl.x, ph.x, pm.x, pl.x);
      const dsf dy = ds_delta(th.y, td.y, tl.y, ph.y, pm.y, pl.y);
      const dsf dz = ds_delta(th.z, td.z, tl.z, ph.z, pm.z, pl.z);
      if (s.wide || !(fmaf(dx.h, dx.h, fmaf(dy.h, dy.h, dz.h * dz.h)) >= CLOSE2)) {
        if (t0 + k != tc) {
          if (listed == NLIST) form();
          s_list[listed++][threadIdx.x] = t0 + k;
        }
        continue;
      }
      const dsf rinv = ds_rsqrt(dx * dx + dy * dy + dz * dz);
      dsf q[LD];
#pragma unroll
      for (int c = 0; c < LD; ++c) q[c] = dsf{s_qh[k * LD + c], s_ql[k * LD + c]};
      m2m_any<AMOEBA, GRAD>(q, dx, dy, dz, rinv, gradmath::One{}, Q, trq, acc);
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) sum[c] += (double)acc[c].h + (double)acc[c].l;
  }
  form();
  if (!valid) return;
  if (bad) atomicOr(err, 1);
#pragma unroll
  for (int c = 0; c < NV; ++c) partial[((size_t)blockIdx.y * NV + c) * s.m + t] = sum[c];
}

template <bool AMOEBA, bool GRAD>
int resident() {
  static const int r = [] {
    int v = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_m2m<AMOEBA, GRAD>, NT, 0);
    return v < 1 ? 1 : v;
  }();
  return r;
}

}  // namespace

// Source splits (whole quarters of a tile, so that small systems spread over
// the SMs): about four waves of CTAs.
int m2m_pick_split(const DevSites &s, bool grad, int sms) {
  const int r = s.amoeba ? (grad ? resident<true, true>() : resident<true, false>())
                         : (grad ? resident<false, true>() : resident<false, false>());
  const int tblocks = std::max(1, (s.m + NT - 1) / NT);
  return std::max(1, std::min((s.m + 31) / 32, (4 * r * sms + tblocks - 1) / tblocks));
}

void launch_m2m(const DevSites &s, bool grad, double *partial, int nsplit, int *err, cudaStream_t st) {
  add_launch_count(1);
  const int per = ((s.m + nsplit - 1) / nsplit + 31) / 32 * 32;
  const dim3 grid((s.m + NT - 1) / NT, nsplit);
  if (s.amoeba)
    grad ? k_m2m<true, true><<<grid, NT, 0, st>>>(s, partial, per, err)
         : k_m2m<true, false><<<grid, NT, 0, st>>>(s, partial, per, err);
  else
    grad ? k_m2m<false, true><<<grid, NT, 0, st>>>(s, partial, per, err)
         : k_m2m<false, false><<<grid, NT, 0, st>>>(s, partial, per, err);
}

}  // namespace gpu
}  // namespace ommp
