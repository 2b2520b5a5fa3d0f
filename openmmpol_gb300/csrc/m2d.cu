// E_M2D, the field of the static multipoles (charge, dipole, quadrupole for
// AMOEBA; charge for Wang-AL) at the polarizable sites: the all-pairs part of
// elec_prop_M2D (src/mod_electrostatics.F90:2579-2731) at scale 1; the scaled
// pairs are corrected in FP64 by k_m2d_finish (kernels.cu).
//
// In FP64 (40 FP64 operations per pair) the field of 90,000 sites took 0.56 s,
// the FP64 pipe 95 % busy.  All modes now form it in double-single on the FP32
// pipes (ds_pair.cuh), 428 FP32 operations per AMOEBA pair (ncu):
//   E = (q G + (mu.n) F + (n.Q.n) C) n - K mu - H Q n
// with G = y^2, F = 3 y^3, C = 15 y^4, K = y^3, H = 6 y^4 times their factors
// in eps.  Source tiles whose box comes within the damping range test each
// pair; the close and strongly damped ones go to a list of the target's own
// and are formed in FP64 by its thread.  Per tile the double-single sums are
// added to FP64 ones; partial [split][n][3].
// 90,000 sites: 560 -> 108 ms (mixed-ds 128 ms); error against extended
// precision 1.9e-14 to 2.5e-14 for water (FP64 before: 2.9e-14 to 3.2e-14),
// 1.3e-14 for Wang-AL (2.6e-14).  Bound by FP32 issue at 4 CTAs per SM.
//
// Built with --fmad=false -ftz=true: every FMA is explicit.
#include <algorithm>

#include "ds_pair.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int NT = 128;    // targets per CTA, sources per tile
constexpr int NLIST = 32;  // listed sources per target before they are formed

template <bool AMOEBA>
struct M2dRec {
  static constexpr int LD = AMOEBA ? 10 : 1;
  static constexpr int R = (9 + 2 * LD + 3) / 4;  // float4 records of a source
};

__device__ __forceinline__ void m2d_target_ds(const DevSites &s, int tj, float (&tg)[9]) {
  const float4 h = s.pol_split[tj], m = s.pol_split[(size_t)s.n + tj], l = s.pol_split[2 * (size_t)s.n + tj];
  tg[0] = h.x, tg[1] = h.y, tg[2] = h.z, tg[3] = m.x, tg[4] = m.y, tg[5] = m.z, tg[6] = l.x, tg[7] = l.y, tg[8] = l.z;
}

// the record of static site i into the thread's column of the tile
template <bool AMOEBA>
__device__ __forceinline__ void m2d_stage_ds(const DevSites &s, int i, float4 (*s_rec)[NT]) {
  constexpr int LD = M2dRec<AMOEBA>::LD, R = M2dRec<AMOEBA>::R;
  const float4 h = s.mm_split[i], m = s.mm_split[(size_t)s.m + i], l = s.mm_split[2 * (size_t)s.m + i];
  float f[4 * R] = {h.x, h.y, h.z, m.x, m.y, m.z, l.x, l.y, l.z};
#pragma unroll
  for (int c = 0; c < LD; ++c) {
    const dsf q = to_ds(s.mm_q[(size_t)i * LD + c]);
    f[9 + c] = q.h;
    f[9 + LD + c] = q.l;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) s_rec[r][threadIdx.x] = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
}

// a listed pair in FP64; true when the sites coincide
template <bool AMOEBA>
__device__ __forceinline__ bool m2d_close(const DevSites &s, int i, const Pos64 &pt, double at, float2 wat,
                                          float thr2m, double *sum) {
  constexpr int LD = M2dRec<AMOEBA>::LD;
  const Pos64 ps = s.mm_pos[i];
  const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
  if (coincident(fma(dx, dx, fma(dy, dy, dz * dz)))) return true;
  double o[M2D_SLD], acc[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, e[3];
  m2d_stage<AMOEBA>(&s.mm_q[(size_t)i * LD], o);
  m2d_pair_acc<AMOEBA>(dx, dy, dz, pt.w, ps.w, at, AMOEBA ? s.mm_a[i] : 0.0, wat, s.mm_wa32[i], o, s.damp_thr,
                             thr2m, acc);
  m2d_field<AMOEBA>(acc, e[0], e[1], e[2]);
  for (int c = 0; c < 3; ++c) sum[c] += e[c];
  return false;
}

// the field of the staged source f at the target tg added to acc; near: test
// the pair, masked() when it is left to FP64
template <bool AMOEBA, typename MASKED>
__device__ __forceinline__ void m2d_pair_ds(const float (&tg)[9], const float *f, float2 wat, float2 was, bool near,
                                            MASKED masked, dsf *acc) {
  constexpr int LD = M2dRec<AMOEBA>::LD;
  float sc[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) sc[c] = f[c];
  const DspDelta d = dsp_delta(tg, sc);
  float y = d.ri, x = 0.f;
  if (near && dsp_masked<AMOEBA>(d.r2, wat, was, 25.f, x)) {
    y = 0.f;
    masked();
  }
  const DspUnit n = dsp_unit<true>(d, y);
  const float w3 = dsp_power<3>(n.eps);
  const float y2 = y * y, y2l = fmaf(y, y, -y2);
  // the charges of a neutral molecule cancel: their factor is kept to 2^-48
  dsf G = dsp_scaled<3>(y2, y2l, n);
  if (!AMOEBA) {
    const dsf c = dsp_mul(G, dsf{f[9], f[10]});
    dsp_acc(acc[0], c, n.x);
    dsp_acc(acc[1], c, n.y);
    dsp_acc(acc[2], c, n.z);
  } else {
    const float w5 = dsp_power<5>(n.eps), w7 = dsp_power<7>(n.eps);
    const float y3 = y2 * y, y3l = fmaf(y2l, y, fmaf(y2, y, -y3));
    const float y4 = y3 * y, y4l = fmaf(y3l, y, fmaf(y3, y, -y4));
    dsf K = {-y3, -fmaf(y3, w3, y3l)};
    dsf F = dsp_coef(3.f, y3, y3l, w5), H = dsp_coef(-6.f, y4, y4l, w5), C = dsp_coef(15.f, y4, y4l, w7);
    if (x > 0.f) {  // weak damping, within the low parts
      const float e3 = __expf(-x), e5 = fmaf(x, e3, e3), e7 = fmaf(0.6f * x * x, e3, e5);
      G.l = fmaf(-G.h, e3, G.l);
      K.l = fmaf(-K.h, e3, K.l);
      F.l = fmaf(-F.h, e5, F.l);
      H.l = fmaf(-H.h, e5, H.l);
      C.l = fmaf(-C.h, e7, C.l);
    }
    auto q = [&](int c) { return dsf{f[9 + c], f[9 + LD + c]}; };
    const dsf a = dsp_dot(q(1), q(2), q(3), n.x, n.y, n.z);
    const dsf tx = dsp_norm(dsp_dot(q(4), q(5), q(7), n.x, n.y, n.z));
    const dsf ty = dsp_norm(dsp_dot(q(5), q(6), q(8), n.x, n.y, n.z));
    const dsf tz = dsp_norm(dsp_dot(q(7), q(8), q(9), n.x, n.y, n.z));
    const dsf nqn = dsp_dot(tx, ty, tz, n.x, n.y, n.z);
    dsf c = dsp_mul(G, q(0));
    dsp_acc(c, F, a);
    dsp_acc(c, C, nqn);
    c = dsp_norm(c);
    dsp_acc(acc[0], c, n.x);
    dsp_acc(acc[0], K, q(1));
    dsp_acc(acc[0], H, tx);
    dsp_acc(acc[1], c, n.y);
    dsp_acc(acc[1], K, q(2));
    dsp_acc(acc[1], H, ty);
    dsp_acc(acc[2], c, n.z);
    dsp_acc(acc[2], K, q(3));
    dsp_acc(acc[2], H, tz);
  }
  // renormalised every pair: the field is a small remainder of the charges'
#pragma unroll
  for (int c = 0; c < 3; ++c) acc[c] = dsp_norm(acc[c]);
}

template <bool AMOEBA>
__global__ void __launch_bounds__(NT, 4) k_m2d(const __grid_constant__ DevSites s, double *__restrict__ partial,
                                               int per_split, float thr2m, float r2near, int *err_flag) {
  constexpr int LD = M2dRec<AMOEBA>::LD, R = M2dRec<AMOEBA>::R;
  __shared__ float4 s_rec[R][NT];
  __shared__ float2 s_wa[NT];
  __shared__ int s_list[NLIST][NT];
  const int j = blockIdx.x * NT + threadIdx.x;
  const bool valid = j < s.n;
  const int tj = valid ? j : s.n - 1;
  float tg[9];
  m2d_target_ds(s, tj, tg);
  const int tm = s.polar_mm[tj];
  const float2 wat = s.pol_wa32[tj];
  const float4 tlo = s.tile_box32[2 * blockIdx.x], thi = s.tile_box32[2 * blockIdx.x + 1];
  double sum[3] = {0.0, 0.0, 0.0};
  int listed = 0, bad = 0;
  // the listed pairs in FP64
  auto form = [&]() {
    const Pos64 pt = s.pol_pos[tj];
    const double at = AMOEBA ? s.pol_a[tj] : 0.0;
    for (int q = 0; q < listed; ++q) {
      const int i = s_list[q][threadIdx.x];
      if (m2d_close<AMOEBA>(s, i, pt, at, wat, thr2m, sum)) bad = 1;
    }
    listed = 0;
  };
  const int s0 = blockIdx.y * per_split, s1 = min(s.m, s0 + per_split);
  for (int t0 = s0; t0 < s1;) {
    // a tile never crosses a 128-site boundary (its box)
    const int cnt = min(NT - t0 % NT, s1 - t0);
    __syncthreads();
    if (threadIdx.x < cnt) {
      const int i = t0 + threadIdx.x;
      m2d_stage_ds<AMOEBA>(s, i, s_rec);
      s_wa[threadIdx.x] = s.mm_wa32[i];
    }
    __syncthreads();
    const float4 slo = s.mm_tile_box32[2 * (t0 / NT)], shi = s.mm_tile_box32[2 * (t0 / NT) + 1];
    const float gx = fmaxf(0.f, fmaxf(slo.x - thi.x, tlo.x - shi.x));
    const float gy = fmaxf(0.f, fmaxf(slo.y - thi.y, tlo.y - shi.y));
    const float gz = fmaxf(0.f, fmaxf(slo.z - thi.z, tlo.z - shi.z));
    const bool near = !(fmaf(gx, gx, fmaf(gy, gy, gz * gz)) > r2near);  // uniform over the CTA
    dsf acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 1
    for (int k = 0; k < cnt; ++k) {
      float f[4 * R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 v = s_rec[r][k];
        f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
      }
      m2d_pair_ds<AMOEBA>(tg, f, wat, s_wa[k], near, [&]() {
        if (t0 + k == tm) return;
        if (listed == NLIST) form();
        s_list[listed++][threadIdx.x] = t0 + k;
      }, acc);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sum[c] += (double)acc[c].h + (double)acc[c].l;
    t0 += cnt;
  }
  form();
  if (!valid) return;
  if (bad) atomicOr(err_flag, 1);
#pragma unroll
  for (int c = 0; c < 3; ++c) partial[((size_t)blockIdx.y * s.n + j) * 3 + c] = sum[c];
}

// The near field of the FMM's E_M2D: the sources of one column of three
// neighbouring leaves at the targets of a leaf (k_fmm_near of fmm_near.cu with
// static multipoles), every pair tested; partial [kFmmNearSplit][n][3].  In FP64
// (40 operations a pair, one CTA for a leaf and all its neighbours) it was most
// of the FMM's field: 60,000 sites, order 10, with the coordinate update
// 31.4 -> 8.1 ms, 24,000 sites 6.5 -> 3.0 (this kernel 3.2 ms).  FP32 issue.
template <bool AMOEBA>
__global__ void __launch_bounds__(NT, 4) k_m2d_leaf(const __grid_constant__ DevSites s, int L,
                                                    const int *__restrict__ leaf_start, const int *__restrict__ perm,
                                                    const int *__restrict__ leaf_start_t,
                                                    const int *__restrict__ perm_t, double *__restrict__ partial,
                                                    float thr2m, int *err_flag) {
  constexpr int R = M2dRec<AMOEBA>::R;
  __shared__ float4 s_rec[R][NT];
  __shared__ float2 s_wa[NT];
  __shared__ int s_site[NT];
  __shared__ int s_list[NLIST][NT];
  const int c = blockIdx.x, g0 = leaf_start_t[c], g1 = leaf_start_t[c + 1];
  if (g0 == g1) return;
  const int nl = 1 << L;
  const int cz = c % nl, cy = (c / nl) % nl, cx = c / (nl * nl);
  const int X = cx + (int)blockIdx.y / 3 - 1, Y = cy + (int)blockIdx.y % 3 - 1;
  const bool in = X >= 0 && X < nl && Y >= 0 && Y < nl;
  // the leaves of a column are contiguous in z
  const int col = (X * nl + Y) * nl;
  const int r0 = in ? leaf_start[col + max(0, cz - 1)] : 0, r1 = in ? leaf_start[col + min(nl - 1, cz + 1) + 1] : 0;
  int bad = 0;
  for (int b0 = g0; b0 < g1; b0 += NT) {
    const bool valid = b0 + (int)threadIdx.x < g1;
    const bool work = b0 + (int)(threadIdx.x & ~31) < g1;  // warps past the leaf's end only stage
    const int tj = perm_t[valid ? b0 + threadIdx.x : g0];
    float tg[9];
    m2d_target_ds(s, tj, tg);
    const int tm = s.polar_mm[tj];
    const float2 wat = s.pol_wa32[tj];
    double sum[3] = {0.0, 0.0, 0.0};
    int listed = 0;
    auto form = [&]() {
      const Pos64 pt = s.pol_pos[tj];
      const double at = AMOEBA ? s.pol_a[tj] : 0.0;
      for (int q = 0; q < listed; ++q)
        if (m2d_close<AMOEBA>(s, s_list[q][threadIdx.x], pt, at, wat, thr2m, sum)) bad = 1;
      listed = 0;
    };
    for (int t0 = r0; t0 < r1; t0 += NT) {
      const int cnt = min(NT, r1 - t0);
      __syncthreads();
      if ((int)threadIdx.x < cnt) {
        const int i = perm[t0 + threadIdx.x];
        s_site[threadIdx.x] = i;
        m2d_stage_ds<AMOEBA>(s, i, s_rec);
        s_wa[threadIdx.x] = s.mm_wa32[i];
      }
      __syncthreads();
      if (!work) continue;
      dsf acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 1
      for (int k = 0; k < cnt; ++k) {
        float f[4 * R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 v = s_rec[r][k];
          f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
        }
        m2d_pair_ds<AMOEBA>(tg, f, wat, s_wa[k], true, [&]() {
          if (s_site[k] == tm) return;
          if (listed == NLIST) form();
          s_list[listed++][threadIdx.x] = s_site[k];
        }, acc);
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) sum[d] += (double)acc[d].h + (double)acc[d].l;
    }
    form();
    if (valid)
      for (int d = 0; d < 3; ++d) partial[((size_t)blockIdx.y * s.n + tj) * 3 + d] = sum[d];
    __syncthreads();
  }
  if (bad) atomicOr(err_flag, 1);
}

int resident() {
  static const int r = [] {
    int v = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_m2d<true>, NT, 0);
    return v < 1 ? 1 : v;
  }();
  return r;
}

// sources per split: whole quarters of a tile
int per_split(const DevSites &s, int nsplit) { return ((s.m + nsplit - 1) / nsplit + 31) / 32 * 32; }

}  // namespace

// Source splits: about 16 waves of CTAs, so that the last, partly filled wave
// idles few SMs, with the split partials kept below 64 MiB; a split is at
// least 32 sources (small systems: whole 128-site tiles left most SMs idle).
int m2d_pick_split(const DevSites &s, int sms) {
  const long long tblocks = std::max(1, (s.n + NT - 1) / NT);
  long long split = (16LL * resident() * sms + tblocks - 1) / tblocks;
  split = std::min(split, (64LL << 20) / (24LL * (s.n > 0 ? s.n : 1)));
  split = std::min<long long>(split, (s.m + 31) / 32);
  return (int)std::max(1LL, split);
}

size_t m2d_scratch_doubles(const DevSites &s, int nsplit) { return (size_t)nsplit * s.n * 3; }

void launch_m2d(const DevSites &s, double *out, double *scratch, int nsplit, int *err_flag, cudaStream_t st) {
  if (s.n == 0) return;
  add_launch_count(1);
  const int per = per_split(s, nsplit);
  const dim3 grid((s.n + NT - 1) / NT, nsplit);
  const float thr2m = (float)(s.damp_thr * s.damp_thr * (1.0 + 1e-5));
  const float r2near = near_range2(s, s.m2d_r2max32);
  if (s.amoeba)
    k_m2d<true><<<grid, NT, 0, st>>>(s, scratch, per, thr2m, r2near, err_flag);
  else
    k_m2d<false><<<grid, NT, 0, st>>>(s, scratch, per, thr2m, r2near, err_flag);
  launch_m2d_finish(s, out, scratch, nsplit, st);
}

void launch_m2d_leaf(const DevSites &s, int L, const int *leaf_start, const int *perm, const int *leaf_start_t,
                     const int *perm_t, double *partial, int *err_flag, cudaStream_t st) {
  add_launch_count(1);
  const dim3 grid(1 << (3 * L), kFmmNearSplit);
  const float thr2m = (float)(s.damp_thr * s.damp_thr * (1.0 + 1e-5));
  if (s.amoeba)
    k_m2d_leaf<true><<<grid, NT, 0, st>>>(s, L, leaf_start, perm, leaf_start_t, perm_t, partial, thr2m, err_flag);
  else
    k_m2d_leaf<false><<<grid, NT, 0, st>>>(s, L, leaf_start, perm, leaf_start_t, perm_t, partial, thr2m, err_flag);
}

}  // namespace gpu
}  // namespace ommp
