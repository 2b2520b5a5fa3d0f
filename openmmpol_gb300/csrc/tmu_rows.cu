// T.mu of FP64 accuracy over all ordered pairs (TMatVec_otf / field_extD2D,
// src/mod_polarization.F90:459-481, src/mod_electrostatics.F90:1954-2111), for
// the sizes at which a launch over unordered pairs (tmu_sym.cu) leaves the GPU
// idle: a whole row of T, its scaled pairs, the diagonal and the partial sums
// of x.y end in one CTA, so that a product is one launch without accumulators.
//
//   k_rows_f64  one target per CTA, its 128 threads over the sources, in FP64:
//               bound by the FP64 pipe, and by latency below a few hundred
//               sites.
//   k_rows_ds   the arithmetic of tmu_sym.cu, double-single on the FP32 pipes
//               in unit-vector form, ~190 operations per ordered pair; close
//               and strongly damped pairs are listed per target and formed in
//               FP64 by the whole warp.  Lanes run over the sources; a warp
//               holds T targets; a CTA of four warps stages 128 sources at a
//               time; WT of the warps have targets of their own, the 4 / WT
//               others share them and split the sources.  Bound by FP32 issue
//               at 8 to 16 warps per SM and by the FP64 pairs.
// One column, us (f64 / one target per CTA / 8 targets per CTA / symmetric):
// 192 sites 12.6 / 15.1 / 19.4 / 49, 390 22 / 20 / 25 / 62, 600 33 / 23 / 27 /
// 60, 999 72 / 38 / 35 / 67, 2,001 232 / 89 / 72 / 94, 3,003 469 / 156 / 124 /
// 104.  Eight columns (f64 / 8 targets / symmetric): 30 sites 34 / 22 / 92, 192
// 52 / 25 / 86, 999 371 / 98 / 169, 2,001 1,245 / 264 / 328, 3,003 2,526 / 516 /
// 540.
//
// Built with --fmad=false -ftz=true: every FMA is explicit.
#include <algorithm>

#include "ds_pair.cuh"
#include "kernels.h"
#include "pair_math.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int TPB = 128;
constexpr int LIST = 64;  // listed sources of a target before they are formed
constexpr float FAR = 1.0e6f;

// v 2^-ex as two floats (the leading 24 bits truncated, then the other 29
// rounded), by integer operations: the FP64 pipe would take longer over the
// staged dipoles than the FP32 pipes over the pairs.  Values 2^-116 below the
// largest vanish; an infinity or NaN gives NaN.
__device__ __forceinline__ dsf split_scaled(double v, int ex) {
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
  const int e = (hi >> 20) & 0x7ff, fe = e - 1023 - ex + 127;
  if (e == 0x7ff) return {__int_as_float(0x7fc00000), 0.f};
  if (e == 0 || fe < 1) return {0.f, 0.f};
  const unsigned sign = hi & 0x80000000u;
  const unsigned lead = (hi & 0xfffffu) << 3 | lo >> 29;
  const float h = __uint_as_float(sign | (unsigned)fe << 23 | lead);
  const float r = fe > 52 ? (float)(lo & 0x1fffffffu) * __uint_as_float((unsigned)(fe - 52) << 23) : 0.f;
  return {h, sign ? -r : r};
}

template <int G>
struct Rows {
  static constexpr int R = G == 1 ? 4 : 6;  // float4 records of a staged source
};

struct RowsArgs {
  int n, ncol;
  bool dodiag;
  const float4 *split;
  const Pos64 *pos;
  const double *damp;
  const float2 *wa;
  const double *x, *ialpha;
  const int *ri, *src;
  const double *scale;
  double thr;
  float thr2m;
  const unsigned *words;  // largest high word of each column
  double *y, *part;
};

// one pair in FP64, weighted: added to e (scaled dipoles).  Inlined for one
// column; with two its copies cost registers (999 sites, 8 columns: 98 us as a
// function, 112 inlined)
template <int G, bool AMOEBA>
__device__ __forceinline__ void pair64(const RowsArgs &a, const double *x, int j, int i, double w, const int *ex,
                                         double *e) {
  const Pos64 pt = a.pos[j], ps = a.pos[i];
  const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  double k3, k5;
  dd_pair_f64<AMOEBA>(r2, pt.w, ps.w, AMOEBA ? a.damp[j] : 0.0, AMOEBA ? a.damp[i] : 0.0, a.wa[j], a.wa[i], a.thr,
                            a.thr2m, k3, k5);
  k3 *= w;
  k5 *= 3.0 * w;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const double *mu = x + ((size_t)g * a.n + i) * 3;
    const double mx = scale_down(mu[0], ex[g]), my = scale_down(mu[1], ex[g]), mz = scale_down(mu[2], ex[g]);
    const double f = k5 * fma(mx, dx, fma(my, dy, mz * dz));
    e[3 * g] = fma(f, dx, fma(-k3, mx, e[3 * g]));
    e[3 * g + 1] = fma(f, dy, fma(-k3, my, e[3 * g + 1]));
    e[3 * g + 2] = fma(f, dz, fma(-k3, mz, e[3 * g + 2]));
  }
}

template <int G, bool AMOEBA>
__device__ __noinline__ void pair64_call(const RowsArgs &a, const double *x, int j, int i, double w, const int *ex,
                                         double *e) {
  pair64<G, AMOEBA>(a, x, j, i, w, ex, e);
}
template <int G, bool AMOEBA>
__device__ __forceinline__ void rows_pair64(const RowsArgs &a, const double *x, int j, int i, double w, const int *ex,
                                            double *e) {
  if constexpr (G == 1)
    pair64<G, AMOEBA>(a, x, j, i, w, ex, e);
  else
    pair64_call<G, AMOEBA>(a, x, j, i, w, ex, e);
}

__device__ __forceinline__ dsf add(dsf a, dsf b) {
  const dsf s = two_sum(a.h, b.h);
  return dsp_norm({s.h, s.l + (a.l + b.l)});
}

template <int G, bool AMOEBA, int T, int WT>
__global__ void __launch_bounds__(TPB) k_rows_ds(const __grid_constant__ RowsArgs a) {
  constexpr int R = Rows<G>::R, C = 3 * G, WS = 4 / WT;
  static_assert(WT * T * C <= TPB, "one thread per value of the CTA's targets");
  __shared__ float4 s_rec[R][TPB];
  __shared__ float2 s_wa[TPB];
  __shared__ int s_list[4][T][LIST];
  __shared__ dsf s_sum[4][T * C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wt = warp / WS, ws = warp % WS;
  const int n = a.n, col0 = blockIdx.y * G;
  const double *x = a.x + (size_t)col0 * n * 3;
  const int j0 = (blockIdx.x * WT + wt) * T;
  int ex[G];
#pragma unroll
  for (int g = 0; g < G; ++g) ex[g] = dsp_exponent(a.words[col0 + g]);
  float tg[T][9];
  float2 wat[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int j = min(j0 + t, n - 1);
    const float4 h = a.split[j], m = a.split[(size_t)n + j], l = a.split[2 * (size_t)n + j];
    tg[t][0] = h.x, tg[t][1] = h.y, tg[t][2] = h.z, tg[t][3] = m.x, tg[t][4] = m.y, tg[t][5] = m.z, tg[t][6] = l.x,
    tg[t][7] = l.y, tg[t][8] = l.z;
    wat[t] = a.wa[j];
  }
  float ah[T][C], al[T][C];
  double e[T][C];
  int listed[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    listed[t] = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) ah[t][c] = al[t][c] = 0.f, e[t][c] = 0.0;
  }
  const int ntile = (n + TPB - 1) / TPB;
  for (int b = 0; b < ntile; ++b) {
    __syncthreads();
    {
      const int k = b * TPB + tid;
      const bool v = k < n;
      const float4 h = v ? a.split[k] : make_float4(FAR, FAR, FAR, 0.f);
      const float4 m = v ? a.split[(size_t)n + k] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 l = v ? a.split[2 * (size_t)n + k] : make_float4(0.f, 0.f, 0.f, 0.f);
      float f[4 * R];
      f[0] = h.x, f[1] = h.y, f[2] = h.z, f[3] = m.x, f[4] = m.y, f[5] = m.z, f[6] = l.x, f[7] = l.y, f[8] = l.z;
#pragma unroll
      for (int c = 9 + 2 * C; c < 4 * R; ++c) f[c] = 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const dsf d = v ? split_scaled(x[((size_t)(c / 3) * n + k) * 3 + c % 3], ex[c / 3]) : dsf{0.f, 0.f};
        f[9 + c] = d.h, f[9 + C + c] = d.l;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) s_rec[r][tid] = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
      s_wa[tid] = v ? a.wa[k] : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = 32 * ws + lane; q < TPB; q += 32 * WS) {
      const int k = b * TPB + q;
      float f[4 * R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 v = s_rec[r][q];
        f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
      }
      float s[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) s[c] = f[c];
      const float2 was = s_wa[q];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        bool masked;
        const DsPair p = dsp_geometry<true, AMOEBA>(tg[t], s, wat[t], was, masked);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float mh[3] = {f[9 + 3 * g], f[10 + 3 * g], f[11 + 3 * g]};
          const float ml[3] = {f[9 + C + 3 * g], f[10 + C + 3 * g], f[11 + C + 3 * g]};
          float hh[3] = {ah[t][3 * g], ah[t][3 * g + 1], ah[t][3 * g + 2]};
          float ll[3] = {al[t][3 * g], al[t][3 * g + 1], al[t][3 * g + 2]};
          dsp_column(p, mh, ml, hh, ll);
#pragma unroll
          for (int c = 0; c < 3; ++c) ah[t][3 * g + c] = hh[c], al[t][3 * g + c] = ll[c];
        }
        masked = masked && k < n && k != j0 + t;
        const unsigned any = __ballot_sync(0xffffffffu, masked);
        if (any) {
          if (listed[t] + 32 > LIST) {
            __syncwarp();
            for (int o = lane; o < listed[t]; o += 32)
              rows_pair64<G, AMOEBA>(a, x, min(j0 + t, n - 1), s_list[warp][t][o], 1.0, ex, e[t]);
            __syncwarp();
            listed[t] = 0;
          }
          if (masked) s_list[warp][t][listed[t] + __popc(any & ((1u << lane) - 1u))] = k;
          listed[t] += __popc(any);
        }
      }
    }
    if ((b & 7) == 7) {
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const dsf r = two_sum(ah[t][c], al[t][c]);
          ah[t][c] = r.h, al[t][c] = r.l;
        }
    }
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int j = min(j0 + t, n - 1);
    for (int o = lane; o < listed[t]; o += 32) rows_pair64<G, AMOEBA>(a, x, j, s_list[warp][t][o], 1.0, ex, e[t]);
    if (a.ri)
      for (int o = a.ri[j] + 32 * ws + lane; o < a.ri[j + 1]; o += 32 * WS)
        rows_pair64<G, AMOEBA>(a, x, j, a.src[o], a.scale[o] - 1.0, ex, e[t]);
    // the warp's sums, every lane's to lane 0
#pragma unroll
    for (int c = 0; c < C; ++c) {
      dsf v = add(dsp_norm({ah[t][c], al[t][c]}), to_ds(e[t][c]));
      for (int o = 16; o > 0; o >>= 1) {
        const dsf w{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
        v = add(v, w);
      }
      if (lane == 0) s_sum[warp][t * C + c] = v;
    }
  }
  __syncthreads();
  // one value per thread: WT groups of T targets
  double xy[G];
#pragma unroll
  for (int g = 0; g < G; ++g) xy[g] = 0.0;
  if (tid < WT * T * C) {
    const int w0 = tid / (T * C), r = tid % (T * C), j = (blockIdx.x * WT + w0) * T + r / C, c = r % C;
    if (j < n) {
      double v = 0.0;
      for (int u = 0; u < WS; ++u) v += (double)s_sum[w0 * WS + u][r].h + (double)s_sum[w0 * WS + u][r].l;
      const double field = scale_up(v, ex[G == 2 ? c / 3 : 0]);
      const size_t o = ((size_t)(c / 3) * n + j) * 3 + c % 3;
      const double xv = x[o], yv = a.dodiag ? fma(xv, a.ialpha[j], -field) : -field;
      a.y[(size_t)col0 * n * 3 + o] = yv;
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (c / 3 == g) xy[g] = xv * yv;
    }
  }
  if (!a.part) return;
  __shared__ double s_xy[4][G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    for (int o = 16; o > 0; o >>= 1) xy[g] += __shfl_xor_sync(0xffffffffu, xy[g], o);
    if (lane == 0) s_xy[warp][g] = xy[g];
  }
  __syncthreads();
  if (tid < G) a.part[(size_t)(col0 + tid) * gridDim.x + blockIdx.x] = ((s_xy[0][tid] + s_xy[1][tid]) + s_xy[2][tid]) + s_xy[3][tid];
}

template <int G, bool AMOEBA>
__global__ void __launch_bounds__(128) k_rows_f64(int n, const Pos64 *__restrict__ pos,
                                                  const double *__restrict__ damp, const float2 *__restrict__ wa,
                                                  const double *__restrict__ x, const double *__restrict__ alpha,
                                                  bool dodiag, const int *__restrict__ ri,
                                                  const int *__restrict__ src, const double *__restrict__ scale,
                                                  double thr, float thr2m, double *__restrict__ y) {
  constexpr int C = 3 * G;
  __shared__ double s_sum[4][C];
  const int j = blockIdx.x;
  const Pos64 pt = pos[j];
  const double at = AMOEBA ? damp[j] : 0.0;
  const float2 wat = wa[j];
  double acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = 0.0;
  auto pair = [&](int i, double w) {
    const Pos64 ps = pos[i];
    const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    double k3, k5;
    dd_pair_f64<AMOEBA>(r2, pt.w, ps.w, at, AMOEBA ? damp[i] : 0.0, wat, wa[i], thr, thr2m, k3, k5);
    const double k3w = k3 * w, k5w = 3.0 * w * k5;
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const double *mu = &x[((size_t)r * n + i) * 3];
      const double mx = mu[0], my = mu[1], mz = mu[2];
      const double f = k5w * fma(mx, dx, fma(my, dy, mz * dz));
      acc[3 * r] = fma(f, dx, fma(-k3w, mx, acc[3 * r]));
      acc[3 * r + 1] = fma(f, dy, fma(-k3w, my, acc[3 * r + 1]));
      acc[3 * r + 2] = fma(f, dz, fma(-k3w, mz, acc[3 * r + 2]));
    }
  };
  for (int i = threadIdx.x; i < n; i += 128)
    if (i != j) pair(i, 1.0);
  if (ri)
    for (int k = ri[j] + threadIdx.x; k < ri[j + 1]; k += 128) pair(src[k], scale[k] - 1.0);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5][c] = acc[c];
  }
  __syncthreads();
  if (threadIdx.x < C) {
    const int c = threadIdx.x;
    const double e = ((s_sum[0][c] + s_sum[1][c]) + s_sum[2][c]) + s_sum[3][c];
    const size_t o = ((size_t)(c / 3) * n + j) * 3 + (c % 3);
    y[o] = dodiag ? x[o] / alpha[j] - e : -e;
  }
}

template <int G, int T, int WT>
void launch_ds(const RowsArgs &a, bool amoeba, int groups, cudaStream_t st) {
  const dim3 grid((a.n + T * WT - 1) / (T * WT), groups);
  add_launch_count(1);
  if (amoeba)
    k_rows_ds<G, true, T, WT><<<grid, TPB, 0, st>>>(a);
  else
    k_rows_ds<G, false, T, WT><<<grid, TPB, 0, st>>>(a);
}

template <int G>
void launch_f64(const RowsArgs &a, bool amoeba, const double *alpha, cudaStream_t st) {
  add_launch_count(1);
  if (amoeba)
    k_rows_f64<G, true><<<a.n, 128, 0, st>>>(a.n, a.pos, a.damp, a.wa, a.x, alpha, a.dodiag, a.ri, a.src, a.scale, a.thr,
                                             a.thr2m, a.y);
  else
    k_rows_f64<G, false><<<a.n, 128, 0, st>>>(a.n, a.pos, a.damp, a.wa, a.x, alpha, a.dodiag, a.ri, a.src, a.scale,
                                              a.thr, a.thr2m, a.y);
}

// The kernel by size and columns (times above): FP64 for up to three columns
// of fewer than 300 sites (and for systems wider than the split coordinates
// resolve), one target per CTA for one column of fewer than 800, else 8 targets
// per CTA.
constexpr int kF64Sites = 300, kOneSites = 800;
bool use_f64(const DevSites &s, int ncol) { return s.wide || (s.n < kF64Sites && ncol < 4); }

}  // namespace

int tmu_rows_parts(const DevSites &s, int ncol) {
  if (use_f64(s, ncol)) return 0;
  return ncol == 1 && s.n < kOneSites ? s.n : (s.n + 7) / 8;
}

void launch_tmu_rows(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, const unsigned *words,
                     double *part, cudaStream_t st) {
  if (s.n == 0) return;
  RowsArgs a{};
  a.n = s.n, a.dodiag = dodiag;
  a.split = s.pol_split, a.pos = s.pol_pos, a.damp = s.pol_a, a.wa = s.pol_wa32;
  a.ialpha = s.pol_ialpha;
  a.ri = s.d2d_nnz ? s.d2d_ri : nullptr, a.src = s.d2d_src, a.scale = s.d2d_s;
  a.thr = s.damp_thr;
  a.thr2m = (float)(s.damp_thr * s.damp_thr * (1.0 + 1e-5));
  const bool f64 = use_f64(s, nrhs), one = nrhs == 1 && s.n < kOneSites;
  const int npart = tmu_rows_parts(s, nrhs);
  for (int c = 0; c < nrhs;) {
    const int g = nrhs - c >= 2 ? 2 : 1, groups = g == 2 && !f64 ? (nrhs - c) / 2 : 1;
    a.words = words + c;
    a.x = x + (size_t)c * s.n * 3, a.y = y + (size_t)c * s.n * 3;
    a.part = part ? part + (size_t)c * npart : nullptr;
    if (f64)
      g == 2 ? launch_f64<2>(a, s.amoeba, s.pol_alpha, st) : launch_f64<1>(a, s.amoeba, s.pol_alpha, st);
    else if (g == 2)
      launch_ds<2, 2, 4>(a, s.amoeba, groups, st);
    else if (one)
      launch_ds<1, 1, 1>(a, s.amoeba, 1, st);
    else
      launch_ds<1, 2, 4>(a, s.amoeba, 1, st);
    c += g * groups;
  }
}

}  // namespace gpu
}  // namespace ommp
