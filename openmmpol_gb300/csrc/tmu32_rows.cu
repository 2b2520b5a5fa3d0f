// FP32 T.mu over all ordered pairs with a damping test per pair, for small
// systems: a whole row of T, its scaled pairs, the diagonal and the partial
// sums of x.y end in one CTA, so that the inner iteration's product is one
// launch (field_extD2D, src/mod_electrostatics.F90:2068-2109, and
// TMatVec_otf / TMatVec_diag, src/mod_polarization.F90:459-504).
//
// Lanes run over the sources, a warp holds one target, a CTA of four warps
// stages 128 sources at a time.  A lane's sums are compensated every 32
// sources (FP32), the warp's reduction keeps the rounding errors.  Bound by
// FP32 issue (~30 instructions per ordered pair and column) at 3,003 sites, by
// latency below 1,000.  Times of an inner iteration (with some 27 us of its
// other steps), us, one target per thread before / now: 192 sites 48 / 31, 999
// 56 / 39, 2,001 61 / 45, 3,003 66 / 54; eight columns at 999 sites 69 (tiled) /
// 49.  Also measured: one or two targets shared by the four warps (32 / 31, 40 /
// 39, 56 / 49, 67 / 64), two and four targets per warp (31, 38, 47, 57 and 33,
// 43, 51, 66).
#include <algorithm>

#include "ds_math.cuh"
#include "kernels.h"
#include "pair_math.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int TPB = 128, WARPS = TPB / 32;  // sources per tile; targets per CTA

struct Rows32Args {
  int n;
  const float4 *pos;
  const float *damp, *x;
  const double *ialpha;
  const int *ri, *src;
  const double *scale;
  float thr;
  float *y;
  double *part;
};

__device__ __forceinline__ dsf add(dsf a, dsf b) {
  const dsf s = two_sum(a.h, b.h);
  return fast_two_sum(s.h, s.l + (a.l + b.l));
}

template <int G, bool AMOEBA>
__global__ void __launch_bounds__(TPB) k_rows32(const __grid_constant__ Rows32Args a) {
  constexpr int C = 3 * G;
  __shared__ float4 s_pos[TPB], s_mu[G][TPB];  // s_mu[0].w: damping a
  __shared__ dsf s_sum[WARPS][C];
  __shared__ double s_xy[WARPS][G];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = a.n;
  const size_t col = (size_t)blockIdx.y * G * 3 * n;
  const float *x = a.x + col;
  const int j0 = blockIdx.x * WARPS + warp, j = min(j0, n - 1);
  const float4 pt = a.pos[j];
  const float at = AMOEBA ? a.damp[j] : 0.f;
  float acc[C], sum[C], comp[C];
#pragma unroll
  for (int c = 0; c < C; ++c) acc[c] = sum[c] = comp[c] = 0.f;
  auto flush = [&]() {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float y = acc[c] - comp[c], s = sum[c] + y;
      comp[c] = (s - sum[c]) - y;
      sum[c] = s;
      acc[c] = 0.f;
    }
  };
  const int ntile = (n + TPB - 1) / TPB;
  for (int b = 0; b < ntile; ++b) {
    __syncthreads();
    {
      const int k = b * TPB + tid;
      const bool v = k < n;
      s_pos[tid] = v ? a.pos[k] : make_float4(1.e15f, 1.e15f, 1.e15f, 1.f);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float *m = x + ((size_t)g * n + k) * 3;
        s_mu[g][tid] = v ? make_float4(m[0], m[1], m[2], g == 0 && AMOEBA ? a.damp[k] : 0.f)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    __syncthreads();
    const int self = j0 - b * TPB;
#pragma unroll
    for (int u = 0; u < TPB / 32; ++u) {
      const int q = 32 * u + lane;
      const float4 ps = s_pos[q];
      float4 m[G];
#pragma unroll
      for (int g = 0; g < G; ++g) m[g] = s_mu[g][q];
      const float dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      float k3, k5;
      damped_factors<AMOEBA>(r2, pt.w, ps.w, at, m[0].w, a.thr, k3, k5);
      if (q == self) k3 = k5 = 0.f;
      k5 *= 3.f;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float f = k5 * fmaf(m[g].x, dx, fmaf(m[g].y, dy, m[g].z * dz));
        acc[3 * g] = fmaf(f, dx, fmaf(-k3, m[g].x, acc[3 * g]));
        acc[3 * g + 1] = fmaf(f, dy, fmaf(-k3, m[g].y, acc[3 * g + 1]));
        acc[3 * g + 2] = fmaf(f, dz, fmaf(-k3, m[g].z, acc[3 * g + 2]));
      }
    }
    if ((b & 7) == 7) flush();
  }
  flush();
  double e[C];
#pragma unroll
  for (int c = 0; c < C; ++c) e[c] = 0.0;
  const int o0 = a.ri ? a.ri[j] : 0, o1 = a.ri ? a.ri[j + 1] : 0;
  for (int o = o0 + lane; o < o1; o += 32) {
    const int i = a.src[o];
    const float4 ps = a.pos[i];
    const float dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    float k3, k5;
    damped_factors<AMOEBA>(r2, pt.w, ps.w, at, AMOEBA ? a.damp[i] : 0.f, a.thr, k3, k5);
    const double cs = a.scale[o] - 1.0;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float *m = x + ((size_t)g * n + i) * 3;
      const float mx = m[0], my = m[1], mz = m[2];
      const float f = 3.f * k5 * fmaf(mx, dx, fmaf(my, dy, mz * dz));
      e[3 * g] += cs * (double)fmaf(f, dx, -(k3 * mx));
      e[3 * g + 1] += cs * (double)fmaf(f, dy, -(k3 * my));
      e[3 * g + 2] += cs * (double)fmaf(f, dz, -(k3 * mz));
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    dsf v = fast_two_sum(sum[c], -comp[c]);
    if (o1 > o0) v = add(v, to_ds(e[c]));
    for (int o = 16; o > 0; o >>= 1) {
      const dsf w{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
      v = add(v, w);
    }
    if (lane == 0) s_sum[warp][c] = v;
  }
  __syncthreads();
  double xy[G];
#pragma unroll
  for (int g = 0; g < G; ++g) xy[g] = 0.0;
  if (tid < WARPS * C) {
    const int w0 = tid / C, c = tid % C, j = blockIdx.x * WARPS + w0;
    if (j < n) {
      const double v = (double)s_sum[w0][c].h + (double)s_sum[w0][c].l;
      const size_t o = ((size_t)(c / 3) * n + j) * 3 + c % 3;
      const float xv = x[o], yv = (float)fma((double)xv, a.ialpha[j], -v);
      a.y[col + o] = yv;
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (c / 3 == g) xy[g] = (double)xv * (double)yv;
    }
  }
  if (!a.part) return;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    for (int o = 16; o > 0; o >>= 1) xy[g] += __shfl_xor_sync(0xffffffffu, xy[g], o);
    if (lane == 0) s_xy[warp][g] = xy[g];
  }
  __syncthreads();
  if (tid < G)
    a.part[((size_t)blockIdx.y * G + tid) * gridDim.x + blockIdx.x] =
        ((s_xy[0][tid] + s_xy[1][tid]) + s_xy[2][tid]) + s_xy[3][tid];
}

}  // namespace

int tmu32_rows_parts(int n) { return (n + WARPS - 1) / WARPS; }

void launch_tmu32_rows(const DevSites &s, int ncol, int gmax, const float *x, float *y, double *part, cudaStream_t st) {
  Rows32Args a{};
  a.n = s.n;
  a.pos = s.pol_pos32, a.damp = s.pol_a32, a.ialpha = s.pol_ialpha;
  a.ri = s.d2d_nnz ? s.d2d_ri : nullptr, a.src = s.d2d_src, a.scale = s.d2d_s;
  a.thr = (float)s.damp_thr;
  const int parts = tmu32_rows_parts(s.n);
  for (int c = 0; c < ncol;) {
    const int left = std::min(ncol - c, gmax), g = left >= 4 ? 4 : left >= 2 ? 2 : 1, groups = (ncol - c) / g;
    a.x = x + (size_t)c * 3 * s.n, a.y = y + (size_t)c * 3 * s.n;
    a.part = part ? part + (size_t)c * parts : nullptr;
    add_launch_count(1);
    auto go = [&](auto kernel) { kernel<<<dim3(parts, groups), TPB, 0, st>>>(a); };
    if (g == 4)
      s.amoeba ? go(k_rows32<4, true>) : go(k_rows32<4, false>);
    else if (g == 2)
      s.amoeba ? go(k_rows32<2, true>) : go(k_rows32<2, false>);
    else
      s.amoeba ? go(k_rows32<1, true>) : go(k_rows32<1, false>);
    c += g * groups;
  }
}

}  // namespace gpu
}  // namespace ommp
