// Near field of the fast multipole T.mu: the damped dipole field of the 27
// neighbouring leaves at every polarizable site (elec_prop_D2D's near cells,
// src/mod_electrostatics.F90:1954-2065).
//
// All pairs of neighbouring leaves (about 3,300 sources per site on a
// 60,000-site box) in FP64 took 13.1 ms of a 15.5 ms product, the FP64 pipe
// busy; this kernel takes 1.60 ms.  Here they run in double-single on the FP32
// pipes (ds_pair.cuh), one target per thread; the pairs that are close or strongly damped are masked
// and noted in a list of the target's own, which its thread then forms in
// FP64 (about 18 sources per site in water).  A CTA takes one leaf and one
// column of three neighbours, so that uneven leaves do not hold up the GPU (512
// leaves on 152 SMs); the nine partial fields are added in order by the caller.
//
// Built with --fmad=false -ftz=true: every FMA is explicit.
#include "ds_pair.cuh"

namespace ommp {
namespace gpu {

namespace {

constexpr int NT = 128;    // targets per pass, sources per tile
constexpr int NLIST = 48;  // listed sources per target before they are formed

template <bool AMOEBA>
__global__ void __launch_bounds__(NT, 5) k_fmm_near(const __grid_constant__ FmmNearArgs a, const double *__restrict__ x,
                                                    const unsigned *__restrict__ word, double *__restrict__ partial) {
  __shared__ float4 s_rec[4][NT];
  __shared__ float2 s_wa[NT];
  __shared__ int s_list[NLIST][NT];
  const int n = a.n, col = blockIdx.y, c = blockIdx.x;
  const int s0 = a.leaf_start[c], s1 = a.leaf_start[c + 1];
  if (s0 == s1) return;
  const int nl = 1 << a.L;
  const int cz = c % nl, cy = (c / nl) % nl, cx = c / (nl * nl);
  const int X = cx + (int)blockIdx.z / 3 - 1, Y = cy + (int)blockIdx.z % 3 - 1;
  const int ex = dsp_exponent(word[col]);  // the column's own scale
  const double *xc = x + (size_t)col * n * 3;
  double *out = partial + ((size_t)blockIdx.z * a.ncol + col) * n * 3;
  for (int b0 = s0; b0 < s1; b0 += NT) {
    const int si = b0 + threadIdx.x;
    const bool valid = si < s1;
    // a warp past the end of the leaf only stages: the last pass over a leaf of
    // 140 sites has one warp of work, not four
    const bool work = b0 + (int)(threadIdx.x & ~31) < s1;
    const int ti = valid ? si : s0;
    float tg[9];
    {
      const float4 h = a.split[ti], m = a.split[(size_t)n + ti], l = a.split[2 * (size_t)n + ti];
      tg[0] = h.x, tg[1] = h.y, tg[2] = h.z, tg[3] = m.x, tg[4] = m.y, tg[5] = m.z, tg[6] = l.x, tg[7] = l.y,
      tg[8] = l.z;
    }
    const float2 wat = a.swa[ti];
    double e[3] = {0.0, 0.0, 0.0};
    int listed = 0;
    // the listed pairs in FP64
    auto form = [&]() {
      const Pos64 pt = a.spos[ti];
      const double at = AMOEBA ? a.sa[ti] : 0.0;
      for (int q = 0; q < listed; ++q) {
        const int k = s_list[q][threadIdx.x];
        const Pos64 ps = a.spos[k];
        const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        if (coincident(r2)) continue;
        double k3, k5;
        dd_pair_f64<AMOEBA>(r2, pt.w, ps.w, at, AMOEBA ? a.sa[k] : 0.0, wat, a.swa[k], a.thr, a.thr2m, k3, k5);
        const double *mu = xc + 3 * (size_t)a.perm[k];
        const double mx = scale_down(mu[0], ex), my = scale_down(mu[1], ex), mz = scale_down(mu[2], ex);
        const double f = 3.0 * k5 * fma(mx, dx, fma(my, dy, mz * dz));
        e[0] += fma(f, dx, -(k3 * mx));
        e[1] += fma(f, dy, -(k3 * my));
        e[2] += fma(f, dz, -(k3 * mz));
      }
      listed = 0;
    };
    if (X >= 0 && X < nl && Y >= 0 && Y < nl) {
      // the leaves of a column are contiguous in z
      const int z0 = max(0, cz - 1), z1 = min(nl - 1, cz + 1);
      const int r0 = a.leaf_start[(X * nl + Y) * nl + z0], r1 = a.leaf_start[(X * nl + Y) * nl + z1 + 1];
      for (int t0 = r0; t0 < r1; t0 += NT) {
        __syncthreads();
        const int k = t0 + threadIdx.x;
        if (k < r1) {
          const float4 h = a.split[k], m = a.split[(size_t)n + k], l = a.split[2 * (size_t)n + k];
          const double *mu = xc + 3 * (size_t)a.perm[k];
          const dsf mx = to_ds(scale_down(mu[0], ex)), my = to_ds(scale_down(mu[1], ex)),
                    mz = to_ds(scale_down(mu[2], ex));
          s_rec[0][threadIdx.x] = make_float4(h.x, h.y, h.z, m.x);
          s_rec[1][threadIdx.x] = make_float4(m.y, m.z, l.x, l.y);
          s_rec[2][threadIdx.x] = make_float4(l.z, mx.h, my.h, mz.h);
          s_rec[3][threadIdx.x] = make_float4(mx.l, my.l, mz.l, 0.f);
          s_wa[threadIdx.x] = a.swa[k];
        }
        __syncthreads();
        if (!work) continue;
        const int cnt = min(NT, r1 - t0);
        float ah[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
          const float4 v0 = s_rec[0][q], v1 = s_rec[1][q], v2 = s_rec[2][q], v3 = s_rec[3][q];
          const float s[9] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x};
          const float mh[3] = {v2.y, v2.z, v2.w}, ml[3] = {v3.x, v3.y, v3.z};
          bool masked;
          const DsPair g = dsp_geometry<true, AMOEBA>(tg, s, wat, s_wa[q], masked);
          dsp_column(g, mh, ml, ah, al);
          if (masked && t0 + q != si) {
            if (listed == NLIST) form();
            s_list[listed++][threadIdx.x] = t0 + q;
          }
          if ((q & 31) == 31) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const dsf r = two_sum(ah[d], al[d]);
              ah[d] = r.h;
              al[d] = r.l;
            }
          }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) e[d] += (double)ah[d] + (double)al[d];
      }
    }
    form();
    if (valid) {
      const int pi = a.perm[si];
      for (int d = 0; d < 3; ++d) out[3 * (size_t)pi + d] = scale_up(e[d], ex);
    }
  }
}

}  // namespace

void launch_fmm_near(const FmmNearArgs &a, const double *x, const unsigned *word, double *partial, cudaStream_t st) {
  add_launch_count(1);
  const dim3 grid(1 << (3 * a.L), a.ncol, kFmmNearSplit);
  if (a.amoeba)
    k_fmm_near<true><<<grid, NT, 0, st>>>(a, x, word, partial);
  else
    k_fmm_near<false><<<grid, NT, 0, st>>>(a, x, word, partial);
}

}  // namespace gpu
}  // namespace ommp
