// Conjugate-gradient steps between two T.mu products, for the FP64 solver, the
// FP32 inner solver and (several systems per launch) the multi-system engine.
//
// A CG iteration of one system moves a few hundred kB through vectors that
// stay in L2: it is bound by the number of dependent launches, not by memory.
// The separate dot, reduction, scalar, update and preconditioner kernels took
// 55 us per FP32 iteration of 9,003 sites (11 launches) next to a product of
// 79 us.  Here an iteration is the product, its finishing pass (with the
// partial sums of p.h) and two to four more launches:
//   k_cg_step      every block sums the p.h partials (the same order in each),
//                  forms alpha, updates x and (diagonal preconditioner) r, or
//                  applies the block-Jacobi preconditioner to the new r, which
//                  it recomputes from r, h and alpha over its run of sites.
//   k_cg_near      w = N z, the near-field blocks (8 lanes per row)
//   k_cg_near_sub  r -= alpha h and z -= B^-1 w
//   k_cg_dir       every block sums the r.z partials, forms beta and the new
//                  direction; clears the accumulators of the next product and,
//                  in FP64, takes the largest |p| for its scale.
// A column's scalars (CgCol) are written by block 0 of its column only, and no
// kernel reads a field that it writes: k_cg_step reads `active` and `gnew` (the
// current r.z), writes `gold`, `gama`, `alpha`, `quick`; k_cg_dir reads `gold`,
// `alpha`, writes the rest.
#include <algorithm>

#include "kernels.h"
#include "pair_math.cuh"
#include "pcg.h"

namespace ommp {
namespace gpu {
namespace {
constexpr int TPB = 256;

template <typename J>
struct Table {
  J job[kCgJobs];
};

// The FP64 pipe issues a warp's instruction every 16 cycles per SM, so the
// sums here are taken by as few warps as possible, one thread divides for its
// block, FP32 vectors are updated without that pipe, and 1 / alpha comes from
// memory.

// sum over the block, the same value and order in every thread; nwarp <= 32
__device__ __forceinline__ double block_sum(double v, double *sh, int nwarp) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double s = (int)threadIdx.x < nwarp ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) sh[0] = s;
  }
  __syncthreads();
  return sh[0];
}

// sum of n partial sums, by the first warp
__device__ __forceinline__ double partial_sum(const double *part, int n, double *sh) {
  if (threadIdx.x < 32) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < n; b += 128)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (b + 32 * u < n) v[u] += part[b + 32 * u];
    double s = (v[0] + v[1]) + (v[2] + v[3]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) sh[0] = s;
  }
  __syncthreads();
  const double s = sh[0];
  __syncthreads();
  return s;
}

// a / b (0 when b is 0) by one thread, in every thread
__device__ __forceinline__ double block_ratio(double a, double b, double *sh) {
  __syncthreads();  // sh may still be read
  if (threadIdx.x == 0) sh[0] = b != 0.0 ? a / b : 0.0;
  __syncthreads();
  const double q = sh[0];
  __syncthreads();
  return q;
}

// x + a p.  FP32 vectors: a as two floats, the products and the sum with
// their rounding errors, one rounding of the result as from FP64 arithmetic
struct Scalar {
  double d;
  float h, l;
  __device__ explicit Scalar(double a) : d(a), h((float)a), l((float)(a - (double)(float)a)) {}
};
__device__ __forceinline__ double axpy(double x, const Scalar &a, double p) { return fma(a.d, p, x); }
__device__ __forceinline__ float axpy(float x, const Scalar &a, float p) {
  const float q = __fmul_rn(a.h, p), ql = fmaf(a.l, p, fmaf(a.h, p, -q));
  const float s = __fadd_rn(x, q), t = s - x;
  const float e = (x - (s - t)) + (q - t);
  return s + (e + ql);
}

template <typename T>
__global__ void __launch_bounds__(TPB) k_cg_step(const __grid_constant__ Table<CgJob<T>> tab) {
  __shared__ double sh[TPB / 32];
  const CgJob<T> &jb = tab.job[blockIdx.z];
  const int k = blockIdx.y;
  if (k >= jb.ncol || (int)blockIdx.x >= jb.nb) return;
  CgCol &col = jb.cols[k];
  double al = 0.0;
  bool act = true;
  if (!jb.init) {
    act = col.active != 0;
    const double ph = partial_sum(jb.pa + (size_t)k * jb.na, jb.na, sh);
    const bool quick = act && fabs(ph) < jb.eps;
    const double rho = col.gnew;
    al = block_ratio(act && !quick ? rho : 0.0, ph, sh);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      col.alpha = al;
      if (act) {
        col.gold = rho;
        col.gama = ph;
        if (quick) col.quick = 1;
      }
    }
    act = act && !quick;
  }
  const Scalar pal(al), mal(-al);
  if (blockIdx.x == 0) {
    if (jb.words && k == 0 && threadIdx.x < 3) jb.words[threadIdx.x] = 0ull;
    if (jb.emax && threadIdx.x == 0) jb.emax[k] = 0u;
  }
  const size_t nv = 3 * (size_t)jb.n, off = (size_t)k * nv;
  T *x = jb.x + off, *r = jb.r + off;
  const T *p = jb.p + off, *h = jb.h + off;
  double acc = 0.0;
  if (act) {
    for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < nv; i += (size_t)jb.nb * TPB) {
      T rn = r[i];
      if (jb.init) {
        if (jb.init == kCgInitZero) x[i] = T(0);
      } else {
        x[i] = axpy(x[i], pal, p[i]);
        rn = axpy(rn, mal, h[i]);
      }
      if (jb.mode == 0) {
        if (!jb.init) r[i] = rn;
        const T z = jb.alpha[i / 3] * rn;
        acc += (double)rn * (double)z;
      } else if constexpr (sizeof(T) == 4) {
        const int j = (int)(i / 3);
        const int4 b = jb.info[j];
        const int wd = 3 * b.y;
        const float *rr = r + 3 * (size_t)b.x, *hh = h + 3 * (size_t)b.x;
        const float *m = jb.minv + b.z + (size_t)(3 * b.w + (int)(i - 3 * (size_t)j)) * wd;
        float z = 0.f;
        if (jb.init)
          for (int l = 0; l < wd; ++l) z = fmaf(m[l], rr[l], z);
        else
          for (int l = 0; l < wd; ++l) z = fmaf(m[l], axpy(rr[l], mal, hh[l]), z);
        jb.z[off + i] = z;
        acc += (double)rn * (double)z;
      }
    }
  }
  if (jb.mode == 2) return;  // r.z after the Neumann step
  acc = block_sum(acc, sh, TPB / 32);
  if (threadIdx.x == 0) jb.pb[(size_t)k * jb.nb + blockIdx.x] = acc;
}

// w[j] = sum over the near-field row j of N_ji z[i] (3x3 FP32 blocks)
__global__ void __launch_bounds__(TPB) k_cg_near(const __grid_constant__ Table<CgJob<float>> tab) {
  const CgJob<float> &jb = tab.job[blockIdx.z];
  const int j = (blockIdx.x * TPB + threadIdx.x) >> 3, sub = threadIdx.x & 7, k = blockIdx.y;
  if (k >= jb.ncol || jb.mode != 2 || j >= jb.n) return;
  const size_t co = (size_t)k * 3 * jb.n;
  float y[3] = {0.f, 0.f, 0.f};
  const int e1 = jb.ri[j + 1];
  for (int e = jb.ri[j] + sub; e < e1; e += 8) {
    const float *b = jb.blk + 9 * (size_t)e;
    const float *z = jb.z + co + 3 * (size_t)jb.ci[e];
    const float z0 = z[0], z1 = z[1], z2 = z[2];
#pragma unroll
    for (int c = 0; c < 3; ++c) y[c] = fmaf(b[3 * c], z0, fmaf(b[3 * c + 1], z1, fmaf(b[3 * c + 2], z2, y[c])));
  }
  const unsigned group = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    for (int o = 4; o > 0; o >>= 1) y[c] += __shfl_xor_sync(group, y[c], o);
    if (sub == c) jb.w[co + 3 * (size_t)j + c] = y[c];
  }
}

__global__ void __launch_bounds__(TPB) k_cg_near_sub(const __grid_constant__ Table<CgJob<float>> tab) {
  __shared__ double sh[TPB / 32];
  const CgJob<float> &jb = tab.job[blockIdx.z];
  const int k = blockIdx.y;
  if (k >= jb.ncol || jb.mode != 2 || (int)blockIdx.x >= jb.nb) return;
  const CgCol &col = jb.cols[k];
  const bool act = jb.init || (col.active && !col.quick);
  const Scalar mal(jb.init ? 0.0 : -col.alpha);
  const size_t nv = 3 * (size_t)jb.n, off = (size_t)k * nv;
  double acc = 0.0;
  if (act) {
    for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < nv; i += (size_t)jb.nb * TPB) {
      const int j = (int)(i / 3);
      const int4 b = jb.info[j];
      const int wd = 3 * b.y;
      const float *ww = jb.w + off + 3 * (size_t)b.x;
      const float *m = jb.minv + b.z + (size_t)(3 * b.w + (int)(i - 3 * (size_t)j)) * wd;
      float t = 0.f;
      for (int l = 0; l < wd; ++l) t = fmaf(m[l], ww[l], t);
      const float z = jb.z[off + i] - t;
      jb.z[off + i] = z;
      float r = jb.r[off + i];
      if (!jb.init) {
        r = axpy(r, mal, jb.h[off + i]);
        jb.r[off + i] = r;
      }
      acc += (double)r * (double)z;
    }
  }
  acc = block_sum(acc, sh, TPB / 32);
  if (threadIdx.x == 0) jb.pb[(size_t)k * jb.nb + blockIdx.x] = acc;
}

// another iteration of the captured loop while a column wants one; the last
// column to arrive sets the condition
template <typename T>
__device__ void cg_continue(const CgJob<T> &jb, bool go) {
  if (jb.loop == 0) return;
  if (jb.ncol > 1) {
    if (go) atomicOr(jb.meet + 1, 1u);
    __threadfence();
    if (atomicAdd(jb.meet, 1u) + 1 != (unsigned)jb.ncol) return;
    go = atomicExch(jb.meet + 1, 0u) != 0;
    atomicExch(jb.meet, 0u);
  }
  cudaGraphSetConditional(jb.loop, go ? 1u : 0u);
}

// the scalars of a column after its update: rho = r.z
template <typename T>
__device__ void cg_close(const CgJob<T> &jb, int k, double rho, double beta) {
  CgCol &col = jb.cols[k];
  if (jb.init) {
    CgCol c{};
    c.gnew = rho;
    c.tol = jb.tol;
    c.max_passes = jb.max_passes;
    c.active = jb.init == kCgInitKeep || rho > 0.0 ? 1 : 0;
    col = c;
  } else if (col.active) {
    if (col.quick) {
      col.active = 0;
    } else {
      col.gnew = rho;
      const double rms = sqrt(rho / (3.0 * jb.n));
      col.rms = rms;
      const int it = ++col.iters;
      if (jb.hist && it <= jb.nhist) jb.hist[(size_t)k * jb.nhist + it - 1] = rms;
      if (rms < col.tol) {
        col.converged = 1;
        col.active = 0;
      } else {
        col.beta = beta;
        col.gama = beta;  // the reference reuses gama for the beta ratio
      }
    }
  }
  if (!jb.init) ++col.passes;
  jb.cols_h[k] = col;  // page-locked host memory: read after the stream
  if (!jb.init) cg_continue(jb, col.active && col.passes < col.max_passes);
}

template <typename T>
__global__ void __launch_bounds__(TPB) k_cg_dir(const __grid_constant__ Table<CgJob<T>> tab) {
  __shared__ double sh[TPB / 32];
  const CgJob<T> &jb = tab.job[blockIdx.z];
  const int k = blockIdx.y;
  if (k >= jb.ncol || (int)blockIdx.x >= jb.nb) return;
  const CgCol &col = jb.cols[k];
  const double rho = partial_sum(jb.pb + (size_t)k * jb.nb, jb.nb, sh);
  const double gold = jb.init ? 0.0 : col.gold;
  const Scalar mal(jb.init ? 0.0 : -col.alpha);
  const double beta = block_ratio(rho, gold, sh);
  // one thread closes the column while the others go on
  if (blockIdx.x == 0 && threadIdx.x == TPB - 32) cg_close(jb, k, rho, beta);
  const T bt = (T)beta;
  const size_t nv = 3 * (size_t)jb.n, off = (size_t)k * nv;
  T *p = jb.p + off, *r = jb.r + off;
  unsigned mx = 0;
  for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < nv; i += (size_t)jb.nb * TPB) {
    T z;
    if (jb.mode == 0) {
      z = jb.alpha[i / 3] * r[i];
    } else {
      z = jb.z[off + i];
      if (jb.mode == 1 && !jb.init) r[i] = axpy(r[i], mal, jb.h[off + i]);
    }
    if (!jb.init) z = fma(bt, p[i], z);
    p[i] = z;
    if constexpr (sizeof(T) == 8) mx = max(mx, (unsigned)__double2hiint(z) & 0x7FFFFFFFu);
  }
  if (jb.acc && k == 0)
    for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < jb.nacc; i += (size_t)jb.nb * TPB) jb.acc[i] = 0ull;
  if constexpr (sizeof(T) == 8) {
    if (jb.emax) {
      mx = __reduce_max_sync(0xffffffffu, mx);
      if ((threadIdx.x & 31) == 0 && mx) atomicMax(jb.emax + k, mx);
    }
  }
}

// The whole FP64 iteration after the product in one CTA per column, up to
// kCgSmallSites sites: up to 2 elements of each vector per thread, in
// registers.  Bound by the FP64 pipe of its one SM
// and the latency of its two sums: about 10 us at 192 sites (12 with the
// divisions in every thread), seven launches before.
constexpr int SMALL_TPB = 1024, SMALL_PER = 2;
__global__ void __launch_bounds__(SMALL_TPB) k_cg_small(const __grid_constant__ CgJob<double> jb) {
  __shared__ double sh[SMALL_TPB / 32];
  const int k = blockIdx.x, nv = 3 * jb.n;
  CgCol &col = jb.cols[k];
  if (!col.active) {  // uniform
    __syncthreads();
    if (threadIdx.x == 0) cg_close(jb, k, 0.0, 0.0);
    return;
  }
  const size_t off = (size_t)k * nv;
  double *x = jb.x + off, *r = jb.r + off, *p = jb.p + off;
  const double *h = jb.h + off;
  double pv[SMALL_PER], hv[SMALL_PER], zv[SMALL_PER];
  double acc = 0.0;
#pragma unroll
  for (int u = 0; u < SMALL_PER; ++u) {
    const int i = u * blockDim.x + threadIdx.x;
    pv[u] = i < nv ? p[i] : 0.0;
    hv[u] = i < nv ? h[i] : 0.0;
    if (i < nv) acc = fma(pv[u], hv[u], acc);
  }
  const double ph = block_sum(acc, sh, blockDim.x / 32);
  const double gold = col.gnew;
  const bool quick = fabs(ph) < jb.eps;
  const double al = block_ratio(quick ? 0.0 : gold, ph, sh);
  acc = 0.0;
  if (!quick) {
#pragma unroll
    for (int u = 0; u < SMALL_PER; ++u) {
      const int i = u * blockDim.x + threadIdx.x;
      if (i >= nv) continue;
      x[i] = fma(al, pv[u], x[i]);
      const double rn = fma(-al, hv[u], r[i]);
      r[i] = rn;
      zv[u] = jb.alpha[i / 3] * rn;
      acc = fma(rn, zv[u], acc);
    }
  }
  const double rho = block_sum(acc, sh, blockDim.x / 32);
  const double beta = block_ratio(rho, gold, sh);
  // every thread has read the scalars
  if (threadIdx.x == blockDim.x - 32) {
    col.alpha = al;
    col.gold = gold;
    col.gama = ph;
    if (quick) col.quick = 1;
    cg_close(jb, k, rho, beta);
  }
  __shared__ unsigned s_max;
  unsigned mx = 0;
  if (threadIdx.x == 0) s_max = 0;
  if (!quick) {
#pragma unroll
    for (int u = 0; u < SMALL_PER; ++u) {
      const int i = u * blockDim.x + threadIdx.x;
      if (i < nv) {
        const double v = fma(beta, pv[u], zv[u]);
        p[i] = v;
        mx = max(mx, (unsigned)__double2hiint(v) & 0x7FFFFFFFu);
      }
    }
  }
  if (!jb.emax) return;
  __syncthreads();
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) atomicMax(&s_max, mx);
  __syncthreads();
  if (threadIdx.x == 0) jb.emax[k] = s_max;
}

// partial sums of a.b per column
template <typename T>
__global__ void __launch_bounds__(TPB) k_cg_dot(int nb, size_t nv, const T *__restrict__ a, const T *__restrict__ b,
                                                double *__restrict__ part) {
  __shared__ double sh[TPB / 32];
  const size_t off = (size_t)blockIdx.y * nv;
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < nv; i += (size_t)nb * TPB)
    acc = fma((double)a[off + i], (double)b[off + i], acc);
  acc = block_sum(acc, sh, TPB / 32);
  if (threadIdx.x == 0) part[(size_t)blockIdx.y * nb + blockIdx.x] = acc;
}

// y = -(pair sums + scaled-pair corrections) + x / alpha of an FP32 product,
// L lanes per site: the sums from the fixed-point accumulators (NaN when
// flagged) or from the source-split partials, and the partial sums of x.y.
// L = 4 splits a site's list of scaled pairs below kFinishLanesSites (one
// thread per site left 9,003 sites on 71 CTAs: 21 us with 16 splits); above,
// the chip is full with one lane and four would cost FP64 adds.
template <int L>
__global__ void __launch_bounds__(TPB) k_f32_finish(const __grid_constant__ Table<F32Finish> tab) {
  __shared__ double sh[TPB / 32];
  const F32Finish &jb = tab.job[blockIdx.z];
  const int k = blockIdx.y, n = jb.n;
  if (k >= jb.g || (int)blockIdx.x >= jb.nblk) return;
  const int lane = threadIdx.x % L;
  const bool nan = jb.bad && *jb.bad != 0ull;
  double acc = 0.0;
  for (int j = (blockIdx.x * TPB + threadIdx.x) / L; j < n; j += jb.nblk * (TPB / L)) {
    double e[3] = {0.0, 0.0, 0.0};
    if (jb.ri) {
      const float4 pt = jb.pos[j];
      const float at = jb.amoeba ? jb.damp[j] : 0.f;
      for (int q = jb.ri[j] + lane; q < jb.ri[j + 1]; q += L) {
        const int i = jb.src[q];
        const float4 ps = jb.pos[i];
        const float dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        float k3, k5x3;
        if (jb.amoeba)
          dd_kernel<float, true>(r2, pt.w, ps.w, at, jb.damp[i], jb.thr, k3, k5x3);
        else
          dd_kernel<float, false>(r2, pt.w, ps.w, 0.f, 0.f, jb.thr, k3, k5x3);
        const float *mu = jb.x + ((size_t)k * n + i) * 3;
        const float f = k5x3 * (mu[0] * dx + mu[1] * dy + mu[2] * dz);
        const double cs = jb.scale[q] - 1.0;
        e[0] += cs * (double)(f * dx - k3 * mu[0]);
        e[1] += cs * (double)(f * dy - k3 * mu[1]);
        e[2] += cs * (double)(f * dz - k3 * mu[2]);
      }
      if (L > 1) {
        const unsigned group = ((1u << L) - 1u) << ((threadIdx.x & 31) / L * L);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          for (int o = L / 2; o > 0; o >>= 1) e[c] += __shfl_xor_sync(group, e[c], o);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (L > 1 && lane != c) continue;
      const size_t o = ((size_t)k * n + j) * 3 + c;
      double v = e[c];
      if (jb.lo) {
        v += nan ? __longlong_as_double(0x7ff8000000000000ll) : fixed_value(jb.lo[o], jb.hi[o]);
      } else {
        const float *pp = jb.partial + o;
        const size_t st = 3 * (size_t)jb.g * n;
        float sum = 0.f, err = 0.f;
#pragma unroll 4
        for (int s = 0; s < jb.nsplit; ++s) {
          const float q = pp[s * st], t = sum + q, u = t - sum;
          err += (sum - (t - u)) + (q - u);
          sum = t;
        }
        v += (double)sum + (double)err;
      }
      const float xv = jb.x[o], yv = (float)fma((double)xv, jb.ialpha[j], -v);
      jb.y[o] = yv;
      acc = fma((double)xv, (double)yv, acc);
    }
  }
  if (!jb.part) return;
  acc = block_sum(acc, sh, TPB / 32);
  if (threadIdx.x == 0) jb.part[(size_t)k * jb.nblk + blockIdx.x] = acc;
}

// r (refinement residual) of one column block and the partial sums of
// r.(alpha r): rhs - t (t = T mu), or r - scale t32, or r as it is
__global__ void __launch_bounds__(TPB) k_refine(int nb, size_t nv, const double *__restrict__ rhs,
                                                const double *__restrict__ t, const float *__restrict__ t32,
                                                const double *__restrict__ scale, const double *__restrict__ alpha,
                                                double *__restrict__ r, double *__restrict__ part) {
  __shared__ double sh[TPB / 32];
  const int k = blockIdx.y;
  const size_t off = (size_t)k * nv;
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < nv; i += (size_t)nb * TPB) {
    double v;
    if (t32)
      v = r[off + i] - scale[k] * (double)t32[off + i];
    else
      v = t ? rhs[off + i] - t[off + i] : rhs[off + i];
    r[off + i] = v;
    acc = fma(v, alpha[i / 3] * v, acc);
  }
  acc = block_sum(acc, sh, TPB / 32);
  if (threadIdx.x == 0) part[(size_t)k * nb + blockIdx.x] = acc;
}

// one block per column; the sums also to page-locked host memory
__global__ void __launch_bounds__(TPB) k_sum_partials(int nb, const double *__restrict__ part,
                                                      double *__restrict__ out_h) {
  __shared__ double sh[TPB / 32];
  const double s = partial_sum(part + (size_t)blockIdx.x * nb, nb, sh);
  if (threadIdx.x == 0) out_h[blockIdx.x] = s;
}

// f(table, jobs, grid.x, grid.y) for every kCgJobs of the jobs
template <typename J, typename Blocks, typename Cols, typename F>
void for_tables(const J *jobs, int njob, Blocks blocks, Cols cols, F f) {
  for (int b = 0; b < njob; b += kCgJobs) {
    Table<J> tab{};
    const int m = std::min(kCgJobs, njob - b);
    int gx = 0, gy = 0;
    for (int q = 0; q < m; ++q) {
      tab.job[q] = jobs[b + q];
      gx = std::max(gx, blocks(jobs[b + q]));
      gy = std::max(gy, cols(jobs[b + q]));
    }
    if (gx > 0 && gy > 0) f(tab, dim3(gx, gy, m));
  }
}
}  // namespace

int cg_blocks(int n, int ncol, size_t partial_len) {
  const size_t want = (3 * (size_t)n + TPB - 1) / TPB, cap = partial_len / (2 * (size_t)ncol);
  return (int)std::max<size_t>(1, std::min(want, std::min<size_t>(cap, 4 * kRedBlocks)));
}

namespace {
// the near-field launches of the jobs of a table with the Neumann step
void launch_near(const Table<CgJob<float>> &tab, dim3 grid, cudaStream_t st) {
  int near = 0;
  for (unsigned q = 0; q < grid.z; ++q)
    if (tab.job[q].mode == 2) near = std::max(near, tab.job[q].n);
  if (!near) return;
  add_launch_count(2);
  k_cg_near<<<dim3((near + TPB / 8 - 1) / (TPB / 8), grid.y, grid.z), TPB, 0, st>>>(tab);
  k_cg_near_sub<<<grid, TPB, 0, st>>>(tab);
}
}  // namespace

void launch_precondition(const CgJob<float> &job, double *rz_h, cudaStream_t st) {
  Table<CgJob<float>> tab{};
  tab.job[0] = job;
  tab.job[0].init = kCgInitKeep;
  const dim3 grid(job.nb, job.ncol, 1);
  add_launch_count(2);
  k_cg_step<float><<<grid, TPB, 0, st>>>(tab);
  launch_near(tab, grid, st);
  k_sum_partials<<<job.ncol, TPB, 0, st>>>(job.nb, job.pb, rz_h);
}

template <typename T>
void launch_cg_steps(const CgJob<T> *jobs, int njob, cudaStream_t st) {
  for_tables(
      jobs, njob, [](const CgJob<T> &j) { return j.n ? j.nb : 0; }, [](const CgJob<T> &j) { return j.ncol; },
      [&](const Table<CgJob<T>> &tab, dim3 grid) {
        add_launch_count(2);
        k_cg_step<T><<<grid, TPB, 0, st>>>(tab);
        if constexpr (sizeof(T) == 4) launch_near(tab, grid, st);
        k_cg_dir<T><<<grid, TPB, 0, st>>>(tab);
      });
}
template void launch_cg_steps<float>(const CgJob<float> *, int, cudaStream_t);
template void launch_cg_steps<double>(const CgJob<double> *, int, cudaStream_t);

void launch_cg_small(const CgJob<double> &job, cudaStream_t st) {
  add_launch_count(1);
  const int nv = 3 * job.n;
  const int threads = nv <= SMALL_TPB ? (nv + 31) / 32 * 32 : SMALL_TPB;
  k_cg_small<<<job.ncol, threads, 0, st>>>(job);
}

template <typename T>
void launch_cg_dot(int ncol, int nb, size_t nv, const T *a, const T *b, double *part, cudaStream_t st) {
  add_launch_count(1);
  k_cg_dot<T><<<dim3(nb, ncol), TPB, 0, st>>>(nb, nv, a, b, part);
}
template void launch_cg_dot<double>(int, int, size_t, const double *, const double *, double *, cudaStream_t);
template void launch_cg_dot<float>(int, int, size_t, const float *, const float *, double *, cudaStream_t);

F32Finish f32_finish(const DevSites &s, int g, const float *x, float *y) {
  F32Finish j{};
  j.n = s.n, j.g = g, j.amoeba = s.amoeba ? 1 : 0;
  j.pos = s.pol_pos32, j.damp = s.pol_a32, j.x = x, j.ialpha = s.pol_ialpha;
  j.ri = s.d2d_nnz ? s.d2d_ri : nullptr, j.src = s.d2d_src, j.scale = s.d2d_s;
  j.thr = (float)s.damp_thr;
  j.y = y;
  const int lanes = s.n < kFinishLanesSites ? 4 : 1;
  j.nblk = (int)(((size_t)s.n * lanes + TPB - 1) / TPB);
  return j;
}

void launch_f32_finish(const F32Finish *jobs, int njob, cudaStream_t st) {
  // systems of either side of the lane rule in launches of their own
  for (int many = 0; many < 2; ++many) {
    F32Finish sel[kCgJobs];
    int m = 0;
    for (int q = 0; q < njob; ++q) {
      if (jobs[q].n && (jobs[q].n < kFinishLanesSites) == (many == 1)) sel[m++] = jobs[q];
      if (m == kCgJobs || (q == njob - 1 && m)) {
        for_tables(
            sel, m, [](const F32Finish &j) { return j.nblk; }, [](const F32Finish &j) { return j.g; },
            [&](const Table<F32Finish> &tab, dim3 grid) {
              add_launch_count(1);
              if (many)
                k_f32_finish<4><<<grid, TPB, 0, st>>>(tab);
              else
                k_f32_finish<1><<<grid, TPB, 0, st>>>(tab);
            });
        m = 0;
      }
    }
  }
}

void launch_refine(int ncol, int nb, size_t nv, const double *rhs, const double *t, const float *t32,
                   const double *scale, const double *alpha, double *r, double *part, double *out_h, cudaStream_t st) {
  add_launch_count(2);
  k_refine<<<dim3(nb, ncol), TPB, 0, st>>>(nb, nv, rhs, t, t32, scale, alpha, r, part);
  k_sum_partials<<<ncol, TPB, 0, st>>>(nb, part, out_h);
}

}  // namespace gpu
}  // namespace ommp
