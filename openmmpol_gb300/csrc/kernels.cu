// GB300 (sm_103a) kernels of the induced-point-dipole path.
//
// Finishing passes of the pair kernels (whose pair tensor math is not a dense
// contraction, so no tensor cores), dense T, LU and BLAS-1:
//   k_m2d_finish     fixed-order reduction of the source-split partials plus
//                    the scaled-pair correction pass: for every listed pair
//                    (s - 1) * f_ij is added, which equals the reference's
//                    "skip when s == 0, multiply when s != 1" rule.
//   k_tmu_finish     the FMM's finishing pass: u-scale correction, sign and the
//                    1/alpha diagonal of TMatVec_otf/TMatVec_diag
//                    (src/mod_polarization.F90:459-504).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <type_traits>
#include <vector>

#include "kernels.h"
#include "pair_math.cuh"
#include "pcg.h"

namespace ommp {
namespace gpu {

namespace {
constexpr int TILE = 128;  // sources per tile of the FP32 operator

// Reduce partials and apply the scaled-pair corrections; out [n_ipd][n][3]
// with set 0 = D (direct field, d-scale) and set 1 = P (p-scale) for AMOEBA.
template <bool AMOEBA>
__global__ void k_m2d_finish(int n, int nsplit, const double *__restrict__ partial,
                             const Pos64 *__restrict__ pol_pos, const double *__restrict__ pol_a,
                             const Pos64 *__restrict__ mm_pos, const double *__restrict__ mm_a,
                             const double *__restrict__ mm_q, const float2 *__restrict__ pol_wa,
                             const float2 *__restrict__ mm_wa, const int *__restrict__ ri,
                             const int *__restrict__ src, const double *__restrict__ sP,
                             const double *__restrict__ sD, double thr, float thr2m,
                             double *__restrict__ out) {
  constexpr int LD = AMOEBA ? 10 : 1;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  double e[3] = {0, 0, 0};
  for (int s = 0; s < nsplit; ++s)
    for (int c = 0; c < 3; ++c) e[c] += partial[((size_t)s * n + j) * 3 + c];
  double eP[3] = {e[0], e[1], e[2]}, eD[3] = {e[0], e[1], e[2]};
  Pos64 pt = pol_pos[j];
  double at = AMOEBA ? pol_a[j] : 0.0;
  float2 wat = pol_wa[j];
  for (int k = ri[j]; k < ri[j + 1]; ++k) {
    int i = src[k];
    Pos64 ps = mm_pos[i];
    double q[LD];
    for (int c = 0; c < LD; ++c) q[c] = mm_q[(size_t)i * LD + c];
    double fx = 0, fy = 0, fz = 0;
    // the same reciprocal distance as the pair pass: the excluded pairs are
    // the largest terms and have to cancel
    m2d_pair_f64<AMOEBA>(pt.x - ps.x, pt.y - ps.y, pt.z - ps.z, pt.w, ps.w, at,
                         AMOEBA ? mm_a[i] : 0.0, wat, mm_wa[i], q, thr, thr2m, fx, fy, fz);
    double cp = sP[k] - 1.0, cd = sD[k] - 1.0;
    eP[0] += cp * fx;
    eP[1] += cp * fy;
    eP[2] += cp * fz;
    eD[0] += cd * fx;
    eD[1] += cd * fy;
    eD[2] += cd * fz;
  }
  if (AMOEBA) {
    for (int c = 0; c < 3; ++c) {
      out[(size_t)j * 3 + c] = eD[c];
      out[((size_t)n + j) * 3 + c] = eP[c];
    }
  } else {
    for (int c = 0; c < 3; ++c) out[(size_t)j * 3 + c] = eP[c];
  }
}

// y[r][j] = -(field + scaled-pair corrections) (+ x/alpha): the FMM's finishing pass
template <bool AMOEBA>
__global__ void k_tmu_finish(int n, const double *__restrict__ field, const Pos64 *__restrict__ pos,
                             const double *__restrict__ damp, const float2 *__restrict__ wa,
                             const double *__restrict__ x, const double *__restrict__ alpha, bool dodiag,
                             const int *__restrict__ ri, const int *__restrict__ src,
                             const double *__restrict__ scale, double thr, float thr2m, double *__restrict__ y) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int r = blockIdx.y;
  if (j >= n) return;
  double e[3];
  for (int c = 0; c < 3; ++c) e[c] = field[((size_t)r * n + j) * 3 + c];
  if (ri) {
    const Pos64 pt = pos[j];
    const double at = AMOEBA ? damp[j] : 0.0;
    const float2 wat = wa[j];
    for (int k = ri[j]; k < ri[j + 1]; ++k) {
      int i = src[k];
      const Pos64 ps = pos[i];
      const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      double k3, k5;
      // every operation as in the near field (fmm_near.cu): the excluded pairs
      // are the largest terms and have to cancel
      dd_pair_f64<AMOEBA>(r2, pt.w, ps.w, at, AMOEBA ? damp[i] : 0.0, wat, wa[i], thr, thr2m, k3, k5);
      const double *mu = &x[((size_t)r * n + i) * 3];
      const double f = 3.0 * k5 * fma(mu[0], dx, fma(mu[1], dy, mu[2] * dz));
      const double cs = scale[k] - 1.0;
      e[0] = fma(cs, fma(f, dx, -(k3 * mu[0])), e[0]);
      e[1] = fma(cs, fma(f, dy, -(k3 * mu[1])), e[1]);
      e[2] = fma(cs, fma(f, dz, -(k3 * mu[2])), e[2]);
    }
  }
  const double *xj = &x[((size_t)r * n + j) * 3];
  double *yj = &y[((size_t)r * n + j) * 3];
  double ia = dodiag ? 1.0 / alpha[j] : 0.0;
  for (int c = 0; c < 3; ++c) yj[c] = -e[c] + (dodiag ? xj[c] * ia : 0.0);
}

// ---------------------------------------------------------------------------
// dense T matrix (create_tmat / dipole_T, src/mod_polarization.F90:327-435)
// ---------------------------------------------------------------------------
template <bool AMOEBA>
__global__ void k_build_tmat(int n, const Pos64 *__restrict__ pos, const double *__restrict__ damp,
                             const double *__restrict__ alpha, double thr, double *__restrict__ T) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;  // row block (target)
  int i = blockIdx.y;                             // column block (source)
  if (j >= n) return;
  size_t nn = 3 * (size_t)n;
  double blk[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (i == j) {
    double ia = 1.0 / alpha[j];
    blk[0][0] = blk[1][1] = blk[2][2] = ia;
  } else {
    Pos64 pt = pos[j], ps = pos[i];
    double d[3] = {pt.x - ps.x, pt.y - ps.y, pt.z - ps.z};
    double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    double k3, k5x3;
    dd_kernel<double, AMOEBA>(r2, pt.w, ps.w, AMOEBA ? damp[j] : 0.0, AMOEBA ? damp[i] : 0.0, thr,
                              k3, k5x3);
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) blk[a][b] = (a == b ? k3 : 0.0) - k5x3 * d[a] * d[b];
  }
  for (int b = 0; b < 3; ++b)
    for (int a = 0; a < 3; ++a) T[(3 * (size_t)i + b) * nn + 3 * (size_t)j + a] = blk[a][b];
}

// multiply the listed off-diagonal blocks by their u-scale
__global__ void k_scale_tmat(int n, const int *__restrict__ ri, const int *__restrict__ src,
                             const double *__restrict__ scale, double *__restrict__ T) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  size_t nn = 3 * (size_t)n;
  for (int k = ri[j]; k < ri[j + 1]; ++k) {
    int i = src[k];
    double s = scale[k];
    for (int b = 0; b < 3; ++b)
      for (int a = 0; a < 3; ++a) T[(3 * (size_t)i + b) * nn + 3 * (size_t)j + a] *= s;
  }
}

// LU: pivot search in column k (one block), swap, update, scale
__global__ void k_lu_pivot(int nn, int k, double *A, int *piv, int *info) {
  __shared__ double sv[1024];
  __shared__ int si[1024];
  double best = -1.0;
  int bi = k;
  for (int r = k + threadIdx.x; r < nn; r += blockDim.x) {
    double v = fabs(A[(size_t)k * nn + r]);
    if (v > best) {
      best = v;
      bi = r;
    }
  }
  sv[threadIdx.x] = best;
  si[threadIdx.x] = bi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      double o = sv[threadIdx.x + s];
      int oi = si[threadIdx.x + s];
      if (o > sv[threadIdx.x] || (o == sv[threadIdx.x] && oi < si[threadIdx.x])) {
        sv[threadIdx.x] = o;
        si[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    piv[k] = si[0];
    if (sv[0] == 0.0 && *info == 0) *info = k + 1;
  }
}

__global__ void k_lu_swap(int nn, int k, double *A, const int *piv) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  int p = piv[k];
  if (c >= nn || p == k) return;
  double t = A[(size_t)c * nn + k];
  A[(size_t)c * nn + k] = A[(size_t)c * nn + p];
  A[(size_t)c * nn + p] = t;
}

__global__ void k_lu_update(int nn, int k, double *A, const int *info) {
  if (*info) return;
  int r = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;
  int c = k + 1 + blockIdx.y;
  if (r >= nn || c >= nn) return;
  double l = A[(size_t)k * nn + r] / A[(size_t)k * nn + k];
  A[(size_t)c * nn + r] -= l * A[(size_t)c * nn + k];
}

__global__ void k_lu_scale(int nn, int k, double *A, const int *info) {
  if (*info) return;
  int r = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nn) return;
  A[(size_t)k * nn + r] /= A[(size_t)k * nn + k];
}

// forward/back substitution for one rhs (single block)
__global__ void k_lu_solve(int nn, const double *A, const int *piv, double *b) {
  for (int k = 0; k < nn; ++k) {  // apply the row interchanges in order
    if (threadIdx.x == 0) {
      int p = piv[k];
      if (p != k) {
        double t = b[k];
        b[k] = b[p];
        b[p] = t;
      }
    }
  }
  __syncthreads();
  for (int k = 0; k < nn; ++k) {
    double bk = b[k];
    for (int r = k + 1 + threadIdx.x; r < nn; r += blockDim.x) b[r] -= A[(size_t)k * nn + r] * bk;
    __syncthreads();
  }
  for (int k = nn - 1; k >= 0; --k) {
    if (threadIdx.x == 0) b[k] /= A[(size_t)k * nn + k];
    __syncthreads();
    double bk = b[k];
    for (int r = threadIdx.x; r < k; r += blockDim.x) b[r] -= A[(size_t)k * nn + r] * bk;
    __syncthreads();
  }
}

// The source-split partials [nsplit][total] summed into the first block: 32
// values per block, its 8 warps take every eighth split, added in warp order.
// One thread per value was a chain of nsplit loads in kernels of a few blocks:
// 83 us for the static sums' finishing pass at 6,000 sites (39 to 65 splits),
// 90 us for 40 external points (282 splits).
__global__ void __launch_bounds__(256) k_sum_splits(size_t total, int nsplit, double *partial) {
  __shared__ double sh[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t k = (size_t)blockIdx.x * 32 + lane;
  double s = 0.0;
  if (k < total) {
#pragma unroll 4
    for (int p = w; p < nsplit; p += 8) s += partial[(size_t)p * total + k];
  }
  sh[w][lane] = s;
  __syncthreads();
  if (w || k >= total) return;
  for (int v = 1; v < 8; ++v) s += sh[v][lane];
  partial[k] = s;
}

// ---------------------------------------------------------------------------
// BLAS-1 with deterministic two-stage reductions
// ---------------------------------------------------------------------------
// Columns run side by side (blockIdx.y = column), not one after another
// inside a block, and each thread sums about 8 elements of its column with
// four independent loads in flight: a block-serial column loop with ~2
// elements per thread left the 64-column dots of a batch latency-bound (1.4
// TB/s).  gridDim.x blocks of a column write partial[b][k]; the rows from
// gridDim.x to kRedBlocks are zeroed so that the fixed-order reduction over
// kRedBlocks rows is unchanged.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_dots(int ncol, size_t n, const T *__restrict__ a,
                                                      const T *__restrict__ b, size_t bstride,
                                                      double *__restrict__ partial) {
  __shared__ double sh[kRedThreads / 32];
  const int k = blockIdx.y;
  const T *ak = a + (size_t)k * n;
  const T *bk = b + (size_t)k * bstride;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] += (double)ak[i + u * stride] * (double)bk[i + u * stride];
  }
  for (; i < n; i += stride) acc[0] += (double)ak[i] * (double)bk[i];
  double s0 = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  for (int o = 16; o > 0; o >>= 1) s0 += __shfl_down_sync(0xffffffffu, s0, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s0;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kRedThreads / 32; ++w) s += sh[w];
    partial[(size_t)blockIdx.x * ncol + k] = s;
  }
  if (blockIdx.x == 0)
    for (int r = gridDim.x + threadIdx.x; r < kRedBlocks; r += blockDim.x) partial[(size_t)r * ncol + k] = 0.0;
}

// blocks per column of k_dots: about 8 elements per thread
inline int dots_blocks(size_t n) {
  size_t b = (n + (size_t)kRedThreads * 8 - 1) / ((size_t)kRedThreads * 8);
  if (b < 1) b = 1;
  if (b > (size_t)kRedBlocks) b = kRedBlocks;
  return (int)b;
}

__global__ void k_reduce_partials(int ncol, int nb, const double *__restrict__ partial,
                                  double *__restrict__ result) {
  // one warp per column, fixed lane order then fixed tree
  int k = blockIdx.x;
  double acc = 0.0;
  for (int b = threadIdx.x; b < nb; b += 32) acc += partial[(size_t)b * ncol + k];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (threadIdx.x == 0) result[k] = acc;
}

__global__ void k_axpby(size_t n, double a, const double *x, double b, double *y) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}
__global__ void k_add(size_t n, const double *a, const double *b, double *out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = a[i] + b[i];
}
__global__ void k_scale_alpha(int nrhs, int n, const double *alpha, const double *x, double *y) {
  size_t tot = (size_t)nrhs * n * 3;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x)
    y[i] = alpha[(i / 3) % n] * x[i];
}
__global__ void k_to_f32(size_t n, const double *x, const double *scale, float *y) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = (float)(x[i] * (scale ? *scale : 1.0));
}
// ncol columns of nv values, column k scaled by scale[k], in one launch
__global__ void k_to_f32_cols(size_t nv, size_t tot, const double *x, const double *scale, float *y) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x)
    y[i] = (float)(x[i] * scale[i / nv]);
}

__global__ void k_ir_accumulate(int ncol, int n, double *mu, const float *d32, const double *scale) {
  size_t nv = 3 * (size_t)n;
  size_t tot = nv * ncol;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x)
    mu[i] += scale[i / nv] * (double)d32[i];
}

__global__ void k_residual(size_t tot, const double *rhs, const double *tmu, double *r) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x)
    r[i] = rhs[i] - tmu[i];
}

__global__ void k_lincomb(int nvec, size_t n, const double *X, size_t ldx, const double *c, double *out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int v = 0; v < nvec; ++v) acc += c[v] * X[(size_t)v * ldx + i];
    out[i] = acc;
  }
}

__global__ void __launch_bounds__(kRedThreads) k_diff_norms(size_t n, const double *a, const double *b,
                                                            double *partial) {
  __shared__ double s1[kRedThreads / 32], s2[kRedThreads / 32];
  double sq = 0.0, mx = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double d = a[i] - b[i];
    sq += d * d;
    mx = fmax(mx, fabs(d));
  }
  for (int o = 16; o > 0; o >>= 1) {
    sq += __shfl_down_sync(0xffffffffu, sq, o);
    mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) {
    s1[threadIdx.x >> 5] = sq;
    s2[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a1 = 0.0, a2 = 0.0;
    for (int w = 0; w < kRedThreads / 32; ++w) {
      a1 += s1[w];
      a2 = fmax(a2, s2[w]);
    }
    partial[2 * blockIdx.x] = a1;
    partial[2 * blockIdx.x + 1] = a2;
  }
}

__global__ void k_reduce_norms(int nb, const double *partial, double *out) {
  double a1 = 0.0, a2 = 0.0;
  for (int b = threadIdx.x; b < nb; b += 32) {
    a1 += partial[2 * b];
    a2 = fmax(a2, partial[2 * b + 1]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    a1 += __shfl_down_sync(0xffffffffu, a1, o);
    a2 = fmax(a2, __shfl_down_sync(0xffffffffu, a2, o));
  }
  if (threadIdx.x == 0) {
    out[0] = a1;
    out[1] = a2;
  }
}

__global__ void k_any_diff(size_t n, const double *a, const double *b, int *flag) {
  const unsigned long long *ua = reinterpret_cast<const unsigned long long *>(a);
  const unsigned long long *ub = reinterpret_cast<const unsigned long long *>(b);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (ua[i] != ub[i]) {
      *flag = 1;
      return;
    }
}

// Pipe-throughput calibration: 8 independent FMA chains per thread.
template <typename T>
__global__ void __launch_bounds__(256) k_fma_peak(T *out, int iters, T a, T b) {
  T x0 = (T)threadIdx.x, x1 = x0 + T(1), x2 = x0 + T(2), x3 = x0 + T(3);
  T x4 = x0 + T(4), x5 = x0 + T(5), x6 = x0 + T(6), x7 = x0 + T(7);
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b);
    x1 = fma(x1, a, b);
    x2 = fma(x2, a, b);
    x3 = fma(x3, a, b);
    x4 = fma(x4, a, b);
    x5 = fma(x5, a, b);
    x6 = fma(x6, a, b);
    x7 = fma(x7, a, b);
  }
  T s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == T(-1.2345)) out[blockIdx.x] = s;  // keeps the chains alive
}

// thr^2 with the relative safety margin of the FP32 damping pre-test
inline float damp_thr2_margin(const DevSites &s) {
  return (float)(s.damp_thr * s.damp_thr * (1.0 + 1e-5));
}

inline int blocks_for(size_t n, int tpb, int cap = 4 * 152 * 4) {
  size_t b = (n + tpb - 1) / tpb;
  if (b < 1) b = 1;
  if (b > (size_t)cap) b = cap;
  return (int)b;
}

}  // namespace

// kernels launched by the library: process total, and per host thread (the
// server drives several systems from several threads; a graph capture
// subtracts the kernels its own thread recorded, not those of the others)
static std::atomic<long long> g_launches{0};
static thread_local long long t_launches = 0;
long long launch_count() { return g_launches.load(std::memory_order_relaxed); }
long long thread_launch_count() { return t_launches; }
void add_launch_count(long long k) {
  g_launches.fetch_add(k, std::memory_order_relaxed);
  t_launches += k;
}

double launch_fma_peak(bool fp64, int iters, void *out, cudaStream_t st) {
  int blocks = sm_count() * 8, threads = 256;
  add_launch_count(1);
  if (fp64)
    k_fma_peak<double><<<blocks, threads, 0, st>>>((double *)out, iters, 0.999999, 1e-7);
  else
    k_fma_peak<float><<<blocks, threads, 0, st>>>((float *)out, iters, 0.999999f, 1e-7f);
  return 2.0 * 8.0 * (double)iters * blocks * threads;  // flop
}

int sm_count() {
  static std::atomic<int> cached{0};  // read by several server threads
  int v = cached.load(std::memory_order_relaxed);
  if (!v) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (v <= 0) v = 152;
    cached.store(v, std::memory_order_relaxed);
  }
  return v;
}

int launch_sum_splits(size_t total, int nsplit, double *partial, cudaStream_t st) {
  if (nsplit <= 4 || total == 0) return nsplit;
  add_launch_count(1);
  k_sum_splits<<<(unsigned)((total + 31) / 32), 256, 0, st>>>(total, nsplit, partial);
  return 1;
}

// ---- M2D -----------------------------------------------------------------
// split partials -> FP64 scaled-pair corrections -> D and P sets
static void m2d_finish(const DevSites &s, double *out, const double *scratch, int nsplit, cudaStream_t st) {
  int fb = (s.n + 127) / 128;
  if (s.amoeba)
    k_m2d_finish<true><<<fb, 128, 0, st>>>(s.n, nsplit, scratch, s.pol_pos, s.pol_a, s.mm_pos, s.mm_a, s.mm_q,
                                           s.pol_wa32, s.mm_wa32, s.m2d_ri, s.m2d_src, s.m2d_sP, s.m2d_sD,
                                           s.damp_thr, damp_thr2_margin(s), out);
  else
    k_m2d_finish<false><<<fb, 128, 0, st>>>(s.n, nsplit, scratch, s.pol_pos, s.pol_a, s.mm_pos, s.mm_a,
                                            s.mm_q, s.pol_wa32, s.mm_wa32, s.m2d_ri, s.m2d_src, s.m2d_sP,
                                            s.m2d_sD, s.damp_thr, damp_thr2_margin(s), out);
}

void launch_m2d_finish(const DevSites &s, double *out, double *partial, int nsplit, cudaStream_t st) {
  add_launch_count(1);
  m2d_finish(s, out, partial, launch_sum_splits(3 * (size_t)s.n, nsplit, partial, st), st);
}

// ---- T.mu -----------------------------------------------------------------
int tmu32_max_split(const DevSites &s, int sms) {
  const int tiles = (s.n + TILE - 1) / TILE;
  return std::max(1, std::min(2 * tmu32_pick_split(s, sms), tiles));
}

size_t tmu_scratch_doubles(const DevSites &s, int nrhs, int nsplit) {
  return (size_t)nsplit * nrhs * s.n * 3;
}

// Columns per launch: the widest of 8/4/2/1 not above what is left and gmax.
inline int column_group(int left, int gmax) {
  int g = left < gmax ? left : gmax;
  return g >= 8 ? 8 : (g >= 4 ? 4 : (g >= 2 ? 2 : 1));
}

// the tiled kernel on columns in groups sharing the pair geometry; every
// group has its own [split][g][n][3] block of partials, one after the other
static void tmu_dispatch(const DevSites &s, int nrhs, const float *x, float *partial, int nsplit, int gmax,
                         cudaStream_t st) {
  for (int done = 0; done < nrhs;) {
    const int g = column_group(nrhs - done, gmax), groups = (nrhs - done) / g;
    const size_t xo = (size_t)done * s.n * 3;
    add_launch_count(1);
    launch_tmu32_pairs(s, g, groups, x + xo, partial + nsplit * xo, nsplit, st);
    done += g * groups;
  }
}

void launch_tmu_finish64(const DevSites &s, int nrhs, const double *partial, const double *x, bool dodiag,
                         double *y, cudaStream_t st) {
  add_launch_count(1);
  const dim3 grid((s.n + 127) / 128, nrhs);
  const int *ri = s.d2d_nnz ? s.d2d_ri : nullptr;
  if (s.amoeba)
    k_tmu_finish<true><<<grid, 128, 0, st>>>(s.n, partial, s.pol_pos, s.pol_a, s.pol_wa32, x, s.pol_alpha, dodiag, ri,
                                             s.d2d_src, s.d2d_s, s.damp_thr, damp_thr2_margin(s), y);
  else
    k_tmu_finish<false><<<grid, 128, 0, st>>>(s.n, partial, s.pol_pos, s.pol_a, s.pol_wa32, x, s.pol_alpha, dodiag,
                                              ri, s.d2d_src, s.d2d_s, s.damp_thr, damp_thr2_margin(s), y);
}

int launch_tmu_f32(const DevSites &s, int nrhs, const float *x, float *y, float *scratch, int nsplit, cudaStream_t st,
                   int gmax, int kver, double *sym_scratch, bool prepared, double *part, int max_part) {
  if (s.n == 0) return 0;
  const size_t nv = 3 * (size_t)s.n;
  if (kver == 1) {
    const int parts = tmu32_rows_parts(s.n);
    if (parts > max_part) part = nullptr;
    launch_tmu32_rows(s, nrhs, gmax, x, y, part, st);
    return part ? parts : 0;
  }
  const bool sym = kver == 3 && sym_scratch;
  if (!sym) tmu_dispatch(s, nrhs, x, scratch, nsplit, gmax, st);
  int npart = 0;
  std::vector<F32Finish> fins;
  for (int c = 0; c < nrhs;) {
    const int g = column_group(nrhs - c, sym ? std::min(gmax, 2) : gmax);
    F32Finish fin = f32_finish(s, g, x + c * nv, y + c * nv);
    if (sym) {
      // fixed-point sums, read out by the finishing pass
      const size_t C = 3 * (size_t)g;
      unsigned long long *lo = reinterpret_cast<unsigned long long *>(sym_scratch);
      unsigned long long *hi = lo + C * s.n;
      unsigned long long *bad = lo + 3 * C * s.n;
      if (!prepared) {
        cudaMemsetAsync(lo, 0, 2 * C * s.n * sizeof(unsigned long long), st);
        cudaMemsetAsync(bad, 0, 2 * sizeof(unsigned long long), st);
      }
      SymSlice one{&s, x + c * nv, lo, hi, bad, 0, tmu32_sym_items(s, g)};
      launch_tmu32_sym_multi(g, &one, 1, reinterpret_cast<unsigned *>(bad + 1), st, true);
      fin.lo = lo, fin.hi = hi, fin.bad = bad;
    } else {
      fin.partial = scratch + (size_t)nsplit * c * nv;
      fin.nsplit = nsplit;
    }
    if (part) {
      npart = fin.nblk = std::min(fin.nblk, max_part);
      fin.part = part + (size_t)c * npart;
    }
    if (sym)
      launch_f32_finish(&fin, 1, st);
    else
      fins.push_back(fin);
    c += g;
  }
  launch_f32_finish(fins.data(), (int)fins.size(), st);
  return npart;
}

// Batched right-hand sides, set-major columns: rhs[s*nf + f] = E_M2D[s] + field[f]
__global__ void k_batch_rhs(int n, int nf, int nset, const double *__restrict__ e_m2d,
                            const double *__restrict__ fields, double *__restrict__ rhs) {
  size_t nv = 3 * (size_t)n;
  size_t tot = nv * nf * nset;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x) {
    size_t col = i / nv, e = i % nv;
    size_t set = col / nf, f = col % nf;
    rhs[i] = e_m2d[set * nv + e] + fields[f * nv + e];
  }
}

// out[f][s][n][3] from set-major solution columns; with nsolved == 1 the P
// set repeats the D column (identical systems)
__global__ void k_batch_scatter(int n, int nf, int nipd, int nsolved, const double *__restrict__ x,
                                double *__restrict__ out) {
  size_t nv = 3 * (size_t)n;
  size_t tot = nv * nf * nipd;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x) {
    size_t e = i % nv, rest = i / nv;
    size_t set = rest % nipd, f = rest / nipd;
    size_t src_set = nsolved == 1 ? 0 : set;
    out[i] = x[(src_set * nf + f) * nv + e];
  }
}

void launch_batch_rhs(int n, int nf, int nset, const double *e_m2d, const double *fields, double *rhs,
                      cudaStream_t st) {
  add_launch_count(1);
  k_batch_rhs<<<blocks_for((size_t)3 * n * nf * nset, 256), 256, 0, st>>>(n, nf, nset, e_m2d, fields, rhs);
}

void launch_batch_scatter(int n, int nf, int nipd, int nsolved, const double *x, double *out, cudaStream_t st) {
  add_launch_count(1);
  k_batch_scatter<<<blocks_for((size_t)3 * n * nf * nipd, 256), 256, 0, st>>>(n, nf, nipd, nsolved, x, out);
}

// ---- dense T ------------------------------------------------------------------
void launch_build_tmat(const DevSites &s, double *tmat, cudaStream_t st) {
  add_launch_count(s.d2d_nnz ? 2 : 1);
  dim3 grid((s.n + 127) / 128, s.n);
  if (s.amoeba)
    k_build_tmat<true><<<grid, 128, 0, st>>>(s.n, s.pol_pos, s.pol_a, s.pol_alpha, s.damp_thr, tmat);
  else
    k_build_tmat<false><<<grid, 128, 0, st>>>(s.n, s.pol_pos, s.pol_a, s.pol_alpha, s.damp_thr, tmat);
  if (s.d2d_nnz) k_scale_tmat<<<(s.n + 127) / 128, 128, 0, st>>>(s.n, s.d2d_ri, s.d2d_src, s.d2d_s, tmat);
}

void launch_lu_factor(int nn, double *A, int *piv, int *info, double *work, cudaStream_t st) {
  (void)work;
  cudaMemsetAsync(info, 0, sizeof(int), st);
  for (int k = 0; k < nn; ++k) {
    add_launch_count(nn - k - 1 > 0 ? 4 : 2);
    k_lu_pivot<<<1, 1024, 0, st>>>(nn, k, A, piv, info);
    k_lu_swap<<<(nn + 255) / 256, 256, 0, st>>>(nn, k, A, piv);
    int rows = nn - k - 1;
    if (rows > 0) {
      dim3 g((rows + 127) / 128, rows);
      k_lu_update<<<g, 128, 0, st>>>(nn, k, A, info);
      k_lu_scale<<<(rows + 127) / 128, 128, 0, st>>>(nn, k, A, info);
    }
  }
}

void launch_lu_solve(int nn, const double *A, const int *piv, double *b, cudaStream_t st) {
  add_launch_count(1);
  k_lu_solve<<<1, 1024, 0, st>>>(nn, A, piv, b);
}

// ---- BLAS-1 ---------------------------------------------------------------------
void launch_dots(int ncol, size_t n, const double *a, const double *b, double *partial, cudaStream_t st) {
  if (ncol < 1) return;
  add_launch_count(1);
  k_dots<double><<<dim3(dots_blocks(n), ncol), kRedThreads, 0, st>>>(ncol, n, a, b, n, partial);
}
void launch_dots_bcast(int ncol, size_t n, const double *a, const double *b, double *partial,
                       cudaStream_t st) {
  if (ncol < 1) return;
  add_launch_count(1);
  k_dots<double><<<dim3(dots_blocks(n), ncol), kRedThreads, 0, st>>>(ncol, n, a, b, 0, partial);
}
void launch_reduce_partials(int ncol, const double *partial, double *result, cudaStream_t st) {
  add_launch_count(1);
  k_reduce_partials<<<ncol, 32, 0, st>>>(ncol, kRedBlocks, partial, result);
}
void launch_axpby(size_t n, double a, const double *x, double b, double *y, cudaStream_t st) {
  add_launch_count(1);
  k_axpby<<<blocks_for(n, 256), 256, 0, st>>>(n, a, x, b, y);
}
void launch_add(size_t n, const double *a, const double *b, double *out, cudaStream_t st) {
  add_launch_count(1);
  k_add<<<blocks_for(n, 256), 256, 0, st>>>(n, a, b, out);
}
void launch_scale_by_alpha(int nrhs, int n, const double *alpha, const double *x, double *y, cudaStream_t st) {
  add_launch_count(1);
  k_scale_alpha<<<blocks_for((size_t)nrhs * n * 3, 256), 256, 0, st>>>(nrhs, n, alpha, x, y);
}
void launch_to_f32_cols(int ncol, size_t nv, const double *x, const double *scale, float *y, cudaStream_t st) {
  if (ncol < 1 || nv == 0) return;
  add_launch_count(1);
  const size_t tot = nv * (size_t)ncol;
  k_to_f32_cols<<<blocks_for(tot, 256), 256, 0, st>>>(nv, tot, x, scale, y);
}
void launch_to_f32(size_t n, const double *x, const double *scale, float *y, cudaStream_t st) {
  add_launch_count(1);
  k_to_f32<<<blocks_for(n, 256), 256, 0, st>>>(n, x, scale, y);
}
void launch_ir_accumulate(int ncol, int n, double *mu, const float *d32, const double *scale, cudaStream_t st) {
  add_launch_count(1);
  k_ir_accumulate<<<blocks_for((size_t)ncol * n * 3, 256), 256, 0, st>>>(ncol, n, mu, d32, scale);
}
void launch_residual(size_t total, const double *rhs, const double *tmu, double *r, cudaStream_t st) {
  add_launch_count(1);
  k_residual<<<blocks_for(total, 256), 256, 0, st>>>(total, rhs, tmu, r);
}
void launch_lincomb(int nvec, size_t n, const double *X, size_t ldx, const double *c, double *out,
                    cudaStream_t st) {
  add_launch_count(1);
  k_lincomb<<<blocks_for(n, 256), 256, 0, st>>>(nvec, n, X, ldx, c, out);
}
void launch_diff_norms(size_t n, const double *a, const double *b, double *partial, cudaStream_t st) {
  add_launch_count(1);
  k_diff_norms<<<kRedBlocks, kRedThreads, 0, st>>>(n, a, b, partial);
}
void launch_reduce_norms(const double *partial, double *out, cudaStream_t st) {
  add_launch_count(1);
  k_reduce_norms<<<1, 32, 0, st>>>(kRedBlocks, partial, out);
}
void launch_any_diff(size_t n, const double *a, const double *b, int *flag, cudaStream_t st) {
  add_launch_count(1);
  k_any_diff<<<blocks_for(n, 256), 256, 0, st>>>(n, a, b, flag);
}

}  // namespace gpu
}  // namespace ommp
