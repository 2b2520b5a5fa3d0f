// Dense T (in-core product and the inversion solver): y = T x, and the
// solution of T x = b by an FP32 inverse refined in FP64.
//
// The reference's inversion solver factors T in double precision
// (src/mod_solvers.F90:41-84).  On GB300 an FP64 factorisation of the
// 4,500-row matrix of 1,500 sites cannot take less than 25 ms (FP64 pipe), and
// a column at a time, with a division per element, it took 1.15 s.  T is
// symmetric, and positive definite for every physical system, so here its
// inverse is formed once per geometry in FP32 (1/64 of the cost per
// operation) and each right-hand side is refined with FP64 residuals b - T x
// until they stop decreasing (iterative refinement as in LAPACK's dsposv):
// the result is that of an FP64 solution.  A matrix that is not positive
// definite or a refinement that does not reach FP64 accuracy is left to the
// FP64 LU factorisation (System::inversion64).
//
// The inverse is formed in place by the symmetric block sweep operator: with
// P = A_kk^-1 and C the block column k,
//   A_ij <- A_ij - C_i P C_j^T (i, j != k),  A_ik <- C_i P,  A_kk <- -P,
// which after every block has been swept leaves -A^-1.  Each step is one panel
// kernel (each CTA inverts the 64 x 64 diagonal block for itself and forms
// its rows of C P) and one update of the lower tiles, 64 x 64 x 64 FP32
// multiply-adds each.  The matrix is scaled to a unit diagonal first
// (sqrt(alpha) on both sides) and padded to whole blocks with the identity.
#include <algorithm>
#include <cmath>

#include "kernels.h"

namespace ommp {
namespace gpu {

namespace {

constexpr int SW = 64;      // block size
constexpr int SWT = 256;    // threads: 16 x 16 of 4 x 4 elements
constexpr int SWL = SW + 4; // row length in shared memory (keeps float4 alignment)

__global__ void k_sweep_fill(int nn, int ld, const double *__restrict__ T, const double *__restrict__ s,
                             float *__restrict__ A) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= ld) return;
  float v = i == j ? 1.f : 0.f;
  if (i < nn && j < nn) v = (float)(T[(size_t)i * nn + j] * (s[i] * s[j]));
  A[(size_t)i * ld + j] = v;
}

__global__ void k_sqrt_alpha(int nn, const double *__restrict__ alpha, double *__restrict__ s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nn) s[i] = sqrt(alpha[i / 3]);
}

// acc[4][4] += rows ty of a times rows tx of b (both [SW][SWL], dot over the
// row): a_i . b_j for i = 4 ty + r, j = 4 tx + c
__device__ __forceinline__ void tile_abt(const float (*a)[SWL], const float (*b)[SWL], int ty, int tx,
                                         float (&acc)[4][4]) {
#pragma unroll 4
  for (int k = 0; k < SW; k += 4) {
    float4 u[4], v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      u[r] = *reinterpret_cast<const float4 *>(&a[ty + 16 * r][k]);
      v[r] = *reinterpret_cast<const float4 *>(&b[tx + 16 * r][k]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[r][c] = fmaf(u[r].x, v[c].x, fmaf(u[r].y, v[c].y, fmaf(u[r].z, v[c].z, fmaf(u[r].w, v[c].w, acc[r][c]))));
  }
}

// CTA i: P = A_kk^-1 (every CTA for itself), C_i and W_i = C_i P; i == k: P
__global__ void __launch_bounds__(SWT) k_sweep_panel(int k, int ld, const float *__restrict__ A, float *__restrict__ C,
                                                     float *__restrict__ W, float *__restrict__ P, int *info) {
  __shared__ __align__(16) float sp[SW][SWL], sc[SW][SWL];
  __shared__ float col[2][SW];
  const int i = blockIdx.x, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // the diagonal block, element (ty + 16 r, tx + 16 c) in registers
  float m[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int a = ty + 16 * r, b = tx + 16 * c;
      m[r][c] = A[(size_t)(k * SW + max(a, b)) * ld + k * SW + min(a, b)];
    }
  // this CTA's block of column k
  for (int q = threadIdx.x; q < SW * SW; q += SWT) {
    const int a = q / SW, b = q % SW;
    if (i >= k)
      sc[a][b] = A[(size_t)(i * SW + a) * ld + k * SW + b];
    else
      sc[b][a] = A[(size_t)(k * SW + a) * ld + i * SW + b];
  }
  // sweep the block's columns one by one: m <- -m^-1, symmetric throughout
  bool bad = false;
#pragma unroll
  for (int pc = 0; pc < 4; ++pc)
    for (int pt = 0; pt < 16; ++pt) {
      const int p = pc * 16 + pt;
      if (tx == pt)
#pragma unroll
        for (int r = 0; r < 4; ++r) col[p & 1][ty + 16 * r] = m[r][pc];
      __syncthreads();
      const float piv = col[p & 1][p];
      bad |= !(piv > 0.f) || !(piv < 1e30f);
      const float ip = 1.f / piv;
      float cr[4], cc[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        cr[r] = col[p & 1][ty + 16 * r];
        cc[r] = col[p & 1][tx + 16 * r];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const bool ir = ty + 16 * r == p, ic = tx + 16 * c == p;
          m[r][c] = ir && ic ? -ip : ir ? cc[c] * ip : ic ? cr[r] * ip : fmaf(-cr[r] * ip, cc[c], m[r][c]);
        }
    }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) sp[ty + 16 * r][tx + 16 * c] = -m[r][c];
  __syncthreads();
  if (i == k) {
    if (bad) atomicExch(info, 1);
    for (int q = threadIdx.x; q < SW * SW; q += SWT) P[q] = sp[q / SW][q % SW];
    return;
  }
  float acc[4][4] = {};
  tile_abt(sc, sp, ty, tx, acc);  // P is symmetric
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) W[(size_t)(i * SW + ty + 16 * r) * SW + tx + 16 * c] = acc[r][c];
  for (int q = threadIdx.x; q < SW * SW; q += SWT) C[(size_t)i * SW * SW + q] = sc[q / SW][q % SW];
}

// lower tile (ti, tj): A_ij -= W_i C_j^T; the tiles of block k take W and -P
__global__ void __launch_bounds__(SWT) k_sweep_update(int k, int ld, float *__restrict__ A,
                                                      const float *__restrict__ C, const float *__restrict__ W,
                                                      const float *__restrict__ P) {
  __shared__ __align__(16) float sw[SW][SWL], sc[SW][SWL];
  const int t = blockIdx.x;
  int ti = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  while (ti * (ti + 1) / 2 > t) --ti;
  const int tj = t - ti * (ti + 1) / 2;
  float *tile = A + (size_t)ti * SW * ld + tj * SW;
  if (ti == k || tj == k) {
    for (int q = threadIdx.x; q < SW * SW; q += SWT) {
      const int a = q / SW, b = q % SW;
      tile[(size_t)a * ld + b] = ti == tj ? -P[q]
                                 : tj == k ? W[(size_t)(ti * SW + a) * SW + b]
                                           : W[(size_t)(tj * SW + b) * SW + a];
    }
    return;
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int q = threadIdx.x; q < SW * SW / 4; q += SWT) {
    const int a = q / (SW / 4), b = 4 * (q % (SW / 4));
    *reinterpret_cast<float4 *>(&sw[a][b]) = *reinterpret_cast<const float4 *>(&W[(size_t)(ti * SW + a) * SW + b]);
    *reinterpret_cast<float4 *>(&sc[a][b]) = *reinterpret_cast<const float4 *>(&C[(size_t)(tj * SW + a) * SW + b]);
  }
  __syncthreads();
  float acc[4][4] = {};
  tile_abt(sw, sc, ty, tx, acc);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) tile[(size_t)(ty + 16 * r) * ld + tx + 16 * c] -= acc[r][c];
}

// -A^-1 in the lower tiles -> A^-1 in all of A
__global__ void __launch_bounds__(SWT) k_sweep_finish(int ld, float *__restrict__ A) {
  __shared__ float s[SW][SW + 1];
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  for (int q = threadIdx.x; q < SW * SW; q += SWT)
    s[q / SW][q % SW] = -A[(size_t)(ti * SW + q / SW) * ld + tj * SW + q % SW];
  __syncthreads();
  for (int q = threadIdx.x; q < SW * SW; q += SWT) {
    const int a = q / SW, b = q % SW;
    A[(size_t)(ti * SW + a) * ld + tj * SW + b] = s[a][b];
    if (ti != tj) A[(size_t)(tj * SW + a) * ld + ti * SW + b] = s[b][a];
  }
}

// r32 = s r scale (zero in the padding)
__global__ void k_refine_rhs(int nn, int ld, const double *__restrict__ r, const double *__restrict__ s, double scale,
                             float *__restrict__ r32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ld) r32[i] = i < nn ? (float)(r[i] * s[i] * scale) : 0.f;
}

// x += s (A^-1 r32) / scale, one warp per row
__global__ void __launch_bounds__(256) k_refine_step(int nn, int ld, const float *__restrict__ A,
                                                     const float *__restrict__ r32, const double *__restrict__ s,
                                                     double inv_scale, double *__restrict__ x) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= nn) return;
  const float4 *a = reinterpret_cast<const float4 *>(A + (size_t)row * ld);
  const float4 *v = reinterpret_cast<const float4 *>(r32);
  float acc = 0.f;
#pragma unroll 4
  for (int c = lane; c < ld / 4; c += 32) {
    const float4 p = a[c], q = v[c];
    acc = fmaf(p.x, q.x, fmaf(p.y, q.y, fmaf(p.z, q.z, fmaf(p.w, q.w, acc))));
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) x[row] += s[row] * ((double)acc * inv_scale);
}

// y = T x (rhs null) or y = rhs - T x, one warp per row: T is symmetric, so the
// row is read as the contiguous column; !dodiag leaves the diagonal 1 / alpha
// out.  Memory (8 bytes per element) and the FP64 pipe are near balance; one
// thread per row left most SMs without work below ~20,000 rows.
__global__ void __launch_bounds__(256) k_gemv(int nn, const double *__restrict__ T, const double *__restrict__ x,
                                              const double *__restrict__ rhs, double *__restrict__ y, bool dodiag,
                                              const double *__restrict__ alpha) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= nn) return;
  const double *t = T + (size_t)row * nn;
  const double *xv = x + (size_t)blockIdx.y * nn;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  int c = lane;
  for (; c + 96 < nn; c += 128)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = fma(t[c + 32 * u], xv[c + 32 * u], acc[u]);
  for (; c < nn; c += 32) acc[0] = fma(t[c], xv[c], acc[0]);
  double s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    if (!dodiag) s -= xv[row] / alpha[row / 3];
    const size_t k = (size_t)blockIdx.y * nn + row;
    y[k] = rhs ? rhs[k] - s : s;
  }
}

}  // namespace

void launch_gemv(int nn, const double *T, const double *x, double *y, bool dodiag, const double *alpha, int nrhs,
                 cudaStream_t st) {
  add_launch_count(1);
  k_gemv<<<dim3((nn + 7) / 8, nrhs), 256, 0, st>>>(nn, T, x, nullptr, y, dodiag, alpha);
}

void launch_dense_residual(int nn, const double *T, const double *x, const double *rhs, double *r, cudaStream_t st) {
  add_launch_count(1);
  k_gemv<<<dim3((nn + 7) / 8, 1), 256, 0, st>>>(nn, T, x, rhs, r, true, nullptr);
}

int inverse32_ld(int nn) { return (nn + SW - 1) / SW * SW; }
size_t inverse32_floats(int nn) {
  const size_t ld = inverse32_ld(nn);
  // the matrix, C and W panels, P, a right-hand side
  return ld * ld + 2 * ld * SW + SW * SW + ld;
}

void launch_inverse32(int nn, const double *T, const double *alpha, double *s, float *buf, int *info,
                      cudaStream_t st) {
  const int ld = inverse32_ld(nn), nb = ld / SW;
  float *A = buf, *C = A + (size_t)ld * ld, *W = C + (size_t)ld * SW, *P = W + (size_t)ld * SW;
  cudaMemsetAsync(info, 0, sizeof(int), st);
  add_launch_count(3 + 2 * nb);
  k_sqrt_alpha<<<(nn + 255) / 256, 256, 0, st>>>(nn, alpha, s);
  k_sweep_fill<<<dim3((ld + 255) / 256, ld), 256, 0, st>>>(nn, ld, T, s, A);
  for (int k = 0; k < nb; ++k) {
    k_sweep_panel<<<nb, SWT, 0, st>>>(k, ld, A, C, W, P, info);
    k_sweep_update<<<nb * (nb + 1) / 2, SWT, 0, st>>>(k, ld, A, C, W, P);
  }
  k_sweep_finish<<<dim3(nb, nb), SWT, 0, st>>>(ld, A);
}

void launch_inverse32_step(int nn, float *buf, const double *s, const double *r, double scale, double *x,
                           cudaStream_t st) {
  const int ld = inverse32_ld(nn);
  float *r32 = buf + (size_t)ld * ld + 2 * (size_t)ld * SW + SW * SW;
  add_launch_count(2);
  k_refine_rhs<<<(ld + 255) / 256, 256, 0, st>>>(nn, ld, r, s, scale, r32);
  k_refine_step<<<(nn + 7) / 8, 256, 0, st>>>(nn, ld, buf, r32, s, 1.0 / scale, x);
}

}  // namespace gpu
}  // namespace ommp
