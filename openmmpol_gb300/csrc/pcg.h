// Fused conjugate-gradient steps (pcg.cu) of the FP64 and FP32 solvers and of
// the multi-system engine.
#pragma once
#include "kernels.h"

namespace ommp {
namespace gpu {

constexpr int kCgJobs = 16;          // systems per launch
constexpr int kCgSmallSites = 682;   // one CTA per column up to here (2 x 1024 elements)
enum { kCgInitZero = 1, kCgInitKeep = 2 };

template <typename T>
struct CgJob {
  int n, ncol;
  int mode;  // preconditioner: 0 diagonal, 1 block Jacobi, 2 with the Neumann step
  int init;  // 0: an iteration after a product; else the start: r.z and p = z,
             // with x cleared (kCgInitZero) or kept (kCgInitKeep)
  int na, nb;  // partial sums per column of p.h and of r.z
  int nhist;
  int max_passes;   // iterations of the loop (put into the columns at the start, as tol)
  double eps, tol;  // |p.h| of the quick exit; convergence threshold
  T *x, *r, *p, *h, *z, *w;  // [ncol][n][3]; z and w of modes 1 and 2
  const T *alpha;            // polarizability, mode 0
  const int4 *info;
  const float *minv;
  const int *ri, *ci;
  const float *blk;
  double *pa, *pb;  // [ncol][na], [ncol][nb]
  CgCol *cols, *cols_h;
  double *hist;
  // the next product's accumulators and control words (or null)
  unsigned long long *acc, *words;
  size_t nacc;
  // largest high word of |p| of each column for the next FP64 product (or null)
  unsigned *emax;
  // loop on the device: the condition of the captured loop (0: none), and two
  // words, zero between iterations, where the columns meet to set it
  cudaGraphConditionalHandle loop;
  unsigned *meet;
};

struct F32Finish {
  int n, g, amoeba, nsplit, nblk;
  float thr;
  const float4 *pos;
  const float *damp, *x;
  const double *ialpha;
  const int *ri, *src;
  const double *scale;
  const unsigned long long *lo, *hi, *bad;  // fixed-point sums, or null and:
  const float *partial;                     // [nsplit][g][n][3]
  float *y;
  double *part;  // [g][nblk] or null
};

// blocks (and partial sums) per column of the steps; two sets of partial sums
// of ncol columns fit into partial_len doubles
int cg_blocks(int n, int ncol, size_t partial_len);
// the launches of one iteration (or of the start) after the product
template <typename T>
void launch_cg_steps(const CgJob<T> *jobs, int njob, cudaStream_t st);
// z = M^-1 r of modes 1 and 2, and r.z per column (any mode) to pinned memory
void launch_precondition(const CgJob<float> &job, double *rz_h, cudaStream_t st);
void launch_cg_small(const CgJob<double> &job, cudaStream_t st);
template <typename T>
void launch_cg_dot(int ncol, int nb, size_t nv, const T *a, const T *b, double *part, cudaStream_t st);
// finishing pass of an FP32 product (sums, partial sums of x.y set by the caller)
F32Finish f32_finish(const DevSites &s, int g, const float *x, float *y);
void launch_f32_finish(const F32Finish *jobs, int njob, cudaStream_t st);
// refinement residual and its preconditioned norms (squared) to pinned memory
void launch_refine(int ncol, int nb, size_t nv, const double *rhs, const double *t, const float *t32,
                   const double *scale, const double *alpha, double *r, double *part, double *out_h, cudaStream_t st);

}  // namespace gpu
}  // namespace ommp
