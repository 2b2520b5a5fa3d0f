// Launch interface of the GB300 kernels (implemented in kernels.cu).
//
// Layout conventions (device memory, all 0-based):
//   site arrays are structure-of-arrays or packed Pos64 (x, y, z, w);
//   field / dipole vectors are [nrhs][n][3] contiguous (C order), the same
//   as the reference's Fortran (3, n, n_ipd) arrays seen from C.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace ommp {
namespace gpu {

// One site: position and a per-site scalar, 32-byte aligned so that a tile
// load is two 16-byte transactions per thread.
struct __align__(32) Pos64 {
  double x, y, z, w;
};

// Immutable per-geometry device data of one system.
constexpr int kNoExponent = -4096;
// 2^e of a scaling of values of the exponent e: nothing to scale when there are
// none or they are within 2^-4 to 2^4 (a few bits more or less are not missed)
__host__ __device__ inline int scaling_exponent(int e) { return e == kNoExponent || (e >= -4 && e < 4) ? 0 : e; }

struct DevSites {
  int n = 0;      // polarizable sites
  int m = 0;      // MM (static) sites
  bool amoeba = false;
  // polarizable sites
  Pos64 *pol_pos = nullptr;   // x, y, z, 1/thole
  double *pol_a = nullptr;      // Thole damping a
  double *pol_alpha = nullptr;  // polarizability
  double *pol_ialpha = nullptr;  // and its reciprocal
  int *polar_mm = nullptr;      // mm index of each polarizable site
  float4 *pol_pos32 = nullptr;  // centred FP32 copy: x, y, z, 1/thole
  float *pol_a32 = nullptr;
  float2 *pol_wa32 = nullptr;   // (1/thole)^2, a^2 in FP32: damping pre-test of the FP64 kernels
  float2 *mm_wa32 = nullptr;    // same for the static sites (inf when not polarizable)
  // static sites
  Pos64 *mm_pos = nullptr;    // x, y, z, thole (0 when not polarizable)
  double *mm_a = nullptr;       // damping a of the source (AMOEBA)
  double *mm_q = nullptr;       // [m][ld] lab-frame multipoles
  // their largest magnitude is in [2^q_e, 2^(q_e + 1)) (before the rotation of
  // the frames, which changes a value at most threefold); kNoExponent: all zero
  int q_e = kNoExponent;
  int ld = 1;
  // scaled pairs, target-major
  int *m2d_ri = nullptr, *m2d_src = nullptr;
  double *m2d_sP = nullptr, *m2d_sD = nullptr;
  int m2d_nnz = 0;
  int *d2d_ri = nullptr, *d2d_src = nullptr;
  double *d2d_s = nullptr;
  int d2d_nnz = 0;
  double damp_thr = 50.0;       // AMOEBA: damping applied when a u^3 < 50
  // FP32 operator: per 128-site tile the bounding box of pol_pos32 (lo, hi
  // pairs, [2*ntile]) and the squared distance beyond which no pair is damped
  float4 *tile_box32 = nullptr;
  int ntile = 0;
  // symmetric FP64 product: coordinates split into three floats [3][n]
  // (launch_split) and the bounding boxes of 32 sites
  float4 *pol_split = nullptr, *sub_box32 = nullptr;
  // the same split of the static sites [3][m] (one grid for both)
  float4 *mm_split = nullptr, *mm_sub_box32 = nullptr;  // and their 32-site boxes
  // a site is farther than kGridReach from the grid's origin: every pair in FP64
  // (the damping pre-test data have (1/thole)^2 = 0, so that no pair passes it)
  bool wide = false;
  float damp_r2max32 = 0.f;
  // tile boxes of the static sites and the squared distance beyond which no
  // M2D pair is damped
  float4 *mm_tile_box32 = nullptr;
  float m2d_r2max32 = 0.f;
};

// ---- pair kernels ---------------------------------------------------------
// Permanent-multipole field at the polarizable sites (E_M2D), n_ipd sets:
// out [n_ipd][n][3]; scratch holds split partials (m2d_scratch_doubles()).
size_t m2d_scratch_doubles(const DevSites &s, int nsplit);
int m2d_pick_split(const DevSites &s, int sm_count);
void launch_m2d(const DevSites &s, double *out, double *scratch, int nsplit, int *err_flag,
                cudaStream_t st);
// the finishing pass alone: split partials [nsplit][n][3] summed, the
// scaled-pair corrections, out [n_ipd][n][3]
void launch_m2d_finish(const DevSites &s, double *out, double *partial, int nsplit, cudaStream_t st);
// split partials [nsplit][total] summed into the first block (few splits are
// left to the reader); returns the splits left
int launch_sum_splits(size_t total, int nsplit, double *partial, cudaStream_t st);

// y = T x (dodiag) or y = -E_dd(x) (no diagonal); x,y [nrhs][n][3], FP64.
size_t tmu_scratch_doubles(const DevSites &s, int nrhs, int nsplit);
// All ordered pairs to FP64 accuracy in one launch (tmu_rows.cu); words: the
// largest high word of each column (launch_max_words).  part: partial sums of
// x.y, tmu_rows_parts per column (0: this size gives none).
int tmu_rows_parts(const DevSites &s, int ncol);
void launch_tmu_rows(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, const unsigned *words,
                     double *part, cudaStream_t st);
// The finishing pass alone on a field partial [nrhs][n][3] (one split): the
// u-scaled pair corrections, the sign and the 1/alpha diagonal
void launch_tmu_finish64(const DevSites &s, int nrhs, const double *partial, const double *x, bool dodiag,
                         double *y, cudaStream_t st);
// Same product with each unordered pair evaluated once (deterministic
// half-shell schedule, tmu_sym.cu): near pairs in FP64, the others in
// double-single; scratch of tmu_sym_scratch_doubles(s, nrhs_max).  The product
// of every mode from kSymMinSites sites (launch_tmu_rows below).
constexpr int kSymMinSites = 2400;
// the finishing passes give a site four lanes below this many sites, one above
constexpr int kFinishLanesSites = 32768;
// squared distances within which a pair always runs in FP64 (AMOEBA pairs
// also while the damping is strong, a u^3 < 20)
constexpr float kSymNear2 = 36.f, kSymNear2Wang = 64.f;
// The three floats of a coordinate on a grid as wide as 2^e resolve 2^(e - 71)
// bohr: up to 2^22 that is 2^-49, below the rounding of a coordinate of 8 bohr.
// Wider grids lose it (one external point at 1e10 bohr left the others with
// 1e-10, a water molecule at 1e12 the solve of 300 others with 4e-7).
constexpr double kGridReach = 4194304.0;
// squared distance of boxes within which their pairs are tested one by one
inline float near_range2(const DevSites &s, float damped) {
  const float close = s.amoeba ? kSymNear2 : kSymNear2Wang;
  return s.wide ? INFINITY : damped > close ? damped : close;
}
size_t tmu_sym_scratch_doubles(const DevSites &s, int nrhs);
void launch_tmu_f64_sym(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, double *scratch,
                        cudaStream_t st);
// the same for many columns: as many pairs of columns per launch as fill the
// GPU (tmu_sym_groups; one for large systems), scratch of
// tmu_sym_groups(s, nrhs) * tmu_sym_scratch_doubles(s, 2)
int tmu_sym_groups(const DevSites &s, int nrhs);
void launch_tmu_f64_sym_groups(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, double *scratch,
                               cudaStream_t st);
// its passes for callers that spread a product over launches: accumulators
// [g][n][3] (lo, then hi) and the two words from bad zeroed and the scales of
// the columns of x found (before the first share), and the sums read out into y = T x, with
// at most max_part partial sums of x.y per column (part [g][*npart])
void launch_tmu_sym_prepare(const DevSites &s, int g, const double *x, unsigned long long *lo,
                            unsigned long long *bad, cudaStream_t st);
void launch_tmu_sym_finish(const DevSites &s, int g, const unsigned long long *lo, const unsigned long long *hi,
                           const unsigned long long *bad, const double *x, bool dodiag, double *y, cudaStream_t st,
                           double *part = nullptr, int max_part = 0, int *npart = nullptr, size_t group_words = 0);
// the largest high word of |x| (the scale of the double-single products)
void launch_max_word(size_t total, const double *x, unsigned *word, cudaStream_t st, bool zeroed = false);
void launch_max_words(int ncol, size_t nv, const double *x, unsigned *words, cudaStream_t st);
// near field of the FMM (fmm_near.cu): the dipoles x [col][n][3] of the 27
// neighbouring leaves at every site, sites sorted by leaf (split coordinates
// [3][n], spos, sa, swa; perm the polarizable index); partial
// [kFmmNearSplit][col][n][3] in polarizable order, word from launch_max_words
struct FmmNearArgs {
  int n, L, ncol;
  bool amoeba;
  const int *leaf_start, *perm;
  const float4 *split;
  const Pos64 *spos;
  const double *sa;
  const float2 *swa;
  double thr;
  float thr2m;
};
constexpr int kFmmNearSplit = 9;
void launch_fmm_near(const FmmNearArgs &a, const double *x, const unsigned *word, double *partial, cudaStream_t st);
// the same for the field of the static multipoles (m2d.cu): sources and targets
// sorted by leaf (perm: static site, perm_t: polarizable site); partial
// [kFmmNearSplit][n][3] in polarizable order
void launch_m2d_leaf(const DevSites &s, int L, const int *leaf_start, const int *perm, const int *leaf_start_t,
                     const int *perm_t, double *partial, int *err_flag, cudaStream_t st);
// coordinates of the sites pos about a centre as three floats each, out [3][n],
// on the grid of a step for the largest of them
double split_step(double extent);
void launch_split(int n, const Pos64 *pos, const double centre[3], double g1, float4 *out, cudaStream_t st);
void split_coordinates(int n, const Pos64 *pos, const double centre[3], double g1, float4 *out);  // on the host
// The pairwise FP32 product (tmu32_rows.cu): columns in groups of up to gmax
// (4); part: partial sums of x.y, tmu32_rows_parts per column
int tmu32_rows_parts(int n);
void launch_tmu32_rows(const DevSites &s, int ncol, int gmax, const float *x, float *y, double *part, cudaStream_t st);
// FP32 inner operator with compensated cross-tile sums; x,y float.  Columns
// go through the pair kernel in groups of up to gmax (8, 4, 2 or 1) sharing
// the pair geometry; scratch holds nsplit * nrhs * n * 3 floats.
// kver 1: lanes over the sources, per-pair damping test (tmu32_rows.cu; scratch unused);
// kver 2: the tile-classified kernel of tmu32.cu.
// kver 3: the symmetric kernel of tmu32.cu (each unordered pair once),
// columns in groups of gmax (1 or 2), sums in sym_scratch (laid out as for
// launch_tmu_f64_sym, tmu_sym_scratch_doubles(s, 2)); scratch unused.
// prepared: the accumulators of a kver-3 product in one column group are
// zero already.  part: partial sums of x.y, at most max_part per column; their
// number is returned (part [nrhs][number]).
int launch_tmu_f32(const DevSites &s, int nrhs, const float *x, float *y, float *scratch, int nsplit, cudaStream_t st,
                   int gmax = 4, int kver = 2, double *sym_scratch = nullptr, bool prepared = false,
                   double *part = nullptr, int max_part = 0);

// ---- multi-system symmetric products --------------------------------------
// One system's share of a launch that serves several systems (the products
// of uneven systems in one persistent kernel): the items [item0, item0 +
// count) of its product, whose item space (super-tile, chunk of slots) is
// fixed per system and product kind (*_sym_items), so that a product may be
// spread over several launches; its fixed-point accumulators [g][n][3] and
// error flag are zeroed by the caller before the first share.
// round_pairs: the pairs one round of a caller that spreads products over
// launches spends on this product kind; items are then cut to about a
// quarter of a resident CTA's share of such a round, so that a round keeps
// every CTA busy (0: items sized for one launch of the whole product).  The
// value is part of the item space and stays fixed for a product.
struct SymSlice {
  const DevSites *s;
  const void *x;  // [g][n][3]: float for the FP32 product, double otherwise
  unsigned long long *lo, *hi, *bad;
  int item0, count;
  double round_pairs = 0.0;
};
constexpr int kMaxSymSlices = 32;  // systems per launch
int tmu32_sym_items(const DevSites &s, int g, double round_pairs = 0.0);
// next: a device counter of the launch (zeroed by the launcher unless it is
// zero already)
void launch_tmu32_sym_multi(int g, const SymSlice *sl, int nsl, unsigned *next, cudaStream_t st, bool zeroed = false);
// symmetric product of FP64 accuracy (g = 1 or 2; one damping kind per
// launch; launch_tmu_sym_prepare before a product's first share)
int tmu_f64_sym_items(const DevSites &s, int g, double round_pairs = 0.0);
void launch_tmu_f64_sym_multi(int g, bool amoeba, const SymSlice *sl, int nsl, unsigned *next, cudaStream_t st,
                              bool zeroed = false);
void launch_tmu32_pairs(const DevSites &s, int g, int groups, const float *x, float *partial, int nsplit,
                        cudaStream_t st);
// source splits an FP32 scratch must hold (per column)
int tmu32_max_split(const DevSites &s, int sm_count);
// Split of the source range for the FP32 operator (tmu32.cu) and its tile
// boxes / undamped distance, computed on the host from the FP32 positions.
int tmu32_pick_split(const DevSites &s, int sm_count);
void tile_boxes32(const float4 *pos32, int n, float4 *boxes /*[2*ceil(n/tile)]*/, int tile = 128);
float damp_r2max32(bool amoeba, double damp_thr, const double *inv_thole, const double *a, int n);
float m2d_r2max32(bool amoeba, double damp_thr, const double *pol_w, const double *pol_a, int n, const double *mm_w,
                  const double *mm_a, int m);
// Static-static pair sums (m2m.cu), energy or gradient: partial
// [nsplit][10 or 12 (Wang-AL 1 or 3)][m]
int m2m_pick_split(const DevSites &s, bool grad, int sm_count);
void launch_m2m(const DevSites &s, bool grad, double *partial, int nsplit, int *err, cudaStream_t st);
// Pair pass of the polarization gradient (grad_sym.cu): buf of
// grad_sym_doubles(s) receives fixed-point sums lo [m][6 or 3] (force, for
// AMOEBA torque), hi, then the non-finite flag, the work counter and the
// scale word; polar one bit per static site
size_t grad_sym_doubles(const DevSites &s);
void launch_grad_sym(const DevSites &s, const double *ipd, const int *mm_polar, const unsigned *polar, double *buf,
                     int *err, cudaStream_t st);
// batched fields: rhs[s*nf+f] = E_M2D[s] + field[f]; solution scatter to [f][s]
void launch_batch_rhs(int n, int nf, int nset, const double *e_m2d, const double *fields, double *rhs,
                      cudaStream_t st);
void launch_batch_scatter(int n, int nf, int nipd, int nsolved, const double *x, double *out, cudaStream_t st);

// ---- block CG (block_cg.cu) -----------------------------------------------
// out[a][b] = sum_i U[ua[a]][i] V[vb[b]][i], b < sb, then V2[vb2[b]], b < sb2
// (rows of sb + sb2; FP32 tiles, FP64 across tiles, fixed order); partial of
// block_cg_gram_doubles(smax)
size_t block_cg_gram_doubles(int smax);
int block_cg_max_columns();
void launch_gram(size_t nv, int sa, const float *U, const int *ua, int sb, const float *V, const int *vb, int sb2,
                 const float *V2, const int *vb2, double *partial, double *out, cudaStream_t st);
// out[oc[k]] = base[bc[k]] + sum_j in[ic[j]] C[j][k], C [nin][nout] (device);
// with in2 also out2[oc[k]] -= sum_j in2[ic[j]] C[j][k]
void launch_combine(size_t nv, int nin, const float *in, const int *ic, int nout, float *out, const int *oc,
                    const float *base, const int *bc, const float *C, cudaStream_t st, const float *in2 = nullptr,
                    float *out2 = nullptr);
void launch_scale_alpha32(int ncol, int n, const float *alpha, const float *r, float *z, cudaStream_t st);

// ---- dense T (incore matvec / inversion) ---------------------------------
void launch_build_tmat(const DevSites &s, double *tmat, cudaStream_t st);  // [3n][3n] col-major
void launch_gemv(int nn, const double *A, const double *x, double *y, bool dodiag,
                 const double *alpha, int nrhs, cudaStream_t st);
// r = rhs - T x
void launch_dense_residual(int nn, const double *T, const double *x, const double *rhs, double *r, cudaStream_t st);
// FP32 inverse of the symmetric positive definite T (dense.cu): buf of
// inverse32_floats(nn), s [nn] the square roots of the polarizabilities; info
// (device int) 0 = ok.  launch_inverse32_step: x += T^-1 r with it (scale:
// about the inverse of r's size, so that r fits FP32).
size_t inverse32_floats(int nn);
void launch_inverse32(int nn, const double *T, const double *alpha, double *s, float *buf, int *info,
                      cudaStream_t st);
void launch_inverse32_step(int nn, float *buf, const double *s, const double *r, double scale, double *x,
                           cudaStream_t st);
// LU with partial pivoting in place (column major); info (device int) 0 = ok.
void launch_lu_factor(int nn, double *A, int *piv, int *info, double *work, cudaStream_t st);
void launch_lu_solve(int nn, const double *A, const int *piv, double *b, cudaStream_t st);

// ---- BLAS-1 and reductions (deterministic) --------------------------------
constexpr int kRedBlocks = 456;  // 3 x 152 SMs
constexpr int kRedThreads = 256;
// partial[b][k] for k < ncol: sum over i of a[k*n+i]*b[k*n+i]
void launch_dots(int ncol, size_t n, const double *a, const double *b, double *partial,
                 cudaStream_t st);
// partial[b][k] = sum_i a[k*n+i] * v[i]  (one vector against ncol columns)
void launch_dots_bcast(int ncol, size_t n, const double *a, const double *v, double *partial,
                       cudaStream_t st);
// result[k] = sum_b partial[b][k]  (fixed order)
void launch_reduce_partials(int ncol, const double *partial, double *result, cudaStream_t st);

// misc elementwise
void launch_axpby(size_t n, double a, const double *x, double b, double *y, cudaStream_t st);
void launch_add(size_t n, const double *a, const double *b, double *out, cudaStream_t st);
void launch_scale_by_alpha(int nrhs, int n, const double *alpha, const double *x, double *y,
                           cudaStream_t st);
void launch_to_f32(size_t n, const double *x, const double *scale, float *y, cudaStream_t st);
// y[k][i] = x[k][i] * scale[k] for ncol columns of nv values (one launch)
void launch_to_f32_cols(int ncol, size_t nv, const double *x, const double *scale, float *y, cudaStream_t st);

// Multi-column PCG state kept on the device (one entry per column).
struct CgCol {
  double gold, gama, alpha, gnew, rms, beta;
  double tol;     // convergence threshold of this column (kept on the device
                  // so that a captured iteration graph stays valid)
  int active;     // column still iterating
  int quick;      // left through |p.Tp| < eps
  int converged;  // rms < tol
  int iters;
  int passes, max_passes;  // iterations run on the column, active or not, and their limit
};
// cols[k] = {gold = dots[k], tol, active = dots[k] > 0} (inner PCG start)
// mu[k] += scale[k] * dmu32[k]  (IR correction, FP64 accumulate)
void launch_ir_accumulate(int ncol, int n, double *mu, const float *d32, const double *scale,
                          cudaStream_t st);
// r = rhs - Tmu (all columns), into r; and r32 = r / scale
void launch_residual(size_t total, const double *rhs, const double *tmu, double *r,
                     cudaStream_t st);
// DIIS: x_new = sum_i c_i X[:, i]
void launch_lincomb(int nvec, size_t n, const double *X, size_t ldx, const double *c, double *out,
                    cudaStream_t st);
// rms and max of (a - b): out[0] = sum sq, out[1] = max abs (per-block partials then reduce)
void launch_diff_norms(size_t n, const double *a, const double *b, double *partial,
                       cudaStream_t st);
void launch_reduce_norms(const double *partial, double *out, cudaStream_t st);
// NaN / Inf check: flag set to 1 when any entry is not finite
// flag set to 1 when a and b differ in any bit of any entry
void launch_any_diff(size_t n, const double *a, const double *b, int *flag, cudaStream_t st);

// Number of SMs of the current device (cached).
int sm_count();
// Kernels launched by this library since load (all streams); graph replays
// add the kernels of the replayed graph.
long long launch_count();
long long thread_launch_count();
void add_launch_count(long long k);
// FMA-chain kernel for the FP32 / FP64 pipe peak; returns its flop count.
double launch_fma_peak(bool fp64, int iters, void *out, cudaStream_t st);

}  // namespace gpu
}  // namespace ommp
