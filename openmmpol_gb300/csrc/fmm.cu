// Fast multipole method for the FP64 dipole-field product T.mu (the
// reference's FMM path of TMatVec / field_extD2D, src/mod_electrostatics.F90:
// 1954-2065 with src/fast_multipoles/), enabled by ommp_enable_fmm.
//
// GB300 design: a uniform octree over the polarizable sites whose leaf side
// is at least the Thole damping range (every damped pair is a near pair), of
// the depth that minimises near-field pairs plus M2L work; Cartesian Taylor
// expansions of order p (fmm_math.cuh); FP64 but for the FP32 M2L of orders
// <= 10 (k_fmm_m2l_reg) and the near field:
//   k_fmm_p2m     leaf multipoles of the dipoles (one CTA per leaf)
//   k_fmm_m2m     parent multipoles from the 8 children, level by level
//   k_fmm_m2l     local expansions from the well-separated cells of each
//                 level (children of the parent's neighbours that are not
//                 neighbours).  The derivatives of 1/r depend only on the
//                 integer offset of the two cells, so they are tabulated
//                 once per order for the 7^3 offsets at unit cell size and
//                 scaled per level (1/r^(n+1) is homogeneous): the M2L is a
//                 gather of products, its (target term, source term) pairs
//                 spread evenly over the threads, each pair with its own
//                 shared-memory accumulator summed per target term in a
//                 fixed order (deterministic)
//   k_fmm_l2l     children's local expansions from the parent's
//   k_fmm_near    (fmm_near.cu; k_m2d_leaf of m2d.cu for the static multipoles)
//                 the near field of the 27 neighbouring leaves, direct, with
//                 the Thole damping of the direct kernels
//   k_fmm_l2p     far field of the leaf's local expansion at each site
//   k_fmm_add_near  the near field's partial sums added to it
// then the finishing pass of the direct product (scaled-pair corrections
// with exact pair terms, sign, 1/alpha diagonal).  Sites are kept in leaf
// order on the device (a counting sort per geometry).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "engine.h"
#include "fmm_math.cuh"
#include "log.h"
#include "pair_math.cuh"

namespace ommp {

// one octree: its sources and targets sorted by leaf (for T.mu both are the
// polarizable sites and share the arrays)
struct FmmTree {
  int L = -1, ncell = 0, nalloc_cell = 0;
  double h0 = 0.0, ox = 0.0, oy = 0.0, oz = 0.0;
  std::vector<int> off;        // first cell of each level
  bool built = false;
  int *cnt = nullptr, *cnt_t = nullptr;                // sources / targets per cell, every level
  int *leaf_start = nullptr, *leaf_start_t = nullptr;  // [nleaf + 1]
  int *perm = nullptr, *perm_t = nullptr;              // sorted -> site index
  gpu::Pos64 *spos = nullptr, *spos_t = nullptr;       // w = 1/thole (inf without Thole factor)
  double *sa = nullptr;                                // T.mu: Thole damping a
  float2 *swa = nullptr;                               // T.mu: FP32 damping pre-test data
  float4 *split = nullptr;                             // T.mu: split coordinates [3][n] (fmm_near.cu)
  double *sq = nullptr;                                // sorted multipoles [n][ld] (M2D sources)
  double *M = nullptr, *Lc = nullptr;                  // [2][ncell][K]
  float *M32 = nullptr;  // the M2L input [2][ncell][row32(K)] (k_fmm_m32)
  bool shared = false;                                 // targets are the sources
};

struct FmmState {
  int p = 0, K = 0, KD = 0, npairs = 0, nquads = 0;
  short4 *terms = nullptr;     // exponents (a, b, c) and order of each term
  int4 *pairs = nullptr;       // M2L pairs: g, index of g + h in the derivative table, h, (-1)^|g|
  int *hoff = nullptr;         // [K + 1] first pair of each target term h
  int2 *quads = nullptr;       // the pairs by four target terms (build_tables)
  double *dunit = nullptr;     // [343][KD] derivatives of 1/r to order p at unit cell offsets
  float *dunit32 = nullptr;    // the same in FP32, [343][row32(K)] (the FP32 M2L)
  FmmTree d2d, m2d;            // polarizable sites; static sources with polarizable targets
  double *field = nullptr;     // [2][n][3]
  double *near = nullptr;      // T.mu near-field partials [kFmmNearSplit][2][n][3], after field
  unsigned *word = nullptr;    // after near
  size_t field_n = 0;
  // T.mu: the expansions run beside the near field, on a stream of their own
  cudaStream_t far = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  bool built = false;          // d2d tree for the current geometry
};

void free_tree(FmmTree &t) {
  void *b[] = {t.cnt, t.leaf_start, t.perm, t.spos, t.sa, t.swa, t.sq, t.M, t.M32, t.Lc, t.split};
  for (void *p : b)
    if (p) cudaFree(p);
  if (!t.shared) {
    void *c[] = {t.cnt_t, t.leaf_start_t, t.perm_t, t.spos_t};
    for (void *p : c)
      if (p) cudaFree(p);
  }
  t = FmmTree();
}

void free_fmm_state(FmmState *f) {
  if (!f) return;
  void *b[] = {f->terms, f->pairs, f->hoff, f->quads, f->dunit, f->dunit32, f->field};
  for (void *p : b)
    if (p) cudaFree(p);
  free_tree(f->d2d);
  free_tree(f->m2d);
  if (f->far) cudaStreamDestroy(f->far);
  if (f->fork) cudaEventDestroy(f->fork);
  if (f->join) cudaEventDestroy(f->join);
  delete f;
}

namespace gpu {
namespace {

constexpr int FT = 128;  // threads per CTA

// floats of a row of the FP32 M2L's inputs: whole 16-byte copies
__host__ __device__ constexpr int row32(int K) { return (K + 3) & ~3; }


struct FmmArgs {
  int p, K, L, ncell, ncol;
  double h0, ox, oy, oz;
  const int *cnt, *leaf_start, *perm;
  const int *cnt_t;  // targets per cell (M2L / L2L skip cells without targets)
  const Pos64 *spos;
  const short4 *terms;
  const int4 *pairs;
  const int *hoff;
  const int2 *quads;
  int nquads;
  const double *dunit;
  const float *dunit32;
  double *M, *Lc;
  float *M32;
  int KD;
};

// sign of s^m for the child offset s = (b - 1/2) h_c per axis (bit b = 0:
// negative component) and the parities packed in e.y bits 8-10
__device__ __forceinline__ void cell_xyz(int idx, int l, int &x, int &y, int &z) {
  const int n = 1 << l;
  z = idx % n;
  y = (idx / n) % n;
  x = idx / (n * n);
}
__device__ __forceinline__ int cell_idx(int l, int x, int y, int z) {
  const int n = 1 << l;
  return (x * n + y) * n + z;
}
__device__ __forceinline__ int level_off(int l) { return ((1 << (3 * l)) - 1) / 7; }

// leaf multipoles of the dipoles x [col][n][3], one term per thread (blockDim
// covers K): with the powers v^m / m! of a site (X, Y, Z) and the same shifted
// by one and times the dipole (A), a term's share is
//   U[ab] Z[c] + V[ab] Az[c],  U = Ax[a] Y[b] + X[a] Ay[b],  V = X[a] Y[b],
// U and V once per site and pair (a, b): about 2.7 FP64 operations a term
// (five with the sum formed per term, and a division for each power: 283 us at
// 60,000 sites, order 10; now 157, 69 of them the FP64 pipe's).
constexpr int PCH = 16;                                                     // sites per chunk
constexpr int kMaxAB = (fmm::kMaxOrder + 1) * (fmm::kMaxOrder + 2) / 2;  // pairs (a, b), a + b <= p

__global__ void __launch_bounds__(512) k_fmm_p2m(FmmArgs a, const double *__restrict__ x, int n) {
  __shared__ double s_p[3][fmm::kMaxOrder + 1][PCH + 1], s_a[3][fmm::kMaxOrder + 1][PCH + 1];
  __shared__ double s_u[kMaxAB][PCH + 1], s_v[kMaxAB][PCH + 1], s_r[fmm::kMaxOrder + 1];
  __shared__ short2 s_ab[kMaxAB];
  const int c = blockIdx.x, col = blockIdx.y;
  const int s0 = a.leaf_start[c], s1 = a.leaf_start[c + 1];
  if (s0 == s1) return;
  int cx, cy, cz;
  cell_xyz(c, a.L, cx, cy, cz);
  const double h = a.h0 / (1 << a.L);
  const int t = threadIdx.x;
  const short4 e = t < a.K ? a.terms[t] : make_short4(0, 0, 0, 0);
  const int nab = (a.p + 1) * (a.p + 2) / 2, ab = (e.x + e.y) * (e.x + e.y + 1) / 2 + e.y;
  if (t < a.K && e.z == 0) s_ab[ab] = make_short2(e.x, e.y);
  if (t > 0 && t <= a.p) s_r[t] = 1.0 / t;
  double acc = 0.0;
  for (int b0 = s0; b0 < s1; b0 += PCH) {
    const int cnt = min(PCH, s1 - b0);
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * PCH; i += blockDim.x) {
      const int d = i / PCH, k = i % PCH;
      if (k >= cnt) continue;
      const Pos64 ps = a.spos[b0 + k];
      const double v = d == 0 ? ps.x - (a.ox + (cx + 0.5) * h) : d == 1 ? ps.y - (a.oy + (cy + 0.5) * h)
                                                                        : ps.z - (a.oz + (cz + 0.5) * h);
      const double mu = x[((size_t)col * n + a.perm[b0 + k]) * 3 + d];
      double pw = 1.0;
      s_p[d][0][k] = 1.0;
      s_a[d][0][k] = 0.0;
      for (int m = 1; m <= a.p; ++m) {
        s_a[d][m][k] = mu * pw;
        pw = pw * v * s_r[m];
        s_p[d][m][k] = pw;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nab * PCH; i += blockDim.x) {
      const int j = i / PCH, k = i % PCH;
      if (k >= cnt) continue;
      const short2 w = s_ab[j];
      const double X = s_p[0][w.x][k], Y = s_p[1][w.y][k];
      s_u[j][k] = fma(s_a[0][w.x][k], Y, X * s_a[1][w.y][k]);
      s_v[j][k] = X * Y;
    }
    __syncthreads();
    if (t >= a.K) continue;
    double w = 0.0;
    for (int q = 0; q < cnt; ++q) w = fma(s_u[ab][q], s_p[2][e.z][q], fma(s_v[ab][q], s_a[2][e.z][q], w));
    acc += w;
  }
  if (t < a.K) a.M[((size_t)col * a.ncell + level_off(a.L) + c) * a.K + t] = acc;
}

// index of the term (a, b, c); first: that of each order's first term
__device__ __forceinline__ int term_at(const int *first, int a, int b, int c) {
  const int u = b + c;
  return first[a + u] + u * (u + 1) / 2 + c;
}

constexpr int TT = 256;  // threads of the translations

// parents at level l - 1 from their children at level l:
// M_g(parent) = sum_children sum_(k <= g) M_k(child) s^(g - k) / (g - k)!
// One direction after the other (z, y, x), the two children that differ in it
// added on the way: sums of up to p + 1 terms over 4, 2 and 1 sets instead of
// 28 products of three directions on average for each child, their lists read
// from global memory (64 parents at order 10: 166 -> 23 us).
__global__ void __launch_bounds__(TT) k_fmm_m2m(FmmArgs a, int l) {
  extern __shared__ double s_w[];  // [8][K] and [4][K]
  __shared__ int s_first[fmm::kMaxOrder + 1];
  __shared__ double s_c[fmm::kMaxOrder + 1];  // (h_c / 2)^j / j!
  const int pc = blockIdx.x, col = blockIdx.y;
  if (a.cnt[level_off(l - 1) + pc] == 0) return;
  int px, py, pz;
  cell_xyz(pc, l - 1, px, py, pz);
  if ((int)threadIdx.x <= a.p) {
    s_first[threadIdx.x] = fmm::nterms((int)threadIdx.x - 1);
    const double hh = 0.5 * a.h0 / (1 << l);
    double f = 1.0;
    for (int j = 1; j <= (int)threadIdx.x; ++j) f *= hh / j;
    s_c[threadIdx.x] = f;
  }
  for (int i = threadIdx.x; i < 8 * a.K; i += TT) {
    const int ch = i / a.K;
    const int cc = cell_idx(l, 2 * px + (ch >> 2), 2 * py + ((ch >> 1) & 1), 2 * pz + (ch & 1));
    s_w[i] = a.M[((size_t)col * a.ncell + level_off(l) + cc) * a.K + (i - ch * a.K)];  // zero without sources
  }
  __syncthreads();
  // out[o] from in[2 o] (shifted by -h_c / 2 in the direction) and in[2 o + 1]
  auto pass = [&](const double *in, int nout, double *out, int dx, int dy, int dz) {
    for (int i = threadIdx.x; i < nout * a.K; i += TT) {
      const int o = i / a.K, t = i - o * a.K;
      const short4 e = a.terms[t];
      const double *lo = in + 2 * o * a.K, *hi = lo + a.K;
      const int m = dx ? e.x : dy ? e.y : e.z;
      double w = 0.0;
      for (int j = 0; j <= m; ++j) {
        const int k = term_at(s_first, e.x - dx * j, e.y - dy * j, e.z - dz * j);
        w = fma(s_c[j], (j & 1) ? hi[k] - lo[k] : hi[k] + lo[k], w);
      }
      out[i] = w;
    }
    __syncthreads();
  };
  double *s_v = s_w + 8 * a.K;
  pass(s_w, 4, s_v, 0, 0, 1);
  pass(s_v, 2, s_w, 0, 1, 0);
  pass(s_w, 1, a.M + ((size_t)col * a.ncell + level_off(l - 1) + pc) * a.K, 1, 0, 0);
}

// local expansions at level l from the well-separated cells of the level
__global__ void __launch_bounds__(FT) k_fmm_m2l(FmmArgs a, int l) {
  extern __shared__ double sh[];
  double *s_m = sh;               // [K] source multipole scaled by h^-|g|
  double *s_acc = sh + a.K;       // [npairs] per-pair accumulators
  const int npairs = a.hoff[a.K];
  const int tc = blockIdx.x, col = blockIdx.y;
  if (a.cnt_t[level_off(l) + tc] == 0) return;
  int tx, ty, tz;
  cell_xyz(tc, l, tx, ty, tz);
  const int n = 1 << l;
  const double hinv = (1 << l) / a.h0;
  for (int q = threadIdx.x; q < npairs; q += FT) s_acc[q] = 0.0;
  for (int ox = -1; ox <= 1; ++ox)
    for (int oy = -1; oy <= 1; ++oy)
      for (int oz = -1; oz <= 1; ++oz) {
        const int PX = (tx >> 1) + ox, PY = (ty >> 1) + oy, PZ = (tz >> 1) + oz;
        if (PX < 0 || PY < 0 || PZ < 0 || 2 * PX >= n || 2 * PY >= n || 2 * PZ >= n) continue;
        for (int ch = 0; ch < 8; ++ch) {
          const int sx = 2 * PX + (ch >> 2), sy = 2 * PY + ((ch >> 1) & 1), sz = 2 * PZ + (ch & 1);
          const int dx = tx - sx, dy = ty - sy, dz = tz - sz;
          if (abs(dx) <= 1 && abs(dy) <= 1 && abs(dz) <= 1) continue;
          const int sc = cell_idx(l, sx, sy, sz);
          if (a.cnt[level_off(l) + sc] == 0) continue;  // uniform over the CTA
          __syncthreads();
          const double *Ms = a.M + ((size_t)col * a.ncell + level_off(l) + sc) * a.K;
          for (int g = threadIdx.x; g < a.K; g += FT) {
            const int ng = a.terms[g].w;
            double f = 1.0;
            for (int i = 0; i < ng; ++i) f *= hinv;
            s_m[g] = Ms[g] * f;
          }
          __syncthreads();
          const double *D = a.dunit + (size_t)(((dx + 3) * 7 + (dy + 3)) * 7 + (dz + 3)) * a.KD;
          for (int q = threadIdx.x; q < npairs; q += FT) {
            const int4 pr = a.pairs[q];
            s_acc[q] += (pr.w ? -s_m[pr.x] : s_m[pr.x]) * D[pr.y];
          }
        }
      }
  __syncthreads();
  double *Lt = a.Lc + ((size_t)col * a.ncell + level_off(l) + tc) * a.K;
  for (int hh = threadIdx.x; hh < a.K; hh += FT) {
    double s = 0.0;
    for (int q = a.hoff[hh]; q < a.hoff[hh + 1]; ++q) s += s_acc[q];
    const short4 e = a.terms[hh];
    double f = hinv;  // h^-(|h| + 1) / h!
    for (int i = 0; i < e.w; ++i) f *= hinv;
    for (int i = 2; i <= e.x; ++i) f /= i;
    for (int i = 2; i <= e.y; ++i) f /= i;
    for (int i = 2; i <= e.z; ++i) f /= i;
    Lt[hh] += s * f;
  }
}

// The FP32 M2L input: the multipoles of the cells of levels 2..L scaled to
// the cell size, (-1)^|g| M_g h^-|g| (h the level's cell side), in FP32; one
// thread per (column, cell, term of the padded row)
__global__ void k_fmm_m32(FmmArgs a, int first_cell, int ncells) {
  const int row = row32(a.K);
  const size_t total = (size_t)a.ncol * ncells * row;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int g = (int)(i % row);
    const size_t cc = i / row;
    const int col = (int)(cc / ncells);
    const int c = first_cell + (int)(cc % ncells);
    int l = 0;
    while (l < a.L && level_off(l + 1) <= c) ++l;
    const size_t o = (size_t)col * a.ncell + c;
    float v = 0.f;
    if (g < a.K) {
      const int ng = a.terms[g].w;
      const double hinv = (1 << l) / a.h0;
      double f = (ng & 1) ? -1.0 : 1.0;
      for (int r = 0; r < ng; ++r) f *= hinv;
      v = (float)(a.M[o * a.K + g] * f);
    }
    a.M32[o * row + g] = v;
  }
}

// The same M2L in FP32 for the cells of all levels in one launch, the sums of
// the (target term, source term) pairs held in registers: the multipoles
// (scaled to the cell size, with the sign of their order), the unit-offset
// derivatives and the pair sums in FP32, the sum over source terms of each
// local term and the local expansion in FP64.  The FP32 rounding (~1e-6 of a
// local coefficient) is far below the expansion's own truncation error (~1e-4
// at order 10), and GB300 issues FP32 at 64x its FP64 rate.
// A pair is one multiply-add of a multipole and a derivative, both from shared
// memory, so the loads bound the kernel, not the multiply-adds: a thread holds
// QJ quads of pairs, four target terms against one source term, whose
// multipole it loads once (5 loads for 4 multiply-adds instead of 8).  Threads
// of a warp take consecutive source terms of the same target terms: no bank
// conflicts in the multipoles, few in the derivatives.  288 x 3 quads serve
// orders <= 8, 544 x 4 orders <= 10.
// The source cells are listed first and M2L_NB of them are fetched ahead with
// asynchronous 16-byte copies while the previous ones are used.
// 60,000 sites, order 10, one column (both levels, 512 + 64 target cells): 738
// us with a thread's pairs unrelated and 4-byte copies, 299 us now, the same
// sums bit for bit.
constexpr int M2L_NB = 4;

__device__ __forceinline__ void copy_async16(float *dst, const float *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

template <int NT, int QJ, int NCOL>
__global__ void __launch_bounds__(NT) k_fmm_m2l_reg(FmmArgs a) {
  extern __shared__ __align__(16) float sh32[];
  __shared__ int s_src[192], s_off[192], s_n;
  const int row = row32(a.K);        // K == KD
  const int rec = (NCOL + 1) * row;  // multipoles of the columns, derivatives
  float *s_buf = sh32;               // [2][M2L_NB][rec]
  float *s_acc = sh32;               // [npairs], after the last step
  int l = 2;
  while (level_off(l + 1) - level_off(2) <= (int)blockIdx.x) ++l;
  const int tc = blockIdx.x - (level_off(l) - level_off(2));
  if (a.cnt_t[level_off(l) + tc] == 0) return;
  int tx, ty, tz;
  cell_xyz(tc, l, tx, ty, tz);
  const int n = 1 << l;
  const double hinv = (1 << l) / a.h0;
  // the well-separated cells with sources, in a fixed order
  if (threadIdx.x < 32) {
    int cnt = 0;
    for (int b = 0; b < 27 * 8; b += 32) {
      const int i = b + threadIdx.x;
      const int o = i >> 3, ch = i & 7;
      const int sx = 2 * ((tx >> 1) + o / 9 - 1) + (ch >> 2), sy = 2 * ((ty >> 1) + (o / 3) % 3 - 1) + ((ch >> 1) & 1),
                sz = 2 * ((tz >> 1) + o % 3 - 1) + (ch & 1);
      const int dx = tx - sx, dy = ty - sy, dz = tz - sz;
      bool take = i < 27 * 8 && sx >= 0 && sy >= 0 && sz >= 0 && sx < n && sy < n && sz < n &&
                  !(abs(dx) <= 1 && abs(dy) <= 1 && abs(dz) <= 1);
      int sc = 0;
      if (take) {
        sc = cell_idx(l, sx, sy, sz);
        take = a.cnt[level_off(l) + sc] != 0;
      }
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int k = cnt + __popc(m & ((1u << threadIdx.x) - 1u));
        s_src[k] = sc;
        s_off[k] = ((dx + 3) * 7 + (dy + 3)) * 7 + (dz + 3);
      }
      cnt += __popc(m);
    }
    if (threadIdx.x == 0) s_n = cnt;
  }
  int2 qd[QJ];
  float acc[NCOL][QJ][4];
#pragma unroll
  for (int j = 0; j < QJ; ++j) {
    const int q = threadIdx.x + j * NT;
    qd[j] = q < a.nquads ? a.quads[q] : make_int2(-1, -1);
#pragma unroll
    for (int c = 0; c < NCOL; ++c)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[c][j][k] = 0.f;
  }
  __syncthreads();
  const int ns = s_n;
  auto fetch = [&](int b0, int buf) {
    const int chunks = row / 4, total = min(M2L_NB, ns - b0) * (NCOL + 1) * chunks;
    for (int i = threadIdx.x; i < total; i += NT) {
      const int r = i / chunks, ch = i - r * chunks;
      const int k = r / (NCOL + 1), col = r - k * (NCOL + 1);
      const float *src = col < NCOL ? a.M32 + ((size_t)col * a.ncell + level_off(l) + s_src[b0 + k]) * row
                                    : a.dunit32 + (size_t)s_off[b0 + k] * row;
      copy_async16(&s_buf[buf * M2L_NB * rec + r * row + 4 * ch], src + 4 * ch);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, 0);
  for (int b0 = 0, buf = 0; b0 < ns; b0 += M2L_NB, buf ^= 1) {
    fetch(b0 + M2L_NB, buf ^ 1);  // an empty group after the last batch
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const int kn = min(M2L_NB, ns - b0);
    for (int k = 0; k < kn; ++k) {
      const float *s_m = &s_buf[(buf * M2L_NB + k) * rec], *s_d = s_m + NCOL * row;
#pragma unroll
      for (int j = 0; j < QJ; ++j) {
        if (qd[j].x < 0) continue;
        const int g = (qd[j].y >> 10) & 1023;
        const float d0 = s_d[qd[j].x & 1023], d1 = s_d[(qd[j].x >> 10) & 1023], d2 = s_d[qd[j].x >> 20],
                    d3 = s_d[qd[j].y & 1023];
#pragma unroll
        for (int c = 0; c < NCOL; ++c) {
          const float m = s_m[c * row + g];
          acc[c][j][0] += m * d0;
          acc[c][j][1] += m * d1;
          acc[c][j][2] += m * d2;
          acc[c][j][3] += m * d3;
        }
      }
    }
    __syncthreads();  // the buffer is filled again by the next fetch
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int col = 0; col < NCOL; ++col) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < QJ; ++j) {
      if (qd[j].x < 0) continue;
      const int g = (qd[j].y >> 10) & 1023, h = qd[j].y >> 20;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (h + k < a.K && g < a.hoff[h + k + 1] - a.hoff[h + k]) s_acc[a.hoff[h + k] + g] = acc[col][j][k];
    }
    __syncthreads();
    double *Lt = a.Lc + ((size_t)col * a.ncell + level_off(l) + tc) * a.K;
    for (int hh = threadIdx.x; hh < a.K; hh += NT) {
      double s = 0.0;
      for (int q = a.hoff[hh]; q < a.hoff[hh + 1]; ++q) s += (double)s_acc[q];
      const short4 e = a.terms[hh];
      double f = hinv;  // h^-(|h| + 1) / h!
      for (int i = 0; i < e.w; ++i) f *= hinv;
      for (int i = 2; i <= e.x; ++i) f /= i;
      for (int i = 2; i <= e.y; ++i) f /= i;
      for (int i = 2; i <= e.z; ++i) f /= i;
      Lt[hh] += s * f;
    }
  }
}

// children at level l + 1 from their parent at level l:
// L_k(child) += sum_(h >= k) L_h(parent) h! / (k! (h - k)!) t^(h - k)
// One direction after the other, the even and odd powers of t apart, so that
// the two children that differ in it share one sum (512 children at order 10,
// as lists of products per child 128 us, now 23).
__global__ void __launch_bounds__(TT) k_fmm_l2l(FmmArgs a, int l) {
  extern __shared__ double s_w[];  // [1][K], [2][K] and [4][K]
  __shared__ int s_first[fmm::kMaxOrder + 1];
  __shared__ double s_c[(fmm::kMaxOrder + 1) * (fmm::kMaxOrder + 1)];  // [k][j] (k + j over k) (h_c / 2)^j
  const int pc = blockIdx.x, col = blockIdx.y;
  if (a.cnt_t[level_off(l) + pc] == 0) return;
  int px, py, pz;
  cell_xyz(pc, l, px, py, pz);
  const int p1 = a.p + 1;
  if ((int)threadIdx.x < p1) s_first[threadIdx.x] = fmm::nterms((int)threadIdx.x - 1);
  if ((int)threadIdx.x < p1 * p1) {
    const int k = threadIdx.x / p1, m = threadIdx.x % p1;
    const double hh = 0.5 * a.h0 / (1 << (l + 1));
    double b = 1.0, f = 1.0;
    for (int j = 1; j <= m; ++j) {
      b = b * (k + j) / j;
      f *= hh;
    }
    s_c[threadIdx.x] = b * f;
  }
  for (int i = threadIdx.x; i < a.K; i += TT) s_w[i] = a.Lc[((size_t)col * a.ncell + level_off(l) + pc) * a.K + i];
  __syncthreads();
  // term t of the sets 2 o (shifted by -h_c / 2 in the direction) and 2 o + 1 from in[o]
  auto shift = [&](const double *in, int t, int dx, int dy, int dz, double &lo, double &hi) {
    const short4 e = a.terms[t];
    const double *c = s_c + (dx ? e.x : dy ? e.y : e.z) * p1;
    double even = 0.0, odd = 0.0;
    for (int j = 0; j <= a.p - e.w; ++j) {
      const double v = in[term_at(s_first, e.x + dx * j, e.y + dy * j, e.z + dz * j)];
      if (j & 1)
        odd = fma(c[j], v, odd);
      else
        even = fma(c[j], v, even);
    }
    lo = even - odd;
    hi = even + odd;
  };
  double *s_x = s_w + a.K, *s_y = s_x + 2 * a.K;
  for (int t = threadIdx.x; t < a.K; t += TT) shift(s_w, t, 1, 0, 0, s_x[t], s_x[a.K + t]);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * a.K; i += TT) {
    const int o = i / a.K, t = i - o * a.K;
    shift(s_x + o * a.K, t, 0, 1, 0, s_y[2 * o * a.K + t], s_y[(2 * o + 1) * a.K + t]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * a.K; i += TT) {
    const int o = i / a.K, t = i - o * a.K;
    double w[2];
    shift(s_y + o * a.K, t, 0, 0, 1, w[0], w[1]);
    for (int bz = 0; bz < 2; ++bz) {
      const int cc = cell_idx(l + 1, 2 * px + (o >> 1), 2 * py + (o & 1), 2 * pz + bz);
      if (a.cnt_t[level_off(l + 1) + cc]) a.Lc[((size_t)col * a.ncell + level_off(l + 1) + cc) * a.K + t] += w[bz];
    }
  }
}

// position of the term (a, b, c) in the order of nested Horner schemes (a, then
// b, then c from high to low)
__device__ __forceinline__ int horner_pos(int p, int a, int b, int c) {
  const int u = p - a, v = u - b;
  return u * (u + 1) * (u + 2) / 6 + v * (v + 1) / 2 + (v - c);
}
// -grad sum_abc L_abc u^(abc) by nested Horner schemes over s_H (terms in
// horner_pos order): about 3 FP64 operations per term instead of 12 with
// the powers of each component formed apart (791 -> 154 us at 60,000 sites)
__device__ __forceinline__ void horner_field(int p, const double *s_H, double X, double Y, double Z, double *e) {
  double w = 0.0, wx = 0.0, wy = 0.0, wz = 0.0;
  int i = 0;
  for (int a = p; a >= 0; --a) {
    double v = 0.0, vy = 0.0, vz = 0.0;
    for (int b = p - a; b >= 0; --b) {
      double s = 0.0, sz = 0.0;
      for (int c = p - a - b; c >= 0; --c) {
        sz = fma(sz, Z, s);
        s = fma(s, Z, s_H[i++]);
      }
      vy = fma(vy, Y, v);
      vz = fma(vz, Y, sz);
      v = fma(v, Y, s);
    }
    wx = fma(wx, X, w);
    wy = fma(wy, X, vy);
    wz = fma(wz, X, vz);
    w = fma(w, X, v);
  }
  e[0] -= wx;
  e[1] -= wy;
  e[2] -= wz;
}

// far field of the leaf's local expansion at each site of the leaf; field
// [col][n][3]
__global__ void __launch_bounds__(FT) k_fmm_l2p(FmmArgs a, int n, double *__restrict__ field) {
  __shared__ double s_H[fmm::nterms(fmm::kMaxOrder)];
  const int c = blockIdx.x, col = blockIdx.y;
  const int s0 = a.leaf_start[c], s1 = a.leaf_start[c + 1];
  if (s0 == s1) return;
  int cx, cy, cz;
  cell_xyz(c, a.L, cx, cy, cz);
  const double h = a.h0 / (1 << a.L);
  const double *Lt = a.Lc + ((size_t)col * a.ncell + level_off(a.L) + c) * a.K;
  for (int t = threadIdx.x; t < a.K; t += FT) {
    const short4 e = a.terms[t];
    s_H[horner_pos(a.p, e.x, e.y, e.z)] = Lt[t];
  }
  __syncthreads();
  for (int si = s0 + threadIdx.x; si < s1; si += FT) {
    const Pos64 pt = a.spos[si];
    double e[3] = {0.0, 0.0, 0.0};
    horner_field(a.p, s_H, pt.x - (a.ox + (cx + 0.5) * h), pt.y - (a.oy + (cy + 0.5) * h),
                 pt.z - (a.oz + (cz + 0.5) * h), e);
    const size_t o = ((size_t)col * n + a.perm[si]) * 3;
    for (int d = 0; d < 3; ++d) field[o + d] = e[d];
  }
}

// the near field's partial sums (near [kFmmNearSplit][nv], fmm_near.cu) added
// to the far field
__global__ void k_fmm_add_near(size_t nv, const double *__restrict__ near, double *__restrict__ field) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kFmmNearSplit; ++k) s += near[k * nv + i];
  field[i] += s;
}

// leaf multipoles of the static multipoles (charge; dipole and quadrupole
// for AMOEBA, the potential of a quadrupole being sum_kl Q_kl d_k d_l (1/r)
// of its traceless part); one column, one term per thread.  As in k_fmm_p2m the
// products of the x and y powers are formed once per site and pair (a, b), so
// that a term's share is P[ab] Z[c] + Q[ab] Z[c - 1] + S[ab] Z[c - 2] (formed per
// term, with a division for each power, the field of 60,000 sites at order 10
// with its coordinate update took 8.25 ms, now 6.97; this kernel 0.37).  FP64
// pipe.
template <bool AMOEBA>
__global__ void __launch_bounds__(512) k_fmm_p2m_mp(FmmArgs a, const double *__restrict__ sq) {
  constexpr int LD = AMOEBA ? 10 : 1, NS = AMOEBA ? 3 : 1;
  __shared__ double s_p[3][fmm::kMaxOrder + 3][PCH + 1];  // power m at m + 2, below it zeros
  __shared__ double s_u[NS][kMaxAB][PCH + 1], s_q[LD][PCH], s_r[fmm::kMaxOrder + 1];
  __shared__ short2 s_ab[kMaxAB];
  const int c = blockIdx.x;
  const int s0 = a.leaf_start[c], s1 = a.leaf_start[c + 1];
  if (s0 == s1) return;
  int cx, cy, cz;
  cell_xyz(c, a.L, cx, cy, cz);
  const double h = a.h0 / (1 << a.L);
  const int t = threadIdx.x;
  const short4 e = t < a.K ? a.terms[t] : make_short4(0, 0, 0, 0);
  const int nab = (a.p + 1) * (a.p + 2) / 2, ab = (e.x + e.y) * (e.x + e.y + 1) / 2 + e.y;
  if (t < a.K && e.z == 0) s_ab[ab] = make_short2(e.x, e.y);
  if (t > 0 && t <= a.p) s_r[t] = 1.0 / t;
  double acc = 0.0;
  for (int b0 = s0; b0 < s1; b0 += PCH) {
    const int cnt = min(PCH, s1 - b0);
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * PCH; i += blockDim.x) {
      const int d = i / PCH, k = i % PCH;
      if (k >= cnt) continue;
      const Pos64 ps = a.spos[b0 + k];
      const double v = d == 0 ? ps.x - (a.ox + (cx + 0.5) * h) : d == 1 ? ps.y - (a.oy + (cy + 0.5) * h)
                                                                        : ps.z - (a.oz + (cz + 0.5) * h);
      double pw = 1.0;
      s_p[d][0][k] = s_p[d][1][k] = 0.0;
      s_p[d][2][k] = 1.0;
      for (int m = 1; m <= a.p; ++m) {
        pw = pw * v * s_r[m];
        s_p[d][m + 2][k] = pw;
      }
    }
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
      double q[LD];
      for (int d = 0; d < LD; ++d) q[d] = sq[(size_t)(b0 + i) * LD + d];
      if (AMOEBA) {  // traceless part of the quadrupole
        const double t3 = (q[4] + q[6] + q[9]) / 3.0;
        q[4] -= t3;
        q[6] -= t3;
        q[9] -= t3;
      }
      for (int d = 0; d < LD; ++d) s_q[d][i] = q[d];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nab * PCH; i += blockDim.x) {
      const int j = i / PCH, k = i % PCH;
      if (k >= cnt) continue;
      const int ea = s_ab[j].x + 2, eb = s_ab[j].y + 2;
      const double X = s_p[0][ea][k], Y = s_p[1][eb][k], XY = X * Y;
      double w = s_q[0][k] * XY;
      if (AMOEBA) {
        // sum_kl Q_kl v^(g - e_k - e_l) / (g - e_k - e_l)!; Q stored xx xy yy xz yz zz
        const double X1Y = s_p[0][ea - 1][k] * Y, XY1 = X * s_p[1][eb - 1][k];
        w = fma(s_q[1][k], X1Y, fma(s_q[2][k], XY1, w));
        w = fma(s_q[4][k], s_p[0][ea - 2][k] * Y, fma(s_q[6][k], X * s_p[1][eb - 2][k], w));
        w = fma(2.0 * s_q[5][k], s_p[0][ea - 1][k] * s_p[1][eb - 1][k], w);
        s_u[1 % NS][j][k] = fma(s_q[3][k], XY, 2.0 * fma(s_q[7][k], X1Y, s_q[8][k] * XY1));
        s_u[2 % NS][j][k] = s_q[9][k] * XY;
      }
      s_u[0][j][k] = w;
    }
    __syncthreads();
    if (t >= a.K) continue;
    double w = 0.0;
    for (int q = 0; q < cnt; ++q) {
      w = fma(s_u[0][ab][q], s_p[2][e.z + 2][q], w);
      if (AMOEBA) w = fma(s_u[1 % NS][ab][q], s_p[2][e.z + 1][q], fma(s_u[2 % NS][ab][q], s_p[2][e.z][q], w));
    }
    acc += w;
  }
  if (t < a.K) a.M[((size_t)level_off(a.L) + c) * a.K + t] = acc;
}

// the same at targets that are not the sources; field [n][3]
__global__ void __launch_bounds__(FT) k_fmm_l2p_m2d(FmmArgs a, const int *__restrict__ leaf_start_t,
                                                     const int *__restrict__ perm_t, const Pos64 *__restrict__ spos_t,
                                                     double *__restrict__ field) {
  __shared__ double s_H[fmm::nterms(fmm::kMaxOrder)];
  const int c = blockIdx.x;
  const int s0 = leaf_start_t[c], s1 = leaf_start_t[c + 1];
  if (s0 == s1) return;
  int cx, cy, cz;
  cell_xyz(c, a.L, cx, cy, cz);
  const double h = a.h0 / (1 << a.L);
  const double *Lt = a.Lc + ((size_t)level_off(a.L) + c) * a.K;
  for (int t = threadIdx.x; t < a.K; t += FT) {
    const short4 e = a.terms[t];
    s_H[horner_pos(a.p, e.x, e.y, e.z)] = Lt[t];
  }
  __syncthreads();
  for (int si = s0 + threadIdx.x; si < s1; si += FT) {
    const Pos64 pt = spos_t[si];
    double e[3] = {0.0, 0.0, 0.0};
    horner_field(a.p, s_H, pt.x - (a.ox + (cx + 0.5) * h), pt.y - (a.oy + (cy + 0.5) * h),
                 pt.z - (a.oz + (cz + 0.5) * h), e);
    for (int d = 0; d < 3; ++d) field[3 * (size_t)perm_t[si] + d] = e[d];
  }
}

}  // namespace
}  // namespace gpu

namespace {
std::atomic<bool> g_fmm_auto{false};
}  // namespace

void set_fmm_auto(bool on) { g_fmm_auto = on; }
bool fmm_auto() { return g_fmm_auto; }

int System::set_fmm(bool on, int order) {
  int st = set_fmm_order_pol(order);
  if (st) return st;
  st = set_fmm_order_static(order);
  if (st) return st;
  fmm_on_ = on;
  return kOk;
}

int System::set_fmm_order_pol(int order) {
  if (order < 2 || order > fmm::kMaxOrder) {
    set_last_error("FMM expansion order must be between 2 and 12");
    return kErrBadArg;
  }
  if (fmm_ && fmm_->p != order) {
    free_fmm_state(fmm_);
    fmm_ = nullptr;
  }
  fmm_order_ = order;
  return kOk;
}

void System::fmm_drop_static() {
  if (fmms_) fmms_->m2d.built = false;
  if (m2d_method_ == kM2dFMM) m2d_done_ = false;  // a field of the old settings
}

int System::set_fmm_order_static(int order) {
  if (order < 2 || order > fmm::kMaxOrder) {
    set_last_error("FMM expansion order must be between 2 and 12");
    return kErrBadArg;
  }
  if (order == fmm_order_static_) return kOk;
  if (fmms_) {
    free_fmm_state(fmms_);
    fmms_ = nullptr;
  }
  fmm_order_static_ = order;
  fmm_drop_static();
  return kOk;
}

// The reference treats two leaf cells as near when the gap between them is
// below fmm_distance and stops subdividing a cell whose half diagonal is below
// fmm_min_cell_size (src/fast_multipoles/mod_tree.F90:177,
// mod_octatree.F90:98).  Here the near field is the 27 neighbouring leaves of
// a uniform octree, so cells farther apart are separated by at least one leaf
// side: both settings become lower bounds of that side (the min cell size as
// a half diagonal, side = 2 d / sqrt 3), beside the damping range.
double System::fmm_min_leaf() const { return std::max(fmm_dfar_, 2.0 * fmm_mincell_ / std::sqrt(3.0)); }

int System::set_fmm_distance(double d) {
  if (!(d >= 0.0) || !std::isfinite(d)) {
    set_last_error("FMM distance must be a finite non-negative length (bohr)");
    return kErrBadArg;
  }
  fmm_dfar_ = d;
  fmm_invalidate();
  fmm_drop_static();
  return kOk;
}

int System::set_fmm_min_cell_size(double d) {
  if (!(d >= 0.0) || !std::isfinite(d)) {
    set_last_error("FMM minimum cell size must be a finite non-negative length (bohr)");
    return kErrBadArg;
  }
  fmm_mincell_ = d;
  fmm_invalidate();
  fmm_drop_static();
  return kOk;
}

void System::fmm_invalidate() {
  if (fmm_) {
    fmm_->built = false;
    fmm_->d2d.built = false;
  }
  if (fmms_) fmms_->m2d.built = false;
}

namespace {

// shared memory of k_fmm_m2l_reg: two batches of sources, or the pair sums
size_t m2l_smem(const FmmState &f, int ncol) {
  return sizeof(float) * std::max<size_t>(2 * gpu::M2L_NB * (size_t)(ncol + 1) * gpu::row32(f.K), f.npairs);
}

constexpr int kQuadsSmall = 288 * 3, kQuadsLarge = 544 * 4;  // of the two shapes of k_fmm_m2l_reg

int alloc_m32(const FmmState &f, FmmTree &t, int ncol) {
  if (t.M32) cudaFree(t.M32);
  t.M32 = nullptr;
  if (f.nquads > kQuadsLarge) return 0;
  return cudaMalloc((void **)&t.M32, ncol * (size_t)t.ncell * gpu::row32(f.K) * sizeof(float)) != cudaSuccess;
}

// per-order tables: terms, M2L pairs sorted by target term, unit-offset
// derivative tensors
int build_tables(FmmState &f, int p, cudaStream_t st) {
  f.p = p;
  f.K = fmm::nterms(p);
  f.KD = fmm::nterms(p);  // |g| + |h| <= p: derivatives to order p
  std::vector<short4> terms(f.K);
  for (int t = 0; t < f.K; ++t) {
    int a, b, c;
    fmm::exponents(t, a, b, c);
    terms[t] = make_short4((short)a, (short)b, (short)c, (short)(a + b + c));
  }
  std::vector<int4> pairs;
  std::vector<int> hoff(f.K + 1, 0);
  for (int h = 0; h < f.K; ++h) {
    hoff[h] = (int)pairs.size();
    const int nh = terms[h].w;
    for (int g = 0; g < fmm::nterms(p - nh); ++g)
      pairs.push_back(make_int4(g, fmm::term(terms[g].x + terms[h].x, terms[g].y + terms[h].y, terms[g].z + terms[h].z),
                                h, terms[g].w & 1));
  }
  hoff[f.K] = (int)pairs.size();
  f.npairs = (int)pairs.size();
  // Target terms h..h+3 against source term g: x the indexes of g + h, + 1, + 2
  // (10 bits each), y that of g + h + 3, g and h.  Where a quad straddles two
  // orders its later terms may have no pair with g: index 0, sum not used.
  std::vector<int2> quads;
  if (f.npairs <= 4 * kQuadsLarge)
    for (int h = 0; h < f.K; h += 4)
      for (int g = 0; g < hoff[h + 1] - hoff[h]; ++g) {
        int d[4];
        for (int k = 0; k < 4; ++k) d[k] = h + k < f.K && g < hoff[h + k + 1] - hoff[h + k] ? pairs[hoff[h + k] + g].y : 0;
        quads.push_back(make_int2(d[0] | d[1] << 10 | d[2] << 20, d[3] | g << 10 | h << 20));
      }
  f.nquads = quads.empty() ? kQuadsLarge + 1 : (int)quads.size();
  std::vector<double> dunit((size_t)343 * f.KD, 0.0);
  for (int i = -3; i <= 3; ++i)
    for (int j = -3; j <= 3; ++j)
      for (int k = -3; k <= 3; ++k) {
        if (std::abs(i) <= 1 && std::abs(j) <= 1 && std::abs(k) <= 1) continue;
        fmm::derivatives(i, j, k, p, &dunit[(size_t)(((i + 3) * 7 + (j + 3)) * 7 + (k + 3)) * f.KD]);
      }
  auto up = [&](auto *&dst, const auto &v) {
    if (cudaMalloc((void **)&dst, std::max<size_t>(v.size(), 1) * sizeof(v[0])) != cudaSuccess) return 1;
    cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice, st);
    return 0;
  };
  std::vector<float> dunit32((size_t)343 * gpu::row32(f.K), 0.f);
  for (int o = 0; o < 343; ++o)
    for (int k = 0; k < f.KD; ++k) dunit32[(size_t)o * gpu::row32(f.K) + k] = (float)dunit[(size_t)o * f.KD + k];
  int bad = up(f.terms, terms) | up(f.pairs, pairs) | up(f.hoff, hoff) | up(f.quads, quads) |
            up(f.dunit, dunit) | up(f.dunit32, dunit32);
  if (bad) {
    cudaGetLastError();
    set_last_error("out of device memory for the FMM tables");
    return kErrMemory;
  }
  const size_t smem = (f.K + (size_t)f.npairs) * sizeof(double);
  if (smem > 48 * 1024) cudaFuncSetAttribute(gpu::k_fmm_m2l, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  for (int ncol = 1; ncol <= 2; ++ncol) {
    const int b = (int)m2l_smem(f, ncol);
    const void *k[2] = {ncol == 2 ? (const void *)gpu::k_fmm_m2l_reg<288, 3, 2> : (const void *)gpu::k_fmm_m2l_reg<288, 3, 1>,
                        ncol == 2 ? (const void *)gpu::k_fmm_m2l_reg<544, 4, 2> : (const void *)gpu::k_fmm_m2l_reg<544, 4, 1>};
    if (b > 48 * 1024)
      for (const void *fn : k) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  }
  return cudaStreamSynchronize(st) == cudaSuccess ? kOk : kErrCuda;  // host vectors die here
}

// geometry of one tree: sources xs [ns][3] and targets xt [nt][3] (targets
// the sources when xt is null) sorted by leaf, leaf side >= rdamp, depth
// minimising near pairs x 40 + M2L term pairs
struct TreeLayout {
  int L = -1, ncell = 0;
  double side = 0.0, lo[3] = {0, 0, 0};
  std::vector<int> off, start_s, perm_s, start_t, perm_t, cnt_s, cnt_t;
};

bool plan_tree(int ns, const double *xs, int nt, const double *xt, double rdamp, int npairs, TreeLayout &o) {
  const bool same = xt == nullptr;
  if (same) {
    xt = xs;
    nt = ns;
  }
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int pass = 0; pass < 2; ++pass) {
    const double *x = pass ? xt : xs;
    const int m = pass ? nt : ns;
    for (int j = 0; j < m; ++j)
      for (int d = 0; d < 3; ++d) lo[d] = std::min(lo[d], x[3 * (size_t)j + d]), hi[d] = std::max(hi[d], x[3 * (size_t)j + d]);
  }
  double side = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]});
  side = side * (1.0 + 1e-9) + 1e-6;
  if (!std::isfinite(rdamp)) return false;
  auto leaf_of = [&](const double *c, int nl, double h) {
    const int x = std::min(nl - 1, (int)((c[0] - lo[0]) / h)), y = std::min(nl - 1, (int)((c[1] - lo[1]) / h)),
              z = std::min(nl - 1, (int)((c[2] - lo[2]) / h));
    return (x * nl + y) * nl + z;
  };
  int bestL = 0;
  double best = std::numeric_limits<double>::infinity();
  for (int L = 2; L <= 7; ++L) {
    const int nl = 1 << L;
    const double h = side / nl;
    if (h < rdamp) break;
    std::vector<int> cs((size_t)nl * nl * nl, 0), ct((size_t)nl * nl * nl, 0);
    for (int j = 0; j < ns; ++j) cs[leaf_of(&xs[3 * (size_t)j], nl, h)]++;
    for (int j = 0; j < nt; ++j) ct[leaf_of(&xt[3 * (size_t)j], nl, h)]++;
    double near = 0.0, cells = 0.0;
    for (int x = 0; x < nl; ++x)
      for (int y = 0; y < nl; ++y)
        for (int z = 0; z < nl; ++z) {
          const int c = ct[((size_t)x * nl + y) * nl + z];
          if (!c) continue;
          cells += 1.0;
          int nb = 0;
          for (int i = std::max(0, x - 1); i <= std::min(nl - 1, x + 1); ++i)
            for (int j = std::max(0, y - 1); j <= std::min(nl - 1, y + 1); ++j)
              for (int k = std::max(0, z - 1); k <= std::min(nl - 1, z + 1); ++k) nb += cs[((size_t)i * nl + j) * nl + k];
          near += (double)c * nb;
        }
    const double cost = 40.0 * near + 189.0 * cells * 8.0 / 7.0 * npairs;
    if (cost < best) {
      best = cost;
      bestL = L;
    }
  }
  if (bestL == 0) return false;
  const int L = bestL, nl = 1 << L, nleaf = nl * nl * nl;
  const double h = side / nl;
  o.L = L;
  o.side = side;
  for (int d = 0; d < 3; ++d) o.lo[d] = lo[d];
  o.off.assign(L + 2, 0);
  for (int l = 0; l <= L; ++l) o.off[l + 1] = o.off[l] + (1 << (3 * l));
  o.ncell = o.off[L + 1];
  auto sort = [&](int m, const double *x, std::vector<int> &start, std::vector<int> &perm, std::vector<int> &cnt) {
    std::vector<int> leaf(m);
    start.assign(nleaf + 1, 0);
    for (int j = 0; j < m; ++j) {
      leaf[j] = leaf_of(&x[3 * (size_t)j], nl, h);
      start[leaf[j] + 1]++;
    }
    for (int c = 0; c < nleaf; ++c) start[c + 1] += start[c];
    perm.resize(m);
    std::vector<int> fill(start.begin(), start.end() - 1);
    for (int j = 0; j < m; ++j) perm[fill[leaf[j]]++] = j;
    cnt.assign(o.ncell, 0);
    for (int c = 0; c < nleaf; ++c) cnt[o.off[L] + c] = start[c + 1] - start[c];
    for (int l = L; l > 0; --l) {
      const int nc = 1 << l;
      for (int x = 0; x < nc; ++x)
        for (int y = 0; y < nc; ++y)
          for (int z = 0; z < nc; ++z)
            cnt[o.off[l - 1] + ((x >> 1) * (nc >> 1) + (y >> 1)) * (nc >> 1) + (z >> 1)] +=
                cnt[o.off[l] + (x * nc + y) * nc + z];
    }
  };
  sort(ns, xs, o.start_s, o.perm_s, o.cnt_s);
  if (!same) sort(nt, xt, o.start_t, o.perm_t, o.cnt_t);
  return true;
}

template <typename T>
int upload(T *&dst, const std::vector<T> &v, cudaStream_t st) {
  if (dst) cudaFree(dst);
  dst = nullptr;
  if (cudaMalloc((void **)&dst, std::max<size_t>(v.size(), 1) * sizeof(T)) != cudaSuccess) return 1;
  if (!v.empty()) cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
  return 0;
}

void tree_args(const FmmState &f, const FmmTree &t, int ncol, gpu::FmmArgs &a) {
  a = gpu::FmmArgs{};
  a.p = f.p;
  a.K = f.K;
  a.KD = f.KD;
  a.L = t.L;
  a.ncell = t.ncell;
  a.ncol = ncol;
  a.h0 = t.h0;
  a.ox = t.ox, a.oy = t.oy, a.oz = t.oz;
  a.cnt = t.cnt;
  a.cnt_t = t.cnt_t;
  a.leaf_start = t.leaf_start;
  a.perm = t.perm;
  a.spos = t.spos;
  a.terms = f.terms;
  a.pairs = f.pairs;
  a.hoff = f.hoff;
  a.quads = f.quads;
  a.nquads = f.nquads;
  a.dunit = f.dunit;
  a.dunit32 = f.dunit32;
  a.M = t.M;
  a.M32 = t.M32;
  a.Lc = t.Lc;
}

// upward pass from the leaf multipoles, M2L, downward pass (columns of a)
void run_tree(const FmmState &f, const FmmTree &t, const gpu::FmmArgs &a, int ncol, cudaStream_t st) {
  const size_t smem = (f.K + (size_t)f.npairs) * sizeof(double);
  // no cell above level 2 has well-separated neighbours: their multipoles are not needed
  for (int l = t.L; l >= 3; --l)
    gpu::k_fmm_m2m<<<dim3(1 << (3 * (l - 1)), ncol), gpu::TT, 12 * (size_t)f.K * sizeof(double), st>>>(a, l);
  const size_t smem_reg = m2l_smem(f, ncol);
  const bool reg = f.nquads <= kQuadsLarge;
  const int c0 = ((1 << 6) - 1) / 7, nc = t.ncell - c0;  // the cells of levels 2..L
  if (reg && t.L >= 2) {
    gpu::k_fmm_m32<<<gpu::sm_count() * 8, 256, 0, st>>>(a, c0, nc);
    gpu::add_launch_count(1);
  }
  int launches = 1;
  if (f.nquads <= kQuadsSmall) {
    if (ncol == 2)
      gpu::k_fmm_m2l_reg<288, 3, 2><<<nc, 288, smem_reg, st>>>(a);
    else
      gpu::k_fmm_m2l_reg<288, 3, 1><<<nc, 288, smem_reg, st>>>(a);
  } else if (reg) {
    if (ncol == 2)
      gpu::k_fmm_m2l_reg<544, 4, 2><<<nc, 544, smem_reg, st>>>(a);
    else
      gpu::k_fmm_m2l_reg<544, 4, 1><<<nc, 544, smem_reg, st>>>(a);
  } else {
    for (int l = 2; l <= t.L; ++l) gpu::k_fmm_m2l<<<dim3(1 << (3 * l), ncol), gpu::FT, smem, st>>>(a, l);
    launches = t.L - 1;
  }
  for (int l = 2; l < t.L; ++l) gpu::k_fmm_l2l<<<dim3(1 << (3 * l), ncol), gpu::TT, 7 * (size_t)f.K * sizeof(double), st>>>(a, l);
  gpu::add_launch_count(std::max(0, t.L - 2) + launches + std::max(0, t.L - 2));
}

}  // namespace

bool System::fmm_tree() const { return fmm_ && fmm_->built && fmm_->d2d.L >= 0; }

int System::fmm_prepare() {
  if (fmm_ && fmm_->built) return kOk;
  if (!fmm_) {
    fmm_ = new FmmState();
    int st = build_tables(*fmm_, fmm_order_, st_);
    if (st) {
      free_fmm_state(fmm_);
      fmm_ = nullptr;
      return st == kErrCuda ? check(cudaGetLastError(), "FMM tables") : st;
    }
  }
  FmmState &f = *fmm_;
  FmmTree &t = f.d2d;
  const int n = d_.n;
  std::vector<double> xp(3 * (size_t)n);
  for (int j = 0; j < n; ++j)
    for (int d = 0; d < 3; ++d) xp[3 * (size_t)j + d] = m_.cmm[3 * (size_t)m_.polar_mm[j] + d];
  TreeLayout o;
  if (!plan_tree(n, xp.data(), 0, nullptr, std::max((double)std::sqrt(d_.damp_r2max32), fmm_min_leaf()), f.npairs,
                 o)) {
    t.L = -1;  // fewer than four damping ranges across: the direct sums serve
    f.built = true;
    log_msg(kVerbHigh, nullptr, "FMM: system too small for a tree with near field >= damping range; direct sums");
    return kOk;
  }
  std::vector<gpu::Pos64> spos(n);
  std::vector<double> sa(n);
  std::vector<float2> swa(n);
  for (int s = 0; s < n; ++s) {
    const int j = o.perm_s[s];
    const double w = 1.0 / m_.thole[m_.polar_mm[j]];
    spos[s] = gpu::Pos64{xp[3 * (size_t)j], xp[3 * (size_t)j + 1], xp[3 * (size_t)j + 2], w};
    sa[s] = m_.damping[j];
    swa[s] = make_float2(d_.wide ? 0.f : (float)(w * w), (float)(m_.damping[j] * m_.damping[j]));
  }
  double whole[3], extent = 0.0;
  for (int d = 0; d < 3; ++d) whole[d] = std::nearbyint(o.lo[d] + 0.5 * o.side);
  for (int j = 0; j < n; ++j)
    for (int d = 0; d < 3; ++d) extent = std::max(extent, std::fabs(xp[3 * (size_t)j + d] - whole[d]));
  t.L = o.L;
  t.h0 = o.side;
  t.ox = o.lo[0], t.oy = o.lo[1], t.oz = o.lo[2];
  t.off = o.off;
  t.ncell = o.ncell;
  t.shared = true;
  int bad = upload(t.cnt, o.cnt_s, st_) | upload(t.leaf_start, o.start_s, st_) | upload(t.perm, o.perm_s, st_) |
            upload(t.spos, spos, st_) | upload(t.sa, sa, st_) | upload(t.swa, swa, st_);
  if (t.split) cudaFree(t.split);
  t.split = nullptr;
  bad |= cudaMalloc((void **)&t.split, 3 * (size_t)n * sizeof(float4)) != cudaSuccess;
  t.cnt_t = t.cnt, t.leaf_start_t = t.leaf_start, t.perm_t = t.perm, t.spos_t = t.spos;
  if (t.nalloc_cell < t.ncell) {
    if (t.M) cudaFree(t.M);
    if (t.Lc) cudaFree(t.Lc);
    t.M = t.Lc = nullptr;
    bad |= cudaMalloc((void **)&t.M, 2 * (size_t)t.ncell * f.K * sizeof(double)) != cudaSuccess;
    bad |= cudaMalloc((void **)&t.Lc, 2 * (size_t)t.ncell * f.K * sizeof(double)) != cudaSuccess;
    bad |= alloc_m32(f, t, 2);
    t.nalloc_cell = t.ncell;
  }
  if (f.field_n < 6 * (size_t)n) {
    // field, near-field partials and the scales of their two columns of dipoles
    if (f.field) cudaFree(f.field);
    f.field = nullptr;
    const size_t v = 6 * (size_t)n;
    bad |= cudaMalloc((void **)&f.field, ((1 + gpu::kFmmNearSplit) * v + 1) * sizeof(double)) != cudaSuccess;
    f.near = f.field ? f.field + v : nullptr;
    f.word = f.field ? reinterpret_cast<unsigned *>(f.field + (1 + gpu::kFmmNearSplit) * v) : nullptr;
    f.field_n = f.field ? v : 0;
  }
  if (bad) {
    cudaGetLastError();
    t.nalloc_cell = 0;
    set_last_error("out of device memory for the FMM tree");
    return kErrMemory;
  }
  gpu::launch_split(n, t.spos, whole, gpu::split_step(extent), t.split, st_);
  int st = check(cudaStreamSynchronize(st_), "FMM tree upload");  // host vectors die here
  if (st) return st;
  log_msg(kVerbHigh, nullptr, "FMM: order %d, %d levels, leaf side %.2f bohr, %d sites", f.p, t.L, t.h0 / (1 << t.L),
          n);
  t.built = true;
  f.built = true;
  return kOk;
}

// The expansions (P2M to L2P: FP64 and latency bound) and the near field (FP32
// bound) meet only in the sum of the two fields.  They run on two streams, the
// expansions at the highest priority so that their short kernels get in between
// the near field's CTAs: 60,000 sites, a product 2.05 ms (near field alone 1.60;
// the kernels one after the other 2.3).
int System::fmm_tmu(int ncol, const double *x, double *y, bool dodiag) {
  int st = fmm_prepare();
  if (st) return st;
  FmmState &f = *fmm_;
  FmmTree &t = f.d2d;
  if (t.L < 0) {
    set_last_error("FMM: no tree for this system");
    return kErrInput;
  }
  const int n = d_.n;
  const size_t nv = 3 * (size_t)n;
  const float thr2m = (float)(d_.damp_thr * d_.damp_thr * (1.0 + 1e-5));
  if (!f.far) {
    int least = 0, greatest = 0;
    cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (cudaStreamCreateWithPriority(&f.far, cudaStreamNonBlocking, greatest) != cudaSuccess ||
        cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming) != cudaSuccess) {
      st = check(cudaGetLastError(), "FMM streams");
      if (f.fork) cudaEventDestroy(f.fork);
      if (f.far) cudaStreamDestroy(f.far);
      f.far = nullptr;
      f.fork = f.join = nullptr;
      return st;
    }
  }
  for (int c0 = 0; c0 < ncol; c0 += 2) {
    const int g = std::min(2, ncol - c0);
    gpu::FmmArgs a;
    tree_args(f, t, g, a);
    const double *xg = x + c0 * nv;
    cudaEventRecord(f.fork, st_);
    cudaStreamWaitEvent(f.far, f.fork, 0);
    cudaMemsetAsync(t.M, 0, 2 * (size_t)t.ncell * f.K * sizeof(double), f.far);
    cudaMemsetAsync(t.Lc, 0, 2 * (size_t)t.ncell * f.K * sizeof(double), f.far);
    const int nleaf = 1 << (3 * t.L);
    gpu::k_fmm_p2m<<<dim3(nleaf, g), (f.K + 31) / 32 * 32, 0, f.far>>>(a, xg, n);
    run_tree(f, t, a, g, f.far);
    gpu::k_fmm_l2p<<<dim3(nleaf, g), gpu::FT, 0, f.far>>>(a, n, f.field);
    cudaEventRecord(f.join, f.far);
    gpu::launch_max_words(g, nv, xg, f.word, st_);
    gpu::launch_fmm_near({n, t.L, g, m_.amoeba, t.leaf_start, t.perm, t.split, t.spos, t.sa, t.swa, d_.damp_thr, thr2m},
                         xg, f.word, f.near, st_);
    cudaStreamWaitEvent(st_, f.join, 0);
    gpu::k_fmm_add_near<<<(unsigned)((g * nv + 255) / 256), 256, 0, st_>>>(g * nv, f.near, f.field);
    gpu::add_launch_count(3);
    gpu::launch_tmu_finish64(d_, g, f.field, xg, dodiag, y + c0 * nv, st_);
  }
  return check(cudaGetLastError(), "FMM T.mu launch");
}

// E_M2D through the FMM: the static multipoles as sources, the polarizable
// sites as targets; done = false when the system is too small for a tree
int System::fmm_m2d(double *out, bool &done) {
  done = false;
  if (!fmms_) {  // tables of the static order
    fmms_ = new FmmState();
    int st = build_tables(*fmms_, fmm_order_static_, st_);
    if (st) {
      free_fmm_state(fmms_);
      fmms_ = nullptr;
      return st == kErrCuda ? check(cudaGetLastError(), "FMM tables") : st;
    }
  }
  int st = kOk;
  FmmState &f = *fmms_;
  FmmTree &t = f.m2d;
  const int n = d_.n, mm = d_.m, ld = m_.ld_cart;
  if (f.field_n < 3 * (size_t)n) {  // far field, parts of the near field
    if (f.field) cudaFree(f.field);
    f.field = nullptr;
    if (cudaMalloc((void **)&f.field, (1 + gpu::kFmmNearSplit) * 3 * (size_t)n * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      f.field_n = 0;
      set_last_error("out of device memory for the FMM field");
      return kErrMemory;
    }
    f.field_n = 3 * (size_t)n;
  }
  if (!t.built) {
    std::vector<double> xp(3 * (size_t)n);
    for (int j = 0; j < n; ++j)
      for (int d = 0; d < 3; ++d) xp[3 * (size_t)j + d] = m_.cmm[3 * (size_t)m_.polar_mm[j] + d];
    TreeLayout o;
    if (!plan_tree(mm, m_.cmm.data(), n, xp.data(), std::max((double)std::sqrt(d_.m2d_r2max32), fmm_min_leaf()),
                   f.npairs, o)) {
      t.L = -1;
      t.built = true;
      return kOk;
    }
    std::vector<gpu::Pos64> spos(mm), spos_t(n);
    std::vector<double> sq((size_t)mm * ld);
    for (int s = 0; s < mm; ++s) {
      const int i = o.perm_s[s];
      spos[s] = gpu::Pos64{m_.cmm[3 * (size_t)i], m_.cmm[3 * (size_t)i + 1], m_.cmm[3 * (size_t)i + 2], 0.0};
      for (int c = 0; c < ld; ++c) sq[(size_t)s * ld + c] = m_.q[(size_t)i * ld + c];
    }
    for (int s = 0; s < n; ++s) {
      const int j = o.perm_t[s];
      spos_t[s] = gpu::Pos64{xp[3 * (size_t)j], xp[3 * (size_t)j + 1], xp[3 * (size_t)j + 2], 0.0};
    }
    t.L = o.L;
    t.h0 = o.side;
    t.ox = o.lo[0], t.oy = o.lo[1], t.oz = o.lo[2];
    t.off = o.off;
    t.ncell = o.ncell;
    t.shared = false;
    int bad = upload(t.cnt, o.cnt_s, st_) | upload(t.leaf_start, o.start_s, st_) | upload(t.perm, o.perm_s, st_) |
              upload(t.spos, spos, st_) | upload(t.sq, sq, st_) | upload(t.cnt_t, o.cnt_t, st_) |
              upload(t.leaf_start_t, o.start_t, st_) | upload(t.perm_t, o.perm_t, st_) |
              upload(t.spos_t, spos_t, st_);
    if (t.nalloc_cell < t.ncell) {
      if (t.M) cudaFree(t.M);
      if (t.Lc) cudaFree(t.Lc);
      t.M = t.Lc = nullptr;
      bad |= cudaMalloc((void **)&t.M, (size_t)t.ncell * f.K * sizeof(double)) != cudaSuccess;
      bad |= cudaMalloc((void **)&t.Lc, (size_t)t.ncell * f.K * sizeof(double)) != cudaSuccess;
      bad |= alloc_m32(f, t, 1);
      t.nalloc_cell = t.ncell;
    }
    if (bad) {
      cudaGetLastError();
      t.nalloc_cell = 0;
      set_last_error("out of device memory for the FMM tree of the static multipoles");
      return kErrMemory;
    }
    st = check(cudaStreamSynchronize(st_), "FMM M2D tree upload");
    if (st) return st;
    t.built = true;
  }
  if (t.L < 0) return kOk;
  gpu::FmmArgs a;
  tree_args(f, t, 1, a);
  cudaMemsetAsync(t.M, 0, (size_t)t.ncell * f.K * sizeof(double), st_);
  cudaMemsetAsync(t.Lc, 0, (size_t)t.ncell * f.K * sizeof(double), st_);
  const int nleaf = 1 << (3 * t.L);
  if (m_.amoeba)
    gpu::k_fmm_p2m_mp<true><<<nleaf, (f.K + 31) / 32 * 32, 0, st_>>>(a, t.sq);
  else
    gpu::k_fmm_p2m_mp<false><<<nleaf, (f.K + 31) / 32 * 32, 0, st_>>>(a, t.sq);
  run_tree(f, t, a, 1, st_);
  // the finishing pass sums the far field and the near field's parts in order
  gpu::k_fmm_l2p_m2d<<<nleaf, gpu::FT, 0, st_>>>(a, t.leaf_start_t, t.perm_t, t.spos_t, f.field);
  gpu::launch_m2d_leaf(d_, t.L, t.leaf_start, t.perm, t.leaf_start_t, t.perm_t, f.field + 3 * (size_t)n, flag_, st_);
  gpu::add_launch_count(2);
  gpu::launch_m2d_finish(d_, out, f.field, 1 + gpu::kFmmNearSplit, st_);
  done = true;
  return check(cudaGetLastError(), "FMM M2D launch");
}

}  // namespace ommp
