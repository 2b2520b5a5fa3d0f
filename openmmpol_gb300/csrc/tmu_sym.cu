// Symmetric T.mu of FP64 accuracy (TMatVec_otf / field_extD2D,
// src/mod_polarization.F90:459-481, src/mod_electrostatics.F90:1954-2111):
// every unordered pair is evaluated once and both directions are accumulated
// (T_ij = T_ji).
//
// GB300 runs FP64 at 1/64 of its FP32 rate, so a kernel that forms every pair
// on the FP64 pipe (32 FP64 operations per unordered pair) cannot go below
// 2,048 FP32 issue slots per pair and lane; it took 230 ms per product at
// 90,000 sites with that pipe 92 % busy.  Here only the pairs that need FP64
// use it: those that may be Thole-damped (an exponential or a polynomial in
// r) or that are close.  All others are formed on the FP32 pipes in
// double-single arithmetic (ds_math.cuh), 289 FP32 operations per unordered
// pair (ncu), with
//   * coordinates split on a grid into three floats (launch_split), so
//     that the difference of two sites is exact and costs 7 operations;
//   * the unit-length form E = K (mu.n) n - k3 mu of the dipole field
//     (n = d y, y the FP32 reciprocal distance): |n|^2 is within 2^-22 of 1,
//     so its deviation is collected exactly by adding the squares to 2 and
//     r^-3 and 3 r^-5 follow from y^3 by a first- and second-order factor,
//     with no double-single square root;
//   * accumulators renormalised once per 32 sources.
// Errors against extended precision (2-norm, random dipoles): water boxes of
// 900 to 90,000 sites 3.1e-15 to 4.9e-15 (the FP64 kernel: 8.1e-15 to
// 8.7e-15), a Wang-AL system of 10,200 sites 2.1e-15 (2.9e-15).
// Time per product (one column): 917 -> 194 us at 5,001 sites, 2.6 -> 0.50 ms
// at 9,003, 25.6 -> 4.6 ms at 30,000, 230 -> 40.2 ms at 90,000 (4.05e9 pairs:
// 29 T FP32 operations/s of a measured FMA-chain rate of 36 T/s); two columns
// 70.5 ms.  Bound by FP32 issue; 5 CTAs per SM at 96 registers with small
// spills beat 4 at 128 (40.9 ms).
//
// Schedule: sites are grouped in super-tiles of 128 (4 warps x 32 lanes).
// Super-tile I meets the slots k of its half shell J = (I + k) mod ntile,
// k = 0..K (K = ntile / 2); for even ntile the slot k = ntile / 2 is handled
// by the lower of the two tiles only.  Work items (I, a chunk of slots; for
// small systems a quarter of one slot) are handed out by an atomic counter
// to a persistent grid.  Inside a slot each warp tests the bounding boxes of
// its own 32 sites and of each 32-site sub-tile of J: far apart, the 32 x 32
// pairs run without a test; otherwise an FP32 test masks the pairs that may
// be damped or are close and queues them, and the warp then forms the queued
// pairs in FP64, 32 at a time (whole sub-tiles in FP64 kept that pipe busy for
// half of a 9,000-site product: 810 us), so that the FP64 pipe works
// beside the FP32 ones.  A warp meets the 32 sources in 32 rotation steps:
// at step t lane l meets source (l + t) mod 32, the source-side accumulators
// travelling one lane per step by shuffle.  Both sides end in per-site
// 128-bit fixed-point accumulators (2^-80 resolution) with integer atomics:
// the sums do not depend on the order of the CTAs.
//
// The dipoles of each column are scaled by a power of two (sym_prepare: largest
// magnitude of the column in [2^-12, 2^-11)), so that neither the FP32 range nor
// the fixed-point resolution depends on their size or on the other column of
// the group; k_tmu_sym_finish scales back.
//
// Built with --fmad=false -ftz=true: every FMA is explicit.
#include <algorithm>
#include <cmath>

#include "ds_pair.cuh"
#include "kernels.h"
#include "pair_math.cuh"

namespace ommp {
namespace gpu {

namespace {

// x = h + m + l with h a multiple of g1 and m of g1 2^-23 (g1 = 2^-23 of the
// power of two that bounds every coordinate), so that differences of h and of
// m are exact in FP32; the parts a stride apart
__host__ __device__ inline void split_site(const Pos64 &p, double c0, double c1, double c2, double g1, float4 *out,
                                           size_t stride) {
  const double v[3] = {p.x - c0, p.y - c1, p.z - c2}, g2 = g1 * 1.1920928955078125e-7;
  float h[3], m[3], l[3];
  for (int k = 0; k < 3; ++k) {
    const double hk = rint(v[k] / g1) * g1, mk = rint((v[k] - hk) / g2) * g2;
    h[k] = (float)hk, m[k] = (float)mk, l[k] = (float)((v[k] - hk) - mk);
  }
  out[0] = make_float4(h[0], h[1], h[2], 0.f);
  out[stride] = make_float4(m[0], m[1], m[2], 0.f);
  out[2 * stride] = make_float4(l[0], l[1], l[2], 0.f);
}

constexpr int SYM_TILE = 128;
constexpr int SYM_SUB = 32;
// padding sites: no finite distance is 0 and their dipoles are 0
constexpr float SYM_FAR = 1.0e6f;

// A launch serves the products of several systems (same column count and
// damping kind): job j covers the items [item0, item0 + base[j+1] - base[j])
// of its system's product, whose item space is fixed per system, so that a
// product may also be spread over several launches (its fixed-point sums add
// up across them).  A one-job table is the single-system product.
struct SymJob {
  const float4 *g;        // [3][n] coordinate splits
  const Pos64 *pos;
  const double *damp;
  const float2 *wa;
  const float4 *boxes, *subs;  // bounding boxes of 128 and of 32 sites
  const double *x;
  unsigned long long *lo, *hi, *bad;
  int n, ntile, K, chunk, nchunk, quarters, item0;
  double thr;
  float thr2m, r2near;
};
struct SymTable {
  int njobs;
  int base[kMaxSymSlices + 1];
  SymJob job[kMaxSymSlices];
};

// floats of a staged source: 9 coordinate parts, 6 per column
template <int G>
__host__ __device__ constexpr int sym_records() {
  return (9 + 6 * G + 3) / 4;
}

template <int G>
struct SymSmem {
  float4 rec[sym_records<G>()][SYM_TILE];
  double accj[4][3 * G][SYM_TILE];
  float2 wa[SYM_TILE];                         // damping test of the near loops
  unsigned short queue[4][SYM_SUB * SYM_SUB];  // per warp: target lane * 32 + source
};

__device__ __forceinline__ float box_dist2(const float4 &alo, const float4 &ahi, const float4 &blo, const float4 &bhi) {
  const float gx = fmaxf(0.f, fmaxf(blo.x - ahi.x, alo.x - bhi.x));
  const float gy = fmaxf(0.f, fmaxf(blo.y - ahi.y, alo.y - bhi.y));
  const float gz = fmaxf(0.f, fmaxf(blo.z - ahi.z, alo.z - bhi.z));
  return fmaf(gx, gx, fmaf(gy, gy, gz * gz));
}

// the 32 x 32 pairs of a warp's sites and the sub-tile js in double-single;
// NEAR: returns the number of pairs left to FP64 in the warp's queue
template <int G, bool NEAR, bool AMOEBA>
__device__ __forceinline__ int sym_pairs(SymSmem<G> &sm, int js, int warp, int lane, bool self, const float (&tg)[9], float2 wai,
                                         const float (&mih)[G][3], const float (&mil)[G][3],
                                         float (&aih)[G][3], float (&ail)[G][3], float (&ajh)[G][3],
                                         float (&ajl)[G][3]) {
  constexpr int R = sym_records<G>();
  int queued = 0;
#pragma unroll
  for (int c = 0; c < G; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) ajh[c][k] = ajl[c][k] = 0.f;
#pragma unroll 1
  for (int t = 0; t < SYM_SUB; ++t) {
    const int jl = js * SYM_SUB + ((lane + t) & 31);
    float f[4 * R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 v = sm.rec[r][jl];
      f[4 * r] = v.x, f[4 * r + 1] = v.y, f[4 * r + 2] = v.z, f[4 * r + 3] = v.w;
    }
    float s[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = f[k];
    bool masked = false;
    const DsPair g = dsp_geometry<NEAR, AMOEBA>(tg, s, wai, NEAR ? sm.wa[jl] : wai, masked);
    if (NEAR) {
      // a sub-tile with itself meets every pair twice: queued once
      if (self) masked = masked && ((lane + t) & 31) > lane;
      const unsigned m = __ballot_sync(0xffffffffu, masked);
      if (masked)
        sm.queue[warp][queued + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(lane * 32 + ((lane + t) & 31));
      queued += __popc(m);
    }
#pragma unroll
    for (int c = 0; c < G; ++c) {
      const float mh[3] = {f[9 + 6 * c], f[10 + 6 * c], f[11 + 6 * c]};
      const float ml[3] = {f[12 + 6 * c], f[13 + 6 * c], f[14 + 6 * c]};
      dsp_column(g, mh, ml, aih[c], ail[c]);
      dsp_column(g, mih[c], mil[c], ajh[c], ajl[c]);
    }
    // the accumulators of source s move to the lane that meets s next
#pragma unroll
    for (int c = 0; c < G; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        ajh[c][k] = __shfl_sync(0xffffffffu, ajh[c][k], (lane + 1) & 31);
        ajl[c][k] = __shfl_sync(0xffffffffu, ajl[c][k], (lane + 1) & 31);
      }
  }
  // the target sums' low parts stay small against the high ones
#pragma unroll
  for (int c = 0; c < G; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const dsf r = two_sum(aih[c][k], ail[c][k]);
      aih[c][k] = r.h;
      ail[c][k] = r.l;
    }
  return queued;
}

// the queued pairs of target sub-tile at i0 and source sub-tile at j0 in FP64,
// one per lane, both sides straight into the fixed-point sums
template <int G, bool AMOEBA>
__device__ __noinline__ void sym_queued(const unsigned short *queue, int count, int lane, int i0, int j0,
                                        const SymJob &jb, int ex0, int ex1) {
  const int n = jb.n;
  for (int e = lane; e < count; e += 32) {
    const int q = queue[e], i = i0 + (q >> 5), j = j0 + (q & 31);
    if (i >= n || j >= n || i == j) continue;
    const Pos64 pi = jb.pos[i], pj = jb.pos[j];
    const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    double k3, k5;
    dd_pair_f64<AMOEBA>(r2, pi.w, pj.w, AMOEBA ? jb.damp[i] : 0.0, AMOEBA ? jb.damp[j] : 0.0, jb.wa[i], jb.wa[j],
                        jb.thr, jb.thr2m, k3, k5);
    k5 *= 3.0;
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const int ex = r ? ex1 : ex0;
      for (int side = 0; side < 2; ++side) {
        const size_t o = ((size_t)r * n + (side ? i : j)) * 3, d = ((size_t)r * n + (side ? j : i)) * 3;
        const double mx = scale_down(jb.x[o], ex), my = scale_down(jb.x[o + 1], ex), mz = scale_down(jb.x[o + 2], ex);
        const double f = k5 * fma(mx, dx, fma(my, dy, mz * dz));
        fixed_add_int(jb.lo + d, jb.hi + d, fma(f, dx, -(k3 * mx)), jb.bad);
        fixed_add_int(jb.lo + d + 1, jb.hi + d + 1, fma(f, dy, -(k3 * my)), jb.bad);
        fixed_add_int(jb.lo + d + 2, jb.hi + d + 2, fma(f, dz, -(k3 * mz)), jb.bad);
      }
    }
  }
}

template <int G, bool AMOEBA>
__global__ void __launch_bounds__(SYM_TILE, G == 1 ? 5 : 3) k_tmu_sym(const __grid_constant__ SymTable tab,
                                                       unsigned *__restrict__ next) {
  constexpr int C = 3 * G, R = sym_records<G>();
  extern __shared__ float4 sym_dyn[];
  SymSmem<G> &sm = *reinterpret_cast<SymSmem<G> *>(sym_dyn);
  __shared__ int s_item;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total = tab.base[tab.njobs];
  for (;;) {
    __syncthreads();  // every thread has read the previous item
    if (tid == 0) s_item = (int)atomicAdd(next, 1u);
    __syncthreads();
    const int item = s_item;
    if (item >= total) break;
    int jx = 0;
    while (jx + 1 < tab.njobs && tab.base[jx + 1] <= item) ++jx;
    const SymJob &jb = tab.job[jx];
    const int n = jb.n, ntile = jb.ntile, nsub = (n + SYM_SUB - 1) / SYM_SUB;
    const float4 *__restrict__ gc = jb.g;
    const double *__restrict__ x = jb.x;
    const int local = jb.item0 + (item - tab.base[jx]);
    const int q = local % jb.quarters, unit = local / jb.quarters;
    const int js0 = q * (4 / jb.quarters), js1 = js0 + 4 / jb.quarters;
    const int I = unit / jb.nchunk;
    const int ti = I * SYM_TILE + tid;
    const bool vi = ti < n;
    int ex[G];
#pragma unroll
    for (int c = 0; c < G; ++c) ex[c] = dsp_exponent(reinterpret_cast<const unsigned *>(jb.bad + 1)[c]);
    float tg[9], mih[G][3], mil[G][3];
    {
      const float4 h = vi ? gc[ti] : make_float4(SYM_FAR, SYM_FAR, SYM_FAR, 0.f);
      const float4 m = vi ? gc[(size_t)n + ti] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 l = vi ? gc[2 * (size_t)n + ti] : make_float4(0.f, 0.f, 0.f, 0.f);
      tg[0] = h.x, tg[1] = h.y, tg[2] = h.z, tg[3] = m.x, tg[4] = m.y, tg[5] = m.z, tg[6] = l.x, tg[7] = l.y,
      tg[8] = l.z;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const double m = vi ? scale_down(x[((size_t)(c / 3) * n + ti) * 3 + (c % 3)], ex[c / 3]) : 0.0;
      const dsf d = to_ds(m);
      mih[c / 3][c % 3] = d.h;
      mil[c / 3][c % 3] = d.l;
    }
    double sumi[C];
#pragma unroll
    for (int c = 0; c < C; ++c) sumi[c] = 0.0;
    const float4 ilo = jb.boxes[2 * I], ihi = jb.boxes[2 * I + 1];
    const int k0 = (unit - I * jb.nchunk) * jb.chunk;
    const int k1 = min(jb.K + 1, k0 + jb.chunk);
    for (int k = k0; k < k1; ++k) {
      int J = I + k;
      if (J >= ntile) J -= ntile;
      if (k > 0 && 2 * k == ntile && I >= ntile / 2) continue;  // the other tile of the pair owns it
      const bool diag = (k == 0);
      // uniform over the CTA: may the slot hold near pairs?
      const bool near_slot = !(box_dist2(ilo, ihi, jb.boxes[2 * J], jb.boxes[2 * J + 1]) > jb.r2near);
      __syncthreads();
      if (warp >= js0 && warp < js1) {
        const int sj = J * SYM_TILE + tid;
        const bool v = sj < n;
        const float4 h = v ? gc[sj] : make_float4(-SYM_FAR, -SYM_FAR, -SYM_FAR, 0.f);
        const float4 m = v ? gc[(size_t)n + sj] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 l = v ? gc[2 * (size_t)n + sj] : make_float4(0.f, 0.f, 0.f, 0.f);
        float f[4 * R] = {h.x, h.y, h.z, m.x, m.y, m.z, l.x, l.y, l.z};
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const double mu = v ? scale_down(x[((size_t)(c / 3) * n + sj) * 3 + (c % 3)], ex[c / 3]) : 0.0;
          const dsf d = to_ds(mu);
          f[9 + 6 * (c / 3) + c % 3] = d.h;
          f[12 + 6 * (c / 3) + c % 3] = d.l;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) sm.rec[r][tid] = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
        if (near_slot) sm.wa[tid] = v ? jb.wa[sj] : make_float2(0.f, 0.f);
      }
      __syncthreads();
      const int si = 4 * I + warp;  // the warp's own sub-tile
      float aih[G][3], ail[G][3];
#pragma unroll
      for (int c = 0; c < G; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) aih[c][d] = ail[c][d] = 0.f;
      for (int js = js0; js < js1; ++js) {
        const int sj = 4 * J + js;
        const bool skip = si >= nsub || sj >= nsub || (diag && js < warp);
        const bool self = diag && js == warp;
        bool near = false;
        if (!skip && near_slot)
          near = self || !(box_dist2(jb.subs[2 * si], jb.subs[2 * si + 1], jb.subs[2 * sj], jb.subs[2 * sj + 1]) >
                           jb.r2near);
        double outj[C];
        if (skip) {
#pragma unroll
          for (int c = 0; c < C; ++c) outj[c] = 0.0;
        } else {
          float ajh[G][3], ajl[G][3];
          if (near) {
            const float2 wai = vi ? jb.wa[ti] : make_float2(0.f, 0.f);
            const int queued =
                sym_pairs<G, true, AMOEBA>(sm, js, warp, lane, self, tg, wai, mih, mil, aih, ail, ajh, ajl);
            __syncwarp();
            sym_queued<G, AMOEBA>(sm.queue[warp], queued, lane, I * SYM_TILE + warp * 32, J * SYM_TILE + js * 32, jb,
                                  ex[0], ex[G - 1]);
            __syncwarp();
          } else {
            sym_pairs<G, false, AMOEBA>(sm, js, warp, lane, false, tg, make_float2(0.f, 0.f), mih, mil, aih, ail, ajh,
                                        ajl);
          }
#pragma unroll
          for (int c = 0; c < C; ++c) outj[c] = self ? 0.0 : (double)ajh[c / 3][c % 3] + (double)ajl[c / 3][c % 3];
        }
        // after 32 steps lane l holds the sums of source js*32 + l
#pragma unroll
        for (int c = 0; c < C; ++c) sm.accj[warp][c][js * SYM_SUB + lane] = outj[c];
      }
#pragma unroll
      for (int c = 0; c < C; ++c) sumi[c] += (double)aih[c / 3][c % 3] + (double)ail[c / 3][c % 3];
      __syncthreads();
      const int sj = J * SYM_TILE + tid;
      if (warp >= js0 && warp < js1 && sj < n) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const double v = ((sm.accj[0][c][tid] + sm.accj[1][c][tid]) + sm.accj[2][c][tid]) + sm.accj[3][c][tid];
          const size_t o = ((size_t)(c / 3) * n + sj) * 3 + (c % 3);
          fixed_add_int(jb.lo + o, jb.hi + o, v, jb.bad);
        }
      }
    }
    if (vi) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const size_t o = ((size_t)(c / 3) * n + ti) * 3 + (c % 3);
        fixed_add_int(jb.lo + o, jb.hi + o, sumi[c], jb.bad);
      }
    }
  }
}

// column blockIdx.y: its accumulators (if any; the columns' low words, then
// their high words) to zero and its largest high word of |x| (ctl, zeroed
// before: one word per column, or two per group of group_words unsigneds)
__global__ void __launch_bounds__(256) k_sym_prepare(size_t total, const double *__restrict__ x,
                                                     unsigned long long *__restrict__ acc, unsigned *ctl,
                                                     size_t group_words) {
  const size_t col = (size_t)blockIdx.y * total;
  x += col;
  ctl += group_words ? (blockIdx.y / 2) * group_words + blockIdx.y % 2 : blockIdx.y;
  unsigned m = 0;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    if (acc) {
      acc[col + k] = 0ull;
      acc[gridDim.y * total + col + k] = 0ull;
    }
    m = max(m, (unsigned)__double2hiint(x[k]) & 0x7FFFFFFFu);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(ctl, m);
}

// y = -(pair sums + scaled-pair corrections) (+ x / alpha): the fixed-point
// sums read out (NaN when flagged) and scaled back; with part, the partial
// sums of x.y of every block.  L lanes per site share its scaled pairs: four
// below kFinishLanesSites (one thread per site left 5,001 sites on 40 CTAs,
// bound by the latency of its pair list), one above.
constexpr int FIN_TPB = 256;
template <bool AMOEBA, int L>
__global__ void __launch_bounds__(FIN_TPB) k_tmu_sym_finish(
    int n, const unsigned long long *__restrict__ lo, const unsigned long long *__restrict__ hi,
    const unsigned long long *__restrict__ bad, const Pos64 *__restrict__ pos, const double *__restrict__ damp,
    const float2 *__restrict__ wa, const double *__restrict__ x, const double *__restrict__ ialpha, bool dodiag,
    const int *__restrict__ ri, const int *__restrict__ src, const double *__restrict__ scale, double thr, float thr2m,
    double *__restrict__ y, double *__restrict__ part, size_t group_words) {
  __shared__ double s_dot[FIN_TPB / 32];
  const size_t col = (size_t)blockIdx.y * n;
  if (group_words) {  // groups of two columns, each with its own accumulators
    const size_t shift = (blockIdx.y / 2) * group_words;
    lo += shift, hi += shift, bad += shift;
    lo -= (size_t)(blockIdx.y / 2) * 6 * n, hi -= (size_t)(blockIdx.y / 2) * 6 * n;
  }
  const bool nan = *bad != 0ull;
  const int ex = dsp_exponent(reinterpret_cast<const unsigned *>(bad + 1)[blockIdx.y % 2]);
  const int lane = threadIdx.x % L;
  double dot = 0.0;
  for (int j = (blockIdx.x * FIN_TPB + threadIdx.x) / L; j < n; j += gridDim.x * (FIN_TPB / L)) {
    double e[3] = {0.0, 0.0, 0.0};
    if (ri) {
      const Pos64 pt = pos[j];
      const double at = AMOEBA ? damp[j] : 0.0;
      const float2 wat = wa[j];
      for (int k = ri[j] + lane; k < ri[j + 1]; k += L) {
        const int i = src[k];
        const Pos64 ps = pos[i];
        const double dx = pt.x - ps.x, dy = pt.y - ps.y, dz = pt.z - ps.z;
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        double k3, k5;
        dd_pair_f64<AMOEBA>(r2, pt.w, ps.w, at, AMOEBA ? damp[i] : 0.0, wat, wa[i], thr, thr2m, k3, k5);
        const double *mu = &x[(col + i) * 3];
        const double f = 3.0 * k5 * fma(mu[0], dx, fma(mu[1], dy, mu[2] * dz));
        const double cs = scale[k] - 1.0;
        e[0] = fma(cs, fma(f, dx, -(k3 * mu[0])), e[0]);
        e[1] = fma(cs, fma(f, dy, -(k3 * mu[1])), e[1]);
        e[2] = fma(cs, fma(f, dz, -(k3 * mu[2])), e[2]);
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
      const size_t o = (col + j) * 3 + c;
      const double v =
          e[c] + (nan ? __longlong_as_double(0x7ff8000000000000ll) : scale_up(fixed_value(lo[o], hi[o]), ex));
      const double yv = dodiag ? fma(x[o], ialpha[j], -v) : -v;
      y[o] = yv;
      dot = fma(x[o], yv, dot);
    }
  }
  if (!part) return;
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if ((threadIdx.x & 31) == 0) s_dot[threadIdx.x >> 5] = dot;
  __syncthreads();
  if (threadIdx.x == 0) {
    dot = 0.0;
    for (int w = 0; w < FIN_TPB / 32; ++w) dot += s_dot[w];
    part[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = dot;
  }
}

__global__ void __launch_bounds__(256) k_split(int n, const Pos64 *__restrict__ pos, double c0, double c1, double c2,
                                               double g1, float4 *__restrict__ out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) split_site(pos[i], c0, c1, c2, g1, out + i, n);
}

template <int G, bool AMOEBA>
struct SymLaunch {
  int resident = 0;
  SymLaunch() {
    const int smem = (int)sizeof(SymSmem<G>);
    cudaFuncSetAttribute(k_tmu_sym<G, AMOEBA>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_tmu_sym<G, AMOEBA>, SYM_TILE, smem);
    if (resident < 1) resident = 1;
  }
};
template <int G, bool AMOEBA>
int sym_resident() {
  static const SymLaunch<G, AMOEBA> cfg;  // thread-safe one-time set-up
  return cfg.resident;
}
int sym_ctas(int g, bool amoeba) {
  if (g == 2) return (amoeba ? sym_resident<2, true>() : sym_resident<2, false>()) * sm_count();
  return (amoeba ? sym_resident<1, true>() : sym_resident<1, false>()) * sm_count();
}

struct SymPlan {
  int ntile, K, chunk, nchunk, quarters;
  int items() const { return ntile * nchunk * quarters; }
};

// work items: about 16 per resident CTA, each a tile and a chunk of its slots
// (round_pairs > 0: at most a quarter of a CTA's share of round_pairs); with
// fewer than 8 slots per CTA an item is a quarter of one slot
SymPlan sym_plan(int n, int ctas, double round_pairs) {
  SymPlan p;
  p.ntile = (n + SYM_TILE - 1) / SYM_TILE;
  p.K = p.ntile / 2;
  const long long units = (long long)p.ntile * (p.K + 1);
  long long chunk = units / (16LL * ctas);
  if (round_pairs > 0.0) chunk = std::min(chunk, (long long)(round_pairs / (4.0 * ctas * SYM_TILE * SYM_TILE)));
  chunk = std::max(1LL, std::min(chunk, (long long)p.K + 1));
  p.chunk = (int)chunk;
  p.nchunk = (p.K + 1 + p.chunk - 1) / p.chunk;
  p.quarters = units < 8LL * ctas ? 4 : 1;
  return p;
}

template <int G, bool AMOEBA>
void launch_table(const SymTable &tab, unsigned *next, cudaStream_t st, bool zeroed) {
  const int total = tab.base[tab.njobs];
  const int ctas = std::min(sym_resident<G, AMOEBA>() * sm_count(), total);
  if (!zeroed) cudaMemsetAsync(next, 0, sizeof(unsigned), st);
  k_tmu_sym<G, AMOEBA><<<ctas, SYM_TILE, sizeof(SymSmem<G>), st>>>(tab, next);
}

// thr^2 with the relative safety margin of the FP32 damping pre-test
float thr2_margin(const DevSites &s) { return (float)(s.damp_thr * s.damp_thr * (1.0 + 1e-5)); }

}  // namespace

int tmu_f64_sym_items(const DevSites &s, int g, double round_pairs) {
  if (s.n == 0) return 0;
  return sym_plan(s.n, sym_ctas(g, s.amoeba), round_pairs).items();
}

void launch_tmu_f64_sym_multi(int g, bool amoeba, const SymSlice *sl, int nsl, unsigned *next, cudaStream_t st,
                              bool zeroed) {
  SymTable tab{};
  int total = 0;
  for (int k = 0; k < nsl && tab.njobs < kMaxSymSlices; ++k) {
    const DevSites &s = *sl[k].s;
    if (sl[k].count <= 0 || s.n == 0) continue;
    const SymPlan p = sym_plan(s.n, sym_ctas(g, amoeba), sl[k].round_pairs);
    SymJob &j = tab.job[tab.njobs];
    j.g = s.pol_split, j.pos = s.pol_pos, j.damp = s.pol_a, j.wa = s.pol_wa32;
    j.boxes = s.tile_box32, j.subs = s.sub_box32;
    j.x = static_cast<const double *>(sl[k].x);
    j.lo = sl[k].lo, j.hi = sl[k].hi, j.bad = sl[k].bad;
    j.n = s.n, j.ntile = p.ntile, j.K = p.K, j.chunk = p.chunk, j.nchunk = p.nchunk, j.quarters = p.quarters;
    j.item0 = sl[k].item0;
    j.thr = s.damp_thr;
    j.thr2m = thr2_margin(s);
    j.r2near = near_range2(s, s.damp_r2max32);
    tab.base[tab.njobs] = total;
    total += sl[k].count;
    ++tab.njobs;
  }
  tab.base[tab.njobs] = total;
  if (!total) return;
  add_launch_count(1);
  if (g == 2)
    amoeba ? launch_table<2, true>(tab, next, st, zeroed) : launch_table<2, false>(tab, next, st, zeroed);
  else
    amoeba ? launch_table<1, true>(tab, next, st, zeroed) : launch_table<1, false>(tab, next, st, zeroed);
}

void launch_tmu_sym_prepare(const DevSites &s, int g, const double *x, unsigned long long *lo, unsigned long long *bad,
                            cudaStream_t st) {
  const size_t nv = 3 * (size_t)s.n;
  add_launch_count(1);
  cudaMemsetAsync(bad, 0, 2 * sizeof(unsigned long long), st);
  const int blocks = (int)std::min<size_t>((nv + 255) / 256, 1216);
  k_sym_prepare<<<dim3(blocks, g), 256, 0, st>>>(nv, x, lo, reinterpret_cast<unsigned *>(bad + 1), 0);
}

void launch_max_word(size_t total, const double *x, unsigned *word, cudaStream_t st, bool zeroed) {
  add_launch_count(1);
  if (!zeroed) cudaMemsetAsync(word, 0, sizeof(unsigned), st);
  const int blocks = (int)std::min<size_t>((total + 255) / 256, 1216);
  k_sym_prepare<<<blocks, 256, 0, st>>>(total, x, nullptr, word, 0);
}

void launch_tmu_sym_finish(const DevSites &s, int g, const unsigned long long *lo, const unsigned long long *hi,
                           const unsigned long long *bad, const double *x, bool dodiag, double *y, cudaStream_t st,
                           double *part, int max_part, int *npart, size_t group_words) {
  add_launch_count(1);
  const int lanes = s.n < kFinishLanesSites ? 4 : 1;
  int blocks = (int)(((size_t)s.n * lanes + FIN_TPB - 1) / FIN_TPB);
  if (part) blocks = std::min(blocks, max_part);
  if (npart) *npart = blocks;
  const dim3 grid(blocks, g);
  const int *ri = s.d2d_nnz ? s.d2d_ri : nullptr;
  auto go = [&](auto kernel) {
    kernel<<<grid, FIN_TPB, 0, st>>>(s.n, lo, hi, bad, s.pol_pos, s.pol_a, s.pol_wa32, x, s.pol_ialpha, dodiag, ri,
                                     s.d2d_src, s.d2d_s, s.damp_thr, thr2_margin(s), y, part, group_words);
  };
  if (lanes == 4)
    s.amoeba ? go(k_tmu_sym_finish<true, 4>) : go(k_tmu_sym_finish<false, 4>);
  else
    s.amoeba ? go(k_tmu_sym_finish<true, 1>) : go(k_tmu_sym_finish<false, 1>);
}

size_t tmu_sym_scratch_doubles(const DevSites &s, int nrhs) {
  if (s.n == 0) return 0;
  // two 64-bit accumulator words and one value read out (FP32 product) per
  // value of a column group (at most two columns), the error flag, the scales
  // (a 32-bit word per column) and the work counter
  const size_t C = 3 * (size_t)(nrhs < 2 ? nrhs : 2);
  return 3 * C * (size_t)s.n + 3;
}

void launch_tmu_f64_sym(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, double *scratch,
                        cudaStream_t st) {
  if (s.n == 0) return;
  // two columns share the pair geometry
  for (int done = 0; done < nrhs;) {
    const int g = nrhs - done >= 2 ? 2 : 1;
    const size_t C = 3 * (size_t)g;
    unsigned long long *lo = reinterpret_cast<unsigned long long *>(scratch);
    unsigned long long *hi = lo + C * s.n;
    unsigned long long *bad = lo + 3 * C * s.n;
    unsigned *next = reinterpret_cast<unsigned *>(bad + 2);
    const double *xg = x + (size_t)done * s.n * 3;
    launch_tmu_sym_prepare(s, g, xg, lo, bad, st);
    SymSlice one{&s, xg, lo, hi, bad, 0, tmu_f64_sym_items(s, g)};
    launch_tmu_f64_sym_multi(g, s.amoeba, &one, 1, next, st);
    launch_tmu_sym_finish(s, g, lo, hi, bad, xg, dodiag, y + (size_t)done * s.n * 3, st);
    done += g;
  }
}

// Pairs of columns per launch: about 16 slots per resident CTA.  A product of
// two columns of 3,003 sites has 312 slots for 456 CTAs:
// 24 columns took 12 x 176 us one pair after another, 1,436 us in one launch.
int tmu_sym_groups(const DevSites &s, int nrhs) {
  const int pairs = nrhs / 2;
  if (s.n == 0 || pairs < 2) return 1;
  const SymPlan p = sym_plan(s.n, sym_ctas(2, s.amoeba), 0.0);
  const long long units = (long long)p.ntile * (p.K + 1);
  const long long want = (16LL * sym_ctas(2, s.amoeba) + units - 1) / units;
  return (int)std::min<long long>(std::min<long long>(want, pairs), kMaxSymSlices);
}

void launch_tmu_f64_sym_groups(const DevSites &s, int nrhs, const double *x, double *y, bool dodiag, double *scratch,
                               cudaStream_t st) {
  if (s.n == 0) return;
  const int most = tmu_sym_groups(s, nrhs);
  const size_t nv = 3 * (size_t)s.n, words = tmu_sym_scratch_doubles(s, 2);
  unsigned long long *base = reinterpret_cast<unsigned long long *>(scratch);
  int done = 0;
  while (most > 1 && nrhs - done >= 2) {
    const int groups = std::min(most, (nrhs - done) / 2);
    const double *xg = x + done * nv;
    cudaMemsetAsync(scratch, 0, groups * words * sizeof(double), st);
    add_launch_count(1);
    const int blocks = (int)std::min<size_t>((nv + 255) / 256, 1216);
    k_sym_prepare<<<dim3(blocks, 2 * groups), 256, 0, st>>>(nv, xg, nullptr,
                                                            reinterpret_cast<unsigned *>(base + 6 * nv + 1), 2 * words);
    SymSlice sl[kMaxSymSlices];
    const int items = tmu_f64_sym_items(s, 2);
    for (int g = 0; g < groups; ++g) {
      unsigned long long *lo = base + g * words;
      sl[g] = {&s, xg + 2 * g * nv, lo, lo + 2 * nv, lo + 6 * nv, 0, items};
    }
    launch_tmu_f64_sym_multi(2, s.amoeba, sl, groups, reinterpret_cast<unsigned *>(base + 6 * nv + 2), st, true);
    launch_tmu_sym_finish(s, 2 * groups, base, base + 2 * nv, base + 6 * nv, xg, dodiag, y + done * nv, st, nullptr, 0,
                          nullptr, words);
    done += 2 * groups;
  }
  if (done < nrhs) launch_tmu_f64_sym(s, nrhs - done, x + done * nv, y + done * nv, dodiag, scratch, st);
}

// the largest high word of |x| of each column, words zeroed here
void launch_max_words(int ncol, size_t nv, const double *x, unsigned *words, cudaStream_t st) {
  add_launch_count(1);
  cudaMemsetAsync(words, 0, ncol * sizeof(unsigned), st);
  const int blocks = (int)std::min<size_t>((nv + 255) / 256, 1216);
  k_sym_prepare<<<dim3(blocks, ncol), 256, 0, st>>>(nv, x, nullptr, words, 0);
}

double split_step(double extent) {
  int e = 0;
  std::frexp(std::max(1.0, extent), &e);  // extent < 2^e
  return std::ldexp(1.0, e - 23);
}

void split_coordinates(int n, const Pos64 *pos, const double centre[3], double g1, float4 *out) {
  for (int i = 0; i < n; ++i) split_site(pos[i], centre[0], centre[1], centre[2], g1, out + i, n);
}

void launch_split(int n, const Pos64 *pos, const double centre[3], double g1, float4 *out, cudaStream_t st) {
  if (n == 0) return;
  add_launch_count(1);
  k_split<<<(n + 255) / 256, 256, 0, st>>>(n, pos, centre[0], centre[1], centre[2], g1, out);
}

}  // namespace gpu
}  // namespace ommp
