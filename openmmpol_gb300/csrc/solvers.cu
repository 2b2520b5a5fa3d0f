// Iterative solvers on a column workspace, and the batched solve.
//
//   cg64_ws      the reference's preconditioned CG (src/mod_solvers.F90:86-216)
//                for ncol independent columns sharing each T.mu product:
//                zero-norm guess replaced by alpha*x, quick exit when
//                |p.Tp| < 100 eps, convergence on sqrt(r.alpha r / n).
//   pcg32_ws     the FP32 inner solver of the mixed-precision path.
//   run_loop     either loop on the device, as a conditional CUDA graph.
//   mixed_ir_ws  iterative refinement: FP64 residual E - T mu, FP32 PCG on the
//                normalised residual, FP64 accumulation, FP64 convergence test.
//   tune_f32     picks the FP32 kernel, its column-group width and source split
//                by the system's size (kept per width).
//   solve_batch  nf fields at once (64 QM densities, say): one block of
//                columns through the same solvers.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "engine.h"
#include "log.h"

namespace ommp {

namespace {
template <typename T>
int walloc(T *&p, size_t count) {
  return device_alloc((void **)&p, std::max<size_t>(count, 1) * sizeof(T));
}

template <typename T>
void key_add(std::vector<char> &key, const T &v) {
  const char *b = reinterpret_cast<const char *>(&v);
  key.insert(key.end(), b, b + sizeof(T));
}
}  // namespace

void System::free_ws(Workspace &w) {
  w.loop32.drop();
  for (CgLoop &l : w.loop64) l.drop();
  if (w.sym) cudaFree(w.sym);
  w.sym = nullptr, w.sym_len = 0;
  if (!w.owned) return;
  void *b[] = {w.x, w.r, w.p, w.h, w.z, w.rhs, w.fields, w.out, w.x32, w.r32, w.p32, w.h32, w.z32,
               w.scratch32, w.partial, w.dots, w.hist, w.cols, w.t32, w.gram, w.bcoef, w.bidx};
  for (void *p : b)
    if (p) cudaFree(p);
  if (st_) cudaStreamSynchronize(st_);  // read-backs into the pinned buffers
  pinned_free(w.cols_h);
  pinned_free(w.scal_h);
  pinned_free(w.bscal_h);
  pinned_free(w.bcoef_h);
  w = Workspace();
}

int System::ensure_batch_ws(int ncol, int nf) {
  if (wsb_.cap >= ncol && wsb_.fcap >= nf) return kOk;
  cudaStreamSynchronize(st_);
  free_ws(wsb_);
  Workspace &w = wsb_;
  const size_t nv = 3 * (size_t)d_.n;
  const int nipd = m_.n_ipd;
  int s0 = gpu::tmu32_max_split(d_, gpu::sm_count());
  int bad = 0;
  bad |= walloc(w.x, ncol * nv) | walloc(w.r, ncol * nv) | walloc(w.p, ncol * nv) | walloc(w.h, ncol * nv) |
         walloc(w.z, ncol * nv) | walloc(w.rhs, ncol * nv);
  bad |= walloc(w.fields, nf * nv) | walloc(w.out, (size_t)nf * nipd * nv);
  bad |= walloc(w.x32, ncol * nv) | walloc(w.r32, ncol * nv) | walloc(w.p32, ncol * nv) |
         walloc(w.h32, ncol * nv) | walloc(w.z32, ncol * nv);
  bad |= walloc(w.scratch32, (size_t)s0 * ncol * nv);
  w.partial_len = 4 * (size_t)gpu::kRedBlocks * std::max(ncol, nf);
  bad |= walloc(w.partial, w.partial_len) |
         walloc(w.dots, 3 * (size_t)ncol + nf) | walloc(w.cols, ncol + 1);
  // block CG buffers (sized for the widest block)
  const int smax = gpu::block_cg_max_columns();
  bad |= walloc(w.t32, ncol * nv) | walloc(w.gram, gpu::block_cg_gram_doubles(smax)) |
         walloc(w.bcoef, (size_t)smax * smax) | walloc(w.bidx, 2 * (size_t)smax);
  if (bad || pinned_alloc((void **)&w.cols_h, ncol * sizeof(gpu::CgCol)) != cudaSuccess ||
      pinned_alloc((void **)&w.scal_h, (3 * (size_t)ncol + nf) * sizeof(double)) != cudaSuccess ||
      pinned_alloc((void **)&w.bscal_h, (2 * (size_t)smax * smax + smax) * sizeof(double)) != cudaSuccess ||
      pinned_alloc((void **)&w.bcoef_h, (size_t)smax * smax * sizeof(float)) != cudaSuccess) {
    w.owned = true;
    free_ws(w);
    set_last_error("out of device memory for the batch workspace");
    return kErrMemory;
  }
  cudaMemsetAsync(w.cols, 0, (ncol + 1) * sizeof(gpu::CgCol), st_);
  w.cap = ncol;
  w.fcap = nf;
  w.scratch32_nsplit = s0;
  w.owned = true;
  return kOk;
}

// ---------------------------------------------------------------------------
// A CG loop on the device: one iteration captured as the body of a while node
// whose condition the last step sets, so that the host waits once per solve
// instead of once per iteration (about 10 us each).  The loop ends after
// CgCol::max_passes iterations at the latest.  The body holds kernels alone: one
// with memset nodes crashed the host process (the GPU kept answering), so that
// anything else is refused here, whoever captures it.
// ---------------------------------------------------------------------------
namespace {
bool kernels_only(cudaGraph_t g) {
  size_t n = 0;
  if (cudaGraphGetNodes(g, nullptr, &n) != cudaSuccess) return false;
  std::vector<cudaGraphNode_t> nodes(n);
  if (n && cudaGraphGetNodes(g, nodes.data(), &n) != cudaSuccess) return false;
  for (cudaGraphNode_t node : nodes) {
    cudaGraphNodeType type;
    if (cudaGraphNodeGetType(node, &type) != cudaSuccess || type != cudaGraphNodeTypeKernel) return false;
  }
  return n > 0;
}
}  // namespace

bool System::run_loop(CgLoop &loop, const std::vector<char> &key,
                      const std::function<void(cudaGraphConditionalHandle)> &body, int &st) {
  st = kOk;
  if (!use_graphs_) return false;
  if (!loop.exec || loop.key != key) {
    loop.drop();
    cudaGraph_t g = nullptr, captured = nullptr;
    cudaGraphConditionalHandle handle = 0;
    cudaGraphNodeParams par = {};
    cudaGraphNode_t node;
    bool ok = cudaGraphCreate(&g, 0) == cudaSuccess &&
              cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
    if (ok) {
      par.type = cudaGraphNodeTypeConditional;
      par.conditional.handle = handle;
      par.conditional.type = cudaGraphCondTypeWhile;
      par.conditional.size = 1;
      ok = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &par) == cudaSuccess &&
           cudaStreamBeginCaptureToGraph(st_, par.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    }
    if (ok) {
      const long long before = gpu::thread_launch_count();
      body(handle);
      loop.kernels = gpu::thread_launch_count() - before;
      gpu::add_launch_count(-loop.kernels);  // captured, not launched
      ok = cudaStreamEndCapture(st_, &captured) == cudaSuccess && kernels_only(par.conditional.phGraph_out[0]) &&
           cudaGraphInstantiate(&loop.exec, g, 0) == cudaSuccess;
    }
    if (g) cudaGraphDestroy(g);
    if (!ok) {
      loop.exec = nullptr;
      cudaGetLastError();
      log_msg(kVerbHigh, nullptr, "CUDA graph capture of the CG loop failed: launches from the host");
      return false;
    }
    loop.key = key;
  }
  st = check(cudaGraphLaunch(loop.exec, st_), "CG loop");
  if (!st) st = check(cudaStreamSynchronize(st_), "CG loop");
  return true;
}

// ---------------------------------------------------------------------------
// FP64 conjugate gradient (reference algorithm), ncol columns
// ---------------------------------------------------------------------------
int System::cg64_ws(Workspace &w, int matv, int ncol, const double *rhs, double *x, int set0) {
  const int n = d_.n;
  const size_t nv = 3 * (size_t)n;
  log_msg(kVerbLow, nullptr, "Solving linear system with CG solver");
  log_msg(kVerbLow, nullptr, "Max iter: %4d", maxiter_);
  log_msg(kVerbLow, nullptr, "Tolerance: %8.1E", tol_);
  // guess: a zero-norm input is replaced by precnd(x) = alpha * x (:151-157)
  gpu::launch_dots(ncol, nv, x, x, w.partial, st_);
  gpu::launch_reduce_partials(ncol, w.partial, w.dots, st_);
  cudaMemcpyAsync(w.scal_h, w.dots, ncol * sizeof(double), cudaMemcpyDeviceToHost, st_);
  int st = check(cudaStreamSynchronize(st_), "CG start");
  if (st) return st;
  bool all_zero = true;
  for (int k = 0; k < ncol; ++k) {
    if (w.scal_h[k] < kEpsRp) {
      log_msg(kVerbHigh, nullptr, "Input guess has zero norm, generating a guess from preconditioner.");
      gpu::launch_scale_by_alpha(1, n, d_.pol_alpha, x + k * nv, x + k * nv, st_);
    } else {
      log_msg(kVerbHigh, nullptr, "Using input guess as a starting point for iterative solver.");
    }
    if (w.scal_h[k] != 0.0) all_zero = false;
  }
  // r = rhs - T x; an exactly zero x gives T x = 0 without the pair sum
  if (all_zero) {
    cudaMemcpyAsync(w.r, rhs, ncol * nv * sizeof(double), cudaMemcpyDeviceToDevice, st_);
  } else {
    st = matvec64(matv, ncol, x, w.z, true);
    if (st) return st;
    gpu::launch_residual(ncol * nv, rhs, w.z, w.r, st_);
  }
  // z = alpha r, p = z, the first r.z
  const size_t share = w.partial_len / (2 * (size_t)ncol);
  double *hist = (set0 >= 0) ? w.hist : nullptr;
  gpu::CgJob<double> job{};
  job.n = n, job.ncol = ncol;
  job.nb = gpu::cg_blocks(n, ncol, w.partial_len);
  job.eps = kEpsRp, job.tol = tol_;
  job.x = x, job.r = w.r, job.p = w.p, job.h = w.h, job.alpha = d_.pol_alpha;
  job.pa = w.partial, job.pb = w.partial + share * ncol;
  job.cols = w.cols, job.cols_h = w.cols_h;
  job.meet = reinterpret_cast<unsigned *>(w.cols + w.cap);
  job.hist = hist, job.nhist = maxhist_;
  // the direct symmetric product of one column group: its accumulators and
  // scales are prepared by the steps, its finishing pass sums p.h
  const bool sym = direct_symmetric(matv, ncol);
  const size_t C = 3 * (size_t)ncol;
  unsigned long long *lo = reinterpret_cast<unsigned long long *>(sym_scratch_);
  if (sym) {
    job.acc = lo, job.nacc = 2 * C * n, job.words = lo + 3 * C * n;
    job.emax = reinterpret_cast<unsigned *>(job.words + 1);
  }
  // the ordered one: the scale of every column
  const bool rows = !sym && direct_rows(matv, ncol);
  if (rows && gpu::tmu_rows_parts(d_, ncol) > 0) job.emax = row_words_;
  const bool small = !sym && n <= gpu::kCgSmallSites;
  job.max_passes = maxiter_;
  job.init = gpu::kCgInitKeep;
  gpu::launch_cg_steps(&job, 1, st_);
  job.init = 0;
  auto enqueue = [&]() -> int {
    if (sym) {
      KEv e;
      if (ktime_on_) e = kt_begin(0, ncol);
      gpu::SymSlice one{&d_, w.p, lo, lo + C * n, job.words, 0, gpu::tmu_f64_sym_items(d_, ncol)};
      gpu::launch_tmu_f64_sym_multi(ncol, d_.amoeba, &one, 1, reinterpret_cast<unsigned *>(job.words + 2), st_, true);
      gpu::launch_tmu_sym_finish(d_, ncol, lo, lo + C * n, job.words, w.p, true, w.h, st_, job.pa, (int)share, &job.na);
      if (ktime_on_) kt_end(e);
      stats_.f64_matvecs += 1;
    } else if (rows) {
      KEv e;
      if (ktime_on_) e = kt_begin(0, ncol);
      const int parts = gpu::tmu_rows_parts(d_, ncol);
      const bool dot = !small && parts > 0 && (size_t)parts <= share;
      gpu::launch_tmu_rows(d_, ncol, w.p, w.h, true, row_words_, dot ? job.pa : nullptr, st_);
      job.na = dot ? parts : job.nb;
      if (!small && !dot) gpu::launch_cg_dot(ncol, job.nb, nv, w.h, w.p, job.pa, st_);
      if (ktime_on_) kt_end(e);
      stats_.f64_matvecs += 1;
    } else {
      const int rc = matvec64(matv, ncol, w.p, w.h, true);
      if (rc) return rc;
      if (!small) gpu::launch_cg_dot(ncol, job.na = job.nb, nv, w.h, w.p, job.pa, st_);
    }
    if (small)
      gpu::launch_cg_small(job, st_);
    else
      gpu::launch_cg_steps(&job, 1, st_);
    return kOk;
  };
  // the loop of the direct products that are kernels alone (no memset) runs on
  // the device; kernel timing, per-iteration messages, the FMM, the in-core T
  // and symmetric products of more than two columns go from the host
  bool looped = false;
  if (maxiter_ > 0 && !ktime_on_ && log_level() < kVerbHigh && !fmm_on_ && !(matv == kMatvIncore && tmat_ok_) &&
      (sym || rows)) {
    const long long products = stats_.f64_matvecs;
    CgLoop &loop = w.loop64[x == w.x ? 0 : 1];
    std::vector<char> key;
    job.tol = 0.0, job.max_passes = 0;  // those of the start are in w.cols
    key_add(key, d_), key_add(key, job), key_add(key, sym), key_add(key, small), key_add(key, fp64_kernel_);
    key_add(key, sym_scratch_);
    looped = run_loop(loop, key, [&](cudaGraphConditionalHandle hnd) {
      job.loop = hnd;
      enqueue();
    }, st);
    job.loop = 0;
    if (st) return st;
    int passes = 0;
    for (int k = 0; k < ncol; ++k) passes = std::max(passes, w.cols_h[k].passes);
    stats_.f64_matvecs = products + (looped ? passes : 0);
    if (looped) gpu::add_launch_count(loop.kernels * passes);
  }
  for (int it = 1; !looped && it <= maxiter_; ++it) {
    st = enqueue();
    if (st) return st;
    st = check(cudaStreamSynchronize(st_), "CG iteration");
    if (st) return st;
    bool any = false;
    for (int k = 0; k < ncol; ++k) {
      if (w.cols_h[k].active) any = true;
      if (log_level() >= kVerbHigh && w.cols_h[k].iters == it)
        log_msg(kVerbHigh, nullptr, "iter=%4d residual rms norm: %14.4E", it, w.cols_h[k].rms);
    }
    if (!any) break;
  }
  // without an iteration nothing has waited for the start's columns
  if (maxiter_ < 1 && (st = check(cudaStreamSynchronize(st_), "CG start"))) return st;
  std::vector<double> h(maxhist_);
  int rc = kOk;
  for (int k = 0; k < ncol; ++k) {
    const gpu::CgCol &c = w.cols_h[k];
    if (set0 >= 0 && set0 + k < 2) {
      int set = set0 + k;
      stats_.iters[set] = c.iters;
      int nh = std::min(c.iters, maxhist_);
      cudaMemcpy(h.data(), w.hist + (size_t)k * maxhist_, nh * sizeof(double), cudaMemcpyDeviceToHost);
      stats_.hist[set].assign(h.begin(), h.begin() + nh);
    }
    if (c.quick) log_msg(kVerbHigh, nullptr, "Direction vector with zero norm, exiting iterative solver.");
    if (c.converged)
      log_msg(kVerbHigh, nullptr, "Required convergence threshold reached, exiting iterative solver.");
    if (!std::isfinite(c.rms)) {
      set_last_error("non-finite residual in the iterative solver (coincident sites?)");
      rc = kErrNumeric;
    } else if (!c.converged && !c.quick && c.rms > tol_ && std::fabs(c.gama) > kEpsRp) {
      set_last_error("Iterative solver did not converged");
      rc = kErrNotConverged;
    }
  }
  return rc;
}

// ---------------------------------------------------------------------------
// FP32 product with the tuned launch shape
// ---------------------------------------------------------------------------
int System::f32_product(Workspace &w, int ncol, const F32Shape &sh, bool prepared, double *part, int max_part) {
  return gpu::launch_tmu_f32(d_, ncol, w.p32, w.h32, w.scratch32, sh.nsplit, st_, sh.g, sh.kver, sym_scratch_, prepared,
                             part, max_part);
}

// The launch shape by size and columns (forced kernels keep their own shape):
// widest column groups, kernel by the measured time of an inner iteration (all
// its steps), us (pairwise / tiled / symmetric):
//   sites       192       999      2,001      3,003      4,200      6,000        9,003
//   1 column  31/53/48  39/59/53  45/61/56   54/65/60   67/73/65   94/95/82   166/159/119
//   2         34/58/53  41/64/62  51/66/64   61/71/71   80/83/86  110/112/113 206/189/162
//   4         34/48     45/56     58/63      74/74     128/94     164/138     318/247
//   8         37/67     49/69     85/79     114/95     184/141    294/213     555/408
//   24        40/68     72/79    152/130    251/199    415/310    747/537    1549/1095
// (15,000 sites, 8 columns, the product alone: tiled 846, symmetric 1,088.)
// The tiled kernel's source splits: the finer of two candidates, as fine as the
// tiles allow, won everywhere.
int System::tune_f32(Workspace &w, int ncol, F32Shape &shape) {
  auto it = f32_tune_.find(ncol);
  if (it != f32_tune_.end() && it->second.nsplit <= w.scratch32_nsplit) {
    shape = it->second;
    return kOk;
  }
  const int n = d_.n;
  F32Shape pick{ncol >= 8 ? 8 : ncol >= 4 ? 4 : ncol >= 2 ? 2 : 1, 1, fp32_kernel_};
  if (fp32_kernel_ == 0) {
    const int rows = ncol == 1 ? 3600 : ncol < 4 ? 4500 : ncol < 8 ? 3000 : 1500;
    pick.kver = n < rows ? 1 : pick.g >= 4 ? 2 : 3;
    if (pick.kver == 3 && ensure_sym_scratch() != kOk) pick.kver = 2;
  } else if (fp32_kernel_ == 3) {
    const int st = ensure_sym_scratch();
    if (st) return st;
  }
  if (pick.kver == 3) {
    pick.g = std::min(pick.g, 2);
  } else if (pick.kver == 1) {
    pick.g = std::min(pick.g, 4);
  } else {
    pick.nsplit = std::max(1, std::min({2 * gpu::tmu32_pick_split(d_, gpu::sm_count()), w.scratch32_nsplit, (n + 127) / 128}));
  }
  f32_tune_[ncol] = pick;
  shape = pick;
  log_msg(kVerbHigh, nullptr, "FP32 T.mu for %d columns: kernel %d, %d per launch, %d source splits", ncol, pick.kver,
          pick.g, pick.nsplit);
  return kOk;
}

// the CG steps on the FP32 columns of a workspace; prepared: they also clear
// the accumulators of the symmetric product
gpu::CgJob<float> System::inner_job(Workspace &w, int ncol, bool prepared) {
  gpu::CgJob<float> job{};
  job.n = d_.n, job.ncol = ncol;
  // z = M^-1 r: the diagonal, the block-Jacobi blocks, or those with the
  // Neumann step over the near blocks
  job.mode = inner_precond_ >= 1 && blk_info_ ? (near_precond() ? 2 : 1) : 0;
  job.nb = gpu::cg_blocks(d_.n, ncol, w.partial_len);
  job.eps = 1e-300;
  job.x = w.x32, job.r = w.r32, job.p = w.p32, job.h = w.h32, job.z = w.z32;
  job.w = reinterpret_cast<float *>(w.z);  // free during the inner solve
  job.alpha = alpha32_;
  job.info = blk_info_, job.minv = blk_minv_;
  job.ri = near_ri_, job.ci = near_ci_, job.blk = near_blk_;
  job.pa = w.partial, job.pb = w.partial + w.partial_len / (2 * (size_t)ncol) * ncol;
  job.cols = w.cols, job.cols_h = w.cols_h;
  job.meet = reinterpret_cast<unsigned *>(w.cols + w.cap);
  if (prepared) {
    unsigned long long *lo = reinterpret_cast<unsigned long long *>(sym_scratch_);
    job.acc = lo, job.nacc = 2 * 3 * (size_t)ncol * d_.n, job.words = lo + 3 * 3 * (size_t)ncol * d_.n;
  }
  return job;
}

// ---------------------------------------------------------------------------
// FP32 inner PCG on w.r32 (columns normalised to unit rms); result in w.x32
// ---------------------------------------------------------------------------
int System::pcg32_ws(Workspace &w, int ncol, int max_it, double eta) {
  const int n = d_.n;
  F32Shape shape{1, 1, 2};
  int st = tune_f32(w, ncol, shape);
  if (st) return st;
  // the symmetric product of one column group: its accumulators are cleared
  // by the steps
  const bool prepared = shape.kver == 3 && (ncol == 1 || (ncol == 2 && shape.g >= 2));
  gpu::CgJob<float> job = inner_job(w, ncol, prepared);
  const int share = (int)(w.partial_len / (2 * (size_t)ncol));
  job.tol = eta;
  job.max_passes = max_it;
  job.init = gpu::kCgInitZero;
  gpu::launch_cg_steps(&job, 1, st_);
  job.init = 0;
  auto iteration = [&]() {
    job.na = f32_product(w, ncol, shape, prepared, job.pa, share);
    if (job.na == 0) gpu::launch_cg_dot(ncol, job.na = job.nb, 3 * (size_t)n, w.h32, w.p32, job.pa, st_);
    gpu::launch_cg_steps(&job, 1, st_);
  };
  int it = 0;
  if (max_it > 0 && !ktime_on_ && (prepared || shape.kver != 3)) {
    // the loop on the device (the tolerance lives in w.cols)
    job.tol = 0.0, job.max_passes = 0;
    std::vector<char> key;
    key_add(key, d_), key_add(key, job), key_add(key, shape), key_add(key, prepared);
    key_add(key, w.scratch32), key_add(key, sym_scratch_);
    const bool looped = run_loop(w.loop32, key, [&](cudaGraphConditionalHandle hnd) {
      job.loop = hnd;
      iteration();
    }, st);
    job.loop = 0;
    if (st) return st;
    if (looped) {
      for (int k = 0; k < ncol; ++k) it = std::max(it, w.cols_h[k].passes);
      gpu::add_launch_count(w.loop32.kernels * it);
      stats_.f32_matvecs += it;
      stats_.inner_iters += it;
      return kOk;
    }
  }
  for (it = 1; it <= max_it; ++it) {
    KEv ev;
    if (ktime_on_) ev = kt_begin(1, ncol);
    iteration();
    if (ktime_on_) kt_end(ev);
    stats_.f32_matvecs += 1;
    st = check(cudaStreamSynchronize(st_), "inner CG iteration");
    if (st) return st;
    bool any = false;
    for (int k = 0; k < ncol; ++k) any |= w.cols_h[k].active != 0;
    if (!any) break;
  }
  stats_.inner_iters += std::min(it, max_it);
  return kOk;
}

// ---------------------------------------------------------------------------
// Iterative refinement: FP64 residual, FP32 inner PCG, FP64 accumulation
// ---------------------------------------------------------------------------
// The refinement residual after a step may be updated, r -= T d, with the
// FP32 product of the step's correction d (rms times the inner solution)
// instead of recomputing E - T mu: the FP32 operator is within 1e-5 of T
// (relative, the tested bound), so the updated residual is within 1e-5 rms
// of the recomputed one, which must stay below a tenth of the tolerance for
// every unconverged column (a converged column's correction is zero).  The
// first step (r = E) never qualifies: its correction is the whole solution, nor
// does a wide system, whose FP32 positions are farther off.
bool System::update_allowed(const std::vector<double> &rms) const {
  if (!residual_update() || d_.wide) return false;
  for (double r : rms)
    if (r >= tol_ && !(kResidualUpdateRel * r <= 0.1 * tol_)) return false;
  return true;
}

int System::mixed_ir_ws(Workspace &w, int ncol, const double *rhs, double *x, int set0, bool have_guess) {
  const int n = d_.n;
  const size_t nv = 3 * (size_t)n;
  const int max_outer = 30;
  const int cap = w.cap;
  log_msg(kVerbLow, nullptr, "Solving linear system with mixed-precision CG (FP32 inner, FP64 refinement)");
  {
    const int pst = ensure_near();
    if (pst) return pst;
  }
  const int nb = gpu::cg_blocks(n, ncol, w.partial_len);
  if (have_guess) {
    int st0 = matvec_residual(ncol, x, w.h);
    if (st0) return st0;
  } else {
    cudaMemsetAsync(x, 0, ncol * nv * sizeof(double), st_);
  }
  gpu::launch_refine(ncol, nb, nv, rhs, have_guess ? w.h : nullptr, nullptr, nullptr, d_.pol_alpha, w.r, w.partial,
                     w.scal_h, st_);
  if (set0 >= 0)
    for (int k = 0; k < ncol && set0 + k < 2; ++k) stats_.hist[set0 + k].clear();
  std::vector<double> rms(ncol);
  int outer = 0;
  bool done = false;
  while (true) {
    int st = check(cudaStreamSynchronize(st_), "refinement residual");
    if (st) return st;
    done = true;
    for (int k = 0; k < ncol; ++k) {
      rms[k] = std::sqrt(std::max(w.scal_h[k], 0.0) / (double)nv);
      if (set0 >= 0 && set0 + k < 2) stats_.hist[set0 + k].push_back(rms[k]);
      if (!std::isfinite(rms[k])) {
        set_last_error("non-finite residual in the refinement loop (coincident sites?)");
        return kErrNumeric;
      }
      if (!(rms[k] < tol_)) done = false;
      if (log_level() >= kVerbHigh)
        log_msg(kVerbHigh, nullptr, "refinement step %3d column %d residual rms norm: %14.4E", outer, k, rms[k]);
    }
    if (done || outer >= max_outer) break;
    // normalise each unconverged column to unit preconditioned rms; converged
    // columns get a zero right-hand side (the inner CG leaves them at zero)
    double eta = 1e-5;
    for (int k = 0; k < ncol; ++k) {
      w.scal_h[cap + k] = rms[k] < tol_ ? 0.0 : 1.0 / rms[k];
      w.scal_h[2 * cap + k] = rms[k] < tol_ ? 0.0 : rms[k];
      if (rms[k] >= tol_) eta = std::max(eta, std::min(1e-2, 0.3 * tol_ / rms[k]));
    }
    cudaMemcpyAsync(w.dots + cap, w.scal_h + cap, 2 * cap * sizeof(double), cudaMemcpyHostToDevice, st_);
    gpu::launch_to_f32_cols(ncol, nv, w.r, w.dots + cap, w.r32, st_);
    // batches of at least 4 columns share one Krylov space (block CG)
    if (block_cg_ && w.t32 && ncol >= 4 && ncol <= gpu::block_cg_max_columns())
      st = bpcg32_ws(w, ncol, 200, eta);
    else
      st = pcg32_ws(w, ncol, 200, eta);
    if (st) return st;
    gpu::launch_ir_accumulate(ncol, n, x, w.x32, w.dots + 2 * cap, st_);
    if (update_allowed(rms)) {
      // r -= rms T32 x32: the FP32 product of this step's correction
      F32Shape shape{1, 1, 2};
      st = tune_f32(w, ncol, shape);
      if (st) return st;
      cudaMemcpyAsync(w.p32, w.x32, ncol * nv * sizeof(float), cudaMemcpyDeviceToDevice, st_);
      f32_product(w, ncol, shape);
      stats_.f32_matvecs += 1;
      stats_.updates += 1;
      gpu::launch_refine(ncol, nb, nv, rhs, nullptr, w.h32, w.dots + 2 * cap, d_.pol_alpha, w.r, w.partial, w.scal_h,
                         st_);
    } else {
      st = matvec_residual(ncol, x, w.h);
      if (st) return st;
      gpu::launch_refine(ncol, nb, nv, rhs, w.h, nullptr, nullptr, d_.pol_alpha, w.r, w.partial, w.scal_h, st_);
    }
    ++outer;
  }
  stats_.outer += outer;
  if (set0 >= 0)
    for (int k = 0; k < ncol && set0 + k < 2; ++k) stats_.iters[set0 + k] = outer;
  if (!done) {
    set_last_error("Iterative solver did not converged");
    return kErrNotConverged;
  }
  return kOk;
}

// ---------------------------------------------------------------------------
// Batched fields
// ---------------------------------------------------------------------------
int System::solve_batch(int nf, const double *fields, double *out, double *energies) {
  if (nf < 1) {
    set_last_error("batch: the number of fields must be positive");
    return kErrBadArg;
  }
  const int n = d_.n;
  const size_t nv = 3 * (size_t)n;
  if (n == 0) {
    if (energies)
      for (int f = 0; f < nf; ++f) energies[f] = 0.0;
    return kOk;
  }
  int st = ensure_m2d();
  if (st) return st;
  const int nipd = m_.n_ipd;
  int nsets = nipd;
  if (nipd == 2) {
    // identical D and P right-hand sides: one set of columns (see polarization)
    int differ = 1;
    cudaMemsetAsync(flag_, 0, sizeof(int), st_);
    gpu::launch_any_diff(nv, e_m2d_, e_m2d_ + nv, flag_, st_);
    cudaMemcpyAsync(&differ, flag_, sizeof(int), cudaMemcpyDeviceToHost, st_);
    st = check(cudaStreamSynchronize(st_), "batch D/P comparison");
    if (st) return st;
    if (!differ) nsets = 1;
  }
  const int ncol = nf * nsets;
  st = ensure_batch_ws(ncol, nf);
  if (st) return st;
  Workspace &w = wsb_;
  stats_ = SolveStats();
  cudaEventRecord(ev0_, st_);
  gpu::launch_batch_rhs(n, nf, nsets, e_m2d_, fields, w.rhs, st_);
  cudaMemsetAsync(w.x, 0, ncol * nv * sizeof(double), st_);
  if (precision_ != kPrecFP64) {
    st = mixed_ir_ws(w, ncol, w.rhs, w.x, -1, false);
  } else {
    int matv = def_matv_ == kMatvIncore ? kMatvIncore : kMatvDirect;
    if (matv == kMatvIncore && ensure_tmat() != kOk) matv = kMatvDirect;
    st = cg64_ws(w, matv, nf, w.rhs, w.x, -1);
    if (!st && nsets == 2) {
      // P seeded with D (mod_polarization.F90:237-243)
      cudaMemcpyAsync(w.x + nf * nv, w.x, nf * nv * sizeof(double), cudaMemcpyDeviceToDevice, st_);
      st = cg64_ws(w, matv, nf, w.rhs + nf * nv, w.x + nf * nv, -1);
    }
  }
  if (st) return st;
  gpu::launch_batch_scatter(n, nf, nipd, nsets, w.x, out, st_);
  if (energies) {
    // -1/2 ipd(D) . E_M2D(P) per field (AMOEBA), -1/2 ipd . E_M2D otherwise
    const double *ef = m_.amoeba ? e_m2d_ + nv : e_m2d_;
    gpu::launch_dots_bcast(nf, nv, w.x, ef, w.partial, st_);
    gpu::launch_reduce_partials(nf, w.partial, w.dots, st_);
    cudaMemcpyAsync(w.scal_h, w.dots, nf * sizeof(double), cudaMemcpyDeviceToHost, st_);
  }
  cudaEventRecord(ev1_, st_);
  st = check(cudaStreamSynchronize(st_), "batch solve");
  if (st) return st;
  if (energies)
    for (int f = 0; f < nf; ++f) energies[f] = -0.5 * w.scal_h[f];
  cudaEventElapsedTime(&last_ms_, ev0_, ev1_);
  return kOk;
}

int System::solve_batch_host(int nf, const double *fields_host, double *out_host, double *energies) {
  if (nf < 1) {
    set_last_error("batch: the number of fields must be positive");
    return kErrBadArg;
  }
  const size_t nv = 3 * (size_t)d_.n;
  const int nsets_max = m_.n_ipd;
  int st = ensure_batch_ws(nf * nsets_max, nf);
  if (st) return st;
  cudaMemcpyAsync(wsb_.fields, fields_host, nf * nv * sizeof(double), cudaMemcpyHostToDevice, st_);
  st = solve_batch(nf, wsb_.fields, wsb_.out, energies);
  if (st) return st;
  cudaMemcpyAsync(out_host, wsb_.out, (size_t)nf * m_.n_ipd * nv * sizeof(double), cudaMemcpyDeviceToHost, st_);
  return check(cudaStreamSynchronize(st_), "batch copy-out");
}

}  // namespace ommp
