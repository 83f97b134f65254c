#include "davidson.hpp"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

namespace c2g {

namespace {
// Offsets in the small device scratch sm_.
constexpr int kMxM = 0;         // 32 x 32 Rayleigh-Ritz matrix (ld 32)
constexpr int kEvecs = 1024;    // its eigenvectors (ld 32)
constexpr int kEvals = 2048;    // eigenvalues, ascending
constexpr int kDots = 2112;     // up to 32 dot products
constexpr int kDotsB = 2144;    // those of the second pass of an orthogonalisation
constexpr int kDots2 = 2176;    // w.t, w.u
constexpr int kOverlap = 2184;  // keep x keep overlap
constexpr int kLowdin = 2200;   // keep x keep Loewdin matrix
constexpr int kSumSq = 2216;    // one sum of squares
constexpr int kLowest = 2217;   // lowest diagonal entry
constexpr int kSmall = 2304;
constexpr int kLd = 32;
// Mixed-precision refinement: cycles, FP32 expansions per cycle, and the residual
// reduction (relative to the cycle's exact first residual) that ends a cycle.
constexpr int kRefineCycles = 8;
constexpr int kRefineExpand = 12;
constexpr double kRefineRel = 1e-3;
// A stall of the reduced-precision phase (no 0.7x residual reduction in 6 iterations)
// with a residual of at most kStallCeiling |theta| is its arithmetic's floor: the
// refinement cycles take over. A stall above it marks a hard step: a residual plateau from
// a poor guess (the first sweep from a random start), on which the FP64 solver may still
// turn to a lower eigenpair after many more products while the reduced-precision one
// settles on an excited state. Such a step, and one that needs more than kLoMaxMatvec
// reduced-precision products, is solved by the FP64 solver from the guess. So is one whose
// reduced-precision Ritz value ends above a diagonal entry, where no lowest eigenvalue is:
// the eigenpair found from such a guess hangs on the arithmetic, and the FP64 mode's is meant.
constexpr double kStallCeiling = 1e-3;
constexpr int kLoMaxMatvec = 1000;
}  // namespace

DeviceDavidson::DeviceDavidson(Runtime& rt, int64_t n, int max_vec, int keep, double rtol, double cutoff)
    : rt_(rt), n_(n), max_vec_(max_vec), keep_(keep), rtol_(rtol), cutoff_(cutoff) {
  if (max_vec > kLd || keep < 1 || keep > 4 || keep >= max_vec)
    throw std::invalid_argument("Davidson: unsupported number of vectors");
  V_ = rt_.alloc(n_ * max_vec_);
  HV_ = rt_.alloc(n_ * max_vec_);
  W_ = rt_.alloc(n_ * (2 + keep_));
  sm_ = rt_.alloc(kSmall);
  rt_.zero(sm_, kSmall);
  host_ = rt_.pinned_scalars();
}

DeviceDavidson::~DeviceDavidson() {
  rt_.release_quiet(V_);
  rt_.release_quiet(HV_);
  rt_.release_quiet(W_);
  rt_.release_quiet(sm_);
}

void DeviceDavidson::multi_dot(const double* A, int ncol, const double* x, double* out) {
  C2G_CUDA(launch_multi_dot(A, n_, ncol, x, n_, rt_.partial(), out, rt_.stream()));
  count_launches(1);
}

double DeviceDavidson::norm2(const double* x) {
  multi_dot(x, 1, x, sm_ + kSumSq);
  return read_sumsq(nullptr);
}

double DeviceDavidson::read_sumsq(double* theta) {
  C2G_CUDA(cudaMemcpyAsync(host_, sm_ + kSumSq, sizeof(double), cudaMemcpyDeviceToHost, rt_.stream()));
  if (theta) C2G_CUDA(cudaMemcpyAsync(host_ + 1, sm_ + kEvals, sizeof(double), cudaMemcpyDeviceToHost, rt_.stream()));
  rt_.sync();
  if (theta) *theta = host_[1];
  return host_[0];
}

// The Ritz value is above the lowest diag entry of guess's support by more than its residual
bool DeviceDavidson::above_diag(const double* diag, const double* guess, double rnorm) {
  if (partial_diag_) return false;
  cudaStream_t s = rt_.stream();
  C2G_CUDA(launch_lowest_entry(diag, guess, n_, rt_.partial(), sm_ + kLowest, s));
  count_launches(1);
  C2G_CUDA(cudaMemcpyAsync(host_, sm_ + kLowest, sizeof(double), cudaMemcpyDeviceToHost, s));
  C2G_CUDA(cudaMemcpyAsync(host_ + 1, sm_ + kEvals, sizeof(double), cudaMemcpyDeviceToHost, s));
  rt_.sync();
  return host_[1] > host_[0] + rnorm;
}

// CheMPS2/Davidson.cpp:216-236 (AddNewVec): t <- t - V V^T t (twice), V[nv] <- t / |t|.
void DeviceDavidson::add_new_vec(double* t, int nv, bool projected) {
  cudaStream_t s = rt_.stream();
  double* partial = rt_.partial();
  if (nv > 0) {
    if (!projected) multi_dot(V_, nv, t, sm_ + kDots);
    C2G_CUDA(launch_subtract(t, V_, n_, sm_ + kDots, nv, n_, false, partial, sm_ + kDotsB, s));
    C2G_CUDA(launch_subtract(t, V_, n_, sm_ + kDotsB, nv, n_, true, partial, sm_ + kSumSq, s));
    count_launches(2);
  } else {
    multi_dot(t, 1, t, sm_ + kSumSq);
  }
  C2G_CUDA(launch_normalize(V(nv), t, sm_ + kSumSq, n_, s));
  count_launches(1);
}

// DiagonalizeSmallMatrixAndCalcResidual (CheMPS2/Davidson.cpp:238-289) with the newest
// product HV(nv); returns the residual norm (and, with theta, the lowest Ritz value).
double DeviceDavidson::ritz(int& nv, double* theta) {
  cudaStream_t s = rt_.stream();
  double* partial = rt_.partial();
  C2G_CUDA(launch_project_row(HV_, n_, nv + 1, V(nv), n_, partial, sm_ + kMxM, kLd, nv, s));
  nv++;
  // warm start when the previous solve was of this matrix's leading block
  C2G_CUDA(launch_small_eig(sm_ + kMxM, nv, kLd, sm_ + kEvals, sm_ + kEvecs, s, eig_n_ == nv - 1));
  eig_n_ = nv;
  C2G_CUDA(launch_ritz(W(0), W(1), HV_, V_, n_, sm_ + kEvecs, nv, sm_ + kEvals, n_, partial, sm_ + kSumSq, s));
  count_launches(3);
  return std::sqrt(read_sumsq(theta));
}

// CalculateNewVec (CheMPS2/Davidson.cpp:291-317) into W(0), and its products with V[0..nproj)
void DeviceDavidson::new_vec(const double* diag, int nproj) {
  cudaStream_t s = rt_.stream();
  double* partial = rt_.partial();
  C2G_CUDA(launch_precond_dots(W(0), W(1), diag, sm_ + kEvals, cutoff_, n_, partial, sm_ + kDots2, s));
  C2G_CUDA(launch_precond(W(0), W(1), diag, sm_ + kEvals, sm_ + kDots2, cutoff_, V_, n_, nproj, n_, partial,
                          sm_ + kDots, s));
  count_launches(2);
}

bool DeviceDavidson::run(const double* diag, const MatVec& matvec, Precision prec, double tol, bool stop_on_stall,
                         DavidsonStats& st) {
  cudaStream_t s = rt_.stream();
  double* t = W(0);
  double* u = W(1);
  auto mv = [&](const double* x, double* y) {
    matvec(x, y, prec);
    st.n_matvec++;
    if (prec != Precision::kFP64) st.n_matvec_fp32++;
  };
  int nv = 0;
  eig_n_ = -1;
  add_new_vec(t, nv);
  mv(V(nv), HV(nv));
  double best = 1e300;
  int since_best = 0;
  const int matvec0 = st.n_matvec;
  for (;;) {
    double theta = 0.0;
    const double rnorm = ritz(nv, stop_on_stall ? &theta : nullptr);
    st.n_iter++;
    st.rnorm = rnorm;
    if (!(rnorm > tol)) break;
    if (stop_on_stall) {  // reduced-precision phase: stop when the residual no longer improves
      if (rnorm < 0.7 * best) {
        best = rnorm;
        since_best = 0;
      } else if (++since_best >= 6) {
        st.lo_stalled = true;
        if (rnorm > kStallCeiling * std::fabs(theta)) return false;
        break;
      }
      if (st.n_matvec - matvec0 >= kLoMaxMatvec) return false;
    }
    // with a deflation next, the basis it is to be orthogonal to does not exist yet
    const bool projected = nv < max_vec_;
    new_vec(diag, projected ? nv : 0);
    if (nv == max_vec_) {
      // Deflation (CheMPS2/Davidson.cpp:319-384): keep the lowest keep_ Ritz vectors
      C2G_CUDA(cudaMemcpyAsync(W(2), u, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
      for (int c = 1; c < keep_; c++) {
        C2G_CUDA(launch_combine(W(2 + c), 0.0, V_, n_, sm_ + kEvecs + kLd * c, nv, n_, s));
        count_launches(1);
      }
      for (int c = 0; c < keep_; c++) multi_dot(W(2), keep_, W(2 + c), sm_ + kOverlap + keep_ * c);
      C2G_CUDA(launch_lowdin(sm_ + kOverlap, keep_, sm_ + kLowdin, s));
      count_launches(1);
      for (int c = 0; c < keep_; c++) {
        C2G_CUDA(launch_combine(V(c), 0.0, W(2), n_, sm_ + kLowdin + keep_ * c, keep_, n_, s));
        count_launches(1);
      }
      for (int c = 0; c < keep_; c++) mv(V(c), HV(c));
      // MxMafterDeflation (CheMPS2/Davidson.cpp:510-536)
      eig_n_ = -1;  // the projected matrix is rebuilt
      for (int j = 0; j < keep_; j++) {
        C2G_CUDA(launch_project_row(V_, n_, j + 1, HV(j), n_, rt_.partial(), sm_ + kMxM, kLd, j, s));
        count_launches(1);
      }
      nv = keep_;
    }
    add_new_vec(t, nv, projected);
    mv(V(nv), HV(nv));
  }
  return true;
}

bool DeviceDavidson::refine_cycle(const double* diag, const MatVec& matvec, double tol, int max_expand, double rel,
                                  DavidsonStats& st, double* r_exact) {
  int nv = 0;
  eig_n_ = -1;
  add_new_vec(W(0), nv);
  matvec(V(0), HV(0), Precision::kFP64);
  st.n_matvec++;
  double r0 = 0.0;
  for (int it = 0;; it++) {
    const double rnorm = ritz(nv, nullptr);
    st.n_iter++;
    st.rnorm = rnorm;
    if (it == 0) {
      // V = {u} with its FP64 product: the exact residual
      r0 = rnorm;
      *r_exact = rnorm;
      if (!(rnorm > tol)) return true;
    } else if (rnorm <= rel * r0 || it >= max_expand || nv >= max_vec_) {
      return false;
    }
    new_vec(diag, nv);
    add_new_vec(W(0), nv, true);
    matvec(V(nv), HV(nv), lo_);
    st.n_matvec++;
    st.n_matvec_fp32++;
  }
}

DavidsonStats DeviceDavidson::solve(double* guess, const double* diag, const MatVec& matvec, bool mixed,
                                    double lo_tol, Precision lo) {
  lo_ = lo;
  cudaStream_t s = rt_.stream();
  DavidsonStats st;
  double* t = W(0);
  double* u = W(1);
  C2G_CUDA(cudaMemcpyAsync(t, guess, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
  // SafetyCheckGuess (CheMPS2/Davidson.cpp:204-214)
  if (norm2(t) == 0.0) {
    std::vector<double> r(n_);
    HostRand libc;
    HostRand& g = rand_ ? *rand_ : libc;
    for (int64_t i = 0; i < n_; i++) r[i] = g.unit();
    C2G_CUDA(cudaMemcpyAsync(t, r.data(), sizeof(double) * n_, cudaMemcpyHostToDevice, s));
    // the start vector also stays in guess (overwritten by the result at the end), for a
    // restart of the mixed solve
    C2G_CUDA(cudaMemcpyAsync(guess, t, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
    rt_.sync();
  }
  bool done = false;
  if (mixed) {
    const bool lo_done = run(diag, matvec, lo_, std::max(lo_tol, rtol_), true, st);
    st.n_lo = st.n_matvec;
    st.lo_rnorm = st.rnorm;
    if (!lo_done || above_diag(diag, guess, st.rnorm)) {  // a hard step: the FP64 solver from the guess
      st.fp64_fallback = true;
      C2G_CUDA(cudaMemcpyAsync(t, guess, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
      run(diag, matvec, Precision::kFP64, rtol_, false, st);
      done = true;
    }
    // refinement cycles from the FP32 Ritz vector; a cycle that cannot improve (for
    // example an FP32 floor above the target) leaves it to the FP64 Davidson below
    double last = 1e300;
    for (int cycle = 0; cycle < kRefineCycles && !done; cycle++) {
      C2G_CUDA(cudaMemcpyAsync(t, u, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
      double r = 0.0;
      st.n_cycles++;
      done = refine_cycle(diag, matvec, rtol_, kRefineExpand, kRefineRel, st, &r);
      if (cycle == 0) st.r_exact0 = r;
      if (!done && r > 0.5 * last) break;  // the exact residual no longer drops
      last = r;
    }
    if (!done) C2G_CUDA(cudaMemcpyAsync(t, u, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
  }
  if (!done) run(diag, matvec, Precision::kFP64, rtol_, false, st);
  C2G_CUDA(cudaMemcpyAsync(guess, u, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
  C2G_CUDA(cudaMemcpyAsync(host_, sm_ + kEvals, sizeof(double), cudaMemcpyDeviceToHost, s));
  rt_.sync();
  st.energy = host_[0];
  return st;
}

}  // namespace c2g
