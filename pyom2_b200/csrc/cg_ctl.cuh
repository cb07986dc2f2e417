// Control flow of congrad_streamfunction (solve_streamfct.f90:153-327) and
// congrad_surf_press (solve_pressure.f90:137-249) on the reduced scalars, and
// the tagged words their reductions and exchanges travel in: shared by the
// resident kernels (cg_res.cu) and the cluster kernel (cg_clu.cu).
#pragma once
#include <math.h>

#include "cg_res.cuh"

namespace pyomgpu {
namespace {

__device__ __forceinline__ unsigned long long tag_lo(unsigned tag, double v) {
  return ((unsigned long long)tag << 32) | (unsigned)__double2loint(v);
}
__device__ __forceinline__ unsigned long long tag_hi(unsigned tag, double v) {
  return ((unsigned long long)tag << 32) | (unsigned)__double2hiint(v);
}
__device__ __forceinline__ bool tag_ok(unsigned long long w, unsigned tag) { return (unsigned)(w >> 32) == tag; }
__device__ __forceinline__ double untag(unsigned long long lo, unsigned long long hi) {
  return __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
}

// The operator and vectors of a solve in the field type T (FP64, or the FP32
// copies of the mixed-precision correction solve).
template <typename T>
__device__ __forceinline__ OpDev<T> res_op(const CGResParams& P) {
  if constexpr (sizeof(T) == 8) return P.op; else return P.op32;
}
template <typename T>
__device__ __forceinline__ const T* res_forc(const CGResParams& P) {
  if constexpr (sizeof(T) == 8) return P.forc; else return P.forc32;
}
template <typename T>
__device__ __forceinline__ T* res_solv(const CGResParams& P) {
  if constexpr (sizeof(T) == 8) return P.sol; else return P.sol32;
}
template <typename T>
__device__ __forceinline__ T* res_resv(const CGResParams& P) {
  if constexpr (sizeof(T) == 8) return P.res; else return P.res32;
}

// ------------------------------------------------------------ control flow
// Scalars of the solve (the reference's congrad_streamfunction variables).  In
// the resident kernels one copy in shared memory, advanced by one thread; in
// the cluster kernel every thread keeps a copy and advances it, so there the
// reduced values must have the same bits in every thread of the cluster.
struct ResCtl {
  double beta, bb, rtol2bb, betam1, betamin, step1, est, bq, alpha;
  int n, status, act, stop_after;
};
constexpr int kRun = 0, kDoneOk = 1, kDoneErr = 2, kNeedMaxp = 3;
constexpr int kStepInit = 0, kStepA = 1, kStepB = 2, kStepInitD = 3, kStepIter = 4, kStepMaxp = 5;
constexpr int kStepInitP = 6, kStepAP = 7, kStepBP = 8;  // congrad_surf_press

__device__ __forceinline__ void ctl_stop(ResCtl& C, int act, int status) {
  C.act = act;
  C.status = status;
}

// Start of iteration C.n: max_it, NaN and divergence tests, beta/betam1.
__device__ __forceinline__ void ctl_begin(ResCtl& C, const CGResParams& P) {
  if (C.n > P.max_it) return ctl_stop(C, kDoneErr, PYOMGPU_MAXITER);  // solve_streamfct.f90:303-304
  if (C.beta != C.beta) {  // early NaN stop (the reference runs on and halts at the end)
    C.est = C.beta;
    return ctl_stop(C, kDoneErr, PYOMGPU_NAN);
  }
  if (C.n == 1) {  // :232-240
    C.betamin = fabs(C.beta);
  } else if (C.n > 2) {
    C.betamin = fmin(C.betamin, fabs(C.beta));
    if (fabs(C.beta) > 100.0 * C.betamin) return ctl_stop(C, kDoneErr, PYOMGPU_DIVERGED);
  }
  C.bq = C.beta / C.betam1;  // :244
}

// v = (Z res, res), sum f^2 and sum res^2 over the unknowns, max|Z res|
__device__ __forceinline__ void ctl_init(ResCtl& C, const CGResParams& P, const double* v) {
  C.beta = v[0];
  C.bb = v[1] > 0.0 ? v[1] : v[2];  // the rtol stop relative to ||res_0|| for a zero forcing
  C.rtol2bb = P.rtol * P.rtol * C.bb;
  C.betam1 = 1.0;
  C.betamin = C.step1 = C.est = C.bq = C.alpha = 0.0;
  C.n = 0;
  C.status = PYOMGPU_OK;
  C.act = kRun;
  C.stop_after = 0;
  if (100.0 * v[3] < P.eps) {  // solve_streamfct.f90:210-213
    C.est = 100.0 * v[3];
    return ctl_stop(C, kDoneOk, PYOMGPU_OK);
  }
  C.n = 1;
  ctl_begin(C, P);
}

// v = (s, As), max|s|.  The quotient is formed first, beside the tests: it is
// what the sweep waits for (a division is ~115 cycles, and every branch before
// it added its own ~30).
__device__ __forceinline__ void ctl_after_a(ResCtl& C, const CGResParams& P, const double* v) {
  const double F_1EM10 = (double)1.e-10f;  // solve_streamfct.f90:262, a default-real literal
  const double sAs = v[0], smax = v[1];
  const double alpha = C.beta / sAs;
  const double step = fabs(alpha) * smax;  // :283-297, decided now, applied after the update
  const bool breakdown = fabs(sAs) < fabs(C.beta) * F_1EM10;  // :262-266
  C.stop_after = 0;
  if (breakdown | (step < P.eps) | (C.n == 1)) {
    if (breakdown) {
      C.est = 100.0 * smax;
      return ctl_stop(C, kDoneOk, PYOMGPU_OK);
    }
    if (C.n == 1) {
      C.step1 = step;
      C.est = step;
      C.stop_after = step < P.eps;
    } else {
      const double rate = exp(log(step / C.step1) / (double)(C.n - 1));
      C.est = step * rate / (1.0 - rate);
      C.stop_after = C.est < P.eps;
    }
  }
  C.alpha = alpha;
}

// v = (Z res, res) and sum res^2 over the unknowns of the updated residual
__device__ __forceinline__ void ctl_after_b(ResCtl& C, const CGResParams& P, const double* v) {
  const double beta_next = v[0], rr_next = v[1];
  const double bq = beta_next / C.beta;  // solve_streamfct.f90:244, of the next iteration
  const double b = fabs(beta_next), low = fmin(C.betamin, b);
  const bool small = P.rtol > 0.0 && (C.bb > 0.0 ? rr_next <= C.rtol2bb : rr_next == 0.0);
  if (small | (C.n < 2) | (C.n >= P.max_it) | !(b <= 100.0 * low)) {  // the last also for a NaN
    if (small) {
      C.est = sqrt(rr_next);
      return ctl_stop(C, kDoneOk, PYOMGPU_OK);
    }
    C.betam1 = C.beta;
    C.beta = beta_next;
    C.n += 1;
    return ctl_begin(C, P);
  }
  C.betam1 = C.beta;
  C.beta = beta_next;
  C.betamin = low;
  C.bq = bq;
  C.n += 1;
}

// congrad_surf_press (solve_pressure.f90:163-232), as cg_ref_kernel<true> runs
// it: products weighted by maskT, no preconditioner, and a convergence test of
// iteration n that needs max|p| of the direction formed after it, so it is
// decided at the next sweep A.
// v = (res, res), (forc, forc) over maskT
__device__ __forceinline__ void ctl_init_sp(ResCtl& C, const CGResParams& P, const double* v) {
  C.beta = v[0];
  C.bb = v[1];
  C.rtol2bb = P.rtol * P.rtol * C.bb;
  C.betam1 = 1.0;
  C.betamin = C.step1 = C.est = C.bq = C.alpha = 0.0;
  C.n = 0;
  C.status = PYOMGPU_OK;
  C.act = kRun;
  C.stop_after = 0;
  if (C.beta == 0.0) return ctl_stop(C, kDoneOk, PYOMGPU_OK);  // solve_pressure.f90:174-177
  C.n = 1;
  if (P.max_it < 1) return ctl_stop(C, kDoneErr, PYOMGPU_MAXITER);
}

// v = (p, Ap), max|p| of the direction of iteration C.n; C.alpha and C.beta are still iteration n-1's step and
// its (res, res)
__device__ __forceinline__ void ctl_after_a_sp(ResCtl& C, const CGResParams& P, const double* v) {
  const double sAs = v[0], smax = v[1];
  const double alpha = C.beta / sAs;  // beside the tests, as in ctl_after_a
  const double step = fabs(C.alpha) * smax;
  const int m = C.n - 1;
  if ((m <= 1) | (step < P.eps) | (C.est != C.est) | (P.rtol > 0.0) | (m >= P.max_it) | (sAs == 0.0)) {
    if (m >= 1) {  // convergence test of iteration n-1 (solve_pressure.f90:209-226)
      bool stop = false;
      if (m == 1) {
        C.step1 = step;
        C.est = step;
        stop = step < P.eps;
      } else if (step < P.eps) {
        const double rate = exp(log(step / C.step1) / (double)(m - 1));
        C.est = step * rate / (1.0 - rate);
        stop = C.est < P.eps;
      }
      if (stop) {
        C.n = m;
        return ctl_stop(C, kDoneOk, PYOMGPU_OK);
      }
      if (C.est != C.est) {
        C.n = m;
        return ctl_stop(C, kDoneErr, PYOMGPU_NAN);
      }
      if (P.rtol > 0.0 && (C.bb > 0.0 ? C.beta <= C.rtol2bb : C.beta == 0.0)) {
        C.est = sqrt(C.beta);
        C.n = m;
        return ctl_stop(C, kDoneOk, PYOMGPU_OK);
      }
      if (m >= P.max_it) {  // solve_pressure.f90:228-229
        C.n = P.max_it + 1;
        return ctl_stop(C, kDoneErr, PYOMGPU_MAXITER);
      }
    }
    if (sAs == 0.0) return ctl_stop(C, kDoneOk, PYOMGPU_OK);  // :185
  }
  C.alpha = alpha;
}

// v = (res, res) over maskT of the updated residual
__device__ __forceinline__ void ctl_after_b_sp(ResCtl& C, const double* v) {
  const double rsnew = v[0];
  C.bq = rsnew / C.beta;  // p = res + rsnew/rsold*p (solve_pressure.f90:190)
  C.beta = rsnew;
  if (C.n == 1) {  // :197-205
    C.betamin = fabs(rsnew);
  } else if (C.n > 2) {
    C.betamin = fmin(C.betamin, fabs(rsnew));
    if (fabs(rsnew) > 100.0 * C.betamin) return ctl_stop(C, kDoneErr, PYOMGPU_DIVERGED);
  }
  C.n += 1;
}

}  // namespace
}  // namespace pyomgpu
