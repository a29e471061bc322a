// The scalar rules of the CG kernels: when a solve ends, and which sums of the next
// residual are formed ahead of it.  Host code without CUDA types (the device takes
// the same functions), so that they can be tested on the CPU: a kernel that runs a
// whole solve in one launch must not depend on the host to stop it.
#pragma once

#include <cmath>

#include "hoefem.h"

#ifdef __CUDACC__
#define HOEFEM_HD __host__ __device__
#else
#define HOEFEM_HD
#endif

namespace hoefem {

// Chunks of `chunk` iterations a solve may take.  Without an iteration limit
// (max_iter < 0) CG is still bounded: 10 n iterations.
inline long long cg_max_chunks(long long max_iter, long long n, long long chunk) {
  const long long cap = max_iter >= 0 ? max_iter : 10 * n;
  return cap / chunk + (cap % chunk != 0) + 2;
}

// The iteration limit of the device state: the caller's, or, without one, that
// of cg_max_chunks.  Never negative.
inline long long cg_iteration_limit(long long max_iter, long long n, long long chunk) {
  return max_iter >= 0 ? max_iter : cg_max_chunks(max_iter, n, chunk) * chunk;
}

// Chunks that a launch of `iterations` iterations stands for (at least one, so
// that a loop over launches ends).
inline long long cg_chunks_of(long long iterations, long long chunk) {
  return iterations > 0 ? iterations / chunk + (iterations % chunk != 0) : 1;
}

// Whether an iteration takes its step alpha = zTr / pAp; the solve is over (status
// set) if not.  With a NaN among the two, every entry of x and r is NaN after the
// step, so no later iteration can change the outcome: this one counts as the last
// that the limit allows.  (One test while all is well.)
HOEFEM_HD inline bool cg_step_begin(double pAp, double zTr, long long limit, long long& iters, int& status) {
  if (pAp > 0.0 && zTr > 0.0) return true;
  if (pAp <= 0.0 || zTr <= 0.0) {
    status = pAp <= 0.0 ? HOEFEM_CG_INDEFINITE_OPERATOR : HOEFEM_CG_INDEFINITE_PRECONDITIONER;
    return false;
  }
  iters = limit - 1;
  return true;
}

// The end of an iteration with the squared residual `rr`: counts it, and whether the
// solve is over (status set).
HOEFEM_HD inline bool cg_iteration_end(double rr, double tol, double bnorm, long long limit, long long& iters,
                                       int& status) {
  iters += 1;
  if (sqrt(rr) <= tol * bnorm) {
    status = HOEFEM_OK;
    return true;
  }
  if (iters < limit) return false;
  status = HOEFEM_CG_MAX_ITERATIONS;
  return true;
}

// r'.r' of r' = r - alpha A p from r.r, r.Ap and Ap.Ap (or z'.r' from the same sums
// with the diagonal); false where they cancel.  The three terms are at most of the
// size of 4 r.r there, so the relative error is about 4 r.r / r'.r' roundings: a
// drop of up to 10 costs one digit (1e-14).  A lower bar would cost as many digits
// as it allows the sum to drop.
HOEFEM_HD inline bool cg_next_sum(double alpha, double rr, double rap, double apap, double& next) {
  next = rr - 2.0 * alpha * rap + alpha * alpha * apap;
  return next > 0.1 * rr;
}

}  // namespace hoefem
