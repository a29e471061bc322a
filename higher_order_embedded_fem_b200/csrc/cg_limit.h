// When a CG solve ends.  Host code without CUDA types (the device takes the
// same functions), so that the ends can be tested on the CPU: a kernel that runs
// a whole solve in one launch must not depend on the host to stop it.
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

// The end of an iteration with step `alpha` and squared residual `rr` after it:
// counts it and decides whether the solve is over (status set if so).  With
// alpha a NaN every entry of x and r is NaN from here on, so no later iteration
// can change the outcome: the solve ends as it would at its limit.
HOEFEM_HD inline bool cg_iteration_end(double alpha, double rr, double tol, double bnorm, long long limit,
                                       long long& iters, int& status) {
  iters += 1;
  if (sqrt(rr) <= tol * bnorm) {
    status = HOEFEM_OK;
    return true;
  }
  if (alpha != alpha) iters = limit;
  if (iters < limit) return false;
  status = HOEFEM_CG_MAX_ITERATIONS;
  return true;
}

}  // namespace hoefem
