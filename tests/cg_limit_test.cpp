// Checks csrc/cg_limit.h: that every solve ends, whatever its numbers, in a model
// of a kernel that iterates until cg_iteration_end and of the host loop around it.
#include "cg_limit.h"

#include <cstdio>
#include <initializer_list>
#include <limits>

using namespace hoefem;

static int fail(const char* what) {
  std::printf("%s\n", what);
  return 1;
}

// One launch: iterations with the given p.Ap, z.r and squared residual until the end;
// false if it has not ended after `most` of them.
static bool launch(double pAp, double zTr, double rr, double tol, long long limit, long long& iters, int& status,
                   long long most) {
  for (long long k = 0; k < most; ++k) {
    if (!cg_step_begin(pAp, zTr, limit, iters, status)) return true;
    if (cg_iteration_end(rr, tol, 1.0, limit, iters, status)) return true;
  }
  return false;
}

int main() {
  const double nan = std::numeric_limits<double>::quiet_NaN(), inf = std::numeric_limits<double>::infinity();
  const long long ns[] = {1, 3, 81, 4095, 132888, 2147483646LL};
  for (long long n : ns)
    for (long long chunk : {1LL, 8LL}) {
      // an explicit limit is kept as it is, 0 and large numbers included
      for (long long m : {0LL, 1LL, 7LL, 8LL, 500LL, std::numeric_limits<long long>::max() / 2}) {
        if (cg_iteration_limit(m, n, chunk) != m) return fail("explicit limit");
        const long long c = cg_max_chunks(m, n, chunk);
        if (c < m / chunk || c > m / chunk + 3) return fail("chunks of a limit");
      }
      // without one: at least 10 n iterations, at most three chunks more
      for (long long m : {-1LL, -2LL, std::numeric_limits<long long>::min()}) {
        const long long l = cg_iteration_limit(m, n, chunk);
        if (l < 10 * n || l > 10 * n + 3 * chunk || l != chunk * cg_max_chunks(m, n, chunk)) return fail("default limit");
      }
    }
  // a NaN anywhere ends a launch at once, with the outcome of the limit
  for (long long m : {-1LL, 20LL}) {
    const long long limit = cg_iteration_limit(m, 300, 8);
    long long iters = 0;
    int status = HOEFEM_OK;
    for (double pAp : {nan, 0.5})
      for (double zTr : {nan, 0.5}) {
        if (pAp == zTr) continue;
        iters = 0;
        status = HOEFEM_OK;
        if (!launch(pAp, zTr, nan, 1e-10, limit, iters, status, 1) || status != HOEFEM_CG_MAX_ITERATIONS || iters != limit)
          return fail("NaN step");
      }
    // an indefinite operator or preconditioner ends it before the step
    for (double bad : {0.0, -1.0, -inf}) {
      iters = 3;
      if (!launch(bad, nan, 1.0, 1e-10, limit, iters, status, 1) || status != HOEFEM_CG_INDEFINITE_OPERATOR || iters != 3)
        return fail("operator");
      if (!launch(nan, bad, 1.0, 1e-10, limit, iters, status, 1) || status != HOEFEM_CG_INDEFINITE_PRECONDITIONER ||
          iters != 3)
        return fail("preconditioner");
    }
    // a residual that never falls (and one that only is a NaN): the limit itself
    for (double rr : {1.0, inf, nan}) {
      iters = 0;
      status = HOEFEM_OK;
      if (!launch(0.5, 0.5, rr, 1e-10, limit, iters, status, limit) || status != HOEFEM_CG_MAX_ITERATIONS || iters != limit)
        return fail("limit");
    }
    iters = limit - 1;  // convergence in the last iteration counts
    if (!launch(0.5, 0.5, 1e-24, 1e-10, limit, iters, status, 1) || status != HOEFEM_OK || iters != limit) return fail("last");
  }
  // a recurrence that reports convergence after every iteration, refuted by the true
  // residual each time: launches until the chunks are used up
  {
    const long long most = cg_max_chunks(-1, 300, 8);
    long long iters = 0, chunks = 0, launches = 0;
    int status = HOEFEM_OK;
    while (chunks < most && launches <= most) {
      const long long it0 = iters;
      if (!launch(0.5, 0.5, 0.0, 1e-17, cg_iteration_limit(-1, 300, 8), iters, status, 1) || status != HOEFEM_OK)
        return fail("claimed convergence");
      chunks += cg_chunks_of(iters - it0, 8);
      ++launches;
    }
    if (launches != most) return fail("launches");
  }
  if (cg_chunks_of(0, 8) != 1 || cg_chunks_of(1, 8) != 1 || cg_chunks_of(8, 8) != 1 || cg_chunks_of(9, 8) != 2)
    return fail("chunks of a launch");
  std::printf("ok\n");
  return 0;
}
