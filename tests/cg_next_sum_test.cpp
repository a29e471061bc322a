// Checks csrc/cg_limit.h: a sum of the next residual that cg_next_sum accepts is exact
// to 1e-14, whatever the drop.
#include "cg_limit.h"

#include <cstdio>
#include <random>
#include <vector>

using namespace hoefem;

int main() {
  std::mt19937 rng(7);
  std::normal_distribution<double> nd;
  const int n = 1000;
  std::vector<double> r(n), ap(n);
  int taken = 0;
  for (double drop = 1.0; drop < 1e7; drop *= 1.3)
    for (int rep = 0; rep < 20; ++rep) {
      // A p = r / alpha up to a part of the size of the next residual
      const double alpha = std::exp(nd(rng)), size = std::sqrt(1.0 / drop);
      long double rr = 0.0L, rap = 0.0L, apap = 0.0L, next = 0.0L;
      for (int i = 0; i < n; ++i) {
        r[i] = nd(rng);
        ap[i] = (r[i] - size * nd(rng)) / alpha;
        rr += (long double)r[i] * r[i];
        rap += (long double)r[i] * ap[i];
        apap += (long double)ap[i] * ap[i];
        const long double q = (long double)r[i] - (long double)alpha * ap[i];
        next += q * q;
      }
      double got;
      if (!cg_next_sum(alpha, (double)rr, (double)rap, (double)apap, got)) continue;
      ++taken;
      const double err = (double)(std::fabs((long double)got - next) / next);
      if (!(err <= 1e-14)) {
        std::printf("drop %g: %g\n", drop, err);
        return 1;
      }
    }
  // a NaN or a sum that is not positive is never taken
  double got;
  if (cg_next_sum(std::nan(""), 1.0, 1.0, 1.0, got) || cg_next_sum(1.0, 0.0, 0.0, 0.0, got) ||
      cg_next_sum(1.0, 1.0, 1.0, 1.0, got)) {
    std::printf("taken\n");
    return 1;
  }
  std::printf(taken > 100 ? "ok\n" : "none taken\n");
  return 0;
}
