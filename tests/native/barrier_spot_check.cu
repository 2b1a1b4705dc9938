// Host-only check of the FP64 lane's barrier thresholds (host_prep.cu): the smallest spot whose rounded
// ratio to the initial spot reaches a barrier does so, and the double below it does not, for initial
// spots over the whole range, ordinary, extreme and absent barriers.  Built and run by
// tests/test_barrier_spot.py against the engine library.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <random>
#include "rg_internal.h"

int main() {
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> expo(-300.0, 300.0), near(0.2, 3.0);
  int bad = 0, checked = 0;
  auto check = [&](double barrier, double init) {
    const double s = rg::smallest_spot(barrier, init);
    const bool ok = s / init >= barrier && (s == 0.0 || !(std::nextafter(s, 0.0) / init >= barrier));
    ++checked;
    if (!ok && ++bad < 10) std::printf("barrier %a initial spot %a: %a\n", barrier, init, s);
  };
  const double inits[] = {5e-324, DBL_MIN, 1e-300, 1e-12, 1e-3, 0.5, 0.73, 0.9, 0.999, 1.0, 1.1, 3.1, 100.0, 1e6, 1e15, 1e300, DBL_MAX};
  const double barriers[] = {5e-324, 1e-310, DBL_MIN, 1e-300, 1e-8, 0.3, 0.6, 0.7, 0.999, 1.0, 1.05, 3.0, 1e8, 1e300, DBL_MAX, INFINITY};
  for (double i : inits)
    for (double b : barriers) check(b, i);
  for (double i : inits)
    for (int k = 0; k < 2000; ++k) check(near(rng), i);
  for (int k = 0; k < 200000; ++k) check(std::pow(10.0, expo(rng)), std::pow(10.0, expo(rng)));
  std::printf("%d thresholds, %d wrong\n", checked, bad);
  return bad != 0;
}
