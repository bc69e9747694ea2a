// Host build of cr_math.cuh's reciprocal, quotient and square root sequences
// beside the IEEE operators (tests/test_rounded_ops.py).
#include <cmath>

#include "cr_math.cuh"

using namespace dgswem;

// mismatches of rcp_from / sqrt_from with 1 / x, sqrt(x) over xs, each with
// `ns` seeds spread over (1 +- err) times the exact one
extern "C" long rounded_rcp(const double* xs, long n, int ns, double err) {
  long bad = 0;
  for (long i = 0; i < n; ++i)
    for (int j = 0; j < ns; ++j)
      if (rcp_from(xs[i], (1.0 / xs[i]) * (1.0 + err * (2.0 * j / (ns - 1) - 1.0))) != 1.0 / xs[i]) ++bad;
  return bad;
}
extern "C" long rounded_sqrt(const double* xs, long n, int ns, double err) {
  long bad = 0;
  for (long i = 0; i < n; ++i)
    for (int j = 0; j < ns; ++j)
      if (sqrt_from(xs[i], (1.0 / std::sqrt(xs[i])) * (1.0 + err * (2.0 * j / (ns - 1) - 1.0))) != std::sqrt(xs[i]))
        ++bad;
  return bad;
}
extern "C" long rounded_quot(const double* a, const double* b, long n) {
  long bad = 0;
  for (long i = 0; i < n; ++i)
    if (quot_from(a[i], b[i], 1.0 / b[i]) != a[i] / b[i]) ++bad;
  return bad;
}
// mismatches of pow_third with the general method; `moved` counts the values
// pow_third_near leaves to it
extern "C" long rounded_pow_third(const double* xs, long n, long* moved) {
  long bad = 0;
  *moved = 0;
  for (long i = 0; i < n; ++i) {
    double r;
    if (!pow_third_try(xs[i], &r)) ++*moved;
    if (pow_third(xs[i]) != pow_third<false>(xs[i])) ++bad;
  }
  return bad;
}
