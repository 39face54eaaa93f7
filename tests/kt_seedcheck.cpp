// kt_seedcheck.cpp -- TEST-ONLY host build of kt_exact.cuh's quotients and
// roots from given seeds, over the whole band of seed errors their bounds
// assume.  Built by test_exact_seeds.py with -ffp-contract=off.
#include <string.h>

#include "../kerrtracecpp2_b200/csrc/kt_exact.cuh"

using namespace kt;

static bool differ(double a, double b) { return memcmp(&a, &b, 8) != 0; }

extern "C" {

// a[i]/b[i] and 1/b[i] from the seed (1 + rel)/b; returns how many differ from
// the divisions (refused denominators left out).
long sc_quot(long n, const double* a, const double* b, double rel) {
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    if (top_ones(b[i]) & kTopBit) continue;
    const Rcp R = make_rcp_seeded(b[i], (1.0 / b[i]) * (1.0 + rel));
    bad += differ(quot_signed(a[i], R), a[i] / b[i]) || differ(quot_one(R), 1.0 / b[i]);
  }
  return bad;
}

// sqrt(x[i]), and a quotient by it and by its square, from the seed
// (1 + rel)/sqrt(x).  *worst: the largest |y sqrt(x) - 1| K, the quantity the
// proof bounds by 3/2, with K = sqrt(x) in units of its ulp.
long sc_sqrt(long n, const double* x, double rel, double* worst) {
  long bad = 0;
  *worst = 0.0;
  for (long i = 0; i < n; ++i) {
    if (top_edge(x[i]) & kTopBit) continue;
    const Root r = make_root_seeded(x[i], (1.0 / sqrt(x[i])) * (1.0 + rel));
    const double s = sqrt(x[i]);
    bad += differ(r.g, s);
    if (!((top_ones(s) | top_ones(s * s)) & kTopBit))
      bad += differ(quot(x[i] + 1.0, make_rcp_from(s, r.y)), (x[i] + 1.0) / s) ||
             differ(quot(x[i] + 1.0, make_rcp_from(s * s, r.y * r.y)), (x[i] + 1.0) / (s * s));
    int e;
    const double K = ldexp(frexp(s, &e), 53);
    const double d = (double)((__float128)r.y * r.y * x[i] - 1.0) / 2.0 * K;
    if (fabs(d) > *worst) *worst = fabs(d);
  }
  return bad;
}
}
