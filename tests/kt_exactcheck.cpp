// kt_exactcheck.cpp -- TEST-ONLY host build of the exact right-hand sides'
// fast forms (kt_exact.cuh, bl_rhs_exact, ktm_sincos_core), compared bit for
// bit with the general forms.  Built by test_exact.py with -ffp-contract=off.
#include <string.h>

#include "../kerrtracecpp2_b200/csrc/kt_machines.cuh"

using namespace kt;

extern "C" {

// Quotients a[i]/b[i] by kt_exact.cuh against the division; returns the
// number that differ, and how many denominators its range test refuses.
long ec_quot(long n, const double* a, const double* b, long* refused) {
  long bad = 0;
  *refused = 0;
  for (long i = 0; i < n; ++i) {
    if (top_ones(b[i]) & kTopBit) {
      ++*refused;
      continue;
    }
    const Rcp R = make_rcp(b[i]);
    const double q = quot_signed(a[i], R), e = a[i] / b[i];
    if (memcmp(&q, &e, 8) != 0) ++bad;
    const double q1 = quot_one(R), e1 = 1.0 / b[i];
    if (memcmp(&q1, &e1, 8) != 0) ++bad;
  }
  return bad;
}

long ec_sincos(long n, const double* x, long* plain) {
  long bad = 0;
  *plain = 0;
  for (long i = 0; i < n; ++i) {
    double s, c, s2, c2;
    ktm_sincos(x[i], &s, &c);
    ktm_sincos_any(x[i], &s2, &c2);
    *plain += ktm_sincos_plain(x[i]);
    if (memcmp(&s, &s2, 8) != 0 || memcmp(&c, &c2, 8) != 0) ++bad;
  }
  return bad;
}

// States y[i] = (r, theta, p_r, p_theta, p_t, p_phi) in one metric: how many
// bl_rhs_exact results differ from bl_rhs; *refused counts those it hands back.
long ec_bl_rhs(double M, double a, double Q, double L, int lam, long n, const double* y,
               long* refused) {
  const Metric g = make_metric(M, a, Q, L);
  long bad = 0;
  *refused = 0;
  for (long i = 0; i < n; ++i) {
    const double* s = y + 6 * i;
    double k[5], e[5];
    const bool ok = lam ? bl_rhs_exact<true>(g, s[0], s[1], s[2], s[3], s[4], s[5], k)
                        : bl_rhs_exact<false>(g, s[0], s[1], s[2], s[3], s[4], s[5], k);
    if (!ok) {
      ++*refused;
      continue;
    }
    bl_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], e);
    if (memcmp(k, e, sizeof k) != 0) ++bad;
  }
  return bad;
}

long ec_sqrt(long n, const double* x, long* refused) {
  long bad = 0;
  *refused = 0;
  for (long i = 0; i < n; ++i) {
    if (top_edge(x[i]) & kTopBit) {
      ++*refused;
      continue;
    }
    const double g = make_root(x[i]).g, e = sqrt(x[i]);
    if (memcmp(&g, &e, 8) != 0) ++bad;
  }
  return bad;
}

// States (X, Y, Z, p_X, p_Y, p_Z, p_T) of the KS chart, as ec_bl_rhs.
long ec_ks_rhs(double M, double a, double Q, long n, const double* y, long* refused) {
  const Metric g = make_metric(M, a, Q, 0.0);
  long bad = 0;
  *refused = 0;
  for (long i = 0; i < n; ++i) {
    const double* s = y + 7 * i;
    double k[6], e[6];
    if (!ks_rhs_exact(g, s[0], s[1], s[2], s[3], s[4], s[5], s[6], k)) {
      ++*refused;
      continue;
    }
    ks_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], s[6], e);
    if (memcmp(k, e, sizeof k) != 0) ++bad;
  }
  return bad;
}

// pow_ctl against ktm_pow for the controllers' exponents.
long ec_pow(long n, const double* x) {
  long bad = 0;
  for (long i = 0; i < n; ++i)
    for (int j = 0; j < 2; ++j) {
      const double y = j ? 0.25 : 0.2, p = pow_ctl(x[i], y), e = ktm_pow(x[i], y);
      if (memcmp(&p, &e, 8) != 0) ++bad;
    }
  return bad;
}

// first_event's quick test: of n cubics (y0, y1, dy0, dy1, h, target), those
// it dismisses although the search (without the test) finds an event;
// *quick counts the dismissed, *none those without an event.
long ec_no_event(long n, const double* v, long* quick, long* none) {
  long bad = 0;
  *quick = *none = 0;
  for (long i = 0; i < n; ++i) {
    const double *c = v + 6 * i, target = c[5];
    bool found = false;
    double f0 = c[0] - target;
    found = fabs(f0) <= 1e-12;
    for (int b = 1; b <= 8 && !found; ++b) {
      const double f1 =
          (b == 8) ? (c[1] - target) : (hermite(c[0], c[1], c[2], c[3], c[4], b / 8.0) - target);
      found = fabs(f1) <= 1e-12 || sign_change(f0, f1);
      f0 = f1;
    }
    const bool no = no_event(c[0], c[1], c[2], c[3], c[4], target);
    *quick += no;
    *none += !found;
    if (no && found) ++bad;
  }
  return bad;
}

// States (r, theta, p_r, p_theta, p_t, p_phi, W[8]) of the bundle right-hand
// side split over two lanes (bundle_half_exact, bundle_combine_exact) against
// bundle_rhs.
long ec_bundle_rhs(double M, double a, double Q, double L, int lam, long n, const double* y,
                   long* refused) {
  const Metric g = make_metric(M, a, Q, L);
  long bad = 0;
  *refused = 0;
  for (long i = 0; i < n; ++i) {
    const double *s = y + 14 * i, *W = s + 6;
    BundleHalf H[2];
    bool ok = true;
    for (int o = 0; o < 2; ++o)
      ok = (lam ? bundle_half_exact<true>(g, s[0], s[1], s[2], s[3], s[4], s[5], o != 0, &H[o])
                : bundle_half_exact<false>(g, s[0], s[1], s[2], s[3], s[4], s[5], o != 0, &H[o])) && ok;
    double k[5], kW[8], e[5], eW[8];
    ok = bundle_combine_exact(H[0], H[1], s[0], s[2], s[3], W, k, kW) && ok;
    if (!ok) {
      ++*refused;
      continue;
    }
    bundle_rhs(g, s[0], s[1], s[2], s[3], s[4], s[5], W, e, eW);
    if (memcmp(k, e, sizeof k) != 0 || memcmp(kW, eW, sizeof kW) != 0) ++bad;
  }
  return bad;
}
}
