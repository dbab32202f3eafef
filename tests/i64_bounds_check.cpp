// Prints "name value" lines: the largest errors of the integer-arithmetic
// functions whose bounds the header states (tests/test_i64_bounds_host.py).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "tp_i64.cuh"

using namespace tp;
typedef long double Q;
static Q val(Sf a) { return ldexpl((Q)a.m, a.e); }

int main() {
  std::mt19937_64 g(3);
  auto rel = [](Q a, Q b) { return (double)fabsl(a / b - 1); };
  double add = 0, rcp = 0, sc = 0;
  long alike = 0, unlike = 0;
  for (int i = 0; i < 2000000; ++i) {
    // mantissas with zero to four leading zeros, small ones often
    Sf a{(g() | (1ull << 63)) >> (g() % 5), (int)(g() % 80) - 100}, b{(g() | (1ull << 63)) >> (g() % 5), 0};
    if (i % 3 == 0) a.m = (1ull << (59 + g() % 5)) | (g() >> 40);
    if (i % 3 == 1) b.m = (1ull << (59 + g() % 5)) | (g() >> 40);
    b.e = a.e + (int)(g() % 140) - 70;
    add = std::max(add, rel(val(sf_add(a, b)), val(a) + val(b)));
    // the step from starts up to 2 ulp off the reciprocal of the upper bits
    const Sf n = sf_norm(a);
    const uint32_t fu = sf_rcp_arg(n);
    float f, y;
    memcpy(&f, &fu, 4);
    y = 1.0f / f;
    for (int d = -2; d <= 2; ++d) {
      uint32_t yu;
      memcpy(&yu, &y, 4);
      yu += d;
      if (yu < 0x3f800000u) continue;  // a reciprocal of [1/2, 1) is at least 1
      rcp = std::max(rcp, rel(val(sf_rcp_step(n, yu)) * val(n), 1));
    }
    // claims of equal rounding: errors of ulps units of 2^-53 of the scale, the
    // value up to 2^22 below it, often next to the middle of two floats
    const double scale = ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 60) - 30);
    uint64_t vb = (g() >> 12) | ((uint64_t)(1023 + ilogb(scale) - (int)(g() % 23)) << 52);
    if (i % 2) vb = (vb & ~0x1fffffffull) | (0x10000000ull + (uint64_t)((int64_t)(g() % (1ull << (g() % 29))) - (int64_t)(g() % 3)) % 0x10000000ull);
    double v;
    memcpy(&v, &vb, 8);
    const int ulps = (int)(g() % 225000);
    if (i64_rounds_alike(v, scale, ulps)) {
      const Q e = ldexpl((Q)ulps, ilogb(scale) - 53);
      ++alike;
      unlike += (float)((Q)v - e) != (float)v || (float)((Q)v + e) != (float)v;
    }
    const double w = (double)(g() >> 11) * 0x1p-53 * (i % 2 ? 7.9999999 : 6.2831853071795862);
    int64_t sn, cs;
    i64_sincos(w, h_i64sin, sn, cs);
    sc = std::max(sc, (double)std::max(fabsl(ldexpl((Q)sn, -62) - sinl((Q)w)), fabsl(ldexpl((Q)cs, -62) - cosl((Q)w))));
  }
  printf("add %g\nrcp %g\nsincos %g\nalike %ld\nunlike %ld\n", add, rcp, sc, alike, unlike);
  return 0;
}
