// Prints "name value" lines: b_kappa nodes and P(ell) terms in integer
// arithmetic over every row that node64_make and pell64_node_make accept,
// against long double (tests/test_i64_domain_host.py). The formulas in long
// double are i64_check.cpp's.
#define main i64_check_main
#include "i64_check.cpp"
#undef main

static std::mt19937_64 rng(7);
static double U() { return (double)(rng() >> 11) * 0x1p-53; }
static double LU(double a, double b) { return exp2(a + U() * (b - a)); }
static double p10(double x) { return pow(10., x); }
static const double LG = 3.32192809488736234787;

// BiHalofit's coefficients of a spectral index n and amplitude s = log10 sigma8 D1
static void bihalofit(double n, double s, Row& r) {
  r.ana = LG * (-2.167 - 2.944 * s - 1.106 * s * s - 2.865 * s * s * s), r.anr = .31 * LG, r.anc = p10(.182 + .57 * n);
  r.bn = p10(-3.428 - 2.681 * s + 1.624 * s * s - .095 * s * s * s), r.cn = p10(.159 - 1.107 * n);
  r.ala = LG * (-4.348 - 3.006 * n - .5745 * n * n), r.ald = LG * p10(-.9 + .2 * n);
  r.betab = p10(-1.731 - 2.845 * n - 1.4995 * n * n - .2811 * n * n * n);
  r.fn = p10(-10.533 - 16.838 * n - 9.3048 * n * n - 1.8263 * n * n * n);
  r.gn = p10(2.787 + 2.405 * n + .4577 * n * n), r.hn = p10(-1.118 - .394 * n);
  r.mn = p10(-2.605 - 2.434 * s + 5.71 * s * s), r.nn = p10(-4.468 - 3.08 * s + 1.035 * s * s);
  r.mun = p10(15.312 + 22.977 * n + 10.9579 * n * n + 1.6586 * n * n * n), r.nun = p10(1.347 + 1.246 * n + .4525 * n * n);
  r.pn = p10(.071 - .433 * n), r.en = p10(-.632 + .646 * n), r.dn = p10(-.483 + .892 * s - .03);
}
// coefficients of any size, unrelated to one another; w the share of the exponents' range
static void unrelated(double w, Row& r) {
  r.ana = (2 * U() - 1) * 899 * w, r.anr = LU(-20, 3.99), r.anc = LU(-20, 4.9), r.bn = LU(-930 * w, 930 * w), r.cn = LU(-60, 60);
  r.ala = rng() % 2 ? -20 * U() : (2 * U() - 1) * 899, r.ald = LU(-20, 4.9), r.betab = LU(-20, 3.95);
  r.fn = LU(-300 * w, 300 * w), r.gn = LU(-300 * w, 300 * w), r.hn = LU(-300 * w, 300 * w);
  r.mn = LU(-930 * w, 930 * w), r.nn = LU(-930 * w, 930 * w), r.mun = LU(-10, 4.99), r.nun = LU(-10, 4.99);
  r.pn = LU(-60, 60), r.en = LU(-60, 60), r.dn = LU(-60, 60);
}

int main() {
  // Omega_m 0.3, Omega_b 0.048, h 0.7: the no-wiggle constants to six digits
  EH e{0.147, 0.853, 0.147, 0.43 * 149.4, 1.00735, 1.85, 3.1e6, .96};
  std::vector<P64Cell> tab(P64_N);
  for (int k = 0; k < P64_N; ++k)
    if (!p64_cell(k, e.omh2, e.sa, e.oms, e.sh043, e.theta2, e.c184, e.ehc, e.ns, h_i64tab, tab[k])) return 2;
  const Cosmo64 C{tab.data(), (uint64_t)i64_fix<59>(1 - 2. / 3 * e.ns), 0, 0, 1, 0};
  // P_lin tables of any Eisenstein & Hu constants that k_node64 and p64_cell accept
  double perr = 0;
  int tables = 0;
  std::vector<P64Cell> pt(P64_N);
  for (int it = 0; it < 600; ++it) {
    const double sa = LU(-6, .3);
    const EH h{LU(-12, 3), sa, 1 - sa, .43 * LU(1, 12), LU(-1, 1), LU(-3, 4), it % 2 ? LU(0, 40) : LU(-90, 90), -1 + 4 * U()};
    bool ok = true;
    for (int k = 0; k < P64_N && ok; ++k)
      ok = p64_cell(k, h.omh2, h.sa, h.oms, h.sh043, h.theta2, h.c184, h.ehc, h.ns, h_i64tab, pt[k]);
    if (!ok) continue;
    ++tables;
    for (int i = 0; i < 2000; ++i) {
      const int64_t k = i64_fix<57>(P64_LO + 0.001 + U() * (P64_HI - P64_LO - 0.002));
      const Q lk = ldexpl((Q)k, -57), t = plin<Q>(h, exp2l(lk), lk);
      perr = std::max(perr, (double)fabsl(val(p64_eval(pt.data(), (uint64_t)k + (64ull << 57), h_i64tab.ex2)) / t - 1));
    }
  }
  // in units of 1e-15, rounded up
  printf("tables %d\nplin_err %ld\n", tables, (long)std::min(1e15, std::ceil(perr * 1e15)));
  // kind 0: BiHalofit rows, 1: unrelated rows. over: nodes whose error exceeds
  // 1e-11 and what the cancellation of F2 makes of it, (l_max / l_min)^2
  for (int kind = 0; kind < 2; ++kind) {
    long rows = 0, used = 0, over = 0;
    for (int it = 0; it < 300000; ++it) {
      Row r;
      r.s = LU(-26.9, 35.9), r.hf = LU(-40, 20);
      if (kind == 0) {
        bihalofit(-4.9 + 5.8 * U(), -4 + 5 * U(), r);
        r.d1sq = LU(-24, 0);
      } else {
        const double w = it % 3 == 0 ? .6 : it % 3 == 1 ? .3 : .05;
        unrelated(w, r);
        r.d1sq = LU(-200 * w, 200 * w);
      }
      Node64 N;
      Tri64 T;
      node64_make(1., r.s, r.hf, r.ana, r.anr, r.anc, r.bn, r.cn, r.ala, r.ald, r.betab, r.fn, r.gn, r.hn, r.mn, r.nn,
                  r.mun, r.nun, r.pn, r.en, r.dn, r.d1sq, false, h_i64tab, N);
      if (!N.ok) continue;
      ++rows;
      // the ell range of k_node64 for this row
      const double a = fmax(-36, P64_LO + .01 - log2(r.hf)), b = fmin(26, P64_HI - .01 - log2(r.hf));
      if (a >= b) continue;
      const double c = a + U() * (b - a), w = it % 2 ? 2 : 40;
      double l[3] = {LU(fmax(a, c - w), fmin(b, c + w)), LU(fmax(a, c - w), fmin(b, c + w)), 0};
      const double ch = cos(U() * 1.57);
      l[2] = sqrt((l[0] - l[1]) * (l[0] - l[1]) + 4 * l[0] * l[1] * ch * ch);
      if (it % 16 == 0) l[1] = l[2] = l[0];
      auto f2 = [](double a, double b, double c) {
        const double m = .5 * (c * c - a * a - b * b) / (a * b);
        return 5. / 7 + .5 * m * (a / b + b / a) + 2. / 7 * m * m;
      };
      const double f[3] = {f2(l[0], l[1], l[2]), f2(l[1], l[2], l[0]), f2(l[2], l[0], l[1])};
      if (!tri64_make(l[0], l[1], l[2], f, exp2(a), exp2(b), h_i64tab, T)) continue;
      const Q t = node<Q>(r, e, l, f);
      const double d = node<double>(r, e, l, f), v = bispec64(N, T, C, h_i64tab.ex2);
      if (!std::isfinite(d) || fabsl(t) < 1e-290L || fabsl(t) > 1e200L) continue;
      ++used;
      const double q = std::max({l[0], l[1], l[2]}) / std::min({l[0], l[1], l[2]});
      over += !(fabsl(v / t - 1) <= 1e-11 + 64 * 2.2e-16 * q * q);
    }
    printf("rows%d %ld\nnodes%d %ld\nover%d %ld\n", kind, rows, kind, used, kind, over);
  }
  // P(ell) terms: exponents and amplitudes over pell64_node_make's fields
  long used = 0, over = 0;
  const double l2h = log2(.7);
  for (int it = 0; it < 300000; ++it) {
    PRow r;
    const double fk = LU(-29, 20), w = it % 2 ? 1 : .2;
    r.fk = fk, r.rs = LU(-29, 29), r.d1 = LU(-24, 0);
    r.a = LU(-199 * w, 199 * w), r.b = LU(-199 * w, 199 * w), r.gam = 3 - (2 * U() - 1) * 14.9 * w;
    r.al = LU(-99 * w, 99 * w), r.be = (2 * U() - 1) * 7.8, r.xnu = LU(-199 * w, 199 * w);
    r.f1 = (2 * U() - 1) * 4.9 * w, r.f2 = (2 * U() - 1) * 14.9 * w;
    r.l2fk = log2(fk), r.l2rs = log2(r.rs), r.l2f3c = (2 * U() - 1) * 29;
    PellNode64 N;
    pell64_node_make(1., r.fk, r.rs, r.d1, r.a, r.b, r.gam, r.al, r.be, r.xnu, r.f1, r.f2, r.l2fk, r.l2rs, r.l2f3c, l2h, h_i64tab, N);
    if (!N.ok) continue;
    double lo = -60, hi = 60;
    pell64_range(r.l2fk, r.l2rs, l2h, lo, hi);
    if (lo >= hi) continue;
    const double ell = LU(lo + .01, hi - .01);
    const Q t = pnode<Q>(r, e, l2h, ell, log2l((Q)ell));
    const double d = pnode<double>(r, e, l2h, ell, log2(ell)), v = pell64(N, pell64_point(ell, h_i64tab), tab.data(), h_i64tab);
    if (!std::isfinite(d) || fabsl(t) < 1e-250L || fabsl(t) > 1e250L) continue;
    ++used;
    over += !(fabsl(v / t - 1) <= 1e-11);
  }
  printf("pells %ld\npell_over %ld\n", used, over);
  return 0;
}
