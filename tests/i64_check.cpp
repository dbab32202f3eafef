// Prints "name value" lines: the errors of the integer-arithmetic functions
// and of one bispectrum node against long double (tests/test_i64_host.py).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "tp_bispec64.cuh"
#include "tp_pell64.cuh"

using namespace tp;
typedef long double Q;

static Q val(Sf a) { return ldexpl((Q)a.m, a.e); }

template <class R> static R e2(R x) { return exp2(x); }
template <> Q e2<Q>(Q x) { return exp2l(x); }
template <class R> static R l2(R x) { return log2(x); }
template <> Q l2<Q>(Q x) { return log2l(x); }

struct EH {
  double omh2, sa, oms, sh043, theta2, c184, ehc, ns;
};
template <class R>
static R plin(const EH& e, R kk, R l2kk) {
  R x = kk * (R)e.sh043, x2 = x * x;
  R geff = (R)e.omh2 * ((R)e.sa + (R)e.oms / (1 + x2 * x2));
  R lq = l2kk + l2<R>((R)e.theta2) - l2<R>(geff);
  R qe = e2<R>(lq), q1 = e2<R>((R)1.11 * lq);
  R L = l2<R>((R)2.718281828 + (R)e.c184 * qe) * (R)0.693147180559945309417232121458L;
  R C = (R)14.4 + (R)325 / (1 + (R)60.5 * q1);
  R r = L / (L + C * qe * qe);
  return (R)e.ehc * e2<R>((R)e.ns * l2kk) * r * r;
}

struct PRow {
  double fk, rs, d1, a, b, gam, al, be, xnu, f1, f2, l2fk, l2rs, l2f3c;
};
// Takahashi et al. 2012 P(k) with the 2017 correction, as pell_node of tp_cov.cuh
template <class R>
static R pnode(const PRow& r, const EH& e, double l2h, double ell, R l2ell) {
  const R k = (R)ell * (R)r.fk, lk = l2ell + (R)r.l2fk, k3 = k * k * k, pi2 = 9.86960440108935861883449099987615113531L;
  const R pl = plin<R>(e, k * e2<R>((R)l2h), lk + (R)l2h) * (R)r.d1 * k3 / (2 * pi2);
  const R ly = lk + (R)r.l2rs, y = k * (R)r.rs, yy = y * y;
  R ph = (R)r.a * e2<R>(3 * (R)r.f1 * ly) / (1 + (R)r.b * e2<R>((R)r.f2 * ly) + e2<R>((3 - (R)r.gam) * ((R)r.l2f3c + ly)));
  ph = ph * yy / (yy + (R)r.xnu);
  const R pq = pl * e2<R>((R)r.be * l2<R>(1 + pl)) / (1 + pl * (R)r.al) * e2<R>(-(y / 4 + yy / 8) * (R)1.442695040888963407359924681L);
  const R c = e2<R>((R)1.3063 * l2<R>(1 + (R)9.5171e-4 * e2<R>((R)-1.3063 * lk)) - (R)0.62793 * l2<R>(1 + (R)5.1543e-3 * e2<R>((R)-1.1475 * lk)));
  return c * (2 * pi2 * (pq + ph) / k3);
}

struct Row {
  double s, hf, ana, anr, anc, bn, cn, ala, ald, betab, fn, gn, hn, mn, nn, mun, nun, pn, en, dn, d1sq;
};
// Takahashi et al. 2020, Eqs. B4-B9, as bispec_eval of tp_bispec.cuh
template <class R>
static R node(const Row& r, const EH& e, const double* l, const double* f2t) {
  R q[3], lq[3], P[3];
  for (int i = 0; i < 3; ++i) q[i] = (R)l[i] * (R)r.s, lq[i] = l2<R>((R)l[i]) + l2<R>((R)r.s);
  double o[3] = {l[0], l[1], l[2]};
  std::sort(o, o + 3);
  const R lr = l2<R>((R)o[0] / (R)o[2]), r2 = ((R)o[1] + (R)o[0] - (R)o[2]) / (R)o[2];
  const R pr2 = e2<R>((R)3.32192809488736234787 * (R)0.007 * r2);
  const R an = e2<R>((R)r.ana - (R)r.anr * e2<R>((R)r.anc * lr));
  R al = e2<R>((R)r.ala + (R)r.ald * r2 * r2);
  al = std::min(al, (R)1 - (R)2 / 3 * (R)e.ns);
  const R be = (R)r.betab * pr2;
  R b1 = 1;
  for (int i = 0; i < 3; ++i) {
    const R cq = (R)r.cn * q[i];
    b1 *= cq / ((an * e2<R>(al * lq[i]) + (R)r.bn * e2<R>(be * lq[i])) * (cq + 1));
    const R A = (1 + (R)r.fn * q[i] * q[i]) / (1 + (R)r.gn * q[i] + (R)r.hn * q[i] * q[i]) * (R)r.d1sq *
                plin<R>(e, (R)l[i] * (R)r.hf, l2<R>((R)l[i]) + l2<R>((R)r.hf));
    const R x = (R)r.pn * q[i], x3 = x * x * x;
    P[i] = A + x3 / (((R)r.mn * e2<R>((R)r.mun * lq[i]) + (R)r.nn * e2<R>((R)r.nun * lq[i])) * (x3 + 1));
  }
  R b3 = 2 * (((R)f2t[0] + (R)r.dn * q[2]) * P[0] * P[1] + ((R)f2t[1] + (R)r.dn * q[0]) * P[1] * P[2] +
              ((R)f2t[2] + (R)r.dn * q[1]) * P[2] * P[0]);
  return b1 + b3 / ((1 + (R)r.en * q[0]) * (1 + (R)r.en * q[1]) * (1 + (R)r.en * q[2]));
}

int main() {
  std::mt19937_64 g(1);
  auto U = [&] { return (double)(g() >> 11) * 0x1p-53; };
  double sc = 0, ex = 0, lg = 0, mu = 0, ad = 0, rc = 0, to = 0, fr = 0, fx = 0;
  auto rel = [](Q a, Q b) { return (double)fabsl(a / b - 1); };
  for (int i = 0; i < 400000; ++i) {
    int64_t x = (int64_t)((U() * 2 - 1) * 1000 * 0x1p52);
    if (i % 8 == 0) x = ((int64_t)(g() % 64) - 32) * (1ll << 44) + (int64_t)(g() % 3) - 1;  // table edges
    const Sf r = i64_exp2(x, h_i64tab.ex2);
    if (!(r.m >> 63)) return 1;
    ex = std::max(ex, rel(val(r), exp2l(ldexpl((Q)x, -52))));
    uint64_t m = g() | (1ull << 63);
    if (i % 4 == 0) m = (1ull << 63) | (g() >> (8 + g() % 50));                  // just above a power of two
    if (i % 4 == 1) m = ~(g() >> (8 + g() % 50));                               // just below
    if (i % 4 == 2) m = (1ull << 63) | ((g() % 256) << 55) | (g() % 2 ? 0 : ~0ull >> 9);  // cell edges
    lg = std::max(lg, (double)fabsl(ldexpl((Q)i64_log2m(m, h_i64tab.rc, h_i64tab.lc), -62) - log2l(ldexpl((Q)m, -63))));
    Sf a{(g() | (1ull << 63)) >> (g() % 5), (int)(g() % 60) - 100}, b{(g() | (1ull << 63)) >> (g() % 5), (int)(g() % 200) - 180};
    if (i % 5 == 0) a.m = 1ull << (59 + g() % 5);
    if (i % 5 == 1) a.m = ~0ull >> (g() % 5);
    rc = std::max(rc, rel(val(sf_rcp(a)) * val(a), 1));
    ad = std::max(ad, rel(val(sf_add(a, b)), val(a) + val(b)));
    const Sf an = sf_norm(a), bn = sf_norm(b);
    mu = std::max(mu, rel(val(sf_mul(an, bn)), val(an) * val(bn)));
    to = std::max(to, rel((Q)sf_to(a), val(a)));
    const double d = exp2((U() * 2 - 1) * 300);
    fr = std::max(fr, rel(val(sf_from(d)), d));
    double w = i % 8 ? U() * 7.999 : ldexp((double)(g() % 652), 0) * 0.012271846303085129838 + (U() - 0.5) * 1e-15;
    if (w < 0) w = 0;
    int64_t sn, cs;
    i64_sincos(w, h_i64sin, sn, cs);
    sc = std::max(sc, (double)std::max(fabsl(ldexpl((Q)sn, -62) - sinl((Q)w)), fabsl(ldexpl((Q)cs, -62) - cosl((Q)w))));
    const double y = (U() * 2 - 1) * exp2(-U() * 60) * 1000;
    fx = std::max(fx, (double)fabsl(ldexpl((Q)i64_fix<52>(y), -52) - (Q)y));
  }
  printf("sincos %g\nexp2 %g\nlog2 %g\nmul %g\nadd %g\nrcp %g\nto_double %g\nfrom_double %g\nfix %g\n", sc, ex, lg, mu, ad, rc, to, fr, fx);

  std::vector<P64Cell> tab(P64_N);
  EH e;
  double im = 0, dm = 0, is = 0, ds = 0;
  const int np = 100000;
  // a cosmology of each end of the box and beyond, the fiducial one last
  const double cs[5][4] = {{0.2, 0.6, 0.048, 0.92}, {0.4, 0.8, 0.048, 1.0}, {0.05, 0.4, 0.03, 0.5}, {1.0, 1.2, 0.5, 1.4}, {0.3, 0.7, 0.048, 0.96}};
  for (int i = 0; i < 5 * np; ++i) {
    if (i % np == 0) {
      const double *c = cs[i / np], om = c[0], h = c[1], ob = c[2];
      // Eisenstein & Hu 1998, the no-wiggle shape
      const double fc = (om - ob) / om, fb = ob / om, th = 2.728 / 2.7, pc = 0.25 * (5 - sqrt(1 + 24 * fc));
      const double o2 = om * h * h, b2 = ob * h * h, zeq = 2.5e4 * o2 / pow(th, 4);
      const double q1 = 0.313 * pow(o2, -0.419) * (1 + 0.607 * pow(o2, 0.674)), q2 = 0.238 * pow(o2, 0.223);
      const double zd = 1291 * pow(o2, 0.251) / (1 + 0.659 * pow(o2, 0.828)) * (1 + q1 * pow(b2, q2));
      const double yd = (1 + zeq) / (1 + zd), sh = 44.5 * log(9.83 / o2) / sqrt(1 + 10 * pow(b2, 0.75));
      const double sa = sqrt(fc * (5 - 2 * pc) / 5 * (1 - 0.553 * fb + 0.126 * fb * fb * fb) * pow(1 + yd, -pc) *
                             (1 + 0.5 * pc * (1 + 1 / (7 * (3 - 4 * pc))) / (1 + yd)));
      e = EH{o2, sa, 1 - sa, 0.43 * sh, th * th, 1.84 * sa / (1 - 0.949 * fb), 3.1e6, c[3]};
      for (int k = 0; k < P64_N; ++k)
        if (!p64_cell(k, e.omh2, e.sa, e.oms, e.sh043, e.theta2, e.c184, e.ehc, e.ns, h_i64tab, tab[k])) return 2;
    }
    // random, and every 8th at a cell's end
    int64_t k = i64_fix<57>(P64_LO + 0.001 + U() * (P64_HI - P64_LO - 0.002));
    if (i % 8 == 0) k = (((k >> 50) + 1) << 50) - 1 - (int64_t)(g() % 2);
    const Q lk = ldexpl((Q)k, -57), t = plin<Q>(e, exp2l(lk), lk);
    const double a = rel(val(p64_eval(tab.data(), (uint64_t)k + (64ull << 57), h_i64tab.ex2)), t);
    const double b = rel((Q)plin<double>(e, exp2((double)lk), (double)lk), t);
    im = std::max(im, a), dm = std::max(dm, b), is += a * a, ds += b * b;
  }
  printf("plin_int_max %g\nplin_dbl_max %g\nplin_int_rms %g\nplin_dbl_rms %g\n", im, dm, sqrt(is / (5 * np)), sqrt(ds / (5 * np)));

  std::vector<double> va, vb;
  const double LG = 3.32192809488736234787;
  auto p10 = [](double x) { return pow(10., x); };
  for (int it = 0; it < 20000; ++it) {
    const double n = -2.9 + U() * 1.6, s = -1.2 + U() * 1.1, D1 = 0.2 + .8 * U();
    Row r;
    r.s = exp2(-18 + U() * 14), r.hf = exp2(-13 + U() * 10);
    r.ana = LG * (-2.167 - 2.944 * s - 1.106 * s * s - 2.865 * s * s * s), r.anr = .31 * LG, r.anc = p10(.182 + .57 * n);
    r.bn = p10(-3.428 - 2.681 * s + 1.624 * s * s - .095 * s * s * s), r.cn = p10(.159 - 1.107 * n);
    r.ala = LG * (-4.348 - 3.006 * n - .5745 * n * n), r.ald = LG * p10(-.9 + .2 * n);
    r.betab = p10(-1.731 - 2.845 * n - 1.4995 * n * n - .2811 * n * n * n);
    r.fn = p10(-10.533 - 16.838 * n - 9.3048 * n * n - 1.8263 * n * n * n);
    r.gn = p10(2.787 + 2.405 * n + .4577 * n * n), r.hn = p10(-1.118 - .394 * n);
    r.mn = p10(-2.605 - 2.434 * s + 5.71 * s * s), r.nn = p10(-4.468 - 3.08 * s + 1.035 * s * s);
    r.mun = p10(15.312 + 22.977 * n + 10.9579 * n * n + 1.6586 * n * n * n), r.nun = p10(1.347 + 1.246 * n + .4525 * n * n);
    r.pn = p10(.071 - .433 * n), r.en = p10(-.632 + .646 * n), r.dn = p10(-.483 + .892 * s - .03), r.d1sq = D1 * D1;
    double l[3] = {exp2(U() * 16), exp2(U() * 16), 0};
    const double ch = cos(U() * 1.57);
    l[2] = sqrt((l[0] - l[1]) * (l[0] - l[1]) + 4 * l[0] * l[1] * ch * ch);
    if (it % 16 == 0) l[1] = l[2] = l[0];
    auto f2 = [](double a, double b, double c) {
      const double m = .5 * (c * c - a * a - b * b) / (a * b);
      return 5. / 7 + .5 * m * (a / b + b / a) + 2. / 7 * m * m;
    };
    const double f[3] = {f2(l[0], l[1], l[2]), f2(l[1], l[2], l[0]), f2(l[2], l[0], l[1])};
    Node64 N;
    Tri64 T;
    node64_make(1., r.s, r.hf, r.ana, r.anr, r.anc, r.bn, r.cn, r.ala, r.ald, r.betab, r.fn, r.gn, r.hn, r.mn, r.nn, r.mun,
                r.nun, r.pn, r.en, r.dn, r.d1sq, false, h_i64tab, N);
    if (!N.ok || !tri64_make(l[0], l[1], l[2], f, 1e-3, 1e7, h_i64tab, T)) continue;
    const Cosmo64 C{tab.data(), (uint64_t)i64_fix<59>(1 - 2. / 3 * e.ns), 0, 0, 1, 0};
    const Q t = node<Q>(r, e, l, f);
    va.push_back(rel((Q)bispec64(N, T, C, h_i64tab.ex2), t));
    vb.push_back(rel((Q)node<double>(r, e, l, f), t));
  }
  std::sort(va.begin(), va.end());
  std::sort(vb.begin(), vb.end());
  const size_t m = va.size();
  printf("nodes %zu\nnode_int_median %g\nnode_dbl_median %g\nnode_int_p99 %g\nnode_dbl_p99 %g\nnode_int_max %g\nnode_dbl_max %g\n", m,
         va[m / 2], vb[m / 2], va[m * 99 / 100], vb[m * 99 / 100], va[m - 1], vb[m - 1]);

  // P(ell) terms over the spectral shapes and scales of a survey's cosmologies
  va.clear(), vb.clear();
  const double l2h = log2(.7);
  for (int it = 0; it < 20000; ++it) {
    const double ne = -2.6 + U() * 1.4, nc = U() * .6, n2 = ne * ne, om = .15 + .85 * U(), fk = exp2(-13 + U() * 10);
    PRow r;
    r.fk = fk, r.rs = exp2(-10 + U() * 14), r.d1 = .04 + .96 * U();
    r.a = p10(1.5222 + 2.8553 * ne + 2.3706 * n2 + .9903 * ne * n2 + .2250 * n2 * n2 - .6038 * nc + .1749 * (1 - om) * (U() - .5));
    r.b = p10(-.5642 + .5864 * ne + .5716 * n2 - 1.5474 * nc + .2279 * (1 - om) * (U() - .5));
    r.gam = .1971 - .0843 * ne + .8460 * nc, r.al = fabs(6.0835 + 1.3373 * ne - .1959 * n2 - 5.5274 * nc);
    r.be = 2.0379 - .7354 * ne + .3157 * n2 + 1.2490 * ne * n2 + .3980 * n2 * n2 - .1682 * nc, r.xnu = p10(5.2105 + 3.6902 * ne);
    r.f1 = pow(om, -.0307), r.f2 = pow(om, -.0585);
    r.l2fk = log2(fk), r.l2rs = log2(r.rs), r.l2f3c = log2(pow(om, .0743) * p10(.3698 + 2.0404 * ne + .8161 * n2 + .5869 * nc));
    PellNode64 N;
    pell64_node_make(1., r.fk, r.rs, r.d1, r.a, r.b, r.gam, r.al, r.be, r.xnu, r.f1, r.f2, r.l2fk, r.l2rs, r.l2f3c, l2h, h_i64tab, N);
    double lo = -60, hi = 60;
    if (N.ok) pell64_range(r.l2fk, r.l2rs, l2h, lo, hi);
    // every eighth point an edge of the range
    const double lg = it % 8 ? fmax(lo, fmin(hi, -1 + U() * 17)) : it % 16 ? lo + .01 : hi - .01, ell = exp2(lg);
    if (!N.ok) continue;
    const Q t = pnode<Q>(r, e, l2h, ell, log2l((Q)ell));
    va.push_back(rel((Q)pell64(N, pell64_point(ell, h_i64tab), tab.data(), h_i64tab) / 1, t));
    vb.push_back(rel((Q)pnode<double>(r, e, l2h, ell, log2(ell)), t));
  }
  std::sort(va.begin(), va.end());
  std::sort(vb.begin(), vb.end());
  const size_t k = va.size();
  printf("pells %zu\npell_int_median %g\npell_dbl_median %g\npell_int_p99 %g\npell_dbl_p99 %g\npell_int_max %g\npell_dbl_max %g\n", k,
         va[k / 2], vb[k / 2], va[k * 99 / 100], vb[k * 99 / 100], va[k - 1], vb[k - 1]);
  return 0;
}
