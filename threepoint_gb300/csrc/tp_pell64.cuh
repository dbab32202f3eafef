// The P_kappa line-of-sight term of one node (pell_node in tp_cov.cuh:
// Takahashi et al. 2012 power spectrum with the Takahashi et al. 2017
// correction) in the 64-bit integer arithmetic of tp_i64.cuh, what the FP64
// covariance integrands of P(ell) products evaluate.
//
// With FP64 instructions a node takes 8 exp2, 4 log2 and 7 divisions of the
// FP64 pipe; here 7 exponentials, 3 logarithms and one reciprocal of the
// integer pipe (all rational factors over one denominator, exponents summed
// before they are raised): two entries of the square-window T2 290 -> 40.9 ms on
// the same clusters (GB300), of the infinite T1 176 -> 24 ms (then 16-CTA clusters: 28.9 and 17.5).
//
// Domain: rows whose exponents fit (PellNode64::ok), a fitted P(k) and ell
// inside the table (pell64_range); everything else keeps the FP64 form.
#pragma once
#include "tp_bispec64.cuh"

namespace tp {

struct PellNode64 {
  int64_t l2fk, l2hf, l2rs;               // log2 1/f_K, h/f_K, r_sigma: Q57
  uint64_t s1, s2, s3, be;                // |slopes| 3 f1, f2, 3 - gamma, beta: Q59
  int64_t k1, k2, k3;                     // offsets: Q52, modulo 2^64 as the exponents' sums are
  int64_t n1, n2, n3, nb;                 // -1 where the slope is negative, else 0
  uint64_t cpl, al, xnu, ys;              // mantissas: D1^2 / (2 pi^2 f_K^3), alpha, 10^xnu, r_sigma / f_K
  int ecpl, eal, exnu, eys;
  double w;                               // 2 pi^2 W f_K^3
  int ok, pad;
};

struct Pell64 {  // a point
  uint64_t lgb, m, m3;  // log2 ell + 64 in Q57, ell, ell^3
  int e, e3;
};

TP_HD bool slope_ok(double c) { return fabs(c) < 15; }
TP_HD uint64_t q59_even(double c) { return (uint64_t)i64_fix<58>(fabs(c)) << 1; }
// log2(c 2^(s (x + l))) = s (x + 64) + k, x the biased logarithm
TP_HD int64_t pell64_off(double l2c, double s, double l, uint64_t sq) {
  const int64_t k = i64_fix<52>(l2c + s * l), b = (int64_t)(sq >> 1);
  return s < 0 ? k + b : k - b;
}

TP_HD void pell64_node_make(double w, double invfk, double rs, double d1sq, double a, double b, double gam, double alpha,
                            double beta, double xnu, double f1, double f2, double l2invfk, double l2rs, double l2f3c,
                            double l2h, const I64Tables& t, PellNode64& N) {
  const double pi2 = 2 * 3.14159265358979323846 * 3.14159265358979323846, fk3 = invfk * invfk * invfk;
  const double s1 = 3.0 * f1, s3 = 3.0 - gam, ys = invfk * rs, cpl = d1sq * fk3 / pi2;
  N.w = w * pi2 / fk3;
  N.ok = fabs(l2invfk) < 30 && fabs(l2invfk + l2h) < 30 && fabs(l2rs) < 30 && fabs(l2f3c) < 30 && slope_ok(s1) &&
         slope_ok(f2) && slope_ok(s3) && fabs(beta) < 7.9 && sf_ok(a) && a > 1e-60 && a < 1e60 && sf_ok(b) &&
         b > 1e-60 && b < 1e60 && sf_ok(cpl) && sf_ok(alpha) && alpha > 1e-30 && alpha < 1e30 && sf_ok(xnu) &&
         xnu > 1e-60 && xnu < 1e60 && sf_ok(ys) && fabs(N.w) < 1e200;
  N.pad = 0;
  if (!N.ok) return;
  N.l2fk = i64_fix<57>(l2invfk);
  N.l2hf = i64_fix<57>(l2invfk + l2h);
  N.l2rs = i64_fix<57>(l2rs);
  N.s1 = q59_even(s1), N.n1 = s1 < 0 ? -1 : 0;
  N.s2 = q59_even(f2), N.n2 = f2 < 0 ? -1 : 0;
  N.s3 = q59_even(s3), N.n3 = s3 < 0 ? -1 : 0;
  N.be = q59_even(beta), N.nb = beta < 0 ? -1 : 0;
  N.k1 = pell64_off(0.0, s1, 0.0, N.s1) + i64_log2_q52(a, t);
  N.k2 = pell64_off(0.0, f2, 0.0, N.s2) + i64_log2_q52(b, t);
  N.k3 = pell64_off(0.0, s3, l2f3c, N.s3);
  Sf v = sf_from(cpl);
  N.cpl = v.m, N.ecpl = v.e;
  v = sf_from(alpha);
  N.al = v.m, N.eal = v.e;
  v = sf_from(xnu);
  N.xnu = v.m, N.exnu = v.e;
  v = sf_from(ys);
  N.ys = v.m, N.eys = v.e;
}

// ell range whose biased logarithms and P table coordinates are inside their
// fields at a row that is ok
TP_HD void pell64_range(double l2invfk, double l2rs, double l2h, double& lo, double& hi) {
  const double a = fmax(fmax(P64_LO + 0.01 - l2invfk - l2h, -31.0 - l2invfk), -60.0 - l2invfk - l2rs);
  const double b = fmin(fmin(P64_HI - 0.01 - l2invfk - l2h, 31.0 - l2invfk), 60.0 - l2invfk - l2rs);
  lo = fmax(lo, a);
  hi = fmin(hi, b);
}

TP_HD Pell64 pell64_point(double ell, const I64Tables& t) {
  const Sf l = sf_from(ell), l3 = sf_norm(sf_mul(sf_norm(sf_mul(l, l)), l));
  return {(uint64_t)i64_log2(ell, t) + (64ull << 57), l.m, l3.m, l.e, l3.e};
}

// Q57 x Q59 with the sign mask n of the second: Q52
TP_HD int64_t pell64_mul(uint64_t x, uint64_t s, int64_t n) { return ((int64_t)i64_mulhi(x, s) ^ n) - n; }
// log2 of x >= 1, Q57
TP_HD uint64_t sf_log2(Sf x, const uint32_t* __restrict__ rc, const uint64_t* __restrict__ lc) {
  x = sf_norm(x);
  return ((uint64_t)(x.e + 63) << 57) + (uint64_t)((i64_log2m(x.m, rc, lc) + 16) >> 5);
}

TP_HD double pell64(const PellNode64& N, const Pell64& p, const P64Cell* __restrict__ ptab, const I64Tables& t) {
  // T17: (1 + c1 k^-a1)^a1 / (1 + c2 k^-a2)^a3
  constexpr uint64_t A1 = 0xa734d6a161e4f80ull, A2 = 0x92e147ae147ae00ull, A3 = 0x5060029f16b11c0ull;       // Q59, even
  constexpr int64_t LC1 = 331311853649588135ll, LC2 = 296516964452189038ll;  // log2 c1 + 64 a1, log2 c2 + 64 a2: Q52
  constexpr uint64_t L2E_4 = 0xb8aa3b295c17f0bcull, L2E_8 = 0xb8aa3b295c17f0bcull;  // log2(e)/4 = m 2^-65, /8 = m 2^-66
  const uint64_t lk = p.lgb + (uint64_t)N.l2fk, ly = lk + (uint64_t)N.l2rs;
  const Sf l = {p.m, p.e}, l3 = {p.m3, p.e3};
  const Sf P = p64_eval(ptab, p.lgb + (uint64_t)N.l2hf, t.ex2);
  const Sf pl = sf_norm(sf_mul(sf_mul({N.cpl, N.ecpl}, P), l3));
  const Sf y = sf_norm(sf_mul({N.ys, N.eys}, l)), y2 = sf_norm(sf_mul(y, y));
  // one-halo: a y^(3 f1) y^2 / ((1 + b y^f2 + (c f3 y)^(3 - gamma)) (y^2 + nu))
  const Sf e1 = i64_exp2(pell64_mul(ly, N.s1, N.n1) + N.k1, t.ex2);
  const Sf d1 = sf_add(sf_add(i64_exp2(pell64_mul(ly, N.s2, N.n2) + N.k2, t.ex2),
                              i64_exp2(pell64_mul(ly, N.s3, N.n3) + N.k3, t.ex2)),
                       sf_one());
  const Sf dh = sf_norm(sf_mul(sf_norm(d1), sf_add(y2, {N.xnu, N.exnu})));
  const Sf nh = sf_norm(sf_mul(e1, y2));
  // two-halo: pl (1 + pl)^beta / (1 + alpha pl) exp(-y/4 - y^2/8)
  const Sf g = sf_norm(sf_add(sf_mul(y, {L2E_4, -65}), sf_mul(y2, {L2E_8, -66})));
  const int64_t gq = g.e > -54 ? 1ll << 62 : (int64_t)i64_shr(g.m, -52 - g.e);  // Q52; 2^-1024 is nothing beside the other
  const uint64_t lp = sf_log2(sf_add(pl, sf_one()), t.rc, t.lc);
  const Sf nq = sf_norm(sf_mul(pl, i64_exp2(pell64_mul(lp, N.be, N.nb) - gq, t.ex2)));
  const Sf dq = sf_norm(sf_add(sf_mul({N.al, N.eal}, pl), sf_one()));
  const Sf num = sf_norm(sf_add(sf_mul(nq, dh), sf_mul(nh, dq)));
  const uint64_t l1 = sf_log2(sf_add(i64_exp2(LC1 - (int64_t)i64_mulhi(lk, A1), t.ex2), sf_one()), t.rc, t.lc);
  const uint64_t l2 = sf_log2(sf_add(i64_exp2(LC2 - (int64_t)i64_mulhi(lk, A2), t.ex2), sf_one()), t.rc, t.lc);
  const Sf c = i64_exp2((int64_t)i64_mulhi(l1, A1) - (int64_t)i64_mulhi(l2, A3), t.ex2);
  const Sf q = sf_mul(sf_mul(num, c), sf_rcp(sf_mul(sf_norm(sf_mul(dh, dq)), l3)));
  return N.w * sf_to(q);
}

}  // namespace tp
