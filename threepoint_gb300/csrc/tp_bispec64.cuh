// The BiHalofit bispectrum of one line-of-sight node (bispec_eval in
// tp_bispec.cuh, Takahashi et al. 2020 Eqs. B4-B9) in the 64-bit integer
// arithmetic of tp_i64.cuh: what the FP64 integrands evaluate.
//
// Why: a node evaluated with FP64 instructions takes about 850 of them (17
// exp2 and 6 log2 of CUDA's FP64 library, 19 divisions), which the FP64 pipe
// (1.6 lanes per clock and SM) bounds at 5.9e8 nodes/s, measured. Here the
// base-2 exponents are fixed point, the factors positive 64-bit-mantissa
// numbers, and 18 FP64 operations are left (the signed tree-level factors and
// the last products), issued beside the integer instructions. P_lin is read
// from a table of log2 P with 128 fifth-order cells per octave; its error and
// that of every step is below the rounding of the FP64 form, which the tests
// measure against long double. Measured (GB300): 2^18 b_kappa points 42.5 ->
// 2.62 ms (9.6e9 nodes/s, about 2500 integer issue slots a node), the ten
// <Map^3> integrals of radii {4, 8, 16}' 608 -> 70 ms, of which ~35 ms are the
// reference passes of the cubature (tp_cubature.cuh), a T4 entry 2.25 -> 0.29 s.
//
// Domain: rows, triangles and cosmologies whose exponents fit the fixed-point
// fields (Node64::ok, Tri64::ok, Cosmo64::ok); everything else (a tabulated
// P(k), z > 10, non-finite coefficients, ell outside the P table) keeps the
// FP64 form.
#pragma once
#include "tp_i64.cuh"

namespace tp {

// cells of the log2 P_lin table: log2(k h) on [P64_LO, P64_HI)
constexpr int P64_PER_OCTAVE = 128, P64_LO = -32, P64_HI = 24;
constexpr int P64_N = (P64_HI - P64_LO) * P64_PER_OCTAVE;

// 4 log2(k h) - log2 P over one cell, T in [0, 1): c0 + T (c1 + T v2),
// v2 = c2 + T (c3 + T (c4 + T c5)); the slope 4 - dlnP/dlnk is positive
struct alignas(16) P64Cell {
  int64_t c0;          // Q52
  uint64_t c1, c2;     // Q64; c2 holds c2 + 2^-12
  int32_t c3, c4, c5;  // Q51, Q52, Q53
  int32_t pad[3];
};
static_assert(sizeof(P64Cell) == 48, "read as three 16-byte loads");

struct Cosmo64 {
  const P64Cell* p;  // [P64_N]
  uint64_t amax;     // 1 - 2/3 n_s, Q59
  double lo, hi;     // ell range whose P table coordinates lie inside at every node
  int ok, bad;       // usable; a P table cell does not fit (set by the table build)
};

struct Node64 {
  int64_t l2s, l2hf;          // log2 s, log2(h / f_K): Q57
  uint64_t anc, ald;          // Q59
  int64_t l2anr, ana, ala;    // Q52
  uint64_t betab;             // Q60
  int64_t l2bn;               // Q52
  uint64_t mun, nun;          // Q59
  int64_t kmn, knn;           // log2 m_n - 64 mu_n, log2 n_n - 64 nu_n: Q52, modulo 2^64 as the exponents' sums are
  uint64_t cns, cns3, fn, d1, hn, gn, pn3;        // mantissas: c_n s, its cube, D1^2 f_n s^2, D1^2, h_n s^2, g_n s, (p_n s)^3
  int ecns, ecns3, efn, ed1, ehn, egn, epn3;      // and exponents
  int ok;
  double w, dns, ens;         // weight, d_n s, e_n s
};

struct Tri64 {
  struct Side {
    uint64_t lgb;        // log2 ell + 64, Q57
    uint64_t m, m2, m3;  // ell, ell^2, ell^3
    int e, e2, e3, pad;
  } s[3];
  uint64_t nlr;   // -log2 r1, Q57
  uint64_t r2;    // r2^2, Q57
  uint64_t pr2;   // 10^(0.007 r2), Q63
  uint64_t lp;    // ell1 ell2 ell3
  int elp, ok;
  double f2t[3];
};

// log2 of a positive normal double in [2^-64, 2^64), Q57, within 2^-57
TP_HD int64_t i64_log2(double x, const I64Tables& t) {
  const Sf a = sf_from(x);
  return (int64_t)(((uint64_t)(a.e + 63) << 57) + (uint64_t)((i64_log2m(a.m, t.rc, t.lc) + 16) >> 5));
}
// of any positive normal double, in units of 2^-(57 - SH)
template <int SH>
TP_HD int64_t i64_log2_sh(double x, const I64Tables& t) {
  const Sf a = sf_from(x);
  return (int64_t)((uint64_t)(int64_t)(a.e + 63) << (57 - SH)) + ((i64_log2m(a.m, t.rc, t.lc) + 16) >> (5 + SH));
}
TP_HD int64_t i64_log2_q52(double x, const I64Tables& t) { return i64_log2_sh<5>(x, t); }

// triangle (ell1, ell2, ell3); f2t = F2_tree(1,2,3), (2,3,1), (3,1,2). Returns
// ok: every ell inside [lo, hi] (and so inside the fixed-point range)
TP_HD bool tri64_make(double l1, double l2, double l3, const double* f2t, double lo, double hi, const I64Tables& t,
                      Tri64& T) {
  const double l[3] = {l1, l2, l3};
  double a = l1, b = l2, c = l3, x;
  if (a < b) { x = a; a = b; b = x; }
  if (a < c) { x = a; a = c; c = x; }
  if (b < c) { x = b; b = c; c = x; }
  for (int i = 0; i < 3; ++i) T.f2t[i] = f2t[i];
  T.ok = c >= lo && a <= hi;
  if (!T.ok) return false;
  uint64_t gmax = 0, gmin = ~0ull;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint64_t g = (uint64_t)i64_log2(l[i], t) + (64ull << 57);
    gmax = g > gmax ? g : gmax;
    gmin = g < gmin ? g : gmin;
    const Sf s = sf_from(l[i]), s2 = sf_norm(sf_mul(s, s)), s3 = sf_norm(sf_mul(s2, s));
    T.s[i].lgb = g;
    T.s[i].m = s.m, T.s[i].e = s.e;
    T.s[i].m2 = s2.m, T.s[i].e2 = s2.e;
    T.s[i].m3 = s3.m, T.s[i].e3 = s3.e;
  }
  T.nlr = gmax - gmin;
  const double r2 = (b + c - a) / a;
  T.r2 = (uint64_t)i64_fix<57>(r2 * r2);
  const Sf p = i64_exp2(i64_fix<52>(0.007 * 3.32192809488736234787 * r2), t.ex2);
  T.pr2 = i64_shr(p.m, -63 - p.e);
  const Sf lp = sf_norm(sf_mul(sf_norm(sf_mul({T.s[0].m, T.s[0].e}, {T.s[1].m, T.s[1].e})), {T.s[2].m, T.s[2].e}));
  T.lp = lp.m;
  T.elp = lp.e;
  return true;
}

TP_HD bool sf_ok(double c) { return c > 1e-280 && c < 1e280; }
TP_HD bool q59_ok(double c) { return c >= 0 && c < 15.9; }
// a c q^m whose base-2 exponent stays inside Q52 over the node's whole range of log2 q (-63 to 63)
TP_HD bool pow_ok(double c, double m) { return sf_ok(c) && m >= 0 && fabs(log2(c)) + 63 * m < 2040; }

// node row from the FP64 coefficients (NC_* values)
TP_HD void node64_make(double w, double s, double hf, double ana, double anr, double anc, double bn, double cn,
                       double ala, double ald, double betab, double fn, double gn, double hn, double mn, double nn,
                       double mun, double nun, double pn, double en, double dn, double d1sq, bool tree,
                       const I64Tables& t, Node64& N) {
  N.w = w;
  N.dns = dn * s;
  N.ens = en * s;
  const double pns = pn * s, cns = cn * s, f = d1sq * fn * s * s, h = hn * s * s, g = gn * s;
  N.ok = !tree && s > 0x1p-27 && s < 0x1p36 && hf > 0x1p-60 && hf < 0x1p60 && sf_ok(anr) && anr < 16 && q59_ok(anc) &&
         q59_ok(ald) && betab >= 0 && betab < 15.5 && mun < 31.9 && nun < 31.9 && pow_ok(bn, betab * 1.017) && pow_ok(mn, mun) &&
         pow_ok(nn, nun) && fabs(ana) < 900 && fabs(ala) < 900 && sf_ok(cns) && cns > 1e-80 && cns < 1e80 && sf_ok(f) && sf_ok(d1sq) &&
         sf_ok(h) && sf_ok(g) && pns > 1e-80 && pns < 1e80;
  if (!N.ok) return;
  N.l2s = i64_log2(s, t);
  N.l2hf = i64_log2(hf, t);
  N.anc = (uint64_t)i64_fix<59>(anc);
  N.ald = (uint64_t)i64_fix<59>(ald);
  N.l2anr = i64_log2_q52(anr, t);
  N.ana = i64_fix<52>(ana);
  N.ala = i64_fix<52>(ala);
  N.betab = (uint64_t)i64_fix<60>(betab * 0.5) << 1;
  N.l2bn = i64_log2_q52(bn, t);
  N.mun = (uint64_t)i64_fix<58>(mun) << 1;
  N.nun = (uint64_t)i64_fix<58>(nun) << 1;
  N.kmn = (int64_t)((uint64_t)i64_log2_q52(mn, t) - (N.mun >> 1));
  N.knn = (int64_t)((uint64_t)i64_log2_q52(nn, t) - (N.nun >> 1));
  Sf v = sf_from(cns);
  N.cns = v.m, N.ecns = v.e;
  v = sf_norm(sf_mul(sf_norm(sf_mul(v, v)), v));
  N.cns3 = v.m, N.ecns3 = v.e;
  v = sf_from(f);
  N.fn = v.m, N.efn = v.e;
  v = sf_from(d1sq);
  N.d1 = v.m, N.ed1 = v.e;
  v = sf_from(h);
  N.hn = v.m, N.ehn = v.e;
  v = sf_from(g);
  N.gn = v.m, N.egn = v.e;
  v = sf_from(pns);
  v = sf_norm(sf_mul(sf_norm(sf_mul(v, v)), v));
  N.pn3 = v.m, N.epn3 = v.e;
}

// one cell of the P table from the Eisenstein & Hu fit (plin in
// tp_bispec.cuh): the polynomial through six points, the rapidly varying
// power law and all logarithms in fixed point. False when a coefficient is
// outside its field (no cosmology of Omega_m 0.05-1, h 0.4-1.2, n_s 0.5-1.4
// comes within a factor 1.5 of that).
TP_HD bool p64_cell(int i, double omh2, double sa, double one_m_sa, double sh043, double theta2, double c184,
                    double ehc, double ns, const I64Tables& t, P64Cell& c) {
  // Chebyshev points of [0, 1], in 1/65536
  const int tk[6] = {1117, 9598, 24287, 41249, 55938, 64419};
  double x[6], d[6];
  int64_t y0 = 0;
  const int64_t l0 = (int64_t)((uint64_t)P64_LO << 57) + ((int64_t)i << 50);
  // log2 P within +-512 (Q51 of eight times it)
  if (!(fabs(log2(ehc)) < 80)) return false;
  const int64_t lehc = i64_log2_sh<3>(ehc, t), nsq = i64_fix<56>(ns);
  for (int k = 0; k < 6; ++k) {
    const int64_t lk = l0 + ((int64_t)tk[k] << 34);  // log2(k h), Q57
    const double kk = sf_to(i64_exp2(lk >> 5, t.ex2));
    const double xx = kk * sh043, x2 = xx * xx;
    const double geff = omh2 * (sa + one_m_sa / (1.0 + x2 * x2));
    const double q = kk * theta2 / geff;
    const double L = log(2.718281828 + c184 * q);
    const double C = 14.4 + 325.0 / (1.0 + 60.5 * exp2(1.11 * log2(q)));
    const double r = L / (L + C * q * q);
    if (!(r > 0x1p-100)) return false;
    // n_s log2 k in Q54 from Q57 and Q56
    const uint64_t al = (uint64_t)(lk < 0 ? -lk : lk), an = (uint64_t)(nsq < 0 ? -nsq : nsq);
    int64_t pw = (int64_t)(i64_mulhi_exact(al, an) << 5) + (int64_t)((al * an) >> 59);
    if ((lk < 0) != (nsq < 0)) pw = -pw;
    const int64_t y = (lk >> 1) - lehc - pw - i64_log2_sh<2>(r, t);  // Q51
    if (k == 0) y0 = y;
    x[k] = tk[k] * 0x1p-16;
    d[k] = (double)(y - y0) * 0x1p-54;
  }
  for (int j = 1; j < 6; ++j)  // divided differences
    for (int k = 5; k >= j; --k) d[k] = (d[k] - d[k - 1]) / (x[k] - x[k - j]);
  double p[6] = {d[5], 0, 0, 0, 0, 0};  // to powers of T
  for (int j = 4; j >= 0; --j) {
    for (int k = 5 - j; k > 0; --k) p[k] = p[k - 1] - x[j] * p[k];
    p[0] = d[j] - x[j] * p[0];
  }
  if (!(p[1] > 0 && p[1] < 0.49 && fabs(p[2]) < 0x1p-12 && fabs(p[3]) < 0x1p-20 && fabs(p[4]) < 0x1p-21 &&
        fabs(p[5]) < 0x1p-22))
    return false;
  c.c0 = ((y0 + 2) >> 2) + i64_fix<52>(p[0]) + (256ll << 52);
  c.c1 = (uint64_t)i64_fix<62>(p[1]) << 2;
  c.c2 = (uint64_t)(i64_fix<64>(p[2] + 0x1p-12));
  c.c3 = (int32_t)i64_fix<51>(p[3]);
  c.c4 = (int32_t)i64_fix<52>(p[4]);
  c.c5 = (int32_t)i64_fix<53>(p[5]);
  c.pad[0] = c.pad[1] = c.pad[2] = 0;
  return true;
}

// P_lin at biased log2(k h) + 64 (Q57)
TP_HD Sf p64_eval(const P64Cell* __restrict__ tab, uint64_t lkb, const uint64_t* __restrict__ ex2) {
  const int i = (int)(lkb >> 50) - (64 + P64_LO) * P64_PER_OCTAVE;
#if defined(__CUDA_ARCH__)
  const uint4* q = reinterpret_cast<const uint4*>(tab + i);
  const uint4 qa = __ldg(q), qb = __ldg(q + 1), qc = __ldg(q + 2);
  P64Cell c;
  c.c0 = (int64_t)(((uint64_t)qa.y << 32) | qa.x);
  c.c1 = ((uint64_t)qa.w << 32) | qa.z;
  c.c2 = ((uint64_t)qb.y << 32) | qb.x;
  c.c3 = (int32_t)qb.z, c.c4 = (int32_t)qb.w, c.c5 = (int32_t)qc.x;
#else
  const P64Cell c = tab[i];
#endif
  const uint64_t r = lkb << 14;                // T, Q64
  const int32_t t = (int32_t)(lkb >> 19) & 0x7fffffff;  // T, Q31
  const int32_t s4 = c.c4 + (int32_t)(((int64_t)t * c.c5) >> 32);   // Q52
  const int32_t s3 = c.c3 + (int32_t)(((int64_t)t * s4) >> 32);     // Q54
  const uint64_t v2 = c.c2 + (uint64_t)(((int64_t)t * s3) >> 18);   // Q64, + 2^-12
  const uint64_t w = c.c1 - (r >> 12) + i64_mulhi(r, v2);
  const int64_t h = c.c0 + (int64_t)(i64_mulhi(r, w) >> 12);
  return i64_exp2((int64_t)(lkb >> 3) - h, ex2);
}

// a_n, alpha_n, beta_n of a triangle shape (B7) as the exponents' coefficients
// and offsets: 2^ka (64 q)^al = a_n q^al
struct Shape64 {
  uint64_t al, be;  // Q59
  uint64_t ka, kb;  // Q52, modulo 2^64
};
TP_HD Shape64 shape64(const Node64& N, uint64_t nlr, uint64_t r2, uint64_t pr2, uint64_t amax,
                      const uint64_t* __restrict__ ex2) {
  Shape64 h;
  const Sf sa = i64_exp2(N.l2anr - (int64_t)i64_mulhi(nlr, N.anc), ex2);
  const int64_t l2an = N.ana - (int64_t)i64_shr(sa.m, -52 - sa.e);
  const Sf sl = i64_exp2(N.ala + (int64_t)i64_mulhi(r2, N.ald), ex2);
  const uint64_t al = sl.e < -63 ? i64_shr(sl.m, -59 - sl.e) : ~0ull;
  h.al = al < amax ? al : amax;
  h.be = i64_mulhi(N.betab, pr2);
  h.ka = (uint64_t)l2an - (h.al >> 1);
  h.kb = (uint64_t)N.l2bn - (h.be >> 1);
  return h;
}

// B of one node (weight not applied) for a triangle shape and its sides:
// S.side(i, lgb, l, l2, l3) gives side i, S.product() ell1 ell2 ell3
template <class S>
TP_HD double bispec64_core(const Node64& N, const Shape64& h, const S& src, const double* f2t,
                           const P64Cell* __restrict__ ptab, const uint64_t* __restrict__ ex2) {
  Sf den1 = sf_one();
  double P[3], f[3], e3 = 1.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint64_t lgb;
    Sf l, l2, l3;
    src.side(i, lgb, l, l2, l3);
    const uint64_t lq = lgb + (uint64_t)N.l2s;
    // 1-halo denominators (B4)
    const Sf d = sf_add(i64_exp2((int64_t)(i64_mulhi(lq, h.al) + h.ka), ex2), i64_exp2((int64_t)(i64_mulhi(lq, h.be) + h.kb), ex2));
    const Sf cq1 = sf_add(sf_mul({N.cns, N.ecns}, l), sf_one());
    den1 = sf_norm(sf_mul(den1, sf_mul(d, cq1)));
    // 3-halo side (B5, B9) over the common denominator
    const Sf num = sf_add(sf_mul({N.fn, N.efn}, l2), {N.d1, N.ed1});
    const Sf den = sf_add(sf_add(sf_mul({N.hn, N.ehn}, l2), sf_mul({N.gn, N.egn}, l)), sf_one());
    const Sf x3 = sf_mul({N.pn3, N.epn3}, l3);
    const Sf mq = sf_add(i64_exp2((int64_t)(i64_mulhi(lq, N.mun) + (uint64_t)N.kmn), ex2),
                         i64_exp2((int64_t)(i64_mulhi(lq, N.nun) + (uint64_t)N.knn), ex2));
    const Sf M = sf_norm(sf_mul(mq, sf_add(x3, sf_one())));
    const Sf pl = p64_eval(ptab, lgb + (uint64_t)N.l2hf, ex2);
    const Sf nm = sf_add(sf_mul(x3, den), sf_mul(sf_mul(num, pl), M));
    P[i] = sf_to(sf_mul(nm, sf_rcp(sf_mul(den, M))));
    const double ld = sf_to(l);
    f[i] = fma(N.dns, ld, f2t[i == 2 ? 0 : i + 1]);
    e3 *= fma(N.ens, ld, 1.0);
  }
  const double b1 = sf_to(sf_mul(sf_mul({N.cns3, N.ecns3}, src.product()), sf_rcp(den1)));
  // F2 of the pairs (0,1), (1,2), (2,0): f[2], f[0], f[1]
  double b3 = f[2] * (P[0] * P[1]);
  b3 = fma(f[0], P[1] * P[2], b3);
  b3 = fma(f[1], P[2] * P[0], b3);
  return fma(2.0 * b3, sf_to(sf_rcp(sf_from(e3))), b1);
}

struct TriSides64 {
  const Tri64& T;
  TP_HD void side(int i, uint64_t& lgb, Sf& l, Sf& l2, Sf& l3) const {
    const Tri64::Side& S = T.s[i];
    lgb = S.lgb;
    l = {S.m, S.e}, l2 = {S.m2, S.e2}, l3 = {S.m3, S.e3};
  }
  TP_HD Sf product() const { return {T.lp, T.elp}; }
};

// T.ok, N.ok and the cosmology's ok hold
TP_HD double bispec64(const Node64& N, const Tri64& T, const Cosmo64& C, const uint64_t* __restrict__ ex2) {
  return bispec64_core(N, shape64(N, T.nlr, T.r2, T.pr2, C.amax, ex2), TriSides64{T}, T.f2t, C.p, ex2);
}

}  // namespace tp
