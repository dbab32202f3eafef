// Natural components Gamma^0..Gamma^3 of the shear three-point correlation
// function: 3-D adaptive cubature over (z, phi, psi) of the Ogata Hankel sum
// of the BiHalofit convergence bispectrum at redshift z.
//
// Reference: gamma0..gamma3 (cuda_version/gamma.cu:98-148), the integrands
// full_integrand_gamma0/1 and one_integrand_gamma0 (:419-482), the triangle
// geometry interior_angle, A, alpha, betabar, prefactor (:484-529), the Ogata
// nodes of compute_weights_bessel (:13-68) and the orthocentre-to-centroid
// rotation (:72-96; CONVERT_TO_CENTROID, gamma.cuh:25).
//
// One job = (triangle, component). A point record holds the z-only BiHalofit
// coefficients of its redshift, the unit triangle shape (cos psi, sin psi,
// ...) and per cyclic term j the scale A_j and complex weight C_j; a
// (point, group) item evaluates 4 Ogata nodes x 3 terms = 12 bispectra.
#include <cuda_runtime.h>

#include <type_traits>

// resident CTAs per SM requested for the FP32 Gamma kernel (2: <= 128
// registers per thread; 1: no register cap, one CTA per SM)
#ifndef TP_GAMMA_MINB
#define TP_GAMMA_MINB 2
#endif

#include <algorithm>
#include <cmath>
#include <complex>
#include <string>
#include <vector>

#include "tp_bispec.cuh"
#include "tp_capi_internal.h"
#include "tp_cubature.cuh"
#include "tp_internal.cuh"
#include "tp_kernels.cuh"

namespace tp {

constexpr int PREC_K = 33;       // int(3.31/0.1) Ogata nodes (index 0 unused), gamma.cuh:29-30
constexpr double PREC_H = 0.1;

struct OgataTab {
  double psi[2][PREC_K], prod[2][PREC_K], l2psi[2][PREC_K];  // [0]: J6 (Gamma0), [1]: J2 (Gamma1)
};
__constant__ OgataTab c_og;

// zeros of J_nu by Newton iteration from McMahon's expansion (s >= 1); s = 0 -> 0
static double bessel_zero(int nu, int s) {
  if (s == 0) return 0.0;
  double mu = 4.0 * nu * nu;
  double b = (s + 0.5 * nu - 0.25) * PI;
  double x = b - (mu - 1) / (8 * b) - 4 * (mu - 1) * (7 * mu - 31) / (3 * pow(8 * b, 3));
  if (s == 1) x = nu + 1.8557571 * cbrt((double)nu) + 1.033150 / cbrt((double)nu);
  for (int it = 0; it < 100; ++it) {
    double J = std::cyl_bessel_j((double)nu, x);
    double dJ = 0.5 * (std::cyl_bessel_j((double)nu - 1, x) - std::cyl_bessel_j((double)nu + 1, x));
    double dx = J / dJ;
    x -= dx;
    if (fabs(dx) < 1e-15 * x) break;
  }
  return x;
}

static void ogata_host(OgataTab& o) {
  for (int pass = 0; pass < 2; ++pass) {
    int nu = pass == 0 ? 6 : 2;
    for (int i = 0; i < PREC_K; ++i) {
      double zr = bessel_zero(nu, i), pz = zr / PI;
      double t = pz * PREC_H;
      double psi = PI * (t * tanh(PI * sinh(t) / 2)) / PREC_H;
      double psip = (sinh(PI * sinh(t)) + PI * t * cosh(t)) / (cosh(PI * sinh(t)) + 1);
      double Jn1 = i == 0 ? 0.0 : std::cyl_bessel_j((double)nu + 1, zr);
      double w = 2 / (PI * zr * Jn1 * Jn1);
      o.psi[pass][i] = psi;
      o.prod[pass][i] = i == 0 ? 0.0 : w * psi * psi * psi * std::cyl_bessel_j((double)nu, psi) * psip;
      o.l2psi[pass][i] = i == 0 ? 0.0 : log2(psi);
    }
  }
}

cudaError_t gamma_upload_constants() {
  static OgataTab o;
  static bool built = false;
  if (!built) {
    ogata_host(o);
    built = true;
  }
  return cudaMemcpyToSymbol(c_og, &o, sizeof(o));
}

// geometry (gamma.cu:491-529), double precision
__host__ __device__ inline double interior_angle(double an1, double an2, double opp) {
  return acos((an1 * an1 + an2 * an2 - opp * opp) / (2.0 * an1 * an2));
}
__host__ __device__ inline double height_of_triangle(double x1, double x2, double x3) {
  return 0.5 * sqrt(2 * x1 * x1 + 2 * x2 * x2 - x3 * x3);
}
__host__ __device__ inline double one_rotation_angle_otc(double x1, double x2, double x3) {
  double psi3 = interior_angle(x1, x2, x3);
  double h3 = height_of_triangle(x1, x2, x3);
  double d = x2 * x2 - x1 * x1;
  double s = x1 * x2 * sin(psi3);
  double c2 = (d * d - 4 * s * s) / ((2 * h3 * x3) * (2 * h3 * x3));
  double s2 = d * x1 * x2 * sin(psi3) / ((h3 * x3) * (h3 * x3));
  return atan2(s2, c2) / 2;
}

struct GammaJobs {
  const double* x;  // [n_tri][3]
  const int* comp;  // [n_jobs]
  const int* tri;   // [n_jobs]
};

template <typename R>
struct GammaPolicy {
  static constexpr int G = 8;     // groups of 4 Ogata nodes
  static constexpr int KPG = 4;
  static constexpr int CH = 4;    // regions per chunk (records are large)
  // FP64: the per-point node coefficients; FP32: the folded NF_* row
  // (bispec_fast_row), an odd number of words (57) per record
  struct RefD {
    double zc[NC_COUNT];
    Tri<double> tri;  // unit-scale triangle (cos psi, sin psi, ell3/psi_k)
    double invA[3], l2A[3];
    double cre[3], cim[3];
    double bmin;
    int live;
  };
  struct FastD {
    Node64 N;
    Shape64 h;
    uint64_t lgb[3], m[3], lp;  // log2 ell + 64 (Q57), mantissas of ell_i and ell1 ell2 ell3 at unit scale
    int e[3], elp;
    double f2t[3];
    int64_t l2ia[3];  // log2 (1 / A_j), Q57
    uint64_t iam[3];  // 1 / A_j
    int iae[3], pad;
    double cre[3], cim[3];
  };
  // FP64: the integer-arithmetic form, or (f64form) the FP64 instructions'; 59
  // 64-bit words, conflict-free across lanes
  struct RecD {
    union {
      FastD f;
      RefD d;
    };
    int live, f64form;
  };
  struct RecF {
    float nf[NCP];
    TriF tri;
    float invA[3], l2A[3];
    float cre[3], cim[3];
    float bmin;
    int live;
  };
  typedef typename std::conditional<sizeof(R) == 4, RecF, RecD>::type Rec;
  static constexpr int REC = (int)sizeof(Rec);
  const int* job_order = nullptr;
  static constexpr int PD = 2;
  static constexpr int NS = 1;
  __device__ static int slot(int) { return 0; }
  // the set-up below and its reference form (the trigonometric one) decide
  // together where the cubature cuts between tied regions
  static constexpr bool REF = true;
  int ref = 0, one = 0;
  // per job: sides and half interior angle of term j, its constant phase
  struct Term {
    double a, b, ch, sh, ce, se;
  };
  static constexpr size_t EX2_BYTES = sizeof(R) == 8 ? sizeof(I64Tables::ex2) : 0;
  static constexpr size_t PSMEM = EX2_BYTES + sizeof(CosmoK<R>) + 3 * sizeof(Term) + 64;
  const uint64_t* s_ex2;
  Term* s_term;

  GammaJobs J;
  const TablesDev* tab;
  const CosmoDev* cosm;
  const CosmoK<R>* ck;
  int cosmo;
  double* out;  // [n_tri][4][2]
  int* status;  // [n_tri]
  // per-job state
  CosmoK<R>* s_ck;
  int which;                      // 0: Gamma0 integrand, 1: Gamma1 integrand
  double x1, x2, x3;              // sides passed to the integrand (permuted for Gamma2/3)
  double vp[3], ph0[3];           // Gamma0: varpsi_j, constant phase of term j
  double p1, p2, p3;              // Gamma1: interior angles
  double zmax;

  __device__ void begin_job(int job, char* psmem, double* xmin, double* xmax) {
    s_ex2 = (const uint64_t*)psmem;
    s_term = (Term*)(psmem + EX2_BYTES);
    s_ck = (CosmoK<R>*)(psmem + EX2_BYTES + 3 * sizeof(Term));
    if (threadIdx.x == 0) *s_ck = ck[cosmo];
    if constexpr (sizeof(R) == 8) {
      for (int i = threadIdx.x; i < 256; i += blockDim.x) ((uint64_t*)psmem)[i] = d_i64tab.ex2[i];
    }
    const int t = J.tri[job], c = J.comp[job];
    double a = J.x[3 * t], b = J.x[3 * t + 1], d = J.x[3 * t + 2];
    which = c == 0 ? 0 : 1;
    if (c <= 1) {
      x1 = a, x2 = b, x3 = d;
    } else if (c == 2) {
      x1 = b, x2 = d, x3 = a;  // gamma2 = gamma1(x2, x3, x1)
    } else {
      x1 = d, x2 = a, x3 = b;  // gamma3 = gamma1(x3, x1, x2)
    }
    const double xs[3][3] = {{x1, x2, x3}, {x2, x3, x1}, {x3, x1, x2}};
    for (int j = 0; j < 3; ++j) {
      vp[j] = interior_angle(xs[j][0], xs[j][1], xs[j][2]);
      ph0[j] = interior_angle(xs[j][1], xs[j][2], xs[j][0]) - interior_angle(xs[j][0], xs[j][2], xs[j][1]);
    }
    p1 = interior_angle(x2, x3, x1);
    p2 = interior_angle(x3, x1, x2);
    p3 = interior_angle(x1, x2, x3);
    if (threadIdx.x < 3) {
      const int j = threadIdx.x;
      Term t;
      if (which == 0) {
        t.a = xs[j][0], t.b = xs[j][1];
        sincos(0.5 * vp[j], &t.sh, &t.ch);
        sincos(ph0[j], &t.se, &t.ce);
      } else {
        t.a = xs[(j + 1) % 3][0], t.b = xs[(j + 1) % 3][1];
        sincos(0.5 * (j == 0 ? p1 : j == 1 ? p2 : p3), &t.sh, &t.ch);
        sincos(j == 0 ? p3 - p2 : j == 1 ? p3 - p1 - 2 * p2 : p1 - p2 + 2 * p3, &t.se, &t.ce);
      }
      s_term[j] = t;
    }
    if constexpr (sizeof(R) == 8) {
      const CosmoK<double>& K = ck[cosmo];
      one = !(K.c64.ok && K.n64[0].ok);
    }
    zmax = cosm[cosmo].zmax;
    xmin[0] = 0;
    xmin[1] = 0;
    xmin[2] = 0;
    xmax[0] = zmax;
    xmax[1] = 2 * PI;
    xmax[2] = PI / 2;
    __syncthreads();
  }

  __device__ bool is_live(const char* recp) const { return ((const Rec*)recp)->live != 0; }

  // the reference form's point: the angles of gamma.cu:419-529 themselves; a
  // function of its own, so that what the compiler contracts in it does not
  // depend on the fast form
  template <class Q>
  __device__ __noinline__ bool setup_ref(const double* x, Q& q) const {
    const double z = x[0], phi = x[1], psi = x[2];
    if constexpr (sizeof(R) == 4) {
      float zc[NC_COUNT];
      q.live = zcoefs<float>(tab[cosmo], cosm[cosmo], z, zc);
      if (q.live) nf_from_nc(zc, q.nf);
    } else {
      q.live = zcoefs<R>(tab[cosmo], cosm[cosmo], z, q.zc);
    }
    if (!q.live) return false;
    // the geometry is evaluated in double: a few dozen operations per point
    // against 96 bispectra
    double cp = cos(psi), sp = sin(psi), s2p = sin(2 * psi), c2p = cos(2 * psi);
    double cph = cos(phi), sph = sin(phi);
    double bb = 0.5 * atan2(c2p * sph, cph + s2p);  // betabar, gamma.cu:524-529
    double b3s = cp * cp + sp * sp + 2 * cp * sp * cph;
    double b3 = b3s <= 0 ? 0.0 : sqrt(b3s);
    q.bmin = (R)fmin(cp, fmin(sp, b3));
    if (!(b3 > 0 && cp > 0 && sp > 0)) {
      q.live = 0;
      return false;
    }
    if constexpr (sizeof(R) == 4) {
      Tri<float> t;
      make_tri_phi_f((float)cp, (float)sp, (float)cph, (float)b3, t);
      trif_from_tri(t, q.tri);
    } else {
      make_tri<R>(cp, sp, b3, q.tri);
    }
    if (which == 0) {
      const double xs[3][2] = {{x1, x2}, {x2, x3}, {x3, x1}};
      for (int j = 0; j < 3; ++j) {
        double a = xs[j][0], b = xs[j][1];
        double ang = phi + vp[j];
        double A = sqrt((cp * b) * (cp * b) + (sp * a) * (sp * a) + s2p * a * b * cos(ang));
        double al = atan2((cp * b - sp * a) * sin(ang / 2), (cp * b + sp * a) * cos(ang / 2));
        double phase = ph0[j] - 6 * al + 2 * bb;
        double mag = s2p * PI / (A * A * A * A);
        q.invA[j] = (R)(1.0 / A);
        q.l2A[j] = (R)log2(A);
        q.cre[j] = (R)(mag * cos(phase));
        q.cim[j] = (R)(mag * sin(phase));
      }
    } else {
      // term order as full_integrand_gamma1: j=0 -> A1, 1 -> A2, 2 -> A3
      const double ab[3][2] = {{x2, x3}, {x3, x1}, {x1, x2}};
      const double vps[3] = {p1, p2, p3};
      double ph[3];
      double alv[3], Av[3];
      for (int j = 0; j < 3; ++j) {
        double a = ab[j][0], b = ab[j][1];
        double ang = phi + vps[j];
        Av[j] = sqrt((cp * b) * (cp * b) + (sp * a) * (sp * a) + s2p * a * b * cos(ang));
        alv[j] = atan2((cp * b - sp * a) * sin(ang / 2), (cp * b + sp * a) * cos(ang / 2));
      }
      ph[0] = p3 - p2 - 2 * (bb + alv[0]);
      ph[1] = p3 - p1 - 2 * p2 + 2 * (bb + phi - alv[1]);
      ph[2] = p1 - p2 + 2 * p3 + 2 * (bb - phi - alv[2]);
      for (int j = 0; j < 3; ++j) {
        double mag = s2p * PI / (Av[j] * Av[j] * Av[j] * Av[j]);
        q.invA[j] = (R)(1.0 / Av[j]);
        q.l2A[j] = (R)log2(Av[j]);
        q.cre[j] = (R)(mag * cos(ph[j]));
        q.cim[j] = (R)(mag * sin(ph[j]));
      }
    }
    return true;
  }

  __device__ bool setup(int p, const double* x, char* recp) {
    (void)p;
    Rec& r = *(Rec*)recp;
    if constexpr (sizeof(R) == 4) {
      return ref || one ? setup_ref(x, r) : setup_f32(x, r);
    } else {
      r.f64form = ref || one || !setup_f64(x, r);
      if (r.f64form) {
        const bool live = setup_ref(x, r.d);
        r.live = live;
      }
      return r.live;
    }
  }

  // The point geometry without inverse functions. With c, s = cos, sin of
  // phi/2, the side of term j is the complex number
  //   w = (cos psi b + sin psi a) cos(phi/2 + vp/2) + i (cos psi b - sin psi a) sin(phi/2 + vp/2),
  // |w| = A_j and arg w = alpha_j (gamma.cu:491-522), and betabar is -arg of
  //   v = (cos psi + sin psi) c + i (sin psi - cos psi) s,  |v| = ell3 / psi_k,
  // so every phase is a product of unit complex numbers. Two sincos and three
  // square roots are left of ~35 FP64 functions a point, which took 4/5 of the
  // FP32 form's time; A_j as a sum of squares does not cancel.
  struct Geo {
    double cp, sp, cph, b3;
    double A2[3], cre[3], cim[3], mag[3], k2[3];  // k2: (cos psi b + sin psi a)^2
    double b2;
  };
  __device__ __forceinline__ bool geometry(double phi, double psi, Geo& G) const {
    double c, s;
    if constexpr (sizeof(R) == 4) {  // on the integer pipe, for arguments in [0, 8)
      // (by the high words: no FP64 instructions; negative numbers and NaN fail)
      if ((uint32_t)__double2hiint(psi) >= 0x40200000u || (uint32_t)__double2hiint(phi) >= 0x40300000u) return false;
      int64_t qs, qc;
      i64_sincos(psi, d_i64sin, qs, qc);
      G.sp = i64_q62(qs), G.cp = i64_q62(qc);
      i64_sincos(0.5 * phi, d_i64sin, qs, qc);
      s = i64_q62(qs), c = i64_q62(qc);
    } else {
      sincos(psi, &G.sp, &G.cp);
      sincos(0.5 * phi, &s, &c);
    }
    const double cp = G.cp, sp = G.sp, s2p = 2 * sp * cp;
    const double vr = (cp + sp) * c, vi = (cp - sp) * s;  // conj v
    const double b2 = vr * vr + vi * vi;
    G.cph = 1 - 2 * s * s;
    G.b2 = b2;
    G.b3 = sqrt(b2);
    if (!(G.b3 > 0 && cp > 0 && sp > 0)) return false;
    const double ib2 = 1 / b2;
    const double ur = (vr * vr - vi * vi) * ib2, ui = 2 * vr * vi * ib2;  // e^(2 i betabar)
    const double fr = G.cph, fi = 2 * s * c;                             // e^(i phi)
    const double f2r = fr * fr - fi * fi, f2i = 2 * fr * fi;             // e^(2 i phi)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const Term& t = s_term[j];
      const double ca = c * t.ch - s * t.sh, sa = s * t.ch + c * t.sh;  // (phi + vp) / 2
      const double wr = (cp * t.b + sp * t.a) * ca, wi = (cp * t.b - sp * t.a) * sa;
      const double A2 = wr * wr + wi * wi, iA2 = 1 / A2;
      G.A2[j] = A2;
      G.k2[j] = (cp * t.b + sp * t.a) * (cp * t.b + sp * t.a);
      const double qr = (wr * wr - wi * wi) * iA2, qi = -2 * wr * wi * iA2;  // e^(-2 i alpha)
      double er, ei;
      if (which == 0) {
        // ph0 - 6 alpha + 2 betabar
        const double q2r = qr * qr - qi * qi, q2i = 2 * qr * qi;
        const double q3r = q2r * qr - q2i * qi, q3i = q2r * qi + q2i * qr;
        er = q3r * ur - q3i * ui;
        ei = q3r * ui + q3i * ur;
      } else {
        // j = 0: -2 (betabar + alpha); 1: 2 (betabar + phi - alpha); 2: 2 (betabar - phi - alpha)
        const double br = ur, bi = j == 0 ? -ui : ui;
        er = qr * br - qi * bi;
        ei = qr * bi + qi * br;
        if (j > 0) {
          const double gi = j == 1 ? f2i : -f2i, xr = er * f2r - ei * gi;
          ei = er * gi + ei * f2r;
          er = xr;
        }
      }
      const double mag = s2p * PI * iA2 * iA2;
      G.mag[j] = mag;
      G.cre[j] = mag * (er * t.ce - ei * t.se);
      G.cim[j] = mag * (er * t.se + ei * t.ce);
    }
    return true;
  }

  // the redshift and shape rows of a point as the reference form makes them
  static __device__ __noinline__ bool zrow_f32(const TablesDev& t, const CosmoDev& c, double z, float* nf) {
    float zc[NC_COUNT];
    const bool live = zcoefs<float>(t, c, z, zc);
    if (live) nf_from_nc(zc, nf);
    return live;
  }
  static __device__ __noinline__ void tri_f32(float cp, float sp, float cph, float b3, TriF& F) {
    Tri<float> t;
    make_tri_phi_f(cp, sp, cph, b3, t);
    trif_from_tri(t, F);
  }

  // The FP32 record rounds the geometry's doubles. Where a value lies so near
  // the middle of two floats that the rounding error of this geometry or of
  // the reference form's (which grows with the cancellation in A_j and betabar)
  // could reach it (i64_rounds_alike with that error in units of 2^-53), the
  // point takes the reference form, so that both make the same floats: ~1 point
  // in 3000.
  __device__ bool setup_f32(const double* x, RecF& r) const {
    Geo G;
    r.live = zrow_f32(tab[cosmo], cosm[cosmo], x[0], r.nf);
    if (!r.live) return false;
    if (!geometry(x[1], x[2], G)) return setup_ref(x, r);
    const double ib2 = 1 / G.b2;
    bool same = ib2 < 1e4 && i64_rounds_alike(G.cp, 1.0, 64) && i64_rounds_alike(G.sp, 1.0, 64) &&
                i64_rounds_alike(G.cph, 1.0, 64) && i64_rounds_alike(G.b3, 64 + (int)(16 * ib2));
    r.bmin = (float)fmin(G.cp, fmin(G.sp, G.b3));
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double A2 = G.A2[j], kap = G.k2[j] / A2;
      same = same && kap < 1e3 && A2 > 1e-60 && A2 < 1e60 &&
             (uint32_t)__double2hiint(G.mag[j]) > 0x39c00000u;  // 2^-99: cre, cim normal floats
      const int m = 128 + (int)(64 * fmin(kap, 1e3) + 16 * fmin(ib2, 1e4));
      const int64_t la = i64_log2(A2, d_i64tab) / 2;  // log2 A_j, Q57
      const double l2 = (double)la * 0x1p-57, ia = sf_to(i64_exp2(-(la >> 5), d_i64tab.ex2));
      same = same && i64_rounds_alike(ia, m) && i64_rounds_alike(l2, 2.0, m) && i64_rounds_alike(G.cre[j], G.mag[j], m) &&
             i64_rounds_alike(G.cim[j], G.mag[j], m);
      r.invA[j] = (float)ia;
      r.l2A[j] = (float)l2;
      r.cre[j] = (float)G.cre[j];
      r.cim[j] = (float)G.cim[j];
    }
    if (!same) return setup_ref(x, r);
    tri_f32((float)G.cp, (float)G.sp, (float)G.cph, (float)G.b3, r.tri);
    return true;
  }

  // false: outside the integer form's domain
  __device__ bool setup_f64(const double* x, RecD& r) const {
    FastD& f = r.f;
    const CosmoK<double>& K = *(const CosmoK<double>*)s_ck;
    r.live = 0;
    if (!zrow64(tab[cosmo], cosm[cosmo], K, x[0], s_ex2, f.N)) return true;
    if (!f.N.ok) return false;
    Geo G;
    if (!geometry(x[1], x[2], G)) return true;
    const double l[3] = {G.cp, G.sp, G.b3};
    f2_trees(G.cp, G.sp, G.b3, f.f2t);
    double a = l[0], b = l[1], c = l[2], t;
    if (a < b) { t = a; a = b; b = t; }
    if (a < c) { t = a; a = c; c = t; }
    if (b < c) { t = b; b = c; c = t; }
    if (!(c > 1e-12)) return false;
    int64_t lmin = 0, lmax = 0, amin = 0, amax = 0;
    Sf lp = sf_one();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int64_t g = i64_log2(l[i], d_i64tab);
      lmin = i == 0 || g < lmin ? g : lmin;
      lmax = i == 0 || g > lmax ? g : lmax;
      const Sf v = sf_from(l[i]);
      f.lgb[i] = (uint64_t)g + (64ull << 57);
      f.m[i] = v.m, f.e[i] = v.e;
      lp = sf_norm(sf_mul(lp, v));
      const double A2 = G.A2[i];
      if (!(A2 > 1e-60 && A2 < 1e60)) return false;
      const int64_t la = i64_log2(A2, d_i64tab) / 2;
      f.l2ia[i] = -la;
      amin = i == 0 || la < amin ? la : amin;
      amax = i == 0 || la > amax ? la : amax;
      const Sf ia = sf_norm(sf_from(1.0 / sqrt(A2)));
      f.iam[i] = ia.m, f.iae[i] = ia.e;
      f.cre[i] = G.cre[i], f.cim[i] = G.cim[i];
    }
    f.lp = lp.m, f.elp = lp.e;
    // every ell of the 96 evaluations inside the integer form's domain
    const double lo = (double)(lmin - amax) * 0x1p-57 + c_og.l2psi[which][1];
    const double hi = (double)(lmax - amin) * 0x1p-57 + c_og.l2psi[which][PREC_K - 1];
    const double hf = (double)f.N.l2hf * 0x1p-57, ss = (double)f.N.l2s * 0x1p-57;
    if (!(lo > -33.2 && hi < 40 && lo + hf > P64_LO + 0.01 && hi + hf < P64_HI - 0.01 && lo + ss > -63 && hi + ss < 63))
      return false;
    const double r2 = (b + c - a) / a;
    const Sf pr = i64_exp2(i64_fix<52>(LOG2_10 * 0.007 * r2), s_ex2);
    f.h = shape64(f.N, (uint64_t)(lmax - lmin), (uint64_t)i64_fix<57>(r2 * r2), i64_shr(pr.m, -63 - pr.e), K.c64.amax,
                  s_ex2);
    r.live = 1;
    return true;
  }

  // a point's triangle scaled by sc
  struct Scaled {
    const FastD& f;
    Sf sc;
    uint64_t l2sc;
    __device__ __forceinline__ void side(int i, uint64_t& lgb, Sf& l, Sf& l2, Sf& l3) const {
      lgb = f.lgb[i] + l2sc;
      l = sf_norm(sf_mul({f.m[i], f.e[i]}, sc));
      l2 = sf_norm(sf_mul(l, l));
      l3 = sf_norm(sf_mul(l2, l));
    }
    __device__ __forceinline__ Sf product() const {
      return sf_norm(sf_mul({f.lp, f.elp}, sf_norm(sf_mul(sf_norm(sf_mul(sc, sc)), sc))));
    }
  };

  // the reference form's group (FP64 instructions)
  static __device__ __noinline__ void group_ref(const RefD& r, int og, int g, const CosmoK<R>& K, double* pv) {
    KSum<R> are, aim;
    const R* zc = r.zc;
    const R s = zc[NC_S], l2s = zc[NC_L2S], hf = zc[NC_HF], l2hf = zc[NC_L2HF], W = zc[NC_W];
    for (int kk = 0; kk < KPG; ++kk) {
      const int k = 1 + g * KPG + kk;
      const R psik = (R)c_og.psi[og][k], l2psik = (R)c_og.l2psi[og][k], prodk = (R)c_og.prod[og][k];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        R sc = psik * r.invA[j];
        if (r.bmin * sc <= (R)1.0e-10) continue;  // integrand_bkappa: ell <= 1e-10 -> 0
        R l2sc = l2psik - r.l2A[j];
        R B = bispec_eval<R>(zc, 1, s * sc, l2s + l2sc, hf * sc, l2hf + l2sc, r.tri, K);
        R v = W * B;
        if (v != v) v = (R)0;  // NaN -> 0 (bispectrum.cu:327-331)
        v *= prodk;
        are.add(r.cre[j] * v);
        aim.add(r.cim[j] * v);
      }
    }
    pv[0] = (double)are.s;
    pv[1] = (double)aim.s;
  }

  __device__ void group(const char* recp, int g, double* pv) {
    const Rec& r = *(const Rec*)recp;
    typename std::conditional<sizeof(R) == 4, const CosmoK<R>, const CosmoK<R>&>::type K = *s_ck;
    const int og = which;
    KSum<R> are, aim;
    if constexpr (sizeof(R) == 4) {
      const float* c = r.nf;
      const float W = c[NF_W];
      for (int kk = 0; kk < KPG; ++kk) {
        const int k = 1 + g * KPG + kk;
        const float psik = (float)c_og.psi[og][k], l2psik = (float)c_og.l2psi[og][k], prodk = (float)c_og.prod[og][k];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float sc = psik * r.invA[j];
          if (r.bmin * sc <= 1.0e-10f) continue;  // integrand_bkappa: ell <= 1e-10 -> 0
          const TriF T = trif_scaled(r.tri, sc, l2psik - r.l2A[j]);
          float v = W * bispec_fast_row(c, T, K);
          if (v != v) v = 0.f;  // NaN -> 0 (bispectrum.cu:327-331)
          v *= prodk;
          are.add(r.cre[j] * v);
          aim.add(r.cim[j] * v);
        }
      }
    } else {
      if (r.f64form) return group_ref(r.d, og, g, K, pv);
      const FastD& f = r.f;
#pragma unroll 1
      for (int kk = 0; kk < KPG; ++kk) {
        const int k = 1 + g * KPG + kk;
        const Sf psi = sf_from(c_og.psi[og][k]);
        const uint64_t l2psi = (uint64_t)i64_fix<57>(c_og.l2psi[og][k]);
        const double wk = f.N.w * c_og.prod[og][k];
#pragma unroll 1
        for (int j = 0; j < 3; ++j) {
          const Scaled S = {f, sf_norm(sf_mul(psi, {f.iam[j], f.iae[j]})), l2psi + (uint64_t)f.l2ia[j]};
          double v = wk * bispec64_core(f.N, f.h, S, f.f2t, K.c64.p, s_ex2);
          if (v != v) v = 0;  // NaN -> 0 (bispectrum.cu:327-331)
          are.add(f.cre[j] * v);
          aim.add(f.cim[j] * v);
        }
      }
    }
    pv[0] = (double)are.s;
    pv[1] = (double)aim.s;
  }

  __device__ void finalize(const char* recp, const double* sum, double* fv) {
    const Rec& r = *(const Rec*)recp;
    fv[0] = r.live ? sum[0] : 0.0;
    fv[1] = r.live ? sum[1] : 0.0;
  }

  __device__ void end_job(int job, const double* V, const double* E, long long nev, int st) {
    (void)E;
    (void)nev;
    if (threadIdx.x != 0) return;
    const int t = J.tri[job], c = J.comp[job];
    double re = V[0], im = V[1];
    // orthocentre -> centroid (gamma.cu:83-91); Gamma1..3 conjugate phi1
    double a1 = one_rotation_angle_otc(x2, x3, x1), a2 = one_rotation_angle_otc(x3, x1, x2),
           a3 = one_rotation_angle_otc(x1, x2, x3);
    if (c != 0) a1 = -a1;
    double ang = -2. * (a1 + a2 + a3);
    double cr = re * cos(ang) - im * sin(ang), ci = re * sin(ang) + im * cos(ang);
    double om = cosm[cosmo].om;
    double f = 27. / 8. * om * om * om * pow(100. / 299792., 5.0) / 3. / (2 * pow(2 * PI, 3.0));
    out[8 * t + 2 * c] = cr * f;
    out[8 * t + 2 * c + 1] = ci * f;
    if (status && st) atomicOr(&status[t], st);
  }
};

// CS > 1: one cluster of CS CTAs per integral (cooperative adaptive_body)
template <typename R, int NT, int CS>
__global__ void __launch_bounds__(NT, sizeof(R) == 4 ? TP_GAMMA_MINB : 2) k_gamma(GammaPolicy<R> pol_in, int njobs, int* job_counter, EngineCfg cfg,
                                              char* scratch, size_t slot_bytes) {
  GammaPolicy<R> pol = pol_in;
  adaptive_body<3, 2, NT, GammaPolicy<R>, CS>(pol, njobs, job_counter, cfg, scratch, slot_bytes);
}

// The Gamma integrand at caller-given points (no cubature): the policy's
// point set-up and its node groups, summed over the groups, one thread per
// point; dynamic shared memory GammaPolicy<R>::PSMEM.
template <typename R>
__global__ void k_gamma_points(GammaPolicy<R> pol, const double* pts, int n, double* out) {
  extern __shared__ __align__(16) char psmem_[];
  double xmin[3], xmax[3];
  pol.begin_job(0, psmem_, xmin, xmax);
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    alignas(16) char rec[GammaPolicy<R>::REC];
    double sum[2] = {0.0, 0.0}, fv[2];
    if (pol.setup(p, pts + 3 * p, rec)) {
      for (int g = 0; g < GammaPolicy<R>::G; ++g) {
        double pv[2];
        pol.group(rec, g, pv);
        sum[0] += pv[0];
        sum[1] += pv[1];
      }
    }
    pol.finalize(rec, sum, fv);
    out[2 * p] = fv[0];
    out[2 * p + 1] = fv[1];
  }
}

template <typename R>
static size_t gamma_smem_bytes() {
  return engine_smem_bytes<3, 2, GammaPolicy<R>>();
}

constexpr int GAMMA_NT = 256;
constexpr int GAMMA_CLUSTER = 8;

// max_stores: region stores the launch may use (one per CTA, or per cluster),
// 0 = no limit beyond ctx->max_ctas. A batch with no more integrals than CTA
// slots runs one GAMMA_CLUSTER-CTA cluster per integral.
template <typename R>
static int run_gamma(tp_ctx* ctx, int cosmo, const double* d_x, const int* d_comp, const int* d_tri, int njobs,
                     double rel_tol, double* d_out, int* d_status, int cap, int max_stores) {
  size_t smem = gamma_smem_bytes<R>();
  cudaError_t e =
      cudaFuncSetAttribute(k_gamma<R, GAMMA_NT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return tp_cuda(ctx, e, "gamma attribute");
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gamma<R, GAMMA_NT, 1>, GAMMA_NT, smem);
  if (e != cudaSuccess || per_sm < 1) return tp_cuda(ctx, e == cudaSuccess ? cudaErrorInvalidConfiguration : e, "gamma occupancy");
  int slots = sms * per_sm;
  if (ctx->max_ctas > 0 && slots > ctx->max_ctas) slots = ctx->max_ctas;
  int cluster = 1, units = slots;
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = GAMMA_CLUSTER;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.blockDim = dim3(GAMMA_NT);
  lc.dynamicSmemBytes = smem;
  lc.stream = ctx->stream;
  lc.attrs = attr;
  lc.numAttrs = 1;
  if (njobs <= slots && slots >= GAMMA_CLUSTER) {
    int ncl = 0;
    lc.gridDim = dim3(GAMMA_CLUSTER);
    e = cudaFuncSetAttribute(k_gamma<R, GAMMA_NT, GAMMA_CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveClusters(&ncl, (const void*)k_gamma<R, GAMMA_NT, GAMMA_CLUSTER>, &lc);
    cudaGetLastError();
    ncl = std::min(ncl, slots / GAMMA_CLUSTER);
    if (e == cudaSuccess && ncl >= 1) {
      cluster = GAMMA_CLUSTER;
      units = ncl;
    }
  }
  if (max_stores > 0 && units > max_stores) units = max_stores;
  if (units > njobs) units = njobs;
  size_t slot = Slot<3, 2>::bytes(cap);
  int st = ctx->ensure_scratch((size_t)units * slot);
  if (st) return st;
  GammaPolicy<R> pol;
  pol.J.x = d_x;
  pol.J.comp = d_comp;
  pol.J.tri = d_tri;
  pol.tab = ctx->d_tab;
  pol.cosm = ctx->d_cos;
  pol.ck = (const CosmoK<R>*)(sizeof(R) == 8 ? ctx->d_ck64 : ctx->d_ck32);
  pol.cosmo = cosmo;
  pol.one = ctx->reference_forms;
  pol.out = d_out;
  pol.status = d_status;
  EngineCfg cfg{0.0, rel_tol, TP_NORM_L1, cap, 2000};
  e = cudaMemsetAsync(ctx->d_counter, 0, sizeof(int), ctx->stream);
  if (e == cudaSuccess) {
    if (cluster > 1) {
      lc.gridDim = dim3(units * GAMMA_CLUSTER);
      e = cudaLaunchKernelEx(&lc, k_gamma<R, GAMMA_NT, GAMMA_CLUSTER>, pol, njobs, ctx->d_counter, cfg,
                             ctx->d_scratch, slot);
    } else {
      k_gamma<R, GAMMA_NT, 1><<<units, GAMMA_NT, smem, ctx->stream>>>(pol, njobs, ctx->d_counter, cfg, ctx->d_scratch,
                                                                    slot);
      e = cudaGetLastError();
    }
  }
  return tp_cuda(ctx, e, "gamma launch");
}

}  // namespace tp

using namespace tp;

extern "C" int tp_ogata_weights(double* out) {
  if (!out) return TP_ERR_ARG;
  OgataTab o;
  ogata_host(o);
  for (int k = 0; k < PREC_K; ++k) {
    out[k] = o.psi[0][k];
    out[PREC_K + k] = k == 0 ? NAN : o.prod[0][k];
    out[2 * PREC_K + k] = o.psi[1][k];
    out[3 * PREC_K + k] = k == 0 ? NAN : o.prod[1][k];
  }
  return TP_OK;
}

extern "C" int tp_gamma_integrand_points(tp_ctx* ctx, int cosmo_index, const double* x, int which, const double* pts,
                                         int n, int precision, double* out) {
  TpRange nvtx_range("tp_gamma_integrand_points");
  if (!ctx || !x || !pts || !out || n < 0 || (which != 0 && which != 1)) return TP_ERR_ARG;
  if (precision != TP_FP64 && precision != TP_FP32) return TP_ERR_ARG;
  if (cosmo_index < 0 || cosmo_index >= ctx->n_cosmo) return tp_fail(ctx, TP_ERR_STATE, "no such cosmology");
  if (!(x[0] > 0 && x[1] > 0 && x[2] > 0)) return tp_fail(ctx, TP_ERR_ARG, "triangle sides must be > 0");
  if (n == 0) return TP_OK;
  cudaSetDevice(ctx->device);
  cudaError_t e = gamma_upload_constants();
  if (e != cudaSuccess) return tp_cuda(ctx, e, "ogata constants");
  if (precision == TP_FP64) {
    const int st64 = ctx->ensure_i64();
    if (st64) return st64;
  }
  const int jc[2] = {which, 0};  // job 0: component `which` of triangle 0
  const size_t o_c = 256, o_p = 512, o_o = o_p + ((sizeof(double) * 3 * n + 255) & ~size_t(255));
  int st = ctx->ensure_io(o_o + sizeof(double) * 2 * n + 256);
  if (st) return st;
  char* b = ctx->d_io;
  cudaStream_t s = ctx->stream;
  e = cudaMemcpyAsync(b, x, sizeof(double) * 3, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(b + o_c, jc, sizeof(jc), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(b + o_p, pts, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return tp_cuda(ctx, e, "gamma points upload");
  const int nt = 128;
  if (precision == TP_FP64) {
    GammaPolicy<double> pol;
    pol.J.x = (const double*)b;
    pol.J.comp = (const int*)(b + o_c);
    pol.J.tri = (const int*)(b + o_c) + 1;
    pol.tab = ctx->d_tab;
    pol.cosm = ctx->d_cos;
    pol.ck = (const CosmoK<double>*)ctx->d_ck64;
    pol.cosmo = cosmo_index;
    pol.one = ctx->reference_forms;
    pol.out = nullptr;
    pol.status = nullptr;
    k_gamma_points<double><<<1, nt, GammaPolicy<double>::PSMEM, s>>>(pol, (const double*)(b + o_p), n,
                                                                      (double*)(b + o_o));
  } else {
    GammaPolicy<float> pol;
    pol.J.x = (const double*)b;
    pol.J.comp = (const int*)(b + o_c);
    pol.J.tri = (const int*)(b + o_c) + 1;
    pol.tab = ctx->d_tab;
    pol.cosm = ctx->d_cos;
    pol.ck = (const CosmoK<float>*)ctx->d_ck32;
    pol.cosmo = cosmo_index;
    pol.one = ctx->reference_forms;
    pol.out = nullptr;
    pol.status = nullptr;
    k_gamma_points<float><<<1, nt, GammaPolicy<float>::PSMEM, s>>>(pol, (const double*)(b + o_p), n,
                                                                    (double*)(b + o_o));
  }
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, b + o_o, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return tp_cuda(ctx, e, "gamma points");
}

// One pass of the Gamma integrals of n triangles (components of comp_mask)
// at region cap `cap` on at most max_ctas CTAs (0: all resident); out is
// [n][4] complex as 8 doubles, status_out[n] the OR of the triangle's
// components' engine status (bit 1: region cap reached).
static int gamma_pass(tp_ctx* ctx, int cosmo_index, const double* x, int n, int comp_mask, double rel_tol,
                      int precision, int cap, int max_ctas, double* out, int* status_out) {
  std::vector<int> comp, tri;
  for (int t = 0; t < n; ++t)
    for (int c = 0; c < 4; ++c)
      if (comp_mask & (1 << c)) {
        comp.push_back(c);
        tri.push_back(t);
      }
  const int nj = (int)comp.size();
  size_t o_x = 0, o_c = (sizeof(double) * 3 * n + 255) & ~size_t(255);
  size_t o_t = o_c + ((sizeof(int) * nj + 255) & ~size_t(255));
  size_t o_o = o_t + ((sizeof(int) * nj + 255) & ~size_t(255));
  size_t o_s = o_o + ((sizeof(double) * 8 * n + 255) & ~size_t(255));
  int st = ctx->ensure_io(o_s + sizeof(int) * n + 256);
  if (st) return st;
  char* b = ctx->d_io;
  cudaStream_t s = ctx->stream;
  cudaError_t e = cudaMemcpyAsync(b + o_x, x, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(b + o_c, comp.data(), sizeof(int) * nj, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(b + o_t, tri.data(), sizeof(int) * nj, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b + o_o, 0, sizeof(double) * 8 * n, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b + o_s, 0, sizeof(int) * n, s);
  if (e != cudaSuccess) return tp_cuda(ctx, e, "gamma upload");
  st = precision == TP_FP64
           ? run_gamma<double>(ctx, cosmo_index, (double*)(b + o_x), (int*)(b + o_c), (int*)(b + o_t), nj, rel_tol,
                               (double*)(b + o_o), (int*)(b + o_s), cap, max_ctas)
           : run_gamma<float>(ctx, cosmo_index, (double*)(b + o_x), (int*)(b + o_c), (int*)(b + o_t), nj, rel_tol,
                              (double*)(b + o_o), (int*)(b + o_s), cap, max_ctas);
  if (st) return st;
  e = cudaMemcpyAsync(out, b + o_o, sizeof(double) * 8 * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(status_out, b + o_s, sizeof(int) * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return tp_cuda(ctx, e, "gamma");
}

// The reference integrates Gamma with an unbounded hcubature_v (maxEval = 0,
// gamma.cu:110). Triangles whose integrals reach the context's region cap are
// integrated again, from the start, with a cap 16 times larger on as many
// CTAs as fit GAMMA_ESCALATE_BYTES of region stores, up to the context's
// escalation cap (at most GAMMA_CAP_MAX regions per integral); the adaptive
// sequence is deterministic, so the larger cap continues exactly where the
// smaller one stopped. Only what still reaches the last cap is reported.
constexpr int GAMMA_CAP_MAX = 1 << 24;
constexpr size_t GAMMA_ESCALATE_BYTES = size_t(32) << 30;

extern "C" int tp_gamma_batch(tp_ctx* ctx, int cosmo_index, const double* x, int n, int comp_mask, double rel_tol,
                              int precision, double* out, int* status_out) {
  TpRange nvtx_range("tp_gamma_batch: Gamma");
  if (!ctx || !x || !out || n < 0 || (comp_mask & ~0xF) || comp_mask == 0) return TP_ERR_ARG;
  if (precision != TP_FP64 && precision != TP_FP32) return TP_ERR_ARG;
  if (!(rel_tol > 0)) return TP_ERR_ARG;
  if (cosmo_index < 0 || cosmo_index >= ctx->n_cosmo) return tp_fail(ctx, TP_ERR_STATE, "no such cosmology");
  for (int i = 0; i < 3 * n; ++i)
    if (!(x[i] > 0)) return tp_fail(ctx, TP_ERR_ARG, "triangle sides must be > 0");
  for (int t = 0; t < n; ++t) {
    double a = x[3 * t], b = x[3 * t + 1], c = x[3 * t + 2];
    if (a > b + c || b > a + c || c > a + b) return tp_fail(ctx, TP_ERR_ARG, "sides violate the triangle inequality");
  }
  if (n == 0) return TP_OK;
  cudaSetDevice(ctx->device);
  cudaError_t e = gamma_upload_constants();
  if (e != cudaSuccess) return tp_cuda(ctx, e, "ogata constants");
  if (precision == TP_FP64) {
    const int st64 = ctx->ensure_i64();
    if (st64) return st64;
  }
  std::vector<int> hst(n);
  int st = gamma_pass(ctx, cosmo_index, x, n, comp_mask, rel_tol, precision, ctx->region_cap, ctx->max_ctas, out,
                      hst.data());
  if (st) return st;
  for (int cap = ctx->region_cap; cap < std::min(GAMMA_CAP_MAX, ctx->escalate_cap);) {
    std::vector<int> again;
    for (int t = 0; t < n; ++t)
      if (hst[t] & 1) again.push_back(t);
    if (again.empty()) break;
    cap = (int)std::min<long>((long)cap * 16, std::min(GAMMA_CAP_MAX, ctx->escalate_cap));
    const int nj = (int)again.size() * __builtin_popcount((unsigned)comp_mask);
    int ctas = (int)std::max<size_t>(1, GAMMA_ESCALATE_BYTES / Slot<3, 2>::bytes(cap));
    if (ctx->max_ctas > 0) ctas = std::min(ctas, ctx->max_ctas);
    ctas = std::min(ctas, nj);
    std::vector<double> xs(3 * again.size()), os(8 * again.size());
    std::vector<int> ss(again.size());
    for (size_t k = 0; k < again.size(); ++k)
      for (int q = 0; q < 3; ++q) xs[3 * k + q] = x[3 * again[k] + q];
    st = gamma_pass(ctx, cosmo_index, xs.data(), (int)again.size(), comp_mask, rel_tol, precision, cap, ctas,
                    os.data(), ss.data());
    if (st) return st;
    for (size_t k = 0; k < again.size(); ++k) {
      for (int q = 0; q < 8; ++q) out[8 * again[k] + q] = os[8 * k + q];
      hst[again[k]] = ss[k];
    }
  }
  // region stores grown by the escalation are released again
  if (ctx->scratch_bytes > (size_t(4) << 30)) {
    cudaFree(ctx->d_scratch);
    ctx->d_scratch = nullptr;
    ctx->scratch_bytes = 0;
  }
  int bad = 0;
  for (int t = 0; t < n; ++t) {
    if (status_out) status_out[t] = hst[t];
    bad += hst[t] != 0;
  }
  if (bad) return tp_fail(ctx, TP_ERR_CAPACITY, std::to_string(bad) + " Gamma integrals hit a region or sweep cap");
  return TP_OK;
}
