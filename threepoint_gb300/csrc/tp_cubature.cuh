// Device-side h-adaptive cubature for batches of independent integrals.
//
// Semantics follow the reference's vendored Gladwell-parallel hcubature_v
// (cuda_version/hcubature.cpp:456-617 rule, 620-780 1-D rule, 904-1067
// driver; converged.h): every sweep evaluates all regions split in the
// previous sweep; a sweep splits the largest-error regions, in decreasing
// order of their maximum component error, until the remaining error meets the
// tolerance; a region is halved along the dimension of largest fourth
// difference; the lower half keeps the parent volume * 0.5 and the upper half
// recomputes the product of its widths.
//
// GB300 mapping: one CTA owns one integral for its whole adaptive life (a
// persistent grid pulls integrals from an atomic job counter), so no CTA ever
// waits on another; for small batches the CTAs of a thread-block cluster own
// one integral together (adaptive_body with CS > 1, below), synchronised by
// the hardware cluster barrier only. Region state lives in a per-CTA (per
// cluster) slot of HBM scratch (structure of arrays, FP64). Inside a sweep the CTA evaluates the new
// regions' cubature points in chunks; each point's integrand is split into G
// independent partial sums (for the line-of-sight integrands: G groups of
// nodes), giving (point x group) parallelism even for one-region sweeps. The
// region choice is a radix select on the bit pattern of the FP64 error keys
// (8 passes of 256-bin shared-memory histograms) followed by a block-wide
// stream compaction; no sort and no host round trip.
#pragma once
#include <cooperative_groups.h>
#include <stdint.h>

#include <type_traits>

#include "tp_internal.cuh"

namespace tp {

// Genz-Malik generators sqrt(9/70), sqrt(9/10), sqrt(9/19) (correctly rounded)
// and ratio = l2^2 / l4^2 as computed in double from them.
struct GM {
  static constexpr double l2 = 0x1.6f2c9a420071ep-2;
  static constexpr double l4 = 0x1.e5b9d136c6d96p-1;
  static constexpr double l5 = 0x1.6061efecf8ae9p-1;
  static constexpr double ratio = 0x1.2492492492493p-3;
};

// 15-point Kronrod abscissae, 7-point Gauss weights and 15-point Kronrod
// weights (QUADPACK qk15 constants)
__device__ __forceinline__ double gk_xgk(int i) {
  const double v[8] = {0.991455371120812639206854697526329, 0.949107912342758524526189684047851,
                       0.864864423359769072789712788640926, 0.741531185599394439863864773280788,
                       0.586087235467691130294144838258730, 0.405845151377397166906606412076961,
                       0.207784955007898467600689403773245, 0.000000000000000000000000000000000};
  return v[i];
}
__device__ __forceinline__ double gk_wg(int i) {
  const double v[4] = {0.129484966168869693270611432679082, 0.279705391489276667901467771423780,
                       0.381830050505118944950369775488975, 0.417959183673469387755102040816327};
  return v[i];
}
__device__ __forceinline__ double gk_wgk(int i) {
  const double v[8] = {0.022935322010529224963732008058970, 0.063092092629978553290700663189204,
                       0.104790010322250183839876322541518, 0.140653259715525918745189590510238,
                       0.169004726639267902826583426598550, 0.190350578064785409913256402421014,
                       0.204432940075298892414161999234649, 0.209482141084727828012999174891714};
  return v[i];
}

template <int DIM>
struct GMRule {
  static constexpr int NP = (DIM == 1) ? 15 : 1 + 4 * DIM + 2 * DIM * (DIM - 1) + (1 << DIM);
};

struct EngineCfg {
  double abs_tol, rel_tol;
  int norm;        // TP_NORM_*; fdim == 1 always behaves as INDIVIDUAL
  int cap;         // regions per integral
  int max_sweeps;
};

// Policies with P::REF: the region's axis, its values come from the reference
// form of the integrand; its two largest fourth differences tie
constexpr int SPLIT_AXIS = 7, SPLIT_AXIS_REF = 32, SPLIT_REF = 64, SPLIT_TIE = 128;

template <class P, class = void>
struct EngineRef {
  static constexpr bool value = false;
};
template <class P>
struct EngineRef<P, std::enable_if_t<P::REF>> {
  static constexpr bool value = true;
};

// per-CTA region store
template <int DIM, int FDIM>
struct Slot {
  double* cen;    // [DIM][cap]
  double* hw;     // [DIM][cap]
  double* vol;    // [cap]
  double* val;    // [FDIM][cap]
  double* err;    // [FDIM][cap]
  double* emax;   // [cap]
  int* pend;      // [cap]
  uint8_t* split; // [cap] axis | SPLIT_*
  int cap;
  __host__ __device__ static constexpr size_t bytes(int cap) {
    return (size_t)cap * (sizeof(double) * (2 * DIM + 2 + 2 * FDIM) + sizeof(int) + 1) + 256;
  }
  __device__ void init(char* base, int c) {
    cap = c;
    double* d = (double*)base;
    cen = d;
    hw = cen + (size_t)DIM * cap;
    vol = hw + (size_t)DIM * cap;
    val = vol + cap;
    err = val + (size_t)FDIM * cap;
    emax = err + (size_t)FDIM * cap;
    pend = (int*)(emax + cap);
    split = (uint8_t*)(pend + cap);
  }
};

// ---------------------------------------------------------------------------
// cubature point p of a region (same ordering as the reference rules)
template <int DIM>
__device__ inline void rule_point(int p, const double* c, const double* h, double* x) {
#pragma unroll
  for (int d = 0; d < DIM; ++d) x[d] = c[d];
  if constexpr (DIM == 1) {
    // center, then +-xgk[1], +-xgk[3], +-xgk[5], then +-xgk[0], +-xgk[2], +-xgk[4], +-xgk[6]
    if (p == 0) return;
    int q = p - 1;
    int j = q >> 1;
    int idx = j < 3 ? 2 * j + 1 : 2 * (j - 3);
    double w = h[0] * gk_xgk(idx);
    x[0] = (q & 1) ? c[0] + w : c[0] - w;
  } else {
    if (p == 0) return;
    if (p < 1 + 4 * DIM) {
      int k = (p - 1) >> 2, s = (p - 1) & 3;
      double r = (s < 2 ? GM::l2 : GM::l4) * h[k];
      x[k] = (s & 1) ? c[k] + r : c[k] - r;
      return;
    }
    int q = p - (1 + 4 * DIM);
    if (q < 2 * DIM * (DIM - 1)) {
      int pr = q >> 2, s = q & 3;
      int i = 0, j = 1, cnt = 0;
      for (int a = 0; a < DIM - 1; ++a)
        for (int b = a + 1; b < DIM; ++b) {
          if (cnt == pr) {
            i = a;
            j = b;
          }
          ++cnt;
        }
      double ri = GM::l4 * h[i], rj = GM::l4 * h[j];
      // (-,-), (+,-), (+,+), (-,+)
      x[i] = (s == 1 || s == 2) ? c[i] + ri : c[i] - ri;
      x[j] = (s >= 2) ? c[j] + rj : c[j] - rj;
      return;
    }
    int m = q - 2 * DIM * (DIM - 1);
    int gray = m ^ (m >> 1);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      double r = GM::l5 * h[d];
      x[d] = ((gray >> d) & 1) ? c[d] - r : c[d] + r;
    }
  }
}

// relative difference below which two errors (or fourth differences) count as
// a tie of mirror-image regions (axes) that rounding decides: rounding moves
// them by up to ~1e-9, and unrelated regions come this close with a
// probability of ~1e-4 per cut
constexpr double TIE_REL = 1e-6;

// axis of the largest fourth difference, from the centre and the 4 DIM axis
// points (the rule's first points); tie: another axis comes within TIE_REL
template <int DIM, int FDIM>
__device__ inline void rule_axis(const double* f, int* split, bool* split_tie) {
  double diff[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) diff[d] = 0;
  for (int k = 0; k < FDIM; ++k) {
    auto V = [&](int i) { return f[i * FDIM + k]; };
    double val0 = V(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      double v0 = V(1 + 4 * d), v1 = V(2 + 4 * d), v2 = V(3 + 4 * d), v3 = V(4 + 4 * d);
      const double da = __dsub_rn(__dadd_rn(v0, v1), 2 * val0), db = __dsub_rn(__dadd_rn(v2, v3), 2 * val0);
      diff[d] += fabs(fma(-GM::ratio, db, da));
    }
  }
  double md = 0;
  int dm = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    if (diff[d] > md) {
      md = diff[d];
      dm = d;
    }
  *split = dm;
  *split_tie = false;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    if (d != dm && diff[d] >= md * (1.0 - TIE_REL)) *split_tie = true;
}

// Apply the embedded rule to one region's NP point values (f[p*FDIM+k]).
template <int DIM, int FDIM>
__device__ inline void rule_combine(const double* f, double vol, double hw0, double* val, double* err, int* split) {
  if constexpr (DIM == 1) {
    auto wg = [](int i) { return gk_wg(i); };
    auto wgk = [](int i) { return gk_wgk(i); };
    for (int k = 0; k < FDIM; ++k) {
      auto V = [&](int i) { return f[i * FDIM + k]; };
      double rg = V(0) * wg(3), rk = V(0) * wgk(7);
      double rabs = fabs(rk);
      int n = 1;
      for (int j = 0; j < 3; ++j) {
        int j2 = 2 * j + 1;
        double v = V(n) + V(n + 1);
        rg += wg(j) * v;
        rk += wgk(j2) * v;
        rabs += wgk(j2) * (fabs(V(n)) + fabs(V(n + 1)));
        n += 2;
      }
      for (int j = 0; j < 4; ++j) {
        int j2 = 2 * j;
        rk += wgk(j2) * (V(n) + V(n + 1));
        rabs += wgk(j2) * (fabs(V(n)) + fabs(V(n + 1)));
        n += 2;
      }
      val[k] = rk * hw0;
      double mean = rk * 0.5;
      double rasc = wgk(7) * fabs(V(0) - mean);
      n = 1;
      for (int j = 0; j < 3; ++j) {
        int j2 = 2 * j + 1;
        rasc += wgk(j2) * (fabs(V(n) - mean) + fabs(V(n + 1) - mean));
        n += 2;
      }
      for (int j = 0; j < 4; ++j) {
        int j2 = 2 * j;
        rasc += wgk(j2) * (fabs(V(n) - mean) + fabs(V(n + 1) - mean));
        n += 2;
      }
      double e = fabs(rk - rg) * hw0;
      rabs *= hw0;
      rasc *= hw0;
      if (rasc != 0 && e != 0) {
        double scale = pow(200 * e / rasc, 1.5);
        e = (scale < 1) ? rasc * scale : rasc;
      }
      const double dmin = 2.2250738585072014e-308, deps = 2.220446049250313e-16;
      if (rabs > dmin / (50 * deps)) {
        double me = 50 * deps * rabs;
        if (me > e) e = me;
      }
      err[k] = e;
    }
    *split = 0;
  } else {
    const double w1 = (double)(12824 - 9120 * DIM + 400 * DIM * DIM) / 19683.0;
    const double w3 = (double)(1820 - 400 * DIM) / 19683.0;
    const double w5 = 6859.0 / 19683.0 / (double)(1u << DIM);
    const double wE1 = (double)(729 - 950 * DIM + 50 * DIM * DIM) / 729.0;
    const double wE3 = (double)(265 - 100 * DIM) / 1458.0;
    const double w2 = 980. / 6561., w4 = 200. / 19683., wE2 = 245. / 486., wE4 = 25. / 729.;
    double diff[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) diff[d] = 0;
    for (int k = 0; k < FDIM; ++k) {
      auto V = [&](int i) { return f[i * FDIM + k]; };
      double val0 = V(0), s2 = 0, s3 = 0, s4 = 0, s5 = 0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        double v0 = V(1 + 4 * d), v1 = V(2 + 4 * d), v2 = V(3 + 4 * d), v3 = V(4 + 4 * d);
        s2 += v0 + v1;
        s3 += v2 + v3;
        const double da = __dsub_rn(__dadd_rn(v0, v1), 2 * val0), db = __dsub_rn(__dadd_rn(v2, v3), 2 * val0);
        diff[d] += fabs(fma(-GM::ratio, db, da));
      }
      int k0 = 1 + 4 * DIM;
      for (int i = 0; i < 2 * DIM * (DIM - 1); ++i) s4 += V(k0 + i);
      k0 += 2 * DIM * (DIM - 1);
      for (int i = 0; i < (1 << DIM); ++i) s5 += V(k0 + i);
      // explicit roundings: what the compiler contracts here would depend on the
      // code around the inlined rule, and bitwise ties of errors decide splits
      const double x7 = fma(w5, s5, fma(w4, s4, fma(w3, s3, fma(w2, s2, __dmul_rn(w1, val0)))));
      const double x5 = fma(wE4, s4, fma(wE3, s3, fma(wE2, s2, __dmul_rn(wE1, val0))));
      const double r7 = __dmul_rn(vol, x7);
      const double dr = fma(vol, x5, -r7);
      val[k] = r7;
      err[k] = fabs(dr);
    }
    double md = 0;
    int dm = 0;
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      if (diff[d] > md) {
        md = diff[d];
        dm = d;
      }
    *split = dm;
  }
}

// rule_combine that also tells whether the axis is a tie
template <int DIM, int FDIM>
__device__ inline void rule_combine_ref(const double* f, double vol, double hw0, double* val, double* err, int* split,
                                        bool* split_tie) {
  rule_combine<DIM, FDIM>(f, vol, hw0, val, err, split);
  *split_tie = false;
  int sp;
  if constexpr (DIM > 1) rule_axis<DIM, FDIM>(f, &sp, split_tie);
}

// ---------------------------------------------------------------------------
// block-wide helpers
template <int NT>
__device__ inline double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x < 32) {
    t = (l < NT / 32) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  t = red[0];
  return t;
}

__device__ inline bool converged_check(int fdim, int norm, const double* V, const double* E, double abs_tol,
                                       double rel_tol) {
  if (fdim == 1 || norm == TP_NORM_INDIVIDUAL) {
    for (int k = 0; k < fdim; ++k)
      if (E[k] > abs_tol && E[k] > fabs(V[k]) * rel_tol) return false;
    return true;
  }
  // L1 (the only multi-component norm used on this path)
  double e = 0, v = 0;
  for (int k = 0; k < fdim; ++k) {
    e += E[k];
    v += fabs(V[k]);
  }
  return e <= abs_tol || e <= v * rel_tol;
}

// Shared scratch of the engine (besides the policy's own)
template <int FDIM>
struct EngineShared {
  int live_list[1024];  // live points of the current chunk; the selection's last candidates
  int nlive_chunk;
  unsigned long long hist[256];
  double red[64];
  int ired[80];
  double V[FDIM], E[FDIM];
  unsigned long long q_above;
  unsigned long long prefix, qtot;
  int digit;
  int job, nlive, npend, status, stop, ktot, sweeps, ref, nband, nref, nfull;
  long long neval;
};

// Dynamic shared memory of adaptive_body for policy P.
template <int DIM, int FDIM, class P>
__host__ __device__ constexpr size_t engine_smem_bytes() {
  return ((P::PSMEM + 15) & ~size_t(15)) + (((size_t)P::CH * GMRule<DIM>::NP * P::REC + 15) & ~size_t(15)) +
         sizeof(double) * (size_t)P::G * P::CH * GMRule<DIM>::NP * P::PD +
         sizeof(double) * (size_t)P::CH * GMRule<DIM>::NP * FDIM + sizeof(EngineShared<FDIM>) + 16;
}


// ---------------------------------------------------------------------------
// One sweep's bookkeeping by the NT threads of one CTA: the totals, the
// convergence test, the choice of the regions to split (every region whose
// error is at least the largest tau that leaves a remaining error within the
// tolerance), and their splitting into S.pend. Sets es->stop, or es->npend,
// es->nlive, es->ref.
//
// The other CTAs of a cluster wait for it, and it is a chain of passes over
// the region store with barriers between them, so its latency counts: the
// error keys are read once and staged in shared memory (stage: the point
// records and partial sums, idle between evaluations) for the radix passes,
// regions above the last 32 candidates are settled by one warp, and the
// chosen regions are split one per thread from a list. Measured with the
// earlier form (keys read again from the region store in each of eight passes,
// a contiguous range of regions split by each thread): a <Map^3> integral's
// sweep of ~1500 regions 60k -> 33k cycles, a Gamma one of ~3000 160k -> 60k;
// 64 FP32 Gamma triangles with the set-up of GammaPolicy 340 -> 240 ms.
template <int DIM, int FDIM, int NT, bool REF>
__device__ __forceinline__ void engine_select(Slot<DIM, FDIM> S, EngineShared<FDIM>* es, EngineCfg cfg,
                                              unsigned long long* stage, int stage_bytes, int sweep, int npend,
                                              int ref, bool ties) {
  constexpr int NP = GMRule<DIM>::NP;
  typedef unsigned long long u64;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0 && !ref) es->neval += (long long)npend * NP;

  // ---------------- totals and convergence ----------------------------
  const int nlive = es->nlive;
  // staged: the key and, with several components, the error sum
  constexpr int SW = FDIM == 1 ? 1 : 2;
  const int nst = min(nlive, stage_bytes / (8 * SW));
  double tv[FDIM], te[FDIM];
#pragma unroll
  for (int k = 0; k < FDIM; ++k) tv[k] = te[k] = 0;
#pragma unroll 4
  for (int i = tid; i < nlive; i += NT) {
    double ev[FDIM];
#pragma unroll
    for (int k = 0; k < FDIM; ++k) {
      tv[k] += S.val[(size_t)k * S.cap + i];
      ev[k] = S.err[(size_t)k * S.cap + i];
      te[k] += ev[k];
    }
    if (i < nst) {
      stage[i] = (u64)__double_as_longlong(S.emax[i]);
      if constexpr (SW == 2) {
        double es_ = 0;
#pragma unroll
        for (int k = 0; k < FDIM; ++k) es_ += ev[k];
        stage[nst + i] = (u64)__double_as_longlong(es_);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < FDIM; ++k) {
    tv[k] = block_sum<NT>(tv[k], es->red);
    te[k] = block_sum<NT>(te[k], es->red);
  }
  auto finish = [&](int bits) {
    if (tid == 0) {
      for (int k = 0; k < FDIM; ++k) {
        es->V[k] = tv[k];
        es->E[k] = te[k];
      }
      es->status |= bits;
      es->sweeps = sweep + 1;
      es->stop = 1;
    }
    __syncthreads();
  };
  const bool conv = converged_check(FDIM, cfg.norm, tv, te, cfg.abs_tol, cfg.rel_tol);
  if (conv || sweep + 1 >= cfg.max_sweeps) return finish(conv ? 0 : 2);
  // tolerance for the Gladwell pop loop
  double etot = 0, vabs = 0;
  bool l1 = !(FDIM == 1 || cfg.norm == TP_NORM_INDIVIDUAL);
#pragma unroll
  for (int k = 0; k < FDIM; ++k) {
    etot += te[k];
    vabs += fabs(tv[k]);
  }
  const double tol = fmax(cfg.abs_tol, (l1 ? vabs : fabs(tv[0])) * cfg.rel_tol);

  // ---------------- radix select of the error threshold ---------------
  // Errors are summed as 62-bit fixed-point fractions of the total error,
  // so the histogram sums (shared-memory integer atomics) are exact and
  // independent of the order of the additions.
  const double qscale = 4.611686018427387904e18 / etot;  // 2^62 / E_tot
  const double tol_q = tol * qscale;
  auto key_of = [&](int i) { return i < nst ? stage[i] : (u64)__double_as_longlong(S.emax[i]); };
  auto q_of = [&](int i, u64 key) {
    double es_;
    if constexpr (FDIM == 1) {
      es_ = __longlong_as_double((long long)key);
    } else if (i < nst) {
      es_ = __longlong_as_double((long long)stage[nst + i]);
    } else {
      es_ = 0;
#pragma unroll
      for (int k = 0; k < FDIM; ++k) es_ += S.err[(size_t)k * S.cap + i];
    }
    return (u64)(es_ * qscale);
  };
  // Digits of the keys, largest first: the first pass takes 255 bins of 1/8
  // octave below the largest key (one byte of the exponent would put all
  // regions into two or three bins, whose shared-memory atomics then queue:
  // 20 us a sweep); a cut below those, and the rest of the key, go by bytes.
  // Keys whose first bits (key >> sh) equal pre are the candidates; they are
  // listed once they fit.
  constexpr int LIST = 1024;
  int hmax = 0;
  for (int i = tid; i < nlive; i += NT) hmax = max(hmax, (int)(key_of(i) >> 32));
  hmax = __reduce_max_sync(0xffffffffu, hmax);
  if (lane == 0) es->ired[warp] = hmax;
  if (tid == 0) {
    es->prefix = 0ull;
    es->q_above = 0ull;
  }
  __syncthreads();
  for (int w = 0; w < NT / 32; ++w) hmax = max(hmax, es->ired[w]);
  const int top = hmax >> 17;  // of key >> 49
  int ncand = -1, sh = 64;
  u64 pre = 0, qtot = 0, tau = 0;
  for (bool octaves = true;; octaves = false) {
    const int w = min(8, sh), nsh = octaves ? 49 : sh - w;
    for (int b = tid; b < 256; b += NT) es->hist[b] = 0ull;
    if (tid == 0) es->nlive_chunk = 0;
    __syncthreads();
    auto count = [&](int i) {
      const u64 key = key_of(i);
      if (octaves) {
        atomicAdd(&es->hist[max(0, 255 - (top - (int)(key >> 49)))], q_of(i, key));
      } else if (sh == 64 || (key >> sh) == pre) {
        atomicAdd(&es->hist[(key >> nsh) & ((1u << w) - 1)], q_of(i, key));
      }
    };
    if (ncand >= 0) {
      for (int c = tid; c < ncand; c += NT) count(es->live_list[c]);
    } else {
      for (int i = tid; i < nlive; i += NT) count(i);
    }
    __syncthreads();
    if (tid < 32) {
      const int l = tid;
      u64 loc[8];
      u64 ls = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        loc[q] = es->hist[8 * l + q];
        ls += loc[q];
      }
      u64 all = ls;
      for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
      // the first pass histograms every region: its sum is the fixed-point total
      const u64 qt = octaves ? all : es->qtot;
      // suffix sum over lanes (lane l: sum of lanes > l)
      u64 suf = ls;
      for (int o = 1; o < 32; o <<= 1) {
        u64 y = __shfl_down_sync(0xffffffffu, suf, o);
        if (l + o < 32) suf += y;
      }
      u64 cum = es->q_above + (suf - ls);
      int best = -1;
      u64 cum_best = 0;
#pragma unroll
      for (int q = 7; q >= 0; --q) {
        cum += loc[q];
        if (best < 0 && (double)(qt > cum ? qt - cum : 0ull) <= tol_q) {
          best = 8 * l + q;
          cum_best = cum;
        }
      }
      int chosen = __reduce_max_sync(0xffffffffu, best);
      bool none = chosen < 0;
      if (none) chosen = 0;
      u64 cb = (best == chosen && !none) ? cum_best : 0ull;
      u64 hb = (best == chosen && !none) ? es->hist[chosen] : 0ull;
      for (int o = 16; o > 0; o >>= 1) {
        cb += __shfl_xor_sync(0xffffffffu, cb, o);
        hb += __shfl_xor_sync(0xffffffffu, hb, o);
      }
      __syncwarp();
      if (l == 0) {
        // bins strictly above the chosen one are selected for sure; when no
        // bin satisfies the tolerance (rounding), take the whole range. The
        // open last bin of the first pass starts again with bytes.
        if (octaves) es->qtot = qt;
        if (!octaves || chosen > 0) es->q_above = none ? es->q_above + all - es->hist[0] : cb - hb;
        es->digit = chosen;
      }
    }
    __syncthreads();
    const int digit = es->digit;
    qtot = es->qtot;
    if (octaves) {
      if (digit == 0) continue;
      pre = (u64)(top - (255 - digit));
    } else {
      pre = (pre << w) | (u64)digit;
    }
    sh = nsh;
    if (sh == 0) {
      tau = pre;
      break;
    }
    if (ncand < 0) {
      for (int i = tid; i < nlive; i += NT)
        if ((key_of(i) >> sh) == pre) {
          const int at = atomicAdd(&es->nlive_chunk, 1);
          if (at < LIST) es->live_list[at] = i;
        }
      __syncthreads();
      ncand = es->nlive_chunk <= LIST ? es->nlive_chunk : -1;
      __syncthreads();
    }
    if (ncand >= 0 && ncand <= 32) {
      // at most one a lane: the largest key whose regions and those above
      // leave a remaining error within the tolerance
      if (tid < 32) {
        u64 key = 0, q = 0;
        bool cand = false;
        if (lane < ncand) {
          const int i = es->live_list[lane];
          key = key_of(i);
          cand = (key >> sh) == pre;
          if (cand) q = q_of(i, key);
        }
        u64 cum = es->q_above;
        for (int o = 0; o < ncand; ++o) {
          const u64 ok = __shfl_sync(0xffffffffu, key, o), oq = __shfl_sync(0xffffffffu, q, o);
          if (ok >= key) cum += oq;
        }
        u64 m = cand && (double)(qtot > cum ? qtot - cum : 0ull) <= tol_q ? key : 0ull;
        for (int o = 16; o > 0; o >>= 1) {
          const u64 y = __shfl_xor_sync(0xffffffffu, m, o);
          m = y > m ? y : m;
        }
        if (lane == 0) es->prefix = m ? m : pre << sh;
      }
      __syncthreads();
      tau = es->prefix;
      break;
    }
  }

  // ---------------- ties that the reference form decides --------------
  if constexpr (REF) {
    // (a job that has the reference form alone has decided them already)
    if (ties && !ref && tau != 0ull) {
      const double kt = __longlong_as_double((long long)tau);
      const double b0 = kt * (1.0 - TIE_REL), b1 = kt * (1.0 + TIE_REL);
      if (tid == 0) es->nband = es->nref = 0;
      __syncthreads();
      // regions at the cut, where there is more than one
      int nb = 0;
      for (int i = tid; i < nlive; i += NT) {
        const double k = __longlong_as_double((long long)key_of(i));
        nb += k >= b0 && k <= b1;
      }
      if (nb) atomicAdd(&es->nband, nb);
      __syncthreads();
      const bool band = es->nband > 1;
      if (band) {
        for (int i = tid; i < nlive; i += NT) {
          const double k = __longlong_as_double((long long)key_of(i));
          if (k >= b0 && k <= b1 && !(S.split[i] & SPLIT_REF)) S.pend[atomicAdd(&es->nref, 1)] = i;
        }
      }
      __syncthreads();
      const int nfl = es->nref;
      __syncthreads();
      // axes of the regions above them
      for (int i = tid; i < nlive; i += NT) {
        const double k = __longlong_as_double((long long)key_of(i));
        if ((band ? k > b1 : k >= kt) && (S.split[i] & (SPLIT_TIE | SPLIT_AXIS_REF)) == SPLIT_TIE)
          S.pend[atomicAdd(&es->nref, 1)] = i;
      }
      __syncthreads();
      if (es->nref > 0) {
        if (tid == 0) {
          es->npend = es->nref;
          es->nfull = nfl;
          es->ref = 1;
          es->nlive_chunk = 0;
        }
        __syncthreads();
        return;  // all ranks evaluate them, then the cut is drawn again
      }
    }
  }

  // ---------------- compaction: split every region with key >= tau ----
  // ranks in the order of the regions: each warp counts, then lists, a
  // contiguous segment
  const int seg = ((nlive + NT - 1) / NT) * 32;
  const int lo = min(warp * seg, nlive), hi = min(lo + seg, nlive);
  int cnt = 0;
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    cnt += __popc(__ballot_sync(0xffffffffu, i < hi && key_of(i) >= tau));
  }
  if (lane == 0) es->ired[warp] = cnt;
  __syncthreads();
  int rank = 0, ktot = 0;
  for (int w = 0; w < NT / 32; ++w) {
    const int c = es->ired[w];
    rank += w < warp ? c : 0;
    ktot += c;
  }
  if (ktot == 0 || nlive + ktot > S.cap) return finish(ktot == 0 ? 4 : 1);
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    const bool sel = i < hi && key_of(i) >= tau;
    const unsigned m = __ballot_sync(0xffffffffu, sel);
    if (sel) S.pend[2 * (rank + __popc(m & ((1u << lane) - 1)))] = i;
    rank += __popc(m);
  }
  __syncthreads();
  for (int k = tid; k < ktot; k += NT) {
    const int i = S.pend[2 * k], u = nlive + k;
    const int d = S.split[i] & SPLIT_AXIS;
    double v = 1;
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
      double cq = S.cen[(size_t)q * S.cap + i];
      double hq = S.hw[(size_t)q * S.cap + i];
      if (q == d) {
        hq *= 0.5;
        S.cen[(size_t)q * S.cap + i] = cq - hq;
        S.hw[(size_t)q * S.cap + i] = hq;
        S.cen[(size_t)q * S.cap + u] = cq + hq;
      } else {
        S.cen[(size_t)q * S.cap + u] = cq;
      }
      S.hw[(size_t)q * S.cap + u] = hq;
      v *= 2 * hq;
    }
    S.vol[i] *= 0.5;
    S.vol[u] = v;
    S.pend[2 * k + 1] = u;
  }
  __syncthreads();
  if (tid == 0) {
    es->nlive = nlive + ktot;
    es->npend = 2 * ktot;
    es->ref = 0;
    es->nlive_chunk = 0;
  }
}

// out of line: its registers are not the evaluation's
template <int DIM, int FDIM, int NT, bool REF>
__device__ __noinline__ void engine_select_call(Slot<DIM, FDIM> S, EngineShared<FDIM>* es, EngineCfg cfg,
                                                unsigned long long* stage, int stage_bytes, int sweep, int npend,
                                                int ref, bool ties) {
  engine_select<DIM, FDIM, NT, REF>(S, es, cfg, stage, stage_bytes, sweep, npend, ref, ties);
}

// ---------------------------------------------------------------------------
// The persistent adaptive-integration kernel body. Policy P provides:
//   static constexpr int G, REC (bytes per point record), CH (regions/chunk)
//   __device__ void begin_job(int job, char* psmem, double* xmin, double* xmax) (all threads; syncs inside)
//   __device__ bool setup(int p, const double* x, char* rec)   (true: point needs its groups)
//   __device__ bool is_live(const char* rec)
//   __device__ void group(const char* rec, int g, double* part /*PD*/)  (live points only)
//   static int slot(int g): sum class of group g (0..NS-1)
//   __device__ void finalize(const char* rec, const double* sum /*FDIM*/, double* fval /*FDIM*/)
//   __device__ void end_job(int job, const double* V, const double* E, long long neval, int status)
//   static constexpr size_t PSMEM (policy shared bytes)
//   static constexpr bool REF (optional): the policy has two forms of the
//   integrand that agree to rounding, a fast one and the reference form
//   (int ref: 0, or not for the reference form; set here; int one: set by
//   begin_job where a job has the reference form alone). An integrand symmetric under an exchange or a
//   reflection of its variables gives mirror-image regions whose errors differ
//   only by rounding, and where a sweep's cut falls between them the reference
//   form's rounding decides whether one or both are split (a bitwise tie splits
//   both); likewise the axis of a region on the mirror plane. Those regions
//   (errors within TIE_REL of the cut; splits with two equal fourth
//   differences) are evaluated again with the reference form before the cut is
//   drawn, so the region sequence, and with it the result to ~1e-15, is the
//   reference form's.
//
// CS > 1 (launch with thread-block clusters of CS CTAs): the CTAs of a
// cluster own one integral together. Every sweep's pending regions are dealt
// out to them in chunks (rank r takes chunks r, r + CS, ...); the region store
// is the cluster's, in HBM; rank 0 alone does the totals, the selection and
// the splitting, and publishes the job, the pending count and the stop flag
// in its shared memory, which the other ranks read through distributed shared
// memory. Two cluster barriers per sweep (after the evaluation, after the
// bookkeeping), with release/acquire ordering of the region store; every rank
// takes the same branches, decided from rank 0's published values after a
// barrier. The region sequence is that of CS = 1.
template <int CS>
__device__ __forceinline__ void engine_cluster_sync() {
  if constexpr (CS > 1) {
    __threadfence();
    cooperative_groups::this_cluster().sync();
  } else {
    __syncthreads();
  }
}

template <int DIM, int FDIM, int NT, class P, int CS = 1>
__device__ void adaptive_body(P& pol, int njobs, int* job_counter, const EngineCfg cfg, char* scratch,
                              size_t slot_bytes) {
  constexpr int NP = GMRule<DIM>::NP;
  constexpr int NPAX = 1 + 4 * DIM;  // the rule's centre and axis points
  constexpr int CH = P::CH;
  constexpr int G = P::G;
  constexpr int PD = P::PD;  // values per group item (>= 1)
  constexpr int NS = P::NS;  // group classes: item g adds into sum class P::slot(g)
  constexpr bool REF = EngineRef<P>::value;
  static_assert(P::CH * NP <= 1024, "live list holds one chunk");
  extern __shared__ __align__(16) char smem[];
  char* psmem = smem;
  char* recs = psmem + ((P::PSMEM + 15) & ~size_t(15));
  double* part = (double*)(recs + (((size_t)CH * NP * P::REC + 15) & ~size_t(15)));  // [G][CH*NP][PD]
  double* fval = part + (size_t)G * CH * NP * PD;                                 // [CH*NP][FDIM]
  EngineShared<FDIM>* es = (EngineShared<FDIM>*)(fval + (size_t)CH * NP * FDIM);
  // the control block every rank follows: rank 0's (distributed shared memory)
  EngineShared<FDIM>* es0 = es;
  int crank = 0;
  if constexpr (CS > 1) {
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    crank = (int)cl.block_rank();
    es0 = cl.map_shared_rank(es, 0);
  }

  const int stage_bytes = (int)((char*)es - recs) & ~15;
  Slot<DIM, FDIM> S;
  S.init(scratch + (size_t)(blockIdx.x / CS) * slot_bytes, cfg.cap);
  const int tid = threadIdx.x;

  for (;;) {
    if (crank == 0 && tid == 0) {
      int k = atomicAdd(job_counter, 1);
      es->job = (k < njobs && pol.job_order) ? pol.job_order[k] : k;
      es->ktot = k;
    }
    engine_cluster_sync<CS>();
    const int job = es0->job;
    if (es0->ktot >= njobs) break;
    double xmin[DIM], xmax[DIM];
    pol.begin_job(job, psmem, xmin, xmax);
    if (tid == 0) es->nlive_chunk = 0;
    if (crank == 0 && tid == 0) {
      for (int d = 0; d < DIM; ++d) {
        S.cen[(size_t)d * S.cap] = 0.5 * (xmin[d] + xmax[d]);
        S.hw[(size_t)d * S.cap] = 0.5 * (xmax[d] - xmin[d]);
      }
      double v = 1;
      for (int d = 0; d < DIM; ++d) v *= 2 * (0.5 * (xmax[d] - xmin[d]));
      S.vol[0] = v;
      S.pend[0] = 0;
      es->nlive = 1;
      es->npend = 1;
      es->status = 0;
      es->stop = 0;
      es->neval = 0;
      es->sweeps = 0;
      es->ref = 0;
    }
    engine_cluster_sync<CS>();

    for (int sweep = 0;;) {
      // ---------------- evaluate the pending regions ----------------------
      const int npend = es0->npend;
      const int ref = REF ? es0->ref : 0;
      if constexpr (REF) pol.ref = ref;
      if constexpr (!REF) {
        // a cluster deals out chunks of CH regions, or single regions while a
        // sweep has fewer than CS * CH of them (all ranks then have work)
        const int step = (CS > 1 && npend < CS * CH) ? 1 : CH;
        for (int base = crank * step; base < npend; base += CS * step) {
          const int nreg = min(step, npend - base);
          const int npts = nreg * NP;
          // (a) point setup; points that need the expensive inner sums are
          //     appended to a compact live list
          for (int p = tid; p < npts; p += NT) {
            int r = S.pend[base + p / NP];
            double c[DIM], h[DIM], x[DIM];
  #pragma unroll
            for (int d = 0; d < DIM; ++d) {
              c[d] = S.cen[(size_t)d * S.cap + r];
              h[d] = S.hw[(size_t)d * S.cap + r];
            }
            rule_point<DIM>(p % NP, c, h, x);
            if (pol.setup(p, x, recs + (size_t)p * P::REC)) es->live_list[atomicAdd(&es->nlive_chunk, 1)] = p;
          }
          __syncthreads();
          // (b) (live point, group) items: equal-cost work for every thread
          const int nl = es->nlive_chunk;
          for (int it = tid; it < nl * G; it += NT) {
            int g = it / nl, q = it - g * nl;
            int p = es->live_list[q];
            double pv[PD];
            pol.group(recs + (size_t)p * P::REC, g, pv);
  #pragma unroll
            for (int k = 0; k < PD; ++k) part[((size_t)g * npts + p) * PD + k] = pv[k];
          }
          __syncthreads();
          // (c) per-point totals (fixed group order -> deterministic)
          for (int p = tid; p < npts; p += NT) {
            double s[NS * PD];
  #pragma unroll
            for (int k = 0; k < NS * PD; ++k) s[k] = 0;
            if (pol.is_live(recs + (size_t)p * P::REC))
              for (int g = 0; g < G; ++g) {
                const int sl = P::slot(g);
  #pragma unroll
                for (int k = 0; k < PD; ++k) s[sl * PD + k] += part[((size_t)g * npts + p) * PD + k];
              }
            pol.finalize(recs + (size_t)p * P::REC, s, fval + (size_t)p * FDIM);
          }
          if (tid == 0) es->nlive_chunk = 0;
          __syncthreads();
          for (int rr = tid; rr < nreg; rr += NT) {
            int r = S.pend[base + rr];
            double v[FDIM], e[FDIM];
            int sp;
            rule_combine<DIM, FDIM>(fval + (size_t)rr * NP * FDIM, S.vol[r], S.hw[r], v, e, &sp);
            double em = 0;
  #pragma unroll
            for (int k = 0; k < FDIM; ++k) {
              S.val[(size_t)k * S.cap + r] = v[k];
              S.err[(size_t)k * S.cap + r] = e[k];
              em = fmax(em, e[k]);
            }
            S.emax[r] = em;
            S.split[r] = (uint8_t)sp;
          }
          __syncthreads();
        }
      } else {
        // as below; a reference pass deals its few regions out evenly and shares
        // their items over the cluster's threads. Its first nfull regions take the
        // whole rule, the others its axis points.
        const int nfull = ref ? es0->nfull : npend;
        const int step = CS == 1 ? CH : ref ? min(CH, (npend + CS - 1) / CS) : npend < CS * CH ? 1 : CH;
        for (int base0 = 0; base0 < npend; base0 += CS * step) {
          const int base = base0 + crank * step;
          const int nreg = max(0, min(step, npend - base));
          auto points = [&](int first, int n) {  // of regions first .. first + n - 1
            const int nf = max(0, min(n, nfull - first));
            return nf * NP + (n - nf) * NPAX;
          };
          const int npts = points(base, nreg), nf = max(0, min(nreg, nfull - base));
          const bool shared = CS > 1 && ref;
          if (!shared && nreg == 0) break;
          // (a) point setup; points that need the expensive inner sums are
          //     appended to a compact live list
          for (int p = tid; p < npts; p += NT) {
            const int pa = p - nf * NP;  // index among the axis points
            int r = S.pend[base + (pa < 0 ? p / NP : nf + pa / NPAX)];
            double c[DIM], h[DIM], x[DIM];
  #pragma unroll
            for (int d = 0; d < DIM; ++d) {
              c[d] = S.cen[(size_t)d * S.cap + r];
              h[d] = S.hw[(size_t)d * S.cap + r];
            }
            rule_point<DIM>(pa < 0 ? p % NP : pa % NPAX, c, h, x);
            if (pol.setup(p, x, recs + (size_t)p * P::REC)) es->live_list[atomicAdd(&es->nlive_chunk, 1)] = p;
          }
          // (b) (live point, group) items: equal-cost work for every thread
          if (!shared) {
            __syncthreads();
            const int nl = es->nlive_chunk;
            for (int it = tid; it < nl * G; it += NT) {
              int g = it / nl, q = it - g * nl;
              int p = es->live_list[q];
              double pv[PD];
              pol.group(recs + (size_t)p * P::REC, g, pv);
  #pragma unroll
              for (int k = 0; k < PD; ++k) part[((size_t)g * npts + p) * PD + k] = pv[k];
            }
            __syncthreads();
          }
          if constexpr (CS > 1) {
            if (shared) {
              cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
              cl.sync();
              // items of rank 0, then of rank 1, ...: records are copied and
              // sums written through distributed shared memory
              int first = 0;
              for (int o = 0; o < CS && base0 + o * step < npend; ++o) {
                EngineShared<FDIM>* eo = cl.map_shared_rank(es, o);
                const char* ro = cl.map_shared_rank(recs, o);
                double* po = cl.map_shared_rank(part, o);
                const int no = points(base0 + o * step, min(step, npend - base0 - o * step)), nl = eo->nlive_chunk;
                const int skip = (crank * NT + tid - first) % (CS * NT);
                for (int it = skip < 0 ? skip + CS * NT : skip; it < nl * G; it += CS * NT) {
                  int g = it / nl, q = it - g * nl;
                  int p = eo->live_list[q];
                  alignas(16) char rec[(P::REC + 15) & ~15];
  #pragma unroll
                  for (int w = 0; w < P::REC / 4; ++w)
                    ((uint32_t*)rec)[w] = ((const uint32_t*)(ro + (size_t)p * P::REC))[w];
                  double pv[PD];
                  pol.group(rec, g, pv);
  #pragma unroll
                  for (int k = 0; k < PD; ++k) po[((size_t)g * no + p) * PD + k] = pv[k];
                }
                first += nl * G;
              }
              cl.sync();
            }
          }
          // (c) per-point totals (fixed group order -> deterministic)
          for (int p = tid; p < npts; p += NT) {
            double s[NS * PD];
  #pragma unroll
            for (int k = 0; k < NS * PD; ++k) s[k] = 0;
            if (pol.is_live(recs + (size_t)p * P::REC))
              for (int g = 0; g < G; ++g) {
                const int sl = P::slot(g);
  #pragma unroll
                for (int k = 0; k < PD; ++k) s[sl * PD + k] += part[((size_t)g * npts + p) * PD + k];
              }
            pol.finalize(recs + (size_t)p * P::REC, s, fval + (size_t)p * FDIM);
          }
          if (tid == 0) es->nlive_chunk = 0;
          __syncthreads();
          for (int rr = tid; rr < nreg; rr += NT) {
            int r = S.pend[base + rr];
            int sp;
            bool tie;
            if constexpr (DIM > 1) {
              if (rr >= nf) {  // the axis alone
                rule_axis<DIM, FDIM>(fval + (size_t)(nf * NP + (rr - nf) * NPAX) * FDIM, &sp, &tie);
                S.split[r] = (uint8_t)((S.split[r] & SPLIT_REF) | SPLIT_AXIS_REF | sp);
                continue;
              }
            }
            double v[FDIM], e[FDIM];
            rule_combine_ref<DIM, FDIM>(fval + (size_t)rr * NP * FDIM, S.vol[r], S.hw[r], v, e, &sp, &tie);
            sp |= ref ? SPLIT_REF | SPLIT_AXIS_REF : tie ? SPLIT_TIE : 0;
            double em = 0;
  #pragma unroll
            for (int k = 0; k < FDIM; ++k) {
              S.val[(size_t)k * S.cap + r] = v[k];
              S.err[(size_t)k * S.cap + r] = e[k];
              em = fmax(em, e[k]);
            }
            S.emax[r] = em;
            S.split[r] = (uint8_t)sp;
          }
          __syncthreads();
        }
      }
      if constexpr (CS > 1) engine_cluster_sync<CS>();
      // rank 0: totals, convergence, selection and splitting (or a reference
      // pass, or a stop)
      if (crank == 0) {
        if constexpr (REF)
          engine_select_call<DIM, FDIM, NT, REF>(S, es, cfg, (unsigned long long*)recs, stage_bytes, sweep, npend, ref,
                                              !pol.one);
        else
          engine_select<DIM, FDIM, NT, REF>(S, es, cfg, (unsigned long long*)recs, stage_bytes, sweep, npend, ref, false);
      }
      engine_cluster_sync<CS>();
      if (es0->stop) break;
      if (!REF || !es0->ref) ++sweep;
    }
    if (crank == 0) pol.end_job(job, es->V, es->E, es->neval, es->status);
    __syncthreads();
  }
  // no rank leaves while another may still read rank 0's shared memory
  if constexpr (CS > 1) cooperative_groups::this_cluster().sync();
}


}  // namespace tp
