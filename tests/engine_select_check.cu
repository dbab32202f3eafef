// One sweep's selection and splitting (engine_select) on given region errors:
// selected sets against a sort on the host (tests/test_gpu_engine_select.py).
// Prints "name ok" or "name ..." with what differs, one line a case.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "tp_cubature.cuh"

using namespace tp;
typedef unsigned long long u64;
constexpr int DIM = 2, NT = 256, STAGE = 32 << 10;

template <int FDIM>
__global__ void k_select(char* store, EngineCfg cfg, int nlive, int stage_bytes, int* out) {
  __shared__ EngineShared<FDIM> es;
  extern __shared__ u64 stage[];
  Slot<DIM, FDIM> S;
  S.init(store, cfg.cap);
  if (threadIdx.x == 0) {
    es.nlive = nlive;
    es.npend = 0;
    es.stop = es.status = es.ref = 0;
    es.neval = 0;
    es.nlive_chunk = 0;
  }
  __syncthreads();
  engine_select<DIM, FDIM, NT, false>(S, &es, cfg, stage, stage_bytes, 0, 0, 0, false);
  __syncthreads();
  if (threadIdx.x == 0) {
    out[0] = es.stop;
    out[1] = es.status;
    out[2] = es.npend;
    out[3] = es.nlive;
  }
  for (int i = threadIdx.x; i < cfg.cap; i += NT) out[4 + i] = es.stop || i >= es.npend ? -1 : S.pend[i];
}

// the region store's layout on the host
template <int FDIM>
struct Store {
  double *cen, *hw, *vol, *val, *err, *emax;
  int* pend;
  uint8_t* split;
  Store(char* base, int cap) {
    cen = (double*)base;
    hw = cen + (size_t)DIM * cap;
    vol = hw + (size_t)DIM * cap;
    val = vol + cap;
    err = val + (size_t)FDIM * cap;
    emax = err + (size_t)FDIM * cap;
    pend = (int*)(emax + cap);
    split = (uint8_t*)(pend + cap);
  }
};

static double as_double(u64 u) {
  double d;
  memcpy(&d, &u, 8);
  return d;
}
static u64 as_u64(double d) {
  u64 u;
  memcpy(&u, &d, 8);
  return u;
}
static int failures = 0;

template <int FDIM>
static void run(const std::string& name, const std::vector<double>& err, double val, double rel_tol, int stage_bytes,
                int cap) {
  const int n = (int)err.size() / FDIM;
  EngineCfg cfg{0.0, rel_tol, TP_NORM_L1, cap, 1000};
  std::vector<char> h(Slot<DIM, FDIM>::bytes(cap), 0);
  char* d;
  int* d_out;
  cudaMalloc(&d, h.size());
  cudaMalloc(&d_out, sizeof(int) * (4 + cap));
  Store<FDIM> S(h.data(), cap);
  for (int i = 0; i < n; ++i) {
    for (int q = 0; q < DIM; ++q) S.cen[(size_t)q * cap + i] = 0.5, S.hw[(size_t)q * cap + i] = 0.25;
    S.vol[i] = 1.0;
    S.emax[i] = 0;
    for (int k = 0; k < FDIM; ++k) {
      S.val[(size_t)k * cap + i] = val / n;
      S.err[(size_t)k * cap + i] = err[(size_t)i * FDIM + k];
      S.emax[i] = fmax(S.emax[i], err[(size_t)i * FDIM + k]);
    }
    S.split[i] = (uint8_t)(i % DIM);
  }
  const std::vector<double> emax(S.emax, S.emax + n);
  cudaMemcpy(d, h.data(), h.size(), cudaMemcpyHostToDevice);
  cudaFuncSetAttribute(k_select<FDIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGE);
  k_select<FDIM><<<1, NT, STAGE>>>(d, cfg, n, stage_bytes, d_out);
  std::vector<int> out(4 + cap);
  const cudaError_t e = cudaMemcpy(out.data(), d_out, sizeof(int) * (4 + cap), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(d_out);
  if (e != cudaSuccess) {
    printf("%s %s\n", name.c_str(), cudaGetErrorString(e));
    exit(1);
  }
  std::string why;
  // regions whose new halves are listed, in order
  std::vector<int> sel;
  if (!out[0]) {
    if (out[2] % 2 || out[3] != n + out[2] / 2 || out[3] > cap) why = "counts";
    for (int k = 0; k < out[2] / 2 && why.empty(); ++k) {
      sel.push_back(out[4 + 2 * k]);
      if (out[4 + 2 * k + 1] != n + k) why = "second half";
      if (sel[k] < 0 || sel[k] >= n || (k && sel[k] <= sel[k - 1])) why = "list";
    }
  }
  double etot = 0;
  for (double v : err) etot += v;
  if (std::isfinite(etot)) {
    // largest key whose regions and those above leave no more than the tolerance,
    // in the same fixed-point fractions of the total
    const double tol = FDIM * fabs(val) * rel_tol, qs = 0x1p62 / etot;
    std::vector<int> at(n);
    for (int i = 0; i < n; ++i) at[i] = i;
    std::sort(at.begin(), at.end(), [&](int a, int b) { return emax[a] > emax[b]; });
    std::vector<u64> below(n + 1, 0);
    for (int k = n; k-- > 0;) {
      double es = 0;
      for (int q = 0; q < FDIM; ++q) es += err[(size_t)at[k] * FDIM + q];
      below[k] = below[k + 1] + (u64)(es * qs);
    }
    double tau = 0;
    for (int k = 0; k < n; ++k)
      if ((k + 1 == n || emax[at[k + 1]] < emax[at[k]]) && (double)below[k + 1] <= tol * qs) {
        tau = emax[at[k]];
        break;
      }
    std::vector<int> want;
    for (int i = 0; i < n; ++i)
      if (emax[i] >= tau) want.push_back(i);
    if (n + (int)want.size() > cap) {
      if (!(out[0] && out[1] == 1)) why = "cap";
    } else if (out[0] || sel != want) {
      why = "selected " + std::to_string(sel.size()) + " want " + std::to_string(want.size()) + " stop " + std::to_string(out[0]);
    }
  } else if (!out[0] && sel.size() > (size_t)n) {
    why = "selected too many";
  }
  printf("%s %s\n", name.c_str(), why.empty() ? "ok" : why.c_str());
  failures += !why.empty();
}

int main() {
  std::mt19937_64 g(5);
  auto U = [&] { return (double)(g() >> 11) * 0x1p-53; };
  auto logu = [&](int n, double lo, double hi) {  // 2^lo .. 2^hi
    std::vector<double> e(n);
    for (double& v : e) v = exp2(lo + U() * (hi - lo));
    return e;
  };
  auto both = [&](const char* name, const std::vector<double>& e, double frac, int cap = 1 << 15) {
    double t = 0;
    for (double v : e) t += v;
    // a tolerance away from the sums' roundings: frac of the total error
    for (int stage : {STAGE, 512, 16})
      run<1>(std::string(name) + "/1/" + std::to_string(stage), e, 1.0, t * frac, stage, cap);
    std::vector<double> e2(2 * e.size());
    double t2 = 0;
    for (size_t i = 0; i < e.size(); ++i) {
      e2[2 * i] = e[i];
      e2[2 * i + 1] = e[i] * (0.25 + 0.5 * U());
      t2 += e2[2 * i] + e2[2 * i + 1];
    }
    for (int stage : {STAGE, 512, 16})
      run<2>(std::string(name) + "/2/" + std::to_string(stage), e2, 1.0, t2 * frac / 2, stage, cap);  // (|V| sums two)
  };
  for (int n : {1, 2, 31, 32, 33, 255, 257, 1023, 1025, 9000}) both(("range" + std::to_string(n)).c_str(), logu(n, -30, 0), 0.1);
  // more candidates than the list holds: keys within 1/16 octave, and within 2^-40
  both("dense", logu(6000, -0.05, 0), 0.437);
  std::vector<double> e(6000);
  for (size_t i = 0; i < e.size(); ++i) e[i] = as_double(as_u64(1.0) + 2 * (g() % 4096));
  both("bits", e, 0.437);
  // a cut below the 255 bins of 1/8 octave: everything but a tiny rest has to go
  both("deep", logu(3000, -200, 0), 1e-12);
  both("deeper", logu(3000, -500, 0), 1e-17);
  {
    std::vector<double> d = logu(2000, -120, -60);
    d.push_back(1.0);
    both("outlier", d, 1e-25);
  }
  // ties: all equal, and two values
  both("equal", std::vector<double>(700, 0.125), 0.31);
  for (size_t i = 0; i < e.size(); ++i) e[i] = i % 3 ? 1.0 : 2.0;
  both("two", e, 0.31);
  // zeros among them, and the cap
  for (size_t i = 0; i < e.size(); ++i) e[i] = i % 2 ? 0.0 : U();
  both("zeros", e, 0.2);
  both("cap", logu(3000, -1, 0), 0.01, 4096);
  // not finite: it ends, with indices of regions
  for (double bad : {(double)INFINITY, (double)NAN}) {
    std::vector<double> d = logu(1500, -10, 0);
    d[700] = bad;
    run<1>(std::isnan(bad) ? "nan/1" : "inf/1", d, 1.0, 1e-3, STAGE, 1 << 14);
    std::vector<double> d2(2 * d.size());
    for (size_t i = 0; i < d.size(); ++i) d2[2 * i] = d[i], d2[2 * i + 1] = 0.5 * U();
    run<2>(std::isnan(bad) ? "nan/2" : "inf/2", d2, 1.0, 1e-3, 512, 1 << 14);
  }
  return failures ? 1 : 0;
}
