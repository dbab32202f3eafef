// FP64-accurate arithmetic on the integer pipe.
//
// GB300 issues FP64 instructions at 1/64 of the FP32 rate (measured per SM and
// clock: DFMA 1.6, IMAD.WIDE 53, IADD 108, SHF/LOP3 57; CUDA's FP64 exp2 0.094,
// log2 0.050, 1/x 0.35), so a 64-bit mantissa product made of three IMAD.WIDE
// is about nine times cheaper than a DMUL. This header holds the pieces the
// FP64 integrands are made of:
//   Sf         a positive number m 2^e with a 64-bit mantissa (sums and products
//              of mantissas with up to four leading zeros are within 2^-57; the
//              exponent has 32 bits, so nothing in between overflows or underflows)
//   Q52        a signed 64-bit fixed-point number in units of 2^-52: the
//              base-2 exponents
//   i64_exp2   2^x of a Q52 by a 256-entry table and a fifth-order polynomial
//              (relative error below 2^-58)
//   i64_log2   log2 of a 64-bit mantissa in Q57 by the same kind of table
// Everything is plain integer arithmetic, the same on host and device, so the
// error bounds are tested on the CPU; sf_rcp's start value alone differs (the
// SFU's on the device), and its steps are tested with starts 2 ulp off.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace tp {

#if defined(__CUDACC__)
#define TP_HD __host__ __device__ __forceinline__
#else
#define TP_HD inline
#endif

// ---- tables (64-bit constants from the definitions) -------------------------
struct I64Tables {
  uint64_t ex2[256];  // 2^(j/256), Q63
  uint64_t lc[256];   // -log2 rc[j], Q62
  uint32_t rc[256];   // 1 / m over the cell [1 + j/256, 1 + (j+1)/256), Q31: 1 at j = 0, 1/2 at j = 255
};

namespace i64detail {
// 64 x 64 -> high 64 bits, rounded to nearest
constexpr uint64_t mulhi_rn(uint64_t a, uint64_t b) {
  const unsigned __int128 p = (unsigned __int128)a * b + ((unsigned __int128)1 << 63);
  return (uint64_t)(p >> 64);
}
// 2^(2^-k), k = 1..8, in Q63
constexpr uint64_t ROOTS[8] = {0xb504f333f9de6484ull, 0x9837f0518db8a96full, 0x8b95c1e3ea8bd6e7ull, 0x85aac367cc487b15ull,
                               0x82cd8698ac2ba1d7ull, 0x8164d1f3bc030773ull, 0x80b1ed4fd999ab6cull, 0x8058d7d2d5e5f6b1ull};
// -log2 of c (Q31 in [1/2, 1]) in Q62, bit by bit: squaring doubles the logarithm
constexpr uint64_t neg_log2(uint32_t c) {
  if (c == 1u << 31) return 0;
  if (c == 1u << 30) return 1ull << 62;
  uint64_t x = (uint64_t)c << 33;  // Q64
  uint64_t bits = 0;               // log2(2 c), Q62
  for (int k = 0; k < 62; ++k) {
    // x: (2 c)^(2^k) / 2 in [1/2, 1), Q64
    const unsigned __int128 s = ((unsigned __int128)x * x + ((unsigned __int128)1 << 62)) >> 63;  // y^2 / 2, Q64: in [1/2, 2)
    bits <<= 1;
    if (s >> 64) {
      bits |= 1;
      x = (uint64_t)(s >> 1);
    } else {
      x = (uint64_t)s;
    }
  }
  return (1ull << 62) - bits;
}
constexpr I64Tables make_tables() {
  I64Tables t{};
  for (int j = 0; j < 256; ++j) {
    uint64_t m = 1ull << 63;
    for (int k = 0; k < 8; ++k)
      if (j & (128 >> k)) m = mulhi_rn(m, ROOTS[k]) << 1;
    t.ex2[j] = m;
  }
  for (int j = 0; j < 256; ++j) {
    // the exact ends keep log2 accurate next to powers of two
    const uint32_t c = j == 0 ? 1u << 31 : j == 255 ? 1u << 30 : (uint32_t)((1ull << 40) / (513 + 2 * j));
    t.rc[j] = c;
    t.lc[j] = neg_log2(c);
  }
  return t;
}
}  // namespace i64detail

// sin(pi (2 k + 1) / 256), Q64
#if defined(__CUDACC__)
static __device__ constexpr uint64_t d_i64sin[64] = {
    0x03243a3f9bd8f08dull, 0x096c32baca2ae68bull, 0x0fb2b73cfc106ff7ull, 0x15f6d00a9aa418c1ull,
    0x1c3785c79ec2d4f6ull, 0x2273e19db5eaed57ull, 0x28aaed62527cb3b6ull, 0x2edbb3bca17e628full,
    0x3505404b6008a13cull, 0x3b269fca8a8622bbull, 0x413ee038dff6b7fdull, 0x474d10fd336cf747ull,
    0x4d50430b860546c3ull, 0x53478909e39da892ull, 0x5931f774fc9f1844ull, 0x5f0ea4c477339c06ull,
    0x64dca98ef24f5cb4ull, 0x6a9b20adb4ff262aull, 0x70492760047b9a7full, 0x75e5dd6e1b8e2555ull,
    0x7b70654bbde35623ull, 0x80e7e43a61f5b6cbull, 0x864b826aec4c74e6ull, 0x8b9a6b1ef6da4502ull,
    0x90d3ccc99f5ac58bull, 0x95f6d92fd79f4fbbull, 0x9b02c58832cf95c0ull, 0x9ff6ca9a2ab6a26dull,
    0xa4d224dcd849c5b0ull, 0xa99414951aacae5full, 0xae3bddf3280c620dull, 0xb2c8c92f83c1eb88ull,
    0xb73a22a755457448ull, 0xbb8f3af81b93095dull, 0xbfc7671ab8bb84c7ull, 0xc3e2007dd175f5a5ull,
    0xc7de651f7ca06749ull, 0xcbbbf7a63eba0dd5ull, 0xcf7a1f794d7ca1b2ull, 0xd31848d817d70e17ull,
    0xd695e4f10ea88570ull, 0xd9f269f7aab88c29ull, 0xdd2d5339ac8692fdull, 0xe046213392aa486cull,
    0xe33c59a4439cd8ecull, 0xe60f879fe7e2e1e5ull, 0xe8bf3ba1f1aedfbcull, 0xeb4b0b9e4f345617ull,
    0xedb29311c504d652ull, 0xeff573116df1555dull, 0xf21352595e0bf351ull, 0xf40bdd5a6688662full,
    0xf5dec646f85ba1c7ull, 0xf78bc51f239e12c6ull, 0xf91297bbb1d6cdbeull, 0xfa7301d859796671ull,
    0xfbaccd1d0903bb0aull, 0xfcbfc926484cd43bull, 0xfdabcb8caeba091cull, 0xfe70afeb6d33d6a2ull,
    0xff0e57e5ead848d1ull, 0xff84ab2c738d6a03ull, 0xffd3977ff7bae4e9ull, 0xfffb10b4dc96dabcull,
};
#endif
static constexpr uint64_t h_i64sin[64] = {
    0x03243a3f9bd8f08dull, 0x096c32baca2ae68bull, 0x0fb2b73cfc106ff7ull, 0x15f6d00a9aa418c1ull,
    0x1c3785c79ec2d4f6ull, 0x2273e19db5eaed57ull, 0x28aaed62527cb3b6ull, 0x2edbb3bca17e628full,
    0x3505404b6008a13cull, 0x3b269fca8a8622bbull, 0x413ee038dff6b7fdull, 0x474d10fd336cf747ull,
    0x4d50430b860546c3ull, 0x53478909e39da892ull, 0x5931f774fc9f1844ull, 0x5f0ea4c477339c06ull,
    0x64dca98ef24f5cb4ull, 0x6a9b20adb4ff262aull, 0x70492760047b9a7full, 0x75e5dd6e1b8e2555ull,
    0x7b70654bbde35623ull, 0x80e7e43a61f5b6cbull, 0x864b826aec4c74e6ull, 0x8b9a6b1ef6da4502ull,
    0x90d3ccc99f5ac58bull, 0x95f6d92fd79f4fbbull, 0x9b02c58832cf95c0ull, 0x9ff6ca9a2ab6a26dull,
    0xa4d224dcd849c5b0ull, 0xa99414951aacae5full, 0xae3bddf3280c620dull, 0xb2c8c92f83c1eb88ull,
    0xb73a22a755457448ull, 0xbb8f3af81b93095dull, 0xbfc7671ab8bb84c7ull, 0xc3e2007dd175f5a5ull,
    0xc7de651f7ca06749ull, 0xcbbbf7a63eba0dd5ull, 0xcf7a1f794d7ca1b2ull, 0xd31848d817d70e17ull,
    0xd695e4f10ea88570ull, 0xd9f269f7aab88c29ull, 0xdd2d5339ac8692fdull, 0xe046213392aa486cull,
    0xe33c59a4439cd8ecull, 0xe60f879fe7e2e1e5ull, 0xe8bf3ba1f1aedfbcull, 0xeb4b0b9e4f345617ull,
    0xedb29311c504d652ull, 0xeff573116df1555dull, 0xf21352595e0bf351ull, 0xf40bdd5a6688662full,
    0xf5dec646f85ba1c7ull, 0xf78bc51f239e12c6ull, 0xf91297bbb1d6cdbeull, 0xfa7301d859796671ull,
    0xfbaccd1d0903bb0aull, 0xfcbfc926484cd43bull, 0xfdabcb8caeba091cull, 0xfe70afeb6d33d6a2ull,
    0xff0e57e5ead848d1ull, 0xff84ab2c738d6a03ull, 0xffd3977ff7bae4e9ull, 0xfffb10b4dc96dabcull,
};

#if defined(__CUDACC__)
static __device__ constexpr I64Tables d_i64tab = i64detail::make_tables();
#endif
static constexpr I64Tables h_i64tab = i64detail::make_tables();

// ---- 64-bit products ----------------------------------------------------------
// high 64 bits of a b without the carry of the low halves: below the true value
// by less than 3
TP_HD uint64_t i64_mulhi(uint64_t a, uint64_t b) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t x = (uint64_t)a1 * b0, y = (uint64_t)a0 * b1;
  return ((uint64_t)a1 * b1 + (x >> 32)) + (y >> 32);
}
TP_HD uint64_t i64_mulhi_exact(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
// high word of a b + c 2^32 (c + the high word must fit)
TP_HD uint32_t i64_mad32(uint32_t a, uint32_t b, uint32_t c) {
  return (uint32_t)(((uint64_t)a * b + ((uint64_t)c << 32)) >> 32);
}

// right shift by any n >= 0
TP_HD uint64_t i64_shr(uint64_t v, int n) {
#if defined(__CUDA_ARCH__)
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));  // amounts above 63 give 0
  return r;
#else
  return n > 63 ? 0 : v >> n;
#endif
}

// ---- positive numbers m 2^e -----------------------------------------------------
struct Sf {
  uint64_t m;
  int e;
};

TP_HD Sf sf_mul(Sf a, Sf b) { return {i64_mulhi(a.m, b.m), a.e + b.e + 64}; }

// the operand with the larger exponent keeps its unit (after one common shift
// that makes room for the carry), the other is shifted to it; both lose less
// than a unit of a result of 2^58 or more
TP_HD Sf sf_add(Sf a, Sf b) {
  const int d = a.e - b.e;
  const int sa = (d < 0 ? -d : 0) + 1, sb = (d > 0 ? d : 0) + 1;
  return {i64_shr(a.m, sa) + i64_shr(b.m, sb), (d > 0 ? a.e : b.e) + 1};
}

TP_HD Sf sf_one() { return {1ull << 63, -63}; }

// positive normal double
TP_HD Sf sf_from(double x) {
#if defined(__CUDA_ARCH__)
  const uint64_t u = (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
#endif
  return {(u << 11) | (1ull << 63), (int)(u >> 52) - 1086};
}

TP_HD int i64_clz(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
TP_HD Sf sf_norm(Sf a) {
  const int z = i64_clz(a.m);
  return {a.m << z, a.e - z};
}

// to double, rounded; results below the normal range give 0, above it inf
TP_HD double sf_to(Sf a) {
#if defined(__CUDA_ARCH__)
  const double v = __ull2double_rn(a.m);
  const int hi = __double2hiint(v), ex = (hi >> 20) + a.e;
  if ((unsigned)(ex - 1) >= 2046u) return ex < 1 ? 0.0 : __longlong_as_double(0x7ff0000000000000ll);
  return __hiloint2double(hi + (a.e << 20), __double2loint(v));
#else
  const double v = (double)a.m;
  uint64_t u;
  memcpy(&u, &v, 8);
  const int ex = (int)(u >> 52) + a.e;
  if ((unsigned)(ex - 1) >= 2046u) return ex < 1 ? 0.0 : HUGE_VAL;
  u += (uint64_t)(int64_t)a.e << 52;
  double r;
  memcpy(&r, &u, 8);
  return r;
#endif
}

// 1 / a: a start of 21 bits or more and one third-order step,
// y (1 + e + e^2) with e = 1 - m y. a normalised, yu the start's float bits
TP_HD Sf sf_rcp_step(Sf a, uint32_t yu) {
  const uint32_t h = (uint32_t)(a.m >> 32);  // m: Q64 in [1/2, 1)
  const uint32_t yq = yu >= 0x40000000u ? 0xffffff00u : 0x80000000u | (yu << 8);  // Q31 in [1, 2)
  const uint64_t my = (uint64_t)h * yq + (((uint64_t)(uint32_t)a.m * yq) >> 32);  // Q63, near 1
  const int64_t e = (int64_t)((1ull << 63) - my);                                 // |e| < 2^-20
  const int32_t eh = (int32_t)(e >> 21);                                          // Q42
  const int64_t s = e + (((int64_t)eh * eh) >> 21);                               // e + e^2, Q63
  const int64_t c = ((int64_t)(int32_t)(s >> 32) * (int64_t)yq) + (int64_t)(((uint64_t)(uint32_t)s * yq) >> 32);
  return {((uint64_t)yq << 31) + (uint64_t)c, -126 - a.e};  // y (1 + s) in Q62
}
// the float of m's upper bits, and 1 / a from its reciprocal
TP_HD uint32_t sf_rcp_arg(Sf a) { return 0x3f000000u | (((uint32_t)(a.m >> 32) << 1) >> 9); }
TP_HD Sf sf_rcp(Sf a) {
  a = sf_norm(a);
  const uint32_t fu = sf_rcp_arg(a);
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fu)));
  const uint32_t yu = __float_as_uint(y);
#else
  uint32_t yu;
  float f, y;
  memcpy(&f, &fu, 4);
  y = 1.0f / f;
  memcpy(&yu, &y, 4);
#endif
  return sf_rcp_step(a, yu);
}

// ---- 2^x -----------------------------------------------------------------------
// mantissa and exponent of 2^x, x in Q52
TP_HD Sf i64_exp2(int64_t x, const uint64_t* __restrict__ tab) {
  // ln2^k / k!
  constexpr uint64_t C1 = 0xb17217f7d1cf79acull, C2 = 0x3d7f7bff058b1d51ull;  // Q64
  constexpr uint32_t C3 = 3814213304u, C4 = 2581847u, C5 = 1398u;            // Q36, Q28, Q20
  const int n = (int)(x >> 52);
  const uint64_t f = (uint64_t)x << 12;
  const uint32_t j = (uint32_t)(f >> 56);
  const uint64_t r = f & 0x00ffffffffffffffull;  // T, Q64, below 2^-8
  const uint32_t t = (uint32_t)(f >> 24);        // T, Q40
  const uint32_t s4 = i64_mad32(t, C5, C4);      // Q28
  const uint32_t v = i64_mad32(t, s4, C3);       // Q36
  const uint64_t u = C2 + (((uint64_t)t * v) >> 12);
  const uint64_t w = C1 + i64_mulhi(r, u);
  const uint64_t p = i64_mulhi(r, w);  // 2^T - 1
  const uint64_t b = tab[j];
  return {b + i64_mulhi(b, p), n - 63};
}

// double to fixed point in units of 2^-B, |x| < 2^(62 - B)
template <int B>
TP_HD int64_t i64_fix(double x) {
#if defined(__CUDA_ARCH__)
  // 2^B enters through the exponent field (x = 0 stays below 2^-900)
  return __double2ll_rn(__hiloint2double(__double2hiint(x) + (B << 20), __double2loint(x)));
#else
  return llrint(ldexp(x, B));
#endif
}

// ---- sine and cosine ---------------------------------------------------------------
// of x in [0, 8), Q62 signed, within 2^-57.6 absolute (two units of 2^-60 turns
// of the argument; 2^-58.7 measured): the quarter turn's 64
// cells by table, sin and cos of the distance d to a cell's centre
// (|d| < pi/256) by their series to d^7 and d^6
TP_HD void i64_sincos(double x, const uint64_t* __restrict__ tab, int64_t& sn, int64_t& cs) {
  constexpr uint64_t INV_2PI = 0x28be60db9391054aull, PI_128 = 0x06487ed5110b4612ull;  // Q64
  constexpr uint64_t R6 = 0x2aaaaaaaaaaaaaabull, R24 = 0x0aaaaaaaaaaaaaabull, R120 = 0x0222222222222222ull;
  const uint64_t xf = (uint64_t)i64_fix<60>(x);
  const uint64_t u = (i64_mulhi_exact(xf, INV_2PI) << 4) | ((xf * INV_2PI) >> 60);  // turns, Q64
  const uint32_t quad = (uint32_t)(u >> 62), k = (uint32_t)(u >> 56) & 63u;
  const int64_t r = (int64_t)((u << 8) ^ (1ull << 63));  // place in the cell minus 1/2, Q64
  const uint64_t d = i64_mulhi((uint64_t)(r < 0 ? -r : r), PI_128 << 1) >> 1;  // (pi/2) / 64 of it
  const uint64_t d2 = i64_mulhi(d, d);
  const uint64_t h = (d2 >> 1) - i64_mulhi(d2, i64_mulhi(d2, R24 - (uint64_t)(((d2 >> 32) * 5965232u))));       // 1 - cos: 2^32 / 720
  const uint64_t s = d - i64_mulhi(d, i64_mulhi(d2, R6 - i64_mulhi(d2, R120 - (uint64_t)((d2 >> 32) * 852176u))));  // sin: 2^32 / 5040
  const uint64_t S = tab[k], C = tab[63 - k];
  const int64_t Sh = (int64_t)(i64_mulhi(S, h) >> 2), Ch = (int64_t)(i64_mulhi(C, h) >> 2);
  int64_t Cs = (int64_t)(i64_mulhi(C, s) >> 2), Ss = (int64_t)(i64_mulhi(S, s) >> 2);
  if (r < 0) Cs = -Cs, Ss = -Ss;
  const int64_t sv = (int64_t)(S >> 2) - Sh + Cs, cv = (int64_t)(C >> 2) - Ch - Ss;
  // quarter turns: (s, c) -> (c, -s)
  const int64_t a = (quad & 1) ? cv : sv, b = (quad & 1) ? sv : cv;
  sn = (quad & 2) ? -a : a;
  cs = ((quad + 1) & 2) ? -b : b;
}
// Q62 to double
TP_HD double i64_q62(int64_t q) { return (double)q * 0x1p-62; }

// ---- rounding of a double to float ------------------------------------------------
// whether every number within ulps units of 2^-52 2^floor(log2 |v|) of v rounds
// to the same float (v a normal float's range)
TP_HD uint64_t i64_bits(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
TP_HD bool i64_rounds_alike(double v, int ulps) {
  const int low = (int)((uint32_t)i64_bits(v) & 0x1fffffffu), d = low - 0x10000000;
  return (d < 0 ? -d : d) > ulps;
}
// the same for an absolute error of ulps units of 2^-53 2^floor(log2 |scale|):
// no value is further than 2^28 units from the middle of two floats, so a larger
// bound is never met (and its shift would leave 32 bits)
TP_HD bool i64_rounds_alike(double v, double scale, int ulps) {
  const int e = ((int)(i64_bits(scale) >> 32) >> 20 & 2047) - ((int)(i64_bits(v) >> 32) >> 20 & 2047) + 1, de = e > 0 ? e : 0;
  return de < 20 && ulps < (0x10000000 >> de) && i64_rounds_alike(v, ulps << de);
}

// ---- log2 -----------------------------------------------------------------------
// log2 of a normalised mantissa m in [1, 2) (Q63): -log2 c + log2(1 + t) with
// t = m c - 1 and c the table's reciprocal of m's 1/256-wide cell; Q62, within 2^-57
TP_HD int64_t i64_log2m(uint64_t m, const uint32_t* __restrict__ rc, const uint64_t* __restrict__ lc) {
  constexpr uint64_t A1 = 0xb8aa3b295c17f0bcull;  // 1 / ln2, Q63
  constexpr uint64_t A2 = 0xb8aa3b295c17f0bcull;  // 1 / (2 ln2), Q64
  constexpr int64_t A3 = 67680425505800;  // 1 / (3 ln2), Q47
  constexpr int32_t A4 = 774541002, A5 = 619632802, A6 = 516360668;  // 1 / (k ln2), Q31
  const uint32_t j = (uint32_t)(m >> 55) & 255u;
  const uint32_t c = rc[j];  // Q31
  const uint64_t mc = (m >> 32) * c + (((m & 0xffffffffull) * c) >> 32);  // Q62
  const int64_t t = (int64_t)((mc - (1ull << 62)) << 2);                  // Q64, |t| <= 2^-8
  const int32_t th = (int32_t)(t >> 25);                                 // Q39
  // s = a3 - t (a4 - t (a5 - t a6)), Q47
  const int32_t s5 = A5 - (int32_t)(((int64_t)th * A6) >> 39);
  const int32_t s4 = A4 - (int32_t)(((int64_t)th * s5) >> 39);
  const uint64_t s3 = (uint64_t)(A3 - (((int64_t)th * s4) >> 23)) << 17;  // Q64
  const uint64_t ta = (uint64_t)(t < 0 ? -t : t);                        // |t|, Q64
  const uint64_t ts = i64_mulhi(ta, s3);
  const uint64_t q = t < 0 ? A2 + ts : A2 - ts;                // a2 - t s: Q64
  const uint64_t tq = i64_mulhi(ta, q) >> 1;                   // |t| q, Q63
  const uint64_t w = t < 0 ? A1 + tq : A1 - tq;                // (log2(1 + t)) / t, Q63
  const int64_t p = (int64_t)(i64_mulhi(ta, w) >> 1);          // Q62
  return (int64_t)lc[j] + (t < 0 ? -p : p);
}

}  // namespace tp
