// salsa_math.cuh -- FP64 division, roots, exp, log and pow with few FP64-pipe instructions.
//
// GB300 issues one FP64 warp instruction per 64 clocks and sub-partition (16 per SM; the
// same for 1 as for 32 active lanes), while its integer and FP32 pipes issue one per one or
// two clocks.  The step, the gradient chain and the sedimentation are bound by the FP64
// pipe, and most of their FP64 instructions sat inside divisions, roots and library
// functions.  The functions here keep FP64 results (errors of about half an ulp: no larger
// than those of the operations they replace) and move the work off that pipe:
//
//   quotients and roots -- a seed of about 40 bits from the FP32 approximation instruction
//     and one Newton step in two-float arithmetic (error-free products, Dekker 1971), put
//     together as a double with integer instructions, then one Newton correction with an
//     FMA residual in FP64 (Markstein 1990): the seed's error e leaves e^2 ~ 2^-80, far
//     below the final rounding;
//   exp, log, pow -- table + polynomial (Tang 1989/1990) in 64-bit fixed point, integers
//     throughout, with at least 9 guard bits; pow takes the logarithm to 63 fractional bits.
//
// Clocks per warp operation on one GB300 SM with 8 warps (latency of one warp in brackets),
// the operator or CUDA function -> the function here:
//   n / d   137 (576) -> 51 (288)      1 / d   86 (364) -> 35 (224)     sqrt  143 (609) -> 51 (319)
//   cbrt    234 (995) -> 83 (526)      exp    304 (1107) -> 70 (461)    log  539 (1991) -> 101 (642)
//   pow    1724 (6226) -> 160 (1016)
// Largest and mean error in ulps over 2 M arguments, CUDA -> here: quotients and square roots
// 0.500, 0.250 (both); cbrt 0.500, 0.250 (both); exp 0.853, 0.258 -> 0.617, 0.253; log 0.542,
// 0.250 -> 0.515, 0.250; pow (|y| <= 3) 1.34, 0.338 -> 0.645, 0.250.
// With them the FP64 step runs 1.19-1.44 times faster (grid384x384x160 block of 1.1 M cells
// 417 -> 299 ms; FP64 instructions per cell 9,620 -> 6,190) and the sedimentation 1.26 times.
//
// Arguments outside the fast range (zero, subnormal, infinite, NaN, extreme exponents) take
// the plain operation, out of line (divc: see there).  A unit that defines SALSA_MATH_PLAIN gets the plain
// operations throughout, one that defines SALSA_MATH_PLAIN_FUNCTIONS CUDA's cbrt, exp, log and pow.
#pragma once
#include <cstdint>
#include "salsa_math_tables.h"

namespace salsa {
namespace {

typedef unsigned long long fm_u64;
typedef unsigned __int128 fm_u128;

__device__ __forceinline__ float fm_rcp32(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float fm_rsqrt32(float x) { float r; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float fm_lg2_32(float x) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float fm_ex2_32(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

#ifdef SALSA_MATH_PLAIN
__device__ __forceinline__ double drcp(double d) { return 1. / d; }
__device__ __forceinline__ double ddiv(double n, double d) { return n / d; }
__device__ __forceinline__ double ddiv_r(double n, double d, double) { return n / d; }
__device__ __forceinline__ double divc(double x, double c) { return x / c; }
__device__ __forceinline__ double dsqrt(double x) { return sqrt(x); }
#else
// the plain operations, out of line: arguments outside the fast ranges
__device__ __noinline__ double fm_div_slow(double n, double d) { return n / d; }
__device__ __noinline__ double fm_sqrt_slow(double x) { return sqrt(x); }

// the double of bits (hi, lo) plus k * unit ulps: the low part of a two-float seed enters as
// an integer, read off a float sum with `magic` (1.5 * 2^e, so that the sum's last bit is
// 2^(e-23))
__device__ __forceinline__ double fm_join(unsigned hi, unsigned lo, float low, float magic, int unit) {
  const int k = __float_as_int(low + magic) - __float_as_int(magic);
  const long long b = (long long)(((fm_u64)hi << 32) | lo) + (long long)k * unit;
  return __longlong_as_double(b);
}

// ---- reciprocal seed: 1/d to about 2^-43, d normal with |exponent| below the caller's limit
__device__ __forceinline__ double fm_rcp_seed(unsigned hi, unsigned lo) {
  const float mf = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);   // top 23 mantissa bits
  const float ml = __int_as_float(((lo >> 6) & 0x7fffffu) | 0x3f800000u) - 1.f;              // the next 23, times 2^23
  const float r0 = fminf(fmaxf(fm_rcp32(mf), 0.5f), 0x1.fffffep-1f);   // in [1/2, 1)
  float e = fmaf(-mf, r0, 1.f);
  e = fmaf(-ml, r0 * 0x1p-23f, e);
  const unsigned b = __float_as_uint(r0);
  // r0's bits as a double, the exponent of d taken off, its sign put on
  const unsigned hr = ((b >> 3) + 0x38000000u + 0x3ff00000u - (hi & 0x7ff00000u)) | (hi & 0x80000000u);
  return fm_join(hr, b << 29, r0 * e, 0x1.8p-21f, 512);
}
// biased exponents 1023 +- 500, as a test on the high word
__device__ __forceinline__ bool fm_mid(unsigned hi) { return ((hi & 0x7fffffffu) - (523u << 20)) < (1000u << 20); }

// 1/d.  d's exponent within +-500.
__device__ __forceinline__ double drcp(double d) {
  const unsigned hi = (unsigned)__double2hiint(d);
  if (!fm_mid(hi)) return fm_div_slow(1., d);
  const double r = fm_rcp_seed(hi, (unsigned)__double2loint(d));
  return fma(fma(-d, r, 1.), r, r);
}

// n/d with r = drcp(d) at hand (several quotients by one denominator).  Exponents within
// +-500; n = 0 too.
__device__ __forceinline__ double ddiv_r(double n, double d, double r) {
  const unsigned hi = (unsigned)__double2hiint(d), hn = (unsigned)__double2hiint(n);
  if (!(fm_mid(hi) && (fm_mid(hn) || ((hn << 1) | (unsigned)__double2loint(n)) == 0u))) return fm_div_slow(n, d);
  const double q = n * r;
  return fma(fma(-d, q, n), r, q);
}

// n/d.  Exponents within +-500; n = 0 too.
__device__ __forceinline__ double ddiv(double n, double d) {
  const unsigned hi = (unsigned)__double2hiint(d), hn = (unsigned)__double2hiint(n);
  if (!(fm_mid(hi) && (fm_mid(hn) || n == 0.))) return fm_div_slow(n, d);
  const double r = fm_rcp_seed(hi, (unsigned)__double2loint(d));
  const double q = n * r;
  return fma(fma(-d, q, n), r, q);
}

// x / c for a positive constant c: the product with 1/c as a sum of two doubles, folded at
// compile time (exact when c is a power of two).  The low product is left out, by a selection
// on integers, where it cannot be formed (x zero, subnormal, above 2^877, infinite or NaN: an
// infinite x against a negative low part gave NaN): one ulp there.
__device__ __forceinline__ double divc(double x, double c) {
  const double r = 1. / c, l = fma(-c, r, 1.) * r;
  if (l == 0.) return x * r;
  const unsigned hi = (unsigned)__double2hiint(x);
  const bool low = (hi & 0x7fffffffu) - (1u << 20) < (1899u << 20);
  return fma(x, r, low ? x * l : __hiloint2double((int)(hi & 0x80000000u), 0));
}
// sqrt(x), x's exponent within +-500, or zero
__device__ __forceinline__ double dsqrt(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (hi - (523u << 20) >= (1000u << 20)) return x == 0. ? x : fm_sqrt_slow(x);
  const unsigned odd = (hi >> 20) & 1u;                    // odd biased exponent: even power of two
  const float sc = __int_as_float(0x40000000u - (odd << 23));   // 1 or 2
  const float mf = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | (0x40000000u - (odd << 23)));   // in [1, 4)
  const float ml = (__int_as_float(((lo >> 6) & 0x7fffffu) | 0x3f800000u) - 1.f) * sc;
  const float y0 = fminf(fmaxf(fm_rsqrt32(mf), 0.5f), 0x1.fffffep-1f);
  const float p = y0 * y0, pe = fmaf(y0, y0, -p);
  float e = fmaf(-mf, p, 1.f);
  e = fmaf(-mf, pe, e);
  e = fmaf(-ml * 0x1p-23f, p, e);
  const float yl = y0 * e * fmaf(0.375f, e, 0.5f);
  const unsigned b = __float_as_uint(y0);
  const unsigned half = (((hi >> 20) + 1u) >> 1) << 20;    // (E' + 512) << 20
  const double y = fm_join((b >> 3) + 0x38000000u + (512u << 20) - half, b << 29, yl, 0x1.8p-20f, 1024);   // 1/sqrt(x)
  const double s = x * y;
  const double hy = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));   // y/2
  return fma(fma(-s, s, x), hy, s);
}

#ifndef SALSA_MATH_PLAIN_FUNCTIONS
__device__ __noinline__ double fm_cbrt_slow(double x) { return cbrt(x); }
__device__ __noinline__ double fm_exp_slow(double x) { return exp(x); }
__device__ __noinline__ double fm_log_slow(double x) { return log(x); }
__device__ __noinline__ double fm_pow_slow(double x, double y) { return pow(x, y); }

// cbrt(x), x positive and normal, or zero
__device__ __forceinline__ double dcbrt(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (hi - 0x00100000u >= 0x7fe00000u) return x == 0. ? x : fm_cbrt_slow(x);
  const unsigned E = (hi >> 20) + 3u;                      // exponent + 3 * 342
  const unsigned k = (E * 43691u) >> 17, rem = E - 3u * k;   // E / 3: x = 2^(3 (k - 342)) m, m in [1, 8)
  const float mf = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | ((127u + rem) << 23));
  const float ml = (__int_as_float(((lo >> 6) & 0x7fffffu) | 0x3f800000u) - 1.f) * __int_as_float((104u + rem) << 23);
  const float z = fm_ex2_32(fm_lg2_32(mf) * (-1.f / 3.f));   // m^(-1/3)
  const float zz = z * z;
  const float c = fminf(fmaxf(mf * zz, 1.f), 0x1.fffffep+0f);
  const float p = c * c, pe = fmaf(c, c, -p);
  float w = zz * (1.f / 3.f);
  w = fmaf(w, fmaf(p, -3.f * w, 1.f), w);                  // 1 / (3 c^2)
  const float q = p * c, qe = fmaf(p, c, -q);
  float e = mf - q;
  e = (e - qe) + fmaf(-pe, c, ml);
  e *= w;
  e = fmaf(e * z, -e, e);                                  // m^(1/3) - c to second order
  const unsigned b = __float_as_uint(c), bw = __float_as_uint(w);
  const double c0 = fm_join((b >> 3) + 0x38000000u, b << 29, e, 0x1.8p-18f, 2048);
  const double wd = __hiloint2double((int)((bw >> 3) + 0x38000000u), (int)(bw << 29));
  const double xm = __hiloint2double((int)((hi & 0x000fffffu) | ((1023u + rem) << 20)), (int)lo);
  const double c2 = c0 * c0, c2l = fma(c0, c0, -c2);
  double r = fma(-c2, c0, xm);
  r = fma(-c2l, c0, r);
  r = fma(r, wd, c0);
  return __hiloint2double(__double2hiint(r) + (int)((k << 20) - (342u << 20)), __double2loint(r));
}

// ---- exponentials ----
// 2^(+-P 2^-(sh + 64)) as a double from the fixed-point magnitude P (sh in [42, 127]); ok is
// false when the result is not a normal number.
__device__ __forceinline__ double fm_exp2_fix(fm_u64 ph, fm_u64 pl, int sh, bool neg, bool &ok) {
  fm_u64 f;
  unsigned ki;
  if (sh < 64) {
    f = (ph << (64 - sh)) | (pl >> sh);
    ki = (unsigned)(ph >> sh);
  } else {
    f = ph >> (sh - 64);
    ki = 0u;
  }
  int k = (int)ki;
  if (neg) {
    k = f ? ~k : -k;
    f = 0ull - f;
  }
  const unsigned j = (unsigned)(f >> 57);
  const fm_u64 T = __ldg(&c_exp2_tab[j]);
  // t = f_low ln2 = u / 128 < 2^-7.5; e^t - 1 = u/2^7 + u^2/2^15 + ... in units of 2^-64.  The
  // terms from the fourth on need no more than 32-bit products.
  const fm_u64 u = __umul64hi(f << 7, 0xb17217f7d1cf79acull);
  const unsigned uh = (unsigned)(u >> 32);
  unsigned h = 0x00444444u + __umulhi(uh, 0x16c1u);
  h = 0xaaaaaaabu + __umulhi(uh, h);
  const fm_u64 h3 = 0x0000015555555555ull + __umulhi(uh, h);
  const fm_u64 h2 = 0x0002000000000000ull + __umul64hi(u, h3);
  const fm_u64 w = (u >> 7) + __umul64hi(__umul64hi(u, u), h2);
  const fm_u64 R = T + __umul64hi(T, w);                      // in [2^63, 2^64)
  ok = (unsigned)(k + 1021) < 2043u;
  return __longlong_as_double((long long)(((fm_u64)(unsigned)(k + 1022) << 52) + (R >> 11) + ((R >> 10) & 1ull)));
}

// exp(x)
__device__ __forceinline__ double dexp(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned ax = hi & 0x7fffffffu;
  if (ax >= 0x40862000u) {                                    // |x| >= 708, infinite or NaN
    if (hi >= 0xc0874a00u && hi < 0xfff00000u) return 0.;     // x < -745.2
    return fm_exp_slow(x);
  }
  const fm_u64 M = ((fm_u64)((ax & 0x000fffffu) | 0x00100000u) << 32) | lo;
  const int sh = min(1074 - (int)(ax >> 20), 127);            // subnormal x: a shift of 127, e^x = 1
  const fm_u64 L = 0xb8aa3b295c17f0bcull;                     // log2(e) 2^63
  bool ok;
  return fm_exp2_fix(__umul64hi(M, L), M * L, sh, (int)hi < 0, ok);
}

// ln(x) 2^117 of a positive normal x as a 128-bit two's complement number (absolute error
// 2^-63; relative 2^-58 near x = 1, where the table's constant and the exponent vanish)
__device__ __forceinline__ fm_u128 fm_log_fix(unsigned hi, unsigned lo) {
  const unsigned i = (hi >> 13) & 127u;
  const unsigned c = __ldg(&c_log_c[i]);
  const fm_u64 l = __ldg(&c_log_l[i]);
  const int E = (int)(hi >> 20) - 1023 + (i == 127u);
  const fm_u64 M = ((fm_u64)((hi & 0x000fffffu) | 0x00100000u) << 32) | lo;
  const long long r = (long long)(M * c) - (1ll << 61);       // m c/512 - 1, exactly, in units of 2^-61
  const bool neg = r < 0;
  const fm_u64 a = neg ? (fm_u64)(-r) : (fm_u64)r;            // below 2^54
  // ln(1 + r)/r = 1 - r/2 + r^2/3 - ... + r^8/9: even and odd parts in b = a^2
  const fm_u64 u = a << 10, b = __umul64hi(u, u);
  const unsigned bh = (unsigned)(b >> 32);
  const fm_u64 e2 = 13743895347ull + __umulhi(bh, 599186u + __umulhi(bh, 28u));
  const fm_u64 ev = __umul64hi(b, 0x0001555555555555ull + (((fm_u64)bh * (unsigned)(e2 >> 2)) >> 30));
  const unsigned o2 = 89478485u + __umulhi(bh, 4096u);
  const fm_u64 o1 = (1ull << 41) + __umulhi(bh, o2);
  const fm_u64 o0 = (1ull << 56) + __umul64hi(b, o1);
  const fm_u64 od = __umul64hi(u, o0);
  const fm_u64 Q = (1ull << 63) + (ev >> 1) + (neg ? (od >> 1) : 0ull - (od >> 1));
  const fm_u64 ph = __umul64hi(a, Q), pl = a * Q;             // |ln(1+r)| 2^124
  fm_u128 S = (((fm_u128)ph << 64) | pl) >> 7;
  if (neg) S = 0 - S;
  // E ln 2 + l in units of 2^-64
  const unsigned Ea = (unsigned)abs(E);
  const fm_u64 p0 = (fm_u64)Ea * 0xd1cf79acu, p1 = (fm_u64)Ea * 0xb17217f7u + (p0 >> 32);
  fm_u128 K = ((fm_u128)(p1 >> 32) << 64) | ((p1 << 32) | (unsigned)p0);
  if (E < 0) K = 0 - K;
  K += l;
  return S + (K << 53);
}

__device__ __forceinline__ bool fm_posnormal(unsigned hi) { return hi - 0x00100000u < 0x7fe00000u; }

// magnitude of a fixed-point logarithm as R 2^(10 - lz - 63), R's leading bit set; S != 0
__device__ __forceinline__ fm_u64 fm_lead(fm_u128 S, bool &neg, int &lz) {
  fm_u64 sh = (fm_u64)(S >> 64), sl = (fm_u64)S;
  neg = (long long)sh < 0;
  if (neg) { sl = 0ull - sl; sh = ~sh + (sl == 0ull); }
  lz = __clzll((long long)sh);
  return lz ? (sh << lz) | (sl >> (64 - lz)) : sh;
}

// log(x)
__device__ __forceinline__ double dlog(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (!fm_posnormal(hi)) return fm_log_slow(x);
  const fm_u128 S = fm_log_fix(hi, lo);
  if (S == 0) return 0.;
  bool neg;
  int lz;
  const fm_u64 R = fm_lead(S, neg, lz);
  const fm_u64 bits = ((fm_u64)(unsigned)(1032 - lz) << 52) + (R >> 11) + ((R >> 10) & 1ull);
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

// pow(x, y) of a positive normal x; |y| up to 512 (the error of the logarithm, 2^-63, is
// multiplied by y)
__device__ __forceinline__ double dpow(double x, double y) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned hy = (unsigned)__double2hiint(y), ly = (unsigned)__double2loint(y), ay = hy & 0x7fffffffu;
  if (fm_posnormal(hi) && ay < 0x40800000u) {
    const fm_u128 S = fm_log_fix(hi, lo);
    if (S == 0) return 1.;
    bool neg, ok;
    int lz;
    const fm_u64 R = __umul64hi(fm_lead(S, neg, lz), 0xb8aa3b295c17f0bcull);   // |log2 x| 2^(62 - 10 + lz)
    const fm_u64 M = ((fm_u64)((ay & 0x000fffffu) | 0x00100000u) << 32) | ly;
    const int sh = min(1063 + lz - (int)(ay >> 20), 127);
    const double p = fm_exp2_fix(__umul64hi(M, R), M * R, max(sh, 42), neg != ((int)hy < 0), ok);
    if (sh >= 42 && ok) return p;
  }
  return fm_pow_slow(x, y);
}

#endif  // SALSA_MATH_PLAIN_FUNCTIONS
#endif  // SALSA_MATH_PLAIN

#if defined(SALSA_MATH_PLAIN) || defined(SALSA_MATH_PLAIN_FUNCTIONS)
__device__ __forceinline__ double dcbrt(double x) { return cbrt(x); }
__device__ __forceinline__ double dexp(double x) { return exp(x); }
__device__ __forceinline__ double dlog(double x) { return log(x); }
__device__ __forceinline__ double dpow(double x, double y) { return pow(x, y); }
#endif

// the float forms of templates written for both types
__device__ __forceinline__ float ddiv(float n, float d) { return n / d; }
__device__ __forceinline__ float divc(float x, float c) { return x / c; }

}  // namespace
}  // namespace salsa
