// flint_fix.cuh -- 64-bit fixed-point evaluation of the kinetics' exponents.
//
// Why fixed point: an SM of this GPU takes one FP64 warp instruction per 16
// cycles (DFMA 16.2, DADD and DMUL 19.1, a conversion 16.3 measured), but a
// 64 x 64 -> high-64 integer multiply per 4.5 and a 64-bit integer add per ~1.
// The kinetics kernels are bound by the FP64 pipe, and most of their FP64 work
// formed the arguments of exponentials (ln k, Gibbs differences) and the
// exponentials themselves.  Those quantities are sums of moderate size whose
// *absolute* error matters, which is what fixed point gives: with 52 fraction
// bits an argument carries an absolute error of about 2^-52, where the FP64
// chain it replaces rounds at every step to 2^-53 of a magnitude of 10-60.
// The result is therefore closer to the exact value, not further from it.
//
// All logarithms are base 2.  Formats (Qn: n fraction bits in a signed 64-bit
// integer):
//   exponents (log2 k, g/RT in octaves)   Q52   |x| < 2^11
//   log2 T - 10                           Q61   T in [129, 8192)
//   1/T (T > 128)                         Q70
//   T/2^13 (high range), T/2^11 (low)     Q63
//   E log2e, a5 (kelvin)                  Q45   |x| < 2^18
//   temperature exponents b               Q55   |x| < 2^8
// A mechanism uses this path when every coefficient and every exponent over
// the temperature range fits its format (ImageLayout::fix, decided when the
// mechanism is packed); a cell outside [fix_Tlo, fix_Thi) takes the FP64 path.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace flint {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ int64_t mulhi_s(int64_t a, int64_t b) { return __mul64hi(a, b); }
__device__ __forceinline__ uint64_t mulhi_u(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
__device__ __forceinline__ int mulhi_i(int a, int b) { return __mulhi(a, b); }
__device__ __forceinline__ int clz64(uint64_t x) { return __clzll((long long)x); }
__device__ __forceinline__ int64_t d_bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double bits_d(int64_t x) { return __longlong_as_double(x); }
#else
inline int64_t mulhi_s(int64_t a, int64_t b) { return (int64_t)(((__int128)a * b) >> 64); }
inline uint64_t mulhi_u(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
inline int mulhi_i(int a, int b) { return (int)(((int64_t)a * b) >> 32); }
inline int clz64(uint64_t x) { return x ? __builtin_clzll(x) : 64; }
inline int64_t d_bits(double x) { int64_t b; __builtin_memcpy(&b, &x, 8); return b; }
inline double bits_d(int64_t x) { double d; __builtin_memcpy(&d, &x, 8); return d; }
#endif

constexpr int64_t ONE52 = 1ll << 52;
constexpr int FIX_EXP2 = 256;    // entries of the exp2 table
constexpr int FIX_LOG2 = 128;    // rows of the log2 table

// 2^x for x in Q52, by a 256-entry table of 2^((j + 1/2)/256) (Q62) and the
// Taylor polynomial of 2^(w/256) - 1, w in [-1/2, 1/2), to degree 5 (the first
// omitted term is below 2^-65): table-driven as P. T. P. Tang, ACM TOMS 15(2),
// 1989.  The two low-order coefficients are applied with 64-bit products, the
// others with 32-bit ones whose weight makes them exact enough (below 2^-59).
// Error below 0.51 ulp of the returned double (tests/test_fix_cpu.py).  Below
// the normal range returns 0, above it inf.  No FP64 instruction: 3 64-bit and
// 3 32-bit products, about 22 cycles per SM and warp where the FP64 form took
// 9 instructions = 150 cycles.
__host__ __device__ __forceinline__ double exp2_q52(int64_t X, const int64_t* __restrict__ tab) {
  constexpr int64_t K1 = 799144290325165979ll;     // ln2/256                   Q68
  constexpr int64_t K2 = 1081884007225522ll;       // (ln2/256)^2 / 2           Q68
  constexpr int K3 = 1907106652;                   // (ln2/256)^3 / 6           Q59
  constexpr int K4 = 1290923;                      // (ln2/256)^4 / 24          Q59
  constexpr int K5 = 699;                          // (ln2/256)^5 / 120         Q59
  const int n = (int)(X >> 52);
  const uint64_t F = (uint64_t)X << 12;
  const int j = (int)(F >> 56);
  const int64_t w = (int64_t)((F << 8) ^ 0x8000000000000000ull);   // Q64, [-1/2, 1/2)
  const int w32 = (int)(w >> 32);
  int t = K4 + mulhi_i(w32, K5);
  t = K3 + mulhi_i(w32, t);
  const int64_t u2 = K2 + (((int64_t)w32 * t) >> 23);
  const int64_t u1 = K1 + mulhi_s(w, u2);
  const int64_t p = mulhi_s(w, u1);                                 // 2^(w/256) - 1, Q68
  const int64_t b = tab[j];
  const int64_t R = b + (mulhi_s(b, p) >> 4);                       // Q62, in [1, 2)
  const int64_t bits = ((int64_t)(n + 1022) << 52) + ((R + 512) >> 10);
  const double r = bits_d(bits);
  return n < -1022 ? 0.0 : (n > 1023 ? bits_d(0x7ff0000000000000ll) : r);
}

// log2 of the significand of a normal positive double, Q62 in [0, 1) up to its
// rounding; e receives the exponent.  128 rows (c, -log2 c), c = 1/(row centre)
// in Q64: r = y c - 1 (|r| < 2^-8) and log2(1 + r) by its Taylor polynomial to
// r^7 (first omitted term below 2^-66), after P. T. P. Tang, ACM TOMS 16(4),
// 1990.  Error below 2^-58.
__host__ __device__ __forceinline__ int64_t log2_q62(double x, const int64_t* __restrict__ tab, int* e) {
  constexpr int64_t A0 = 3326628274461080623ll;    // log2e                     Q61
  constexpr int64_t A1 = -12994641697113596ll;     // -log2e/2 / 2^7            Q61
  constexpr int64_t A2 = 67680425505800ll;         // log2e/3 / 2^14            Q61
  constexpr int A3 = -774541002;                   // -log2e/4 / 2^21           Q52
  constexpr int A4 = 4840881;                      // log2e/5 / 2^28            Q52
  constexpr int A5 = -31516;                       // -log2e/6 / 2^35           Q52
  constexpr int A6 = 211;                          // log2e/7 / 2^42            Q52
  const int64_t b = d_bits(x);
  *e = (int)(b >> 52) - 1023;
  const uint64_t mant = (uint64_t)b & 0xfffffffffffffull;
  const int j = (int)(mant >> 45);
  const uint64_t Y = (mant << 11) | 0x8000000000000000ull;          // Q63
  const uint64_t C = (uint64_t)tab[2 * j];
  const int64_t rs = (int64_t)(mulhi_u(Y, C) - 0x8000000000000000ull) << 7;   // r 2^7, Q63
  const int s = (int)(rs >> 32);
  int t = A5 + (mulhi_i(s, A6) << 1);
  t = A4 + (mulhi_i(s, t) << 1);
  t = A3 + (mulhi_i(s, t) << 1);
  int64_t u = A2 + (((int64_t)s * t) >> 22);
  u = A1 + (mulhi_s(rs, u) << 1);
  u = A0 + (mulhi_s(rs, u) << 1);
  return tab[2 * j + 1] + (mulhi_s(rs, u) >> 5);
}

// log2 x in Q52 (x a normal positive double).
__host__ __device__ __forceinline__ int64_t log2_q52(double x, const int64_t* __restrict__ tab) {
  int e;
  const int64_t f = log2_q62(x, tab, &e);
  return ((int64_t)e << 52) + ((f + 512) >> 10);
}

// A fixed-point value (q fraction bits) as the nearest double.
__host__ __device__ __forceinline__ double fix2d(int64_t X, int q) {
  const uint64_t sgn = (uint64_t)X & 0x8000000000000000ull;
  uint64_t m = (uint64_t)(X < 0 ? -X : X);
  const int lz = clz64(m);
  m = (lz < 64) ? m << lz : 0;
  const int64_t bits = ((int64_t)(1023 + 62 - lz - q) << 52) + (int64_t)((m + 1024) >> 11);
  return X == 0 ? 0.0 : bits_d((int64_t)((uint64_t)bits | sgn));
}

// A double as Q52, saturated to |x| < 2^11 (rounded towards minus infinity
// below 2^-52; NaN saturates).
__host__ __device__ __forceinline__ int64_t d2fix52(double x) {
  const int64_t b = d_bits(x);
  const int e = (int)((b >> 52) & 0x7ff) - 1023;
  int64_t m = (b & 0xfffffffffffffll) | ONE52;
  m = e > 10 ? (2047ll << 52) : (e >= 0 ? m << e : (e > -54 ? m >> -e : 0));
  return b < 0 ? -m : m;
}

// The powers of T that the polynomials and Arrhenius exponents take.
struct FixT {
  int64_t L;     // log2 T - 10, Q61
  int64_t v;     // 1/T, Q70
  int64_t t13;   // T / 2^13, Q63
  int64_t t11;   // T / 2^11, Q63 (meaningful for T < 2048)
};

__host__ __device__ __forceinline__ FixT fix_T(double T, const int64_t* __restrict__ ltab) {
  FixT f;
  int e;
  const int64_t lg = log2_q62(T, ltab, &e);
  f.L = ((int64_t)(e - 10) << 61) + ((lg + 1) >> 1);
  const int64_t b = d_bits(T);
  const uint64_t Y = (((uint64_t)b & 0xfffffffffffffull) << 11) | 0x8000000000000000ull;
  f.t13 = (int64_t)(Y >> (13 - e));
  f.t11 = (int64_t)(e < 11 ? Y >> (11 - e) : Y >> 1);
  // 1/y of the significand y: a single-precision seed r (24 bits) and one
  // third-order (Chebyshev) step r (1 + d + d^2), d = 1 - y r, |d| < 2^-21; d is
  // exact (y and r have 53 and 24 bits, and only the low 64 bits of y r matter)
#ifdef __CUDA_ARCH__
  const float y = __int_as_float((int)(0x3f800000u | (uint32_t)((Y >> 40) & 0x7fffffu)));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  const uint32_t rb = (uint32_t)__float_as_int(r);
#else
  const float y = (float)((double)(Y >> 40) / 8388608.0);
  const float r = 1.0f / y;
  uint32_t rb;
  __builtin_memcpy(&rb, &r, 4);
#endif
  // r in (1/2, 1] as Q24
  const uint32_t r24 = ((rb & 0x7fffffu) | 0x800000u) << ((int)(rb >> 23) - 126);
  const int64_t d = -(int64_t)((Y >> 3) * r24);                              // Q84
  const int d32 = (int)(d >> 32);                                            // Q52
  const int64_t c = (d >> 3) + (((int64_t)d32 * d32) >> 23);                 // Q81
  const int64_t r0 = (int64_t)r24 << 38;                                     // Q62
  f.v = (e <= 8 ? r0 << (8 - e) : r0 >> (e - 8)) + (mulhi_s(r0, c) >> (e + 9));   // Q79 -> Q70
  return f;
}

// 1/x in FP64: the SM's reciprocal approximation (about 2^-20) and one
// third-order (Chebyshev) step r (1 + e + e^2), e = 1 - x r; relative error below
// 2^-52.  Zero, subnormal, huge, inf and NaN take the division.
#ifdef __CUDACC__
static __device__ __noinline__ double recip_slow(double x) { return 1.0 / x; }
__device__ __forceinline__ double recip(double x) {
  const uint32_t eh = ((uint32_t)__double2hiint(x) & 0x7ff00000u);
  if (eh - 0x03000000u >= 0x79000000u) return recip_slow(x);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
#endif

}  // namespace flint
