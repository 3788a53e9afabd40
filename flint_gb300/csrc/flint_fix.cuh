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
// The exponent is therefore closer to the exact value, not further from it.  (Outside
// the exponents the kernels trade a division for a product by a reciprocal, two
// roundings for one; against 64-bit references the rates, Jacobians and right-hand
// sides come out closer all the same.)
//
// All logarithms are base 2.  Formats (Qn: n fraction bits in 64 bits):
//   exponents (log2 k, g/RT in octaves)   Q52 signed   |x| < 2^11
//   log2 T - 7                            Q61 unsigned, T in [129, 8192)
//   log2 c of a factor to a power         Q57 signed within 2^+-63, Q53 beyond
//   orders of such factors                Q60 unsigned, below 16
//   1/T                                   Q70 unsigned (T > 128)
//   T/2^13 (high range), T/2^11 (low)     Q63 unsigned
//   E log2e (kelvin)                      Q45 signed   |x| < 2^18
//   a5, a5 log2e (kelvin)                 Q46 signed   |x| < 2^17
//   temperature exponents b, a0           Q55 signed   |x| < 2^8
// A product is one unsigned 64 x 64 -> high-64 multiplication: a signed factor
// is stored with its sign bit flipped (x + 2^63), which adds exactly half of the
// other, non-negative, factor to the product; that half is a property of the
// cell and is taken off once (a signed product costs twice the instructions).
// A mechanism uses this path when every coefficient and every exponent over
// the temperature range fits its format (ImageLayout::fix, decided when the
// mechanism is packed); a cell outside [fix_Tlo, fix_Thi) takes the FP64 path.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace flint {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint64_t mulhi_u(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
__device__ __forceinline__ uint32_t mulhi_32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ int clz64(uint64_t x) { return __clzll((long long)x); }
__device__ __forceinline__ int64_t d_bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double bits_d(int64_t x) { return __longlong_as_double(x); }
#else
inline uint64_t mulhi_u(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
inline uint32_t mulhi_32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int clz64(uint64_t x) { return x ? __builtin_clzll(x) : 64; }
inline int64_t d_bits(double x) { int64_t b; __builtin_memcpy(&b, &x, 8); return b; }
inline double bits_d(int64_t x) { double d; __builtin_memcpy(&d, &x, 8); return d; }
#endif

// High half of a product without its low x low part: at most 3 too small.
__host__ __device__ __forceinline__ uint64_t mulhi_a(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
}

constexpr int64_t ONE52 = 1ll << 52;
constexpr int FIX_EXP2 = 256;    // entries of the exp2 table
constexpr int FIX_LOG2 = 128;    // rows of the log2 table

// 2^x for x in Q52, by a 256-entry table of 2^(j/256) (Q62, with the rounding
// half of the last double place added) and the Taylor polynomial of 2^(w/256) -
// 1, w in [0, 1), to degree 5 (the first omitted term is below 2^-60):
// table-driven as P. T. P. Tang, ACM TOMS 15(2), 1989.  The low-order
// coefficients are applied with 64-bit products, the others with 32-bit ones
// whose weight makes them exact enough.  Error below 0.53 ulp of the returned
// double (tests/test_fix_cpu.py).  Above the normal range returns inf.  Below it,
// SUB: the value cut to a subnormal one; else 0, for exponents that fix_Tlo keeps
// within the range (SUB costs 5 % of the source terms of 1 M cells, 4.71 -> 4.94
// ms).  No FP64 instruction, where the FP64 form took 9 (150 cycles per SM and
// warp).
template <bool SUB = false>
__host__ __device__ __forceinline__ double exp2_q52(int64_t X, const uint64_t* __restrict__ tab) {
  constexpr uint64_t K1 = 799144290325165979ull;   // ln2/256                   Q68
  constexpr uint64_t K2 = 1081884007225522ull;     // (ln2/256)^2 / 2           Q68
  constexpr uint32_t K3 = 3814213304u;             // (ln2/256)^3 / 6           Q60
  constexpr uint32_t K4 = 2581847u;                // (ln2/256)^4 / 24          Q60
  constexpr uint32_t K5 = 1398u;                   // (ln2/256)^5 / 120         Q60
  const int hi = (int)(X >> 32);
  const int j = (hi >> 12) & 255;
  const uint64_t w = (uint64_t)X << 20;                             // Q64, [0, 1)
  const uint32_t w32 = (uint32_t)(w >> 32);
  uint32_t t = K4 + mulhi_32(w32, K5);
  t = K3 + mulhi_32(w32, t);
  const uint64_t u2 = (uint64_t)mulhi_32(w32, t) * 256u + K2;
  const uint64_t u1 = K1 + mulhi_a(w, u2);
  const uint64_t p = mulhi_a(w, u1);                                // 2^(w/256) - 1, Q68
  const uint64_t b = tab[j];
  const uint64_t R = b + (mulhi_a(b, p) >> 4);                      // Q62, in [1, 2)
  const int n1 = (hi >> 20) + 1022;                                 // biased exponent - 1
  if (SUB) {
    const int e0 = n1 > 0 ? n1 : 0, sh = 10 + e0 - n1;              // 10, more below the normal range
    const double r = bits_d(((int64_t)e0 << 52) + (int64_t)(R >> (sh < 63 ? sh : 63)));
    return n1 <= 2045 ? r : bits_d(0x7ff0000000000000ll);
  }
  const double r = bits_d(((int64_t)n1 << 52) + (int64_t)(R >> 10));
  return (unsigned)n1 <= 2045u ? r : (n1 < 0 ? 0.0 : bits_d(0x7ff0000000000000ll));
}

// log2 of the significand of a normal positive double, Q62 in [0, 1); e receives
// the exponent.  128 rows (c, -log2 c), c just above 1/(1 + j/128) in Q63: r =
// y c - 1 in [0, 2^-7) and log2(1 + r) by its Taylor polynomial to r^8 (first
// omitted term below 2^-65), after P. T. P. Tang, ACM TOMS 16(4), 1990.  Error
// below 2^-59.
__host__ __device__ __forceinline__ int64_t log2_q62(double x, const uint64_t* __restrict__ tab, int* e) {
  constexpr uint64_t A0 = 6653256548922161246ull;  // log2e                     Q62
  constexpr uint64_t A1 = 25989283394227192ull;    // log2e/2 / 2^7             Q62
  constexpr uint64_t A2 = 135360851011600ull;      // log2e/3 / 2^14            Q62
  constexpr uint32_t A3 = 3098164009u;             // log2e/4 / 2^21            Q54
  constexpr uint32_t A4 = 19363525u;               // log2e/5 / 2^28            Q54
  constexpr uint32_t A5 = 126065u;                 // log2e/6 / 2^35            Q54
  constexpr uint32_t A6 = 844u;                    // log2e/7 / 2^42            Q54
  constexpr uint32_t A7 = 6u;                      // log2e/8 / 2^49            Q54
  const int64_t b = d_bits(x);
  *e = (int)(b >> 52) - 1023;
  const uint64_t mant = (uint64_t)b & 0xfffffffffffffull;
  const int j = (int)(mant >> 45);
  const uint64_t Y = (mant << 11) | 0x8000000000000000ull;          // Q63
  const uint64_t s = (mulhi_u(Y, tab[2 * j]) - 0x4000000000000000ull) << 9;   // r 2^7, Q64
  const uint32_t s32 = (uint32_t)(s >> 32);
  uint32_t t = A6 - mulhi_32(s32, A7);
  t = A5 - mulhi_32(s32, t);
  t = A4 - mulhi_32(s32, t);
  t = A3 - mulhi_32(s32, t);
  uint64_t u = A2 - (uint64_t)mulhi_32(s32, t) * 256u;
  u = A1 - mulhi_a(s, u);
  u = A0 - mulhi_a(s, u);
  return (int64_t)(tab[2 * j + 1] + (mulhi_a(s, u) >> 7));
}

// log2 x in Q52 (x a normal positive double).
__host__ __device__ __forceinline__ int64_t log2_q52(double x, const uint64_t* __restrict__ tab) {
  int e;
  const int64_t f = log2_q62(x, tab, &e);
  return ((int64_t)e << 52) + ((f + 512) >> 10);
}

// A fixed-point value (q fraction bits) as the nearest double.  The rounding bit is
// added after the shift: before it the sum of a value just below a power of two would
// leave the 64 bits, and its carry is the next exponent.
__host__ __device__ __forceinline__ double fix2d(int64_t X, int q) {
  const uint64_t sgn = (uint64_t)X & 0x8000000000000000ull;
  uint64_t m = (uint64_t)(X < 0 ? -X : X);
  const int lz = clz64(m);
  m = (lz < 64) ? m << lz : 0;
  const int64_t bits = ((int64_t)(1023 + 62 - lz - q) << 52) + (int64_t)((m >> 11) + ((m >> 10) & 1));
  return X == 0 ? 0.0 : bits_d((int64_t)((uint64_t)bits | sgn));
}

// A double as Q52, saturated to |x| < 2^11 (cut towards zero below 2^-52; NaN
// saturates).
__host__ __device__ __forceinline__ int64_t d2fix52(double x) {
  const int64_t b = d_bits(x);
  const int e = (int)((b >> 52) & 0x7ff) - 1023;
  int64_t m = (b & 0xfffffffffffffll) | ONE52;
  m = e > 10 ? (2047ll << 52) : (e >= 0 ? m << e : (e > -54 ? m >> -e : 0));
  return b < 0 ? -m : m;
}

// The powers of T that the polynomials and Arrhenius exponents take.
struct FixT {
  uint64_t L;     // log2 T - 7, Q61
  uint64_t v;     // 1/T, Q70
  uint64_t t13;   // T / 2^13, Q63
  uint64_t t11;   // T / 2^11, Q63 (meaningful for T < 2048)
  int64_t ka;     // what the flipped signs of b and E add to an Arrhenius exponent
};

__host__ __device__ __forceinline__ FixT fix_T(double T, const uint64_t* __restrict__ ltab) {
  FixT f;
  int e;
  const int64_t lg = log2_q62(T, ltab, &e);
  f.L = ((uint64_t)(e - 7) << 61) + ((uint64_t)(lg + 1) >> 1);
  const int64_t b = d_bits(T);
  const uint64_t Y = (((uint64_t)b & 0xfffffffffffffull) << 11) | 0x8000000000000000ull;
  f.t13 = Y >> (13 - e);
  f.t11 = e < 11 ? Y >> (11 - e) : Y >> 1;
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
  const uint64_t c = (uint64_t)((d >> 3) + (((int64_t)d32 * d32) >> 23)) ^ 0x8000000000000000ull;   // Q81, sign flipped
  const uint64_t r0 = (uint64_t)r24 << 38;                                   // Q62
  const int64_t m = (int64_t)(mulhi_u(r0, c) - (r0 >> 1));                   // Q79
  f.v = (e <= 8 ? r0 << (8 - e) : r0 >> (e - 8)) + (uint64_t)(m >> (e + 9));
  f.ka = -(int64_t)(f.L >> 1) - (int64_t)f.v;
  return f;
}

// log2 A + b log2 T - E log2e/T: a = log2 A + 7 b (Q52); b (Q55) and -E log2e
// (Q45) with their signs flipped.
__host__ __device__ __forceinline__ int64_t fix_arrhenius(int64_t a, uint64_t b, uint64_t e, const FixT& f) {
  return a + f.ka + (int64_t)mulhi_u(b, f.L) + (int64_t)(mulhi_u(e, f.v) << 1);
}

// c1 + t (c2 + t (...)), sign flipped (+ 2^63): coefficients (stride S, signs
// flipped) in Qn, Q(n - 1), ... by order, t in Q63.
template <int N>
__host__ __device__ __forceinline__ uint64_t fix_horner(const uint64_t* __restrict__ c, int S, uint64_t t) {
  uint64_t a = c[(N - 1) * S];
#pragma unroll
  for (int j = N - 2; j >= 0; --j) a = c[j * S] + (mulhi_u(a, t) << 2) - (t << 1);
  return a;
}

// Polynomial of order 4, result in Q52: c[0] plain (Q52), c[1..4] as in
// fix_horner with n = 51.
__host__ __device__ __forceinline__ int64_t fix_poly5(const uint64_t* __restrict__ c, int S, uint64_t t) {
  return (int64_t)(c[0] + (mulhi_u(fix_horner<4>(c + S, S, t), t) << 2) - (t << 1));
}

// g/RT in octaves (Q52): c = constant, a0 (Q55), c1..c4 (Q53...), a5 log2e (Q46).
__host__ __device__ __forceinline__ int64_t fix_gibbs(const uint64_t* __restrict__ c, int S, uint64_t t, const FixT& f) {
  return (int64_t)(c[0] + ((f.L >> 1) + (t >> 1) - (f.v >> 1)) + mulhi_u(c[6 * S], f.v) - mulhi_u(c[S], f.L) -
                   mulhi_u(fix_horner<4>(c + 2 * S, S, t), t));
}

// h/RT (Q52): the polynomial and a5/T.
__host__ __device__ __forceinline__ int64_t fix_enthalpy(const uint64_t* __restrict__ c, int S, uint64_t t, const FixT& f) {
  return fix_poly5(c, S, t) + (int64_t)(mulhi_u(c[5 * S], f.v) - (f.v >> 1));
}

// a / b, correctly rounded, from y = the correctly rounded 1/b: q = a y is within
// one unit of the quotient, its remainder a - b q is exact, and q + r y rounds to
// the quotient (P. W. Markstein, IBM J. Res. Dev. 34(1), 1990).  Needs
// exponents away from the ends; others take the division.
__host__ __device__ inline double div_by(double a, double b, double y) {
#ifdef __CUDA_ARCH__
  const uint32_t ea = (uint32_t)__double2hiint(a) & 0x7ff00000u, eb = (uint32_t)__double2hiint(b) & 0x7ff00000u;
#else
  const uint32_t ea = (uint32_t)(d_bits(a) >> 32) & 0x7ff00000u, eb = (uint32_t)(d_bits(b) >> 32) & 0x7ff00000u;
#endif
  // exponents between -400 and 400, or a = 0
  const bool mid = (ea - 0x26f00000u < 0x32000000u || ((uint64_t)d_bits(a) << 1) == 0) && eb - 0x26f00000u < 0x32000000u;
#ifdef __CUDA_ARCH__
  if (!mid) return __ddiv_rn(a, b);
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
#else
  if (!mid) return a / b;
  const double q = a * y;
  return __builtin_fma(__builtin_fma(-b, q, a), y, q);
#endif
}

// 1/x in FP64: the SM's reciprocal approximation (about 2^-20) and one third-order
// (Chebyshev) step r (1 + e + e^2), e = 1 - x r, whose own error is below 2^-60: the
// result is within 0.51 ulp (tests/test_gpu_recip_sqrt.py; a division's is within
// 0.5).  Zero, subnormal, huge, inf and NaN take the division.
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

// sqrt(x) of a non-negative x: the SM's reciprocal square root r (about 2^-20) and one
// third-order (Householder) step from y = x r on its exact residual d = x - y^2,
// y + d r (1/2 + 3/8 d r^2): 6 FP64 operations where the library's takes about 9
// FP64-pipe slots; within 0.53 ulp.  Zero, subnormal, huge, inf and NaN take the
// library's.
static __device__ __noinline__ double sqrt_slow(double x) { return sqrt(x); }
__device__ __forceinline__ double sqrt_fast(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  if (h - 0x03000000u >= 0x79000000u) return sqrt_slow(x);
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double y = x * r;
  const double w = fma(-y, y, x) * r;
  return fma(w, fma(0.375, w * r, 0.5), y);
}
#endif

}  // namespace flint
