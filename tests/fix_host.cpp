// Host build of the fixed-point primitives (csrc/flint_fix.cuh): largest errors
// against long double over random and edge arguments, printed as key = value.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "flint_fix.cuh"
using namespace flint;

int main() {
  typedef long double ld;
  std::vector<uint64_t> et(FIX_EXP2), lt(2 * FIX_LOG2);
  for (int j = 0; j < FIX_EXP2; ++j) et[j] = (uint64_t)llrintl(ldexpl(exp2l((ld)j / FIX_EXP2), 62)) + 512;
  for (int j = 0; j < FIX_LOG2; ++j) {
    lt[2 * j] = (uint64_t)ldexpl(1.0L / (1.0L + (ld)j / FIX_LOG2), 63) + 1;
    lt[2 * j + 1] = (uint64_t)llrintl(ldexpl(-log2l(ldexpl((ld)lt[2 * j], -63)), 62));
  }
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  ld exp_ulp = 0, lg = 0, L = 0, v = 0, f2d = 0, d2f = 0;
  int exact = 1;
  for (int i = 0; i < 400000; ++i) {
    // exp2: random over the normal range, and around the table's seams
    int64_t X = (int64_t)((U(g) * 2 - 1) * 1020 * std::ldexp(1.0, 52));
    if (i % 3 == 1) X = (X >> 44 << 44) + (i % 7 - 3);
    if (i % 3 == 2) X = ((int64_t)(i % 2000 - 1000) << 52) + (i % 5 - 2);
    const ld ex = exp2l(ldexpl((ld)X, -52));
    exp_ulp = fmaxl(exp_ulp, fabsl((ld)exp2_q52(X, et.data()) - ex) / ldexpl(1.0L, ilogbl(ex) - 52));
    // log2 of a significand, at the ends of the rows too
    double x = 1.0 + U(g);
    if (i % 4 == 1) x = 1.0 + (double)(i % 128) / 128.0 + std::ldexp(1.0, -52) * (i % 3);
    if (i % 4 == 2) x = 2.0 - std::ldexp(1.0, -52) * (1 + i % 1000);
    int e;
    lg = fmaxl(lg, fabsl(ldexpl((ld)log2_q62(x, lt.data(), &e), -62) + e - log2l((ld)x)));
    // the powers of T
    double T = 129.0 + 8063.0 * U(g) * U(g);
    if (i % 5 == 1) T = std::exp2(8 + i % 5);
    if (i % 5 == 2) T = std::nextafter(std::exp2(8 + i % 6), 0.0);
    const FixT t = fix_T(T, lt.data());
    L = fmaxl(L, fabsl(ldexpl((ld)t.L, -61) - (log2l((ld)T) - 7)));
    v = fmaxl(v, fabsl(ldexpl((ld)t.v, -70) - 1.0L / (ld)T));
    exact &= (ld)t.t13 == ldexpl((ld)T, 50) && (T >= 2048 || (ld)t.t11 == ldexpl((ld)T, 52));
    // conversions
    int64_t Z = (int64_t)(g() >> (i % 63));
    if (i & 1) Z = -Z;
    const ld z = ldexpl((ld)Z, -52);
    if (Z) f2d = fmaxl(f2d, fabsl((ld)fix2d(Z, 52) - z) / fabsl(z));
    const double y = (U(g) - 0.5) * 4000.0 * std::exp2(-40.0 * U(g));
    d2f = fmaxl(d2f, fabsl(ldexpl((ld)d2fix52(y), -52) - (ld)y));
  }
  // div_by: the correctly rounded quotient, for divisors like molar masses and any others
  for (int i = 0; i < 4000000; ++i) {
    const double b = i % 2 ? 1.0 + 300.0 * U(g) : std::ldexp(1.0 + U(g), (int)(g() % 900) - 450);
    const double a = (i % 3 ? 1.0 + U(g) : U(g)) * std::ldexp(1.0, (int)(g() % 900) - 450) * (i % 5 ? 1.0 : -1.0);
    exact &= div_by(a, b, 1.0 / b) == a / b;
  }
  exact &= div_by(0.0, 3.0, 1.0 / 3.0) == 0.0 && std::isinf(div_by(INFINITY, 3.0, 1.0 / 3.0)) && std::isnan(div_by(NAN, 3.0, 1.0 / 3.0));
  // ends of the ranges
  exact &= fix2d(0, 52) == 0.0 && d2fix52(0.0) == 0 && d2fix52(1e300) == (2047ll << 52) && d2fix52(-1e300) == -(2047ll << 52);
  exact &= exp2_q52(-(1500ll << 52), et.data()) == 0.0 && std::isinf(exp2_q52(1100ll << 52, et.data()));
  exact &= exp2_q52(0, et.data()) == 1.0;
  std::printf("exp_ulp = %.6Lg\nlog2 = %.6Lg\nL = %.6Lg\nv = %.6Lg\nfix2d = %.6Lg\nd2fix = %.6Lg\nexact = %d\n", exp_ulp, lg, L,
              v, f2d, d2f, exact);
  return 0;
}
