// Host build of the fixed-point primitives (csrc/flint_fix.cuh) at the arguments where
// their rounding carries or leaves the normal range; printed as key = value.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "flint_fix.cuh"
using namespace flint;

// Largest relative error of fix2d over +-(2^k - d), k = 53..63: the values that
// round up to the next power of two, and those just below and above them.
static long double fix2d_carry() {
  long double worst = 0;
  for (int k = 53; k <= 63; ++k)
    for (int q : {0, 45, 52, 57, 70})
      for (int step = 0; step < 2 * k; ++step) {
        const uint64_t far = step < k ? 1ull << step : (1ull << (step - k)) + (step - k) / 2;
        if (far >= 1ull << (k - 1)) continue;
        for (int up = 0; up < 2; ++up) {
          const uint64_t m = up ? (1ull << k) + far : (1ull << k) - far;
          if (m >> 63) continue;
          for (int sign = 0; sign < 2; ++sign) {
            const int64_t Z = sign ? -(int64_t)m : (int64_t)m;
            const long double z = ldexpl((long double)Z, -q);
            worst = fmaxl(worst, fabsl((long double)fix2d(Z, q) - z) / fabsl(z));
          }
        }
      }
  return worst;
}

// Largest error of exp2_q52<true> below the normal range, in units of the least subnormal.
static long double exp2_subnormal() {
  std::vector<uint64_t> et(FIX_EXP2);
  for (int j = 0; j < FIX_EXP2; ++j) et[j] = (uint64_t)llrintl(ldexpl(exp2l((long double)j / FIX_EXP2), 62)) + 512;
  long double worst = 0;
  std::mt19937_64 g(3);
  for (int i = 0; i < 200000; ++i) {
    int64_t X = -(1022ll << 52) - (int64_t)(g() % (70ull << 52));
    if (i % 8 == 0) X = -((1022ll + i % 64) << 52) - i % 3;
    const long double ex = ldexpl(exp2l(ldexpl((long double)X, -52)), 1074);
    worst = fmaxl(worst, fabsl(ldexpl((long double)exp2_q52<true>(X, et.data()), 1074) - ex));
  }
  return worst;
}

int main() {
  std::printf("exp2_subnormal = %.6Lg\n", exp2_subnormal());
  std::printf("fix2d_carry = %.6Lg\n", fix2d_carry());
  std::printf("fix2d_one = %.17g\nfix2d_four = %.17g\nfix2d_minus = %.17g\n", fix2d((1ll << 57) - 1, 57), fix2d((1ll << 54) - 1, 52),
              fix2d(-((1ll << 62) - 1), 62));
  return 0;
}
