// Compares the integer FP64 operations of fp64_int.h with the host's IEEE
// operations on `n` seeded operands of one kind, with the FP32 seeds off by
// RGPU_SEED_ERROR; prints the mismatches of each operation.
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>

static double g_seed_error = 0.0;
#define RGPU_SEED_ERROR g_seed_error
#include "../rhyme_gb300/csrc/fp64_int.h"

using namespace rgpu;

static std::mt19937_64 rng;
static double pick(int kind) {
  uint64_t x = rng();
  const uint64_t near = 1023 - 8 + (x >> 60);
  switch (kind) {
    case 0: break;                                                        // any double
    case 1: x = (x & 0x800fffffffffffffull) | (near << 52); break;        // ordinary magnitudes
    case 2: x = (x & 0x800ffffff0000000ull) | (near << 52); break;        // short significands
    case 3: x = (x & 0x800000000000000full) | (near << 52); break;        // just above a power of two
    case 4: x = (x | 0x000ffffffffffff0ull) & 0x800fffffffffffffull; x |= near << 52; break;  // just below
    default: {
      const double inf = std::numeric_limits<double>::infinity(), s[10] = {0.0, -0.0, 1.0, -1.0, inf, -inf,
          std::numeric_limits<double>::quiet_NaN(), 5e-324, -2.2250738585072014e-308, 1.7976931348623157e308};
      return s[x % 10];
    }
  }
  return f64_from(x);
}
static bool same(double a, double b) { return f64_bits(a) == f64_bits(b) || (a != a && b != b); }

int main(int argc, char** argv) {
  const int kind = atoi(argv[1]);
  const long n = atol(argv[2]);
  g_seed_error = atof(argv[3]);
  rng.seed(1000 + kind);
  long bad[7] = {0};
  for (long i = 0; i < n; ++i) {
    const double a = pick(kind), b = pick(i % 16 ? kind : 5);
    bad[0] += !same(div_rn(a, b), a / b);
    bad[1] += !same(sqrt_rn(a), std::sqrt(a)) + !same(sqrt_rn(std::fabs(b)), std::sqrt(std::fabs(b)));
    // numerators and squares next to a midpoint of the result
    const double m = f64_from((f64_bits(a) & 0x000fffffffffffffull) | 0x3ff0000000000000ull);
    const double d = f64_from((f64_bits(b) & 0x000fffffffffffffull) | 0x3ff0000000000000ull);
    const double near = (double)((long double)d * ((long double)m + 0x1p-53L));
    const double sq = (double)(((long double)m + 0x1p-53L) * ((long double)m + 0x1p-53L));
    bad[2] += !same(div_rn(near, d), near / d) + !same(sqrt_rn(sq), std::sqrt(sq)) + !same(sqrt_rn(m * m), std::sqrt(m * m));
    bad[3] += f64_gt(a, b) != (a > b) || f64_gt(b, a) != (b > a) || f64_gt(a, a) != (a > a) || f64_gt(a, -a) != (a > -a);
    bad[4] += f64_above(a, 0.0) != (a > 0.0) || f64_above(a, 1.0) != (a > 1.0) || f64_negative(a) != (a < 0.0);
    bad[5] += f64_tiny(a) != (std::fabs(a) < std::numeric_limits<double>::min()) || f64_zero(a) != (a == 0.0);
    bad[6] += !same(f64_scale<1>(a), 2.0 * a) || !same(f64_scale<-1>(a), 0.5 * a) || !same(f64_scale<-3>(a), 0.125 * a);
  }
  long all = 0;
  for (int k = 0; k < 7; ++k) {
    printf("%ld ", bad[k]);
    all += bad[k];
  }
  printf("\n");
  return all != 0;
}
