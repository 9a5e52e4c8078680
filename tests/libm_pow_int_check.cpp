// Compares libm_pow_int's powers with libm_pow::pow, bit for bit, on n seeded
// arguments of one kind; prints the mismatches and the calls left to
// libm_pow::pow.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>

#include "../rhyme_gb300/csrc/libm_pow_int.h"

int main(int argc, char** argv) {
  const int kind = atoi(argv[1]);
  const long n = atol(argv[2]);
  std::mt19937_64 rng(kind);
  std::uniform_real_distribution<double> U(0, 1);
  const double gamma[3] = {5 / 3., 7 / 5., 4 / 3.};
  const double inf = std::numeric_limits<double>::infinity();
  const double special[8] = {0.0, -0.0, inf, -1.0, 5e-324, 1e308, std::numeric_limits<double>::quiet_NaN(), 1.0};
  long bad = 0, left = 0;
  for (long i = 0; i < n; ++i) {
    const double g = gamma[i % 3];
    const double ex[6] = {(g - 1) / (2 * g), -(g + 1) / (2 * g), 2 * g / (g - 1), 1 / g, 2 / (g - 1), (U(rng) - 0.5) * 60};
    const double y = ex[(i / 3) % 6], a = U(rng);
    double x;
    switch (kind) {
      case 0: x = 0.3 + 3 * a; break;
      case 1: x = 1 + (a - 0.5) * 0.1; break;
      case 2: x = 1 + (a - 0.5) * 1e-3; break;
      case 3: x = 1 + (a - 0.5) * std::exp2(-50 * U(rng)); break;
      case 4: x = std::exp2((a - 0.5) * 20); break;
      case 5: x = libm_pow::from_bits(rng()); break;
      default: x = special[rng() % 8]; break;
    }
    libm_pow_int::i128 L;
    bool ok = false;
    double r = 0;
    if (libm_pow_int::log_units(x, &L)) r = libm_pow_int::exp_units(L, y, &ok);
    if (!ok) ++left;
    else if (libm_pow::bits(r) != libm_pow::bits(libm_pow::pow(x, y))) ++bad;
  }
  printf("%ld %ld\n", bad, left);
  return 0;
}
