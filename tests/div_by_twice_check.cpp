// Compares div_by_twice of fp64_int.h with the host's a / (2 b) on `n` seeded
// operands of one kind, with the FP32 seed off by RGPU_SEED_ERROR; prints the
// mismatches.
#include <cstdio>
#include <cstdlib>
#include <random>

static double g_seed_error = 0.0;
#define RGPU_SEED_ERROR g_seed_error
#include "../rhyme_gb300/csrc/fp64_int.h"

using namespace rgpu;

int main(int argc, char** argv) {
  const int kind = atoi(argv[1]);
  const long n = atol(argv[2]);
  g_seed_error = atof(argv[3]);
  std::mt19937_64 rng(7 + kind);
  const uint64_t frac = 0x800fffffffffffffull;
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    uint64_t a = rng(), b = rng();
    const uint64_t r = rng();
    if (kind == 0) {  // ordinary magnitudes
      a = (a & frac) | ((1015 + (r & 15)) << 52);
      b = (b & frac) | ((1015 + (r >> 4 & 15)) << 52);
    } else if (kind == 1) {  // a subnormal divisor of any length, a numerator near it
      b = (b & frac) >> (r & 15 ? r & 15 : r >> 4 & 51) | (b & 0x8000000000000000ull);
      a = (a & frac) | ((r >> 12 & 7) << 52);
    } else if (kind == 2) {  // a divisor whose double is the first normal or overflows
      b = (b & frac) | ((r & 1 ? 1 + (r >> 1 & 3) : 2044 + (r >> 1 & 3)) << 52);
      if (r & 8) a = (a & frac) | ((r & 1 ? 1 + (r >> 4 & 7) : 2040 + (r >> 4 & 7)) << 52);
    }  // else any doubles
    const double x = f64_from(a), y = f64_from(b), q = div_by_twice(x, divisor(y)), h = x / (2.0 * y);
    bad += f64_bits(q) != f64_bits(h) && !(q != q && h != h);
  }
  printf("%ld\n", bad);
  return bad != 0;
}
