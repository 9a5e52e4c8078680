// libm_pow_int.h -- libm_pow::pow with most of its FP64 operations in integers.
//
// Why: libm_pow::pow is 43 FP64 operations (59 for two powers of one base),
// each 64 issue cycles of a warp on GB300, and the powers of the Newton
// iteration were two thirds of the FP64 flux kernels' operations. Here the
// logarithm, its product with y and the reduction of the exponential run in
// 64-bit integers and 8 FP64 operations remain: 905 issue cycles a warp
// against 3400, 1460 against 4640 for two powers of one base (chains of
// dependent powers, 32 warps per SM).
//
// How the bits stay libm_pow::pow's. Its result is fma(S, tmp, S) with tmp a
// polynomial of r; every rounding after r is repeated here by the same FP64
// operation. r itself is the double nearest to y log x - k ln2/128 (+ d),
// where d is the rounding error that the subtraction of k NEG_LN2_LO_N
// leaves: the minuend is a multiple of the result's ulp, so d depends on
// k NEG_LN2_LO_N and that ulp alone. So r follows from y log x to about
// 2^-72:
//  * log x as libm_pow's table and polynomial define it (r0 = z INVC - 1 is an
//    exact integer multiple of 2^-61), in units of 2^-78. libm_pow's own
//    roundings put its hi + lo within 2^-76 of that value, truncations here
//    within 2^-75.5 (k ln2 included, |k| <= 7);
//  * times y, a 53-bit integer times a power of two, exactly;
//  * less k ln2/128 (k the nearest integer) plus d, rounded to 53 bits.
// The rounding is known unless the discarded bits lie within the error (16
// units of 2^-78 per unit of |y|, 8 for the rest) of half a unit; then r may
// be off by one ulp, and the result is used only if the last rounding is
// clear of a midpoint by four such ulps (otherwise, and for arguments
// outside the ranges below, libm_pow::pow). Off the ranges' ends that takes
// 0.01 % of the calls. Compared with libm_pow::pow, bit for bit, on 10^8
// arguments on the CPU and 3 10^8 on the GPU; tests/test_libm_pow_int.py
// runs a smaller set.
#pragma once

#include "libm_pow.h"
#include "libm_pow_int_tables.h"

namespace libm_pow_int {

using i128 = __int128;
using u128 = unsigned __int128;
using libm_pow::bits;
using libm_pow::from_bits;

struct LogPiece {
  uint64_t lo;
  int64_t hi;
  int invc;
};
static const LogPiece kLogHost[128] = LIBM_POW_INT_LOG;
#if defined(__CUDACC__)
static __device__ const LogPiece kLogDev[128] = LIBM_POW_INT_LOG;
#endif

LIBM_POW_HD const LogPiece& log_piece(int i) {
#if defined(__CUDA_ARCH__)
  return kLogDev[i];
#else
  return kLogHost[i];
#endif
}
LIBM_POW_HD int64_t mul_hi(int64_t a, int64_t b) {
#if defined(__CUDA_ARCH__)
  return __mul64hi(a, b);
#else
  return (int64_t)(((i128)a * b) >> 64);
#endif
}
LIBM_POW_HD int mul_hi(int a, int b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int)(((int64_t)a * b) >> 32);
#endif
}
LIBM_POW_HD int leading_zeros(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
LIBM_POW_HD i128 of_halves(uint64_t lo, int64_t hi) { return (i128)(((u128)(uint64_t)hi << 64) | lo); }
LIBM_POW_HD int length(u128 v) {  // bits of v
  const uint64_t h = (uint64_t)(v >> 64);
  return h ? 128 - leading_zeros(h) : 64 - leading_zeros((uint64_t)v);
}

constexpr uint64_t kFrac = 0x000fffffffffffffull, kUnit = 0x0010000000000000ull;

// log x in units of 2^-78; false unless x is normal and within 2^-7 .. 2^8
// of OFF.
LIBM_POW_HD bool log_units(double x, i128* out) {
  const uint64_t ix = bits(x), t = ix - libm_pow::kOffBits;
  const int i = (int)((t >> 45) & 127);
  const int k = (int)((int64_t)t >> 52);
  if ((uint32_t)(k + 7) > 14u) return false;
  const uint64_t iz = ix - ((uint64_t)(int64_t)k << 52);
  const LogPiece& e = log_piece(i);
  const uint64_t Z = ((iz & kFrac) | kUnit) << ((uint32_t)(iz >> 52) - 1022u);  // z 2^53
  const int64_t R = (int64_t)(Z * (uint64_t)e.invc - (1ull << 61));            // r 2^61, |r| < 2^-7.4
  const int64_t r70 = (int64_t)((uint64_t)R << 9);
  const int r38 = (int)(R >> 23);
  const int b5 = (int)LIBM_POW_INT_B5 + (mul_hi(r38, (int)LIBM_POW_INT_B6) >> 6);
  const int b4 = (int)LIBM_POW_INT_B4 + (mul_hi(r38, b5) >> 6);
  const int64_t b3 = LIBM_POW_INT_B3 + (((int64_t)r38 * b4) >> 8);
  const int64_t b2 = LIBM_POW_INT_B2 + (mul_hi(r70, b3) >> 6);
  const int64_t b1 = LIBM_POW_INT_B1 + (mul_hi(r70, b2) >> 6);
  const u128 R2 = (u128)((i128)R * R);                              // r^2 2^122
  const int64_t r3 = mul_hi((int64_t)(uint64_t)(R2 >> 46), r70);    // r^3 2^82
  const int64_t p = (mul_hi(r3, b1) >> 3) - (int64_t)(uint64_t)(R2 >> 45);
  i128 L = of_halves(e.lo, e.hi) + ((i128)R << 17) + p;
  if (k) L += of_halves(LIBM_POW_INT_LN2) * k;
  *out = L;
  return true;
}

// x^y from L = log x in units of 2^-78; *ok false: not known, or out of range
// (2^-10 <= |y| < 32, |y log x| < 7.5).
LIBM_POW_HD double exp_units(i128 L, double y, bool* ok) {
  const uint64_t iy = bits(y);
  const int ey = (int)((iy >> 52) & 0x7ff) - 1023;
  *ok = false;
  if ((uint32_t)(ey + 10) > 14u) return 0.0;
  // E = y log x in units of 2^-78: |L| in two parts of 48 and 33 bits
  const uint64_t Y = (iy & kFrac) | kUnit;
  const u128 aL = (u128)(L < 0 ? -L : L);
  const u128 prod = (u128)(uint64_t)(aL >> 48) * Y + (uint64_t)(((u128)((uint64_t)aL & ((1ull << 48) - 1)) * Y) >> 48);
  i128 E = (i128)(prod >> (4 - ey));
  if ((uint64_t)(E >> 64) >= (15ull << 13)) return 0.0;
  if ((L < 0) != (bool)(iy >> 63)) E = -E;
  // k: the nearest integer to E 128/ln2, clear of a half
  const int64_t kk = (int64_t)(E >> 46) * LIBM_POW_INT_INV;
  const int64_t k = (kk + (1LL << 51)) >> 52;
  const int64_t from_half = (kk & ((1LL << 52) - 1)) - (1LL << 51);
  if ((uint64_t)(from_half + (1LL << 36)) < (2ULL << 36)) return 0.0;
  i128 V = E - ((of_halves(LIBM_POW_INT_HL) * k) >> 14);
  // d: the rounding error of subtracting k LO on the result's grid
  const int G = length((u128)(V < 0 ? -V : V)) - 36;  // its ulp is 2^G units of 2^-95
  if (k && G > 0) {
    const int64_t q = (int64_t)(0 - (uint64_t)k * (uint64_t)LIBM_POW_INT_LO);
    const int64_t rem = (int64_t)((uint64_t)q & ((1ull << G) - 1));
    V += (((uint64_t)rem >> (G - 1)) ? (int64_t)(1ull << G) - rem : -rem) >> 17;
  }
  // r = V rounded to 53 bits
  const bool neg = V < 0;
  const u128 aV = (u128)(neg ? -V : V);
  const int s = length(aV) - 53;
  uint64_t m = (uint64_t)aV;
  bool near = true;  // r may be off by an ulp
  if (s > 0) {
    const uint64_t rem = m & ((1ull << s) - 1), half = 1ull << (s - 1);
    const uint64_t tol = (16u << (ey < 0 ? 0 : ey + 1)) + 8u;
    m = (uint64_t)(aV >> s) + (rem >= half ? 1u : 0u);
    near = (rem - half + tol) <= 2 * tol;
  }
  double r = 0.0;
  if (m) r = from_bits(((uint64_t)neg << 63) | (((uint64_t)(s + 996) << 52) + (m << (s > 0 ? 0 : -s))));
  // the exponential's operations (libm_pow::exp_parts)
  const uint64_t* e = libm_pow::exp_tab() + 2 * (k & 127);
  const uint64_t sbits = e[1] + ((uint64_t)k << 45);
  const double tail = from_bits(e[0]);
  using libm_pow::fma3;
  const double r2 = libm_pow::mul(r, r), r4 = libm_pow::mul(r2, r2);
  const double u = fma3(r2, fma3(r, LIBM_POW_C3, LIBM_POW_C2), libm_pow::add(tail, r));
  const double tmp = fma3(r4, fma3(r, LIBM_POW_C5, LIBM_POW_C4), u);
  const double S = from_bits(sbits);
  const double res = fma3(S, tmp, S);
  *ok = true;
  if (near) {
    // the discarded part of S + S tmp in units of 2^-32 of the result's ulp
    const uint64_t it = bits(tmp), ir = bits(res);
    const uint64_t T = (it & kFrac) | kUnit, M = (sbits & kFrac) | kUnit;
    const uint64_t H = (uint64_t)(((u128)(T << 11) * (M << 11)) >> 64);
    const int de = (int)(sbits >> 52) - (int)(ir >> 52);
    const int q = 10 - ((int)((it >> 52) & 0x7ff) - 1023) - de;
    uint32_t f = q >= 96 ? 0u : q >= 32 ? (uint32_t)(H >> (q - 32)) : (uint32_t)(H << (32 - q));
    if (it >> 63) f = 0u - f;
    if (de < 0) f += (uint32_t)(M & 1) << 31;
    const uint32_t tol = (1u << ((s < 0 ? 0 : s) + 9)) + 64u;
    if ((uint32_t)(f - 0x80000000u + tol) <= 2 * tol) *ok = false;
  }
  return res;
}

#if defined(__CUDACC__)
static __device__ __noinline__ double pow_literal(double x, double y) { return libm_pow::pow(x, y); }

// Calls, not inlined: one copy of their instructions serves every warp.
static __device__ __noinline__ double pow(double x, double y) {
  i128 L;
  bool ok = false;
  double r = 0.0;
  if (log_units(x, &L)) r = exp_units(L, y, &ok);
  return ok ? r : pow_literal(x, y);
}

// x**y1 and x**y2 sharing the logarithm.
static __device__ __noinline__ double2 pow2(double x, double y1, double y2) {
  i128 L;
  bool ok1 = false, ok2 = false;
  double a = 0.0, b = 0.0;
  if (log_units(x, &L)) {
    a = exp_units(L, y1, &ok1);
    b = exp_units(L, y2, &ok2);
  }
  return make_double2(ok1 ? a : pow_literal(x, y1), ok2 ? b : pow_literal(x, y2));
}
#endif

}  // namespace libm_pow_int
