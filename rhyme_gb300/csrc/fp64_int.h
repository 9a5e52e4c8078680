// fp64_int.h -- FP64 division, square root, comparison and scaling by powers
// of two in 32-bit integer arithmetic, returning the IEEE results bit for bit.
//
// Why: GB300 issues one FP64 warp instruction per SM sub-partition every 64
// cycles, whatever lanes are active (measured: fma, add and compare alike),
// and a division or a square root takes 9 to 10 of them (550 and 640 cycles a
// warp), while the integer and FP32 pipes idle beside it. In integers the
// same correctly rounded results take 128 and 125 issue cycles (division
// 73 -> 310 G/s, square root 62 -> 317 G/s over the whole GPU), a comparison
// about 6 instead of 64, and the FP64 pipe is left to the sums and products.
//
// Division and square root are the schoolbook digit recurrences on the
// 53-bit significands with two digits of 27 and 28 bits and an exact
// remainder: the reciprocal (root) of the divisor comes from the FP32
// approximation (22 bits or better) and one Newton step in integers, each
// digit is its product with the running remainder rounded down, and the
// remainder after the second digit puts the quotient right by 0, 1 or 2
// units, so that its 56 bits are exactly the leading bits of the true
// quotient. Rounding adds half a unit of the 53rd bit and truncates: neither a quotient
// nor a root of two 53-bit numbers lies exactly between two 53-bit numbers.
// Operands or results outside the normal range take the hardware operation.
//
// Host code can include this header (the FP32 approximations are then
// computed, with RGPU_SEED_ERROR as a relative error added to them).
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define RGPU_HD __host__ __device__ __forceinline__
#define RGPU_CALL static __host__ __device__ __noinline__
#else
#include <cmath>
#define RGPU_HD inline
#define RGPU_CALL inline
#endif

#ifndef RGPU_SEED_ERROR
#define RGPU_SEED_ERROR 0.0
#endif

namespace rgpu {

RGPU_HD uint64_t f64_bits(double d) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(d);
#else
  uint64_t u;
  std::memcpy(&u, &d, sizeof u);
  return u;
#endif
}
RGPU_HD double f64_from(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double d;
  std::memcpy(&d, &u, sizeof d);
  return d;
#endif
}
RGPU_HD uint32_t f64_hi(double d) { return (uint32_t)(f64_bits(d) >> 32); }

namespace fp64_int {

constexpr uint64_t kFrac = 0x000fffffffffffffull, kUnit = 0x0010000000000000ull;
constexpr uint64_t kSign = 0x8000000000000000ull, kInf = 0x7ff0000000000000ull;

RGPU_HD uint32_t mul_hi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
RGPU_HD float f32_from(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, sizeof f);
  return f;
#endif
}
// 2^30 / f and 2^30 / sqrt(f) to 22 bits or better, truncated to integers.
RGPU_HD uint32_t seed_recip(float f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return __float2uint_rz(r * 1073741824.f);
#else
  return (uint32_t)(1073741824.f * (float)((1.0 / f) * (1.0 + RGPU_SEED_ERROR)));
#endif
}
RGPU_HD uint32_t seed_rsqrt(float f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return __float2uint_rz(r * 1073741824.f);
#else
  return (uint32_t)(1073741824.f * (float)((1.0 / std::sqrt((double)f)) * (1.0 + RGPU_SEED_ERROR)));
#endif
}

}  // namespace fp64_int

// A divisor with the reciprocal of its significand: quotients by the same
// number (or by it times a power of two) share the work.
struct Divisor {
  double b;
  uint32_t R;  // 2^83 / B (1 - 2^-29) < R <= 2^83 / B, B the 53-bit significand of b
};

RGPU_HD Divisor divisor(double b) {
  using namespace fp64_int;
  const uint64_t ub = f64_bits(b);
  const uint64_t B = (ub & kFrac) | kUnit;
  // b31 rounded up and every step below rounded down: R never exceeds its
  // real value
  const uint32_t b31 = (uint32_t)(B >> 22) + 1u;
  const uint32_t R0 = seed_recip(f32_from(0x3f800000u | ((uint32_t)(ub >> 29) & 0x7fffffu)));  // 2^60 / b31 (1 - e)
  const int64_t e = (int64_t)((1ull << 60) - (uint64_t)b31 * R0);  // 2^60 e, |e| < 2^-20
  const int64_t c = (int64_t)(int32_t)R0 * (int32_t)(e >> 16);     // 2^44 R0 e
  return {b, 2u * R0 + (uint32_t)(int32_t)(c >> 43)};
}

// a / b, R from divisor(b), rounded to nearest even.
RGPU_HD double div_core(double a, double b, uint32_t R) {
  using namespace fp64_int;
  const uint64_t ua = f64_bits(a), ub = f64_bits(b);
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
  if (ea - 1u < 2046u && eb - 1u < 2046u && ea - eb + 1021u < 2044u) {
    uint64_t A = (ua & kFrac) | kUnit;
    const uint64_t B = (ub & kFrac) | kUnit;
    uint32_t e = ea - eb + 1022u;
    if (A < B) {  // the quotient of the significands in [1, 2)
      A <<= 1;
      e -= 1u;
    }
    const uint32_t q1 = mul_hi((uint32_t)(A >> 22), R) >> 2;  // 2^27 A/B, short by less than 1.75
    const uint64_t r1 = (A << 27) - (uint64_t)q1 * B;
    const uint32_t q2 = mul_hi((uint32_t)(r1 >> 23), R);  // 2^28 r1/B, short by less than 2.4
    const uint64_t r2 = (r1 << 28) - (uint64_t)q2 * B;
    const uint64_t Q = ((uint64_t)q1 << 28) + (q2 + 4u) + (r2 >= B ? 1u : 0u) + (r2 >= 2 * B ? 1u : 0u);
    return f64_from(((ua ^ ub) & kSign) | (((uint64_t)e << 52) + (Q >> 3)));
  }
  if ((ua << 1) == 0 && eb - 1u < 2046u) return f64_from((ua ^ ub) & kSign);
  return a / b;
}

// Calls, not inlined: the interface solve divides at some fifty places, and
// with a copy at each its warps waited for instructions half of the time.
RGPU_CALL double div_with(double a, double b, uint32_t R) { return div_core(a, b, R); }
RGPU_CALL double div_rn(double a, double b) { return div_core(a, b, divisor(b).R); }
RGPU_HD double div_by(double a, const Divisor& d) { return div_with(a, d.b, d.R); }

// sqrt(a), rounded to nearest even.
RGPU_CALL double sqrt_rn(double a) {
  using namespace fp64_int;
  const uint64_t ua = f64_bits(a);
  const uint32_t ea = (uint32_t)(ua >> 52);
  if (ea - 1u < 2046u) {
    const uint32_t odd = (ea & 1u) ^ 1u;  // the exponent is odd: move its unit to the significand
    const uint64_t N = ((ua & kFrac) | kUnit) << odd;  // f 2^52, f in [1, 4)
    const uint32_t n32 = (uint32_t)(N >> 22);
    const uint32_t y0 = seed_rsqrt(f32_from(((uint32_t)(ua >> 29) & 0x7fffffu) | (0x3f800000u + (odd << 23))));
    // Newton: y = 2^31 / sqrt(f) from e = 1 - f y0^2
    const int64_t e = (int64_t)((1ull << 61) - (uint64_t)(uint32_t)(((uint64_t)y0 * y0) >> 29) * n32);
    const uint32_t y = 2u * y0 + (uint32_t)(int32_t)(((int64_t)(int32_t)y0 * (int32_t)(e >> 16)) >> 45);
    // the root 2^28 s1 + s2 of f 2^110: s1 within 1 of 2^27 sqrt(f) so that
    // the neglected square of its error stays below one unit of s2
    const uint32_t s1 = (mul_hi(n32, y) + 2u) >> 2;
    const int64_t r1 = (int64_t)((N << 2) - (uint64_t)s1 * s1);
    const int64_t s2 = (r1 * (int64_t)y) >> 31;
    uint64_t S = ((uint64_t)s1 << 28) + (uint64_t)s2;
    const int64_t r2 = (int64_t)((((uint64_t)r1 << 28) - 2ull * s1 * (uint64_t)s2) << 28) - s2 * s2;
    if (r2 < 0) S -= 1;
    else if (r2 > (int64_t)(2 * S)) S += 1;
    return f64_from(((uint64_t)(((ea + 1023u) >> 1) - 1u) << 52) + ((S + 4) >> 3));
  }
#if defined(__CUDACC__)
  return ::sqrt(a);
#else
  return std::sqrt(a);
#endif
}

// The hardware's operations where an operand is out of the integer forms'
// range: behind an opaque asm on the device, because the compiler would
// otherwise run such a cheap instruction for every lane and select.
RGPU_HD double hw_mul(double a, double b) {
#if defined(__CUDA_ARCH__)
  double r;
  asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
#else
  return a * b;
#endif
}
RGPU_HD bool hw_gt(double a, double b) {
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n setp.gt.f64 p, %1, %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r) : "d"(a), "d"(b));
  return r != 0;
#else
  return a > b;
#endif
}

// a > b. Two non-negative finite numbers order like their bits, others like
// their signed magnitudes; infinities and NaNs take the hardware comparison.
RGPU_HD bool f64_gt(double a, double b) {
  const uint32_t ha = f64_hi(a), hb = f64_hi(b);
  if ((ha > hb ? ha : hb) < 0x7ff00000u) return f64_bits(a) > f64_bits(b);
  const uint32_t ma = ha & 0x7fffffffu, mb = hb & 0x7fffffffu;
  if ((ma > mb ? ma : mb) < 0x7ff00000u) {
    const int64_t ia = (int64_t)f64_bits(a), ib = (int64_t)f64_bits(b);
    const int64_t ka = ia < 0 ? (int64_t)(fp64_int::kSign - (uint64_t)ia) : ia;
    const int64_t kb = ib < 0 ? (int64_t)(fp64_int::kSign - (uint64_t)ib) : ib;
    return ka > kb;
  }
  return hw_gt(a, b);
}
RGPU_HD bool f64_nan(double x) { return (f64_bits(x) << 1) > 0xffe0000000000000ull; }

// x > c for a positive constant c or zero: x in (c, infinity].
RGPU_HD bool f64_above(double x, double c) {
  const uint64_t uc = f64_bits(c);
  return f64_bits(x) - (uc + 1u) < fp64_int::kInf - uc;
}
// x < 0: x in [-infinity, -0).
RGPU_HD bool f64_negative(double x) {
  return f64_bits(x) - (fp64_int::kSign + 1u) < fp64_int::kInf;
}
// x == 0.
RGPU_HD bool f64_zero(double x) { return (f64_bits(x) << 1) == 0; }
// |x| below the smallest normal number.
RGPU_HD bool f64_tiny(double x) { return (f64_hi(x) & 0x7ff00000u) == 0; }

// x 2^K by the exponent field (K small); zeros stay; anything that leaves
// the normal range takes the multiplication.
template <int K>
RGPU_HD double f64_scale(double x) {
  const uint32_t h = f64_hi(x) & 0x7fffffffu;
  constexpr uint32_t lo = (uint32_t)(1 + (K < 0 ? -K : 0)) << 20, hi = (uint32_t)(2047 - (K > 0 ? K : 0)) << 20;
  if (h - lo < hi - lo) return f64_from(f64_bits(x) + ((uint64_t)(int64_t)K << 52));
  if ((f64_bits(x) << 1) == 0) return x;
  return hw_mul(x, K < 0 ? 1.0 / (double)(1 << (K < 0 ? -K : 0)) : (double)(1 << (K > 0 ? K : 0)));
}

// a / (2 b), b given with its reciprocal: the significand of 2 b is b's unless
// b is subnormal (its leading zeros differ from 2 b's).
RGPU_HD double div_by_twice(double a, const Divisor& d) {
  const uint32_t h = f64_hi(d.b) & 0x7fffffffu;
  if (h - 0x00100000u < 0x7fe00000u - 0x00100000u)  // b and 2 b normal
    return div_with(a, f64_from(f64_bits(d.b) + (1ull << 52)), d.R);
  return div_rn(a, hw_mul(2.0, d.b));
}

}  // namespace rgpu
