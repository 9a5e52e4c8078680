// hydro.cuh -- device functions of the MUSCL-Hancock step: ideal-gas EOS,
// slope limiters, half-step extrapolation and the exact Riemann solver.
//
// Templated on NDIM (D) and on the normal axis (AX, compile-time so no state
// vector is indexed dynamically); double for the plain path and the mixed
// path's redone interfaces, float for the FP32 stages of the mixed path. Each
// FP64 routine keeps
// the floating-point evaluation order of the Fortran routine it restates
// (operators of equal precedence left to right), so that with FMA contraction
// disabled the double instantiation performs the same IEEE operations as the
// reference; the only intended difference is that the six p* guesses of
// rhyme_irs_guess_p_star.f90 are evaluated lazily, in order, when the Newton
// iteration from the previous guess fails (identical values, less work).
//
// State vectors are (rho, m_1..m_D, E); reference paths are relative to
// Rhyme's src/.
#pragma once

#include <cfloat>
#include <cstdint>

#include "fp64_int.h"
#include "libm_pow_int.h"

namespace rgpu {

// ---- math by type --------------------------------------------------------
// Double powers return the bits of libm_pow::pow, a restatement of the C
// library's pow that the compiled reference calls for every real `**`, so the
// FP64 path returns the reference's bits even in flows that amplify a one-ulp
// difference; libm_pow_int.h forms them mostly in integers.
__device__ __forceinline__ double m_sqrt(double x) { return sqrt_rn(x); }
__device__ __forceinline__ double m_pow(double x, double y) { return libm_pow_int::pow(x, y); }
// Float powers as 2^(y log2 x) with CUDA's log2f and exp2f: the rounding of
// the product adds a relative error of about 2^-24 |y log2 x| to the result
// (for the positive bases of this path), against powf's ~1 ulp, for a
// fraction of its instructions; two powers of one base share the logarithm.
__device__ __forceinline__ float m_pow(float x, float y) { return exp2f(y * log2f(x)); }
// x**y1 and x**y2 of one base (one logarithm).
__device__ __forceinline__ void m_pow2(double x, double y1, double y2, double& r1, double& r2) {
  const double2 r = libm_pow_int::pow2(x, y1, y2);
  r1 = r.x;
  r2 = r.y;
}
__device__ __forceinline__ void m_pow2(float x, float y1, float y2, float& r1, float& r2) {
  const float l = log2f(x);
  r1 = exp2f(y1 * l);
  r2 = exp2f(y2 * l);
}

// FP64 divisions, comparisons and powers of two through the integer forms of
// fp64_int.h (the same bits; a division or a comparison on the FP64 pipe costs
// 550 or 64 cycles a warp). A Divisor is a divisor used several times.
__device__ __forceinline__ double m_div(double a, const Divisor& d) { return div_by(a, d); }
__device__ __forceinline__ double m_div(double a, double b) { return div_rn(a, b); }
__device__ __forceinline__ bool m_gt(double a, double b) { return f64_gt(a, b); }
__device__ __forceinline__ bool m_neg(double a) { return f64_negative(a); }
__device__ __forceinline__ double m_half(double a) { return f64_scale<-1>(a); }
__device__ __forceinline__ double m_twice(double a) { return f64_scale<1>(a); }

// Fortran MAX/MIN of two reals (same ternary as the CPU oracle).
__device__ __forceinline__ double fmax_ref(double a, double b) { return m_gt(b, a) ? b : a; }
__device__ __forceinline__ double fmin_ref(double a, double b) { return m_gt(a, b) ? b : a; }
// FP32: one instruction, which like the selections above keeps a NaN in a.
__device__ __forceinline__ float fmax_ref(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float fmin_ref(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Ideal-gas constants (rhyme_riemann_problem_init.f90:20-27,
// rhyme_irs_init.f90:21-27) plus the literal quotients the reference
// recomputes at each use (2/gp1, 2/gm1, 1/gm1_2g, gm1/2): the same values.
template <typename T>
struct GasOnly;  // what one of the two forms needs besides
template <>
struct GasOnly<double> {
  Divisor by_gm1, by_gp1, by_kb_amu;
};
template <>
struct GasOnly<float> {
  float gm1_lo, g_gm1;  // what rounding gm1 to FP32 lost; gamma/(gamma-1)
};
template <typename T>
struct Gas : GasOnly<T> {
  T g, gm1, gp1, gm1_gp1, gm1_2g, gp1_2g, g_inv, kb_amu;
  T two_gp1, two_gm1, inv_gm1_2g, gm1_half, half_gm1, g_kb_amu;
};

// Run parameters used inside kernels.
template <typename T>
struct Rp {
  T vac_rho, vac_p, vac_rho_next;  // w_vacuum(rho), w_vacuum(p), nearest(w_vac_rho, +1)
  T tol;  // FP64: the tolerance; FP32: the relative size of a step that ends rp_flux_f32's iteration
  T settle;  // FP32: what the rounded p may move in that step
  int n_iter;
};

// ---- EOS: rhyme_hydro_base / rhyme_ideal_gas ------------------------------

// rhyme_hydro_base_specific_kinetic_energy.f90:9
template <int D>
__device__ __forceinline__ double sp_kin_e(const double* u) {
  double s = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) s = s + u[1 + a] * u[1 + a];
  return m_div(m_half(s), u[0] * u[0]);
}

// rhyme_hydro_base_specific_internal_energy.f90:9; i0: the density as a divisor
template <int D>
__device__ __forceinline__ double sp_int_e(const double* u, const Divisor& i0) {
  return m_div(u[D + 1], i0) - sp_kin_e<D>(u);
}

// rhyme_ideal_gas_pressure.f90:9
template <int D>
__device__ __forceinline__ double pressure(const Gas<double>& G, const double* u, const Divisor& i0) {
  return u[0] * sp_int_e<D>(u, i0) * G.gm1;
}
template <int D>
__device__ __forceinline__ double pressure(const Gas<double>& G, const double* u) {
  return pressure<D>(G, u, divisor(u[0]));
}

// rhyme_ideal_gas_temperature_per_mu.f90:9-10, _speed_of_sound.f90:9
template <int D>
__device__ __forceinline__ double sound_speed(const Gas<double>& G, const double* u, const Divisor& i0) {
  const double t_mu = m_div(sp_int_e<D>(u, i0) * G.gm1, G.by_kb_amu);
  return m_sqrt(G.g_kb_amu * t_mu);
}
template <int D>
__device__ __forceinline__ double sound_speed(const Gas<double>& G, const double* u) {
  return sound_speed<D>(G, u, divisor(u[0]));
}

// The FP32 form of the mixed CFL is the same quantity with fewer divisions:
// p = (E - |m|^2 / (2 rho)) (gamma-1) for rho e_int (gamma-1), cs =
// sqrt(gamma p / rho) for sqrt(gamma kB/amu T/mu). The sweeps' flux and
// interface solve form p so too, from one reciprocal of rho: FP32 division is
// a reciprocal and a multiply plus range handling, and the sweeps divide a lot
// (256^3 mixed step 2.43 -> 2.20 ms, L1(rho) against FP64 a little lower).
template <int D>
__device__ __forceinline__ float sound_speed(const Gas<float>& G, const float* u) {
  float s = 0.f;
#pragma unroll
  for (int a = 0; a < D; ++a) s = s + u[1 + a] * u[1 + a];
  const float p = (u[D + 1] - 0.5f * s / u[0]) * G.gm1;
  return sqrtf(G.g * p / u[0]);
}

// rhyme_ideal_gas_flux.f90:12-23 along axis AX
template <int D, int AX>
__device__ __forceinline__ void flux(const Gas<double>& G, const double* u, double* f) {
  if (f64_tiny(u[0])) {
#pragma unroll
    for (int c = 0; c < D + 2; ++c) f[c] = 0.0;
    return;
  }
  const Divisor i0 = divisor(u[0]);
  const double p = pressure<D>(G, u, i0);
  f[0] = u[1 + AX];
#pragma unroll
  for (int a = 0; a < D; ++a) f[1 + a] = m_div(u[1 + a] * f[0], i0);
  f[1 + AX] = f[1 + AX] + p;
  f[D + 1] = m_div(f[0], i0) * (u[D + 1] + p);
}

// rhyme_ideal_gas_primitive_vars_to_conserved.f90:9-11
template <int D>
__device__ __forceinline__ void prim_vars_to_cons(const Gas<double>& G, double rho, const double* v, double p,
                                                  double* u) {
  u[0] = rho;
  double s = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    u[1 + a] = rho * v[a];
    s = s + v[a] * v[a];
  }
  u[D + 1] = m_half(rho) * s + m_div(p, G.by_gm1);
}

// ---- slope limiter: rhyme_slope_limiter*.f90 -------------------------------

// The FP64 limiter: the reference's operations (xi_r:
// rhyme_slope_limiter_xi_r.f90:11) through the integer forms. With w = 0 (the default) they reduce, with the same
// results, to fewer: 0.5 d_L + 0.5 d_R is half of the rounded sum, xi_r is
// 2/(1+r), and of two quotients with the same divisor the smaller one is
// known from the numerators (rounding is monotonic), so van Leer, minmod
// and superbee need one division after r.
__device__ __forceinline__ double limiter_phi(int type, double w, double r) {  // r > 0
  const double xi = div_rn(2.0, 1.0 - w + (1.0 + w) * r);
  if (type == 1) return fmin_ref(div_rn(f64_scale<1>(r), 1.0 + r), xi);
  if (type == 2) return f64_above(r, 1.0) ? fmin_ref(1.0, xi) : r;
  if (type == 3) return fmin_ref(div_rn(r * (1.0 + r), 1.0 + r * r), xi);
  if (f64_above(r, 1.0)) return fmin_ref(fmin_ref(r, xi), 2.0);
  return f64_above(r, 0.5) ? 1.0 : f64_scale<1>(r);
}

__device__ __forceinline__ double limited_slope_f64(int type, double w, double ul, double u, double ur) {
  const double d_L = u - ul, d_R = ur - u;
  const double r = f64_tiny(d_R) ? 0.0 : div_rn(d_L, d_R);
  if (!f64_above(r, 0.0)) return 0.0;
  // phi first, by integer selections and divisions, then one product with d
  // for every lane
  double d, phi;
  if (f64_zero(w)) {
    d = d_L + d_R;
    // half the sum, exactly, well above the subnormal range
    d = ((f64_hi(d) & 0x7fffffffu) - 0x08000000u < 0x7fe00000u - 0x08000000u) ? f64_scale<-1>(d) : hw_mul(0.5, d_L) + hw_mul(0.5, d_R);
    const bool big = f64_above(r, 1.0);
    if (type == 3 || f64_hi(r) >= 0x7ff00000u) {
      phi = limiter_phi(type, 0.0, r);
    } else if (type == 1) {
      phi = div_rn(big ? 2.0 : f64_scale<1>(r), 1.0 + r);
    } else {
      phi = (type == 2) ? r : f64_above(r, 0.5) ? 1.0 : f64_scale<1>(r);
      if (big) phi = div_rn(2.0, 1.0 + r);
    }
  } else {
    const double h = 0.5 * (1.0 + w);
    d = h * d_L + h * d_R;
    phi = limiter_phi(type, w, r);
  }
  return phi * d;
}

// The FP32 limiter of the mixed sweeps. With w = 0 the products with
// d = 0.5 (d_L + d_R) simplify: xi_r d = 2/(1 + d_L/d_R) d = d_R and
// 2r/(1+r) d = d_L, so van Leer needs no division, minmod and superbee one
// where r <= 1 and r <= 1/2, van Albada two instead of three. The rounding
// errors of the divisions they replace go with them.
// r = d_L/d_R > 0, a denominator below the smallest normal number giving 0:
// d_L with the sign of d_R taken off is positive.
__device__ __forceinline__ bool same_sign_f32(float d_L, float d_R) {
  const float l = __int_as_float(__float_as_int(d_L) ^ (__float_as_int(d_R) & (int)0x80000000u));
  return l > 0.f && fabsf(d_R) >= FLT_MIN;
}

template <int TYPE>
__device__ __forceinline__ float limited_slope_w0_f32(float ul, float u, float ur) {
  const float d_L = u - ul, d_R = ur - u;
  const bool big = fabsf(d_L) > fabsf(d_R);  // r > 1
  float s;
  if (TYPE == 1) {
    s = big ? d_R : d_L;
  } else if (TYPE == 2) {
    s = big ? d_R : __fdividef(d_L, d_R) * (0.5f * (d_L + d_R));
  } else if (TYPE == 3) {
    // r(1+r)/(1+r^2) is 1 to float precision once r > 2^24; beyond ~1.8e19
    // the squares overflow: take the limit (a noise-level d_R against a
    // resolved d_L reaches such r in FP32)
    const float r = __fdividef(d_L, d_R);
    const float half = 0.5f * (d_L + d_R);
    const float a = (r < 1e18f) ? __fdividef(r * (1.f + r), 1.f + r * r) * half : half;
    s = (fabsf(d_R) < fabsf(a)) ? d_R : a;
  } else {
    const float sum = d_L + d_R;
    s = big ? d_R : (2.f * fabsf(d_L) > fabsf(d_R)) ? 0.5f * sum : __fdividef(d_L, d_R) * sum;
  }
  return same_sign_f32(d_L, d_R) ? s : 0.f;
}

__device__ __forceinline__ float limited_slope_w_f32(int type, float w, float ul, float u, float ur) {
  const float d_L = u - ul, d_R = ur - u;
  const bool same = same_sign_f32(d_L, d_R);
  const float r = same ? __fdividef(d_L, d_R) : 0.f;
  const float h = 0.5f * (1.f + w);
  const float d = __fmaf_rn(h, d_L, h * d_R);
  const float xi = __fdividef(2.f, 1.f - w + (1.f + w) * r);
  float phi;
  if (type == 1) phi = fminf(__fdividef(2.f * r, 1.f + r), xi);
  else if (type == 2) phi = (r > 1.f) ? fminf(1.f, xi) : r;
  else if (type == 3) phi = fminf((r < 1e18f) ? __fdividef(r * (1.f + r), 1.f + r * r) : 1.f, xi);
  else phi = (r > 1.f) ? fminf(fminf(r, xi), 2.f) : (r > 0.5f) ? 1.f : 2.f * r;
  return same ? phi * d : 0.f;
}

// r (rhyme_slope_limiter.f90:62-82) and delta of the four limiters
// (van Leer :13-27, minmod :13-29, van Albada :13-27, superbee :13-31) of the
// N components of a cell. FP32: the limiter's type is looked at once per cell
// and axis, not per component. That, the sign test above, one test for a flux
// that is not finite and one-instruction extrema in rp_flux_f32 took a sixth
// of an FP32 sweep's instructions away (3-D 128^3: 65.6e6 -> 54.9e6 warp
// instructions) from kernels that issue in 80 % of their cycles: 256^3, x+y
// 864 -> 753 us, z 704 -> 639.
template <int N>
__device__ __forceinline__ void limited_slopes(int type, double w, const double* ul, const double* u, const double* ur,
                                               double* delta) {
#pragma unroll
  for (int c = 0; c < N; ++c) delta[c] = limited_slope_f64(type, w, ul[c], u[c], ur[c]);
}
// The FP32 quotients by d_R are 0 where it is beyond 2^126 (__fdividef): such
// a cell's density slope becomes a NaN, which makes its face states none that
// the FP32 solve takes, and FP64 redoes both interfaces. The sum of all |d_R|
// tells (four times it is infinite then, and a product with 0 a NaN): six
// instructions of the FP32 pipe where the limiter divides (256^3 superbee, x+y
// 768 -> 774 us; with the largest |d_R|, a comparison and a selection 777).
template <int N>
__device__ __forceinline__ void limited_slopes(int type, float w, const float* ul, const float* u, const float* ur,
                                               float* delta) {
  auto each = [&](auto slope, bool divides) {
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      delta[c] = slope(ul[c], u[c], ur[c]);
      sum = sum + fabsf(ur[c] - u[c]);
    }
    if (divides) delta[0] = __fmaf_rn(__fmul_rn(4.f, sum), 0.f, delta[0]);
  };
  if (w != 0.f) each([&](float a, float b, float c) { return limited_slope_w_f32(type, w, a, b, c); }, true);
  else if (type == 1) each(limited_slope_w0_f32<1>, false);
  else if (type == 2) each(limited_slope_w0_f32<2>, true);
  else if (type == 3) each(limited_slope_w0_f32<3>, true);
  else each(limited_slope_w0_f32<4>, true);
}

// The difference of the FP32 fluxes of l and r (rhyme_ideal_gas_flux.f90:
// 12-23 from one reciprocal of rho each), with the fused product named in
// every sum of two.
template <int D, int AX>
__device__ __forceinline__ void flux_difference_f32(const Gas<float>& G, const float* l, const float* r, float* df) {
  auto terms = [&](const float* u, float& vn, float& p) {
    const bool none = fabsf(u[0]) < FLT_MIN;  // a vanishing density: no flux
    const float inv = none ? 0.f : 1.f / u[0];
    float s = 0.f;
#pragma unroll
    for (int a = 0; a < D; ++a) s = s + u[1 + a] * u[1 + a];
    const float e = u[D + 1] - 0.5f * s * inv;
    // (an FP32 gm1 is off by up to 3e-8 of itself)
    p = none ? 0.f : __fmaf_rn(e, G.gm1, e * G.gm1_lo);
    vn = __fmul_rn(u[1 + AX], inv);
    return none ? 0.f : u[1 + AX];
  };
  float vl, pl, vr, pr;
  const float ml = terms(l, vl, pl), mr = terms(r, vr, pr);
  df[0] = ml - mr;
#pragma unroll
  for (int a = 0; a < D; ++a)
    df[1 + a] = (a == AX) ? __fmaf_rn(l[1 + a], vl, pl) - __fmaf_rn(r[1 + a], vr, pr)
                          : __fmaf_rn(l[1 + a], vl, -__fmul_rn(r[1 + a], vr));
  df[D + 1] = __fmaf_rn(vl, l[D + 1] + pl, -__fmul_rn(vr, r[D + 1] + pr));
}

// rhyme_muscl_hancock_half_step_extrapolation.f90:15-21; hdtdx = (.5*dt)/dx
template <int D, int AX>
__device__ __forceinline__ void half_step(const Gas<double>& G, const double* u, const double* delta, double hdtdx,
                                          double* l, double* r) {
  double fl[D + 2], fr[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    l[c] = u[c] - m_half(delta[c]);
    r[c] = u[c] + m_half(delta[c]);
  }
  flux<D, AX>(G, l, fl);
  flux<D, AX>(G, r, fr);
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    const double df = fl[c] - fr[c];
    l[c] = l[c] + hdtdx * df;
    r[c] = r[c] + hdtdx * df;
  }
}
template <int D, int AX>
__device__ __forceinline__ void half_step(const Gas<float>& G, const float* u, const float* delta, float hdtdx,
                                          float* l, float* r) {
  float df[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    l[c] = u[c] - 0.5f * delta[c];
    r[c] = u[c] + 0.5f * delta[c];
  }
  flux_difference_f32<D, AX>(G, l, r, df);
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    l[c] = l[c] + hdtdx * df[c];
    r[c] = r[c] + hdtdx * df[c];
  }
}

// Face states of one cell along AX from its neighbours um, u0, up.
template <int D, int AX, typename T>
__device__ __forceinline__ void face_states(const Gas<T>& G, int lim, T w, const T* um, const T* u0,
                                            const T* up, T hdtdx, T* l, T* r) {
  T delta[D + 2];
  limited_slopes<D + 2>(lim, w, um, u0, up, delta);
  half_step<D, AX>(G, u0, delta, hdtdx, l, r);
}

// ---- exact Riemann solver (FP64): rhyme_irs_*, rhyme_riemann_problem_* -----
//
// Every operation is the reference's, in its order; what is arranged for the
// GPU is which lanes of a warp run together. Left and right states differ in
// signs and roles only, so where one lane needs a wave of its left side and
// another lane the same kind of wave of its right side, both run it in one
// pass on the side each has picked (a selection of registers is a few
// integer instructions, a pass of the rarefaction's two powers 57 FP64
// ones). Divisors used more than once (a side's density, pressure and sound
// speed) are kept with their reciprocal (Divisor).

// One side's loop-invariant terms of
// rhyme_irs_nonlinear_wave_function.f90:15-23 (Ak, Bk, 2cs/gm1, 1/(rho cs)):
// the reference recomputes them every Newton iteration with the same
// operations, so computing them once gives the same values.
struct WaveSide {
  double p, Ak, Bk, c2g, irc;
  Divisor ip;
};

__device__ __forceinline__ WaveSide wave_side(const Gas<double>& G, double s_rho, double s_p, double s_cs) {
  WaveSide w;
  w.p = s_p;
  w.ip = divisor(s_p);
  w.Ak = m_div(2.0, G.gp1 * s_rho);
  w.Bk = m_div(G.gm1 * s_p, G.by_gp1);
  w.c2g = m_div(m_twice(s_cs), G.by_gm1);
  w.irc = m_div(1.0, s_rho * s_cs);
  return w;
}

// rhyme_irs_nonlinear_wave_function.f90:13-24 of both sides at p.
__device__ __forceinline__ void nonlinear_waves(const Gas<double>& G, const WaveSide& L, const WaveSide& R, double p,
                                                double& l_f, double& l_fp, double& r_f, double& r_fp) {
  const bool l_shock = m_gt(p, L.p), r_shock = m_gt(p, R.p);
  // rarefactions, then shocks: first the left side of a lane if it is of the
  // kind, else the right one; then the right side where both are
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const bool l = pass == 0 && !l_shock;
    if (l || (!r_shock && (pass == 0 || !l_shock))) {
      double y, z;
      const Divisor ip = l ? L.ip : R.ip;
      m_pow2(m_div(p, ip), G.gm1_2g, -G.gp1_2g, y, z);
      const double f = (l ? L.c2g : R.c2g) * (y - 1.0);
      const double fp = (l ? L.irc : R.irc) * z;
      l_f = l ? f : l_f;
      l_fp = l ? fp : l_fp;
      r_f = l ? r_f : f;
      r_fp = l ? r_fp : fp;
    }
  }
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const bool l = pass == 0 && l_shock;
    if (l || (r_shock && (pass == 0 || l_shock))) {
      const double pk = l ? L.p : R.p;
      const double bp = (l ? L.Bk : R.Bk) + p;
      const Divisor ibp = divisor(bp);
      const double dp = p - pk;
      const double factor = m_sqrt(m_div(l ? L.Ak : R.Ak, ibp));
      const double f = dp * factor;
      // (p - pk)/(2 bp): half of the quotient by bp
      const double fp = factor * (1.0 - div_by_twice(dp, ibp));
      l_f = l ? f : l_f;
      l_fp = l ? fp : l_fp;
      r_f = l ? r_f : f;
      r_fp = l ? r_fp : fp;
    }
  }
}

// Guess 0 of rhyme_irs_guess_p_star.f90:14-38 (the adaptive PVRS /
// two-rarefaction / two-shock choice), not yet floored.
__device__ __forceinline__ double guess_p_star_adaptive(const Gas<double>& G, double l_rho, double vl, double l_p,
                                                        double l_cs, double r_rho, double vr, double r_p,
                                                        double r_cs) {
  const double cup = f64_scale<-2>(l_rho + r_rho) * (l_cs + r_cs);
  const double ppv = fmax_ref(m_half(l_p + r_p) + m_half(vl - vr) * cup, 0.0);
  const double p_min = fmin_ref(l_p, r_p);
  const double p_max = fmax_ref(l_p, r_p);
  // q_max = p_max/p_min <= q_user = 2: for normal numbers the quotient
  // rounds to at most 2 exactly where p_max <= 2 p_min
  const bool near2 = (!f64_tiny(p_min) && f64_hi(p_min) < 0x7fe00000u && f64_hi(p_max) < 0x7ff00000u)
                         ? !m_gt(p_max, m_twice(p_min))
                         : p_max / p_min <= 2.0;
  if (near2 && (m_gt(ppv, p_min) && m_gt(p_max, ppv))) return ppv;  // PVRS
  if (m_gt(p_min, ppv)) {                                          // two-rarefaction
    const Divisor icl = divisor(l_cs), icr = divisor(r_cs);
    const double pq = m_pow(m_div(l_p, r_p), G.gm1_2g);
    const double um = m_div(m_div(pq * vl, icl) + m_div(vr, icr) + G.two_gm1 * (pq - 1.0),
                            m_div(pq, icl) + m_div(1.0, icr));
    const double ptl = 1.0 + m_div(G.half_gm1 * (vl - um), icl);
    const double ptr = 1.0 + m_div(G.half_gm1 * (um - vr), icr);
    return m_half(l_p * m_pow(ptl, G.inv_gm1_2g) + r_p * m_pow(ptr, G.inv_gm1_2g));
  }
  // two-shock
  const double gel = m_sqrt(m_div(m_div(G.two_gp1, l_rho), G.gm1_gp1 * l_p + ppv));
  const double ger = m_sqrt(m_div(m_div(G.two_gp1, r_rho), G.gm1_gp1 * r_p + ppv));
  return m_div(gel * l_p + ger * r_p - (vr - vl), gel + ger);
}

// Guess number k (0..5) of rhyme_irs_guess_p_star.f90:14-71, floored at tiny.
static __device__ __noinline__ double guess_p_star(const Gas<double>& G, int k, double l_rho, double vl, double l_p,
                                            double l_cs, double r_rho, double vr, double r_p, double r_cs) {
  double p;
  if (k == 0) {
    p = guess_p_star_adaptive(G, l_rho, vl, l_p, l_cs, r_rho, vr, r_p, r_cs);
  } else if (k == 1) {  // Ramses
    p = (r_rho * r_cs * l_p + l_rho * l_cs * r_p + r_cs * l_cs * (l_rho * vl - r_rho * vr)) /
        (r_rho * r_cs + l_rho * l_cs);
  } else if (k == 2) {  // two-rarefaction approximation
    p = m_pow((l_cs + r_cs - G.gm1_half * (vr - vl)) /
                  (m_pow(l_cs / l_p, G.gm1_2g) + m_pow(r_cs / r_p, G.gm1_2g)),
              G.inv_gm1_2g);
  } else if (k == 3) {  // two-shock approximation; g_K at :74-80
    double l_g = m_sqrt((2.0 / (G.gp1 * l_rho)) / (l_p + G.gm1_gp1 * l_p));
    double r_g = m_sqrt((2.0 / (G.gp1 * r_rho)) / (r_p + G.gm1_gp1 * r_p));
    p = (l_g * l_p + r_g * r_p - (vr - vl)) / (l_g + r_g);
  } else if (k == 4) {  // p_PV
    p = 0.5 * (l_p + r_p) - 0.125 * (vr - vl) * (l_rho + r_rho) * (l_cs + r_cs);
  } else {  // arithmetic mean
    p = 0.5 * (l_p + r_p);
  }
  return fmax_ref(p, DBL_MIN);
}

// rhyme_irs_exec.f90:19-44 with lazily evaluated guesses. l_f / r_f are the
// wave functions at the last iterate before the final update.
//
// A NaN, once there, stays (both wave functions of a NaN are NaN), so the
// iteration ends with the first p* that a NaN gave: what the cap of n_iter
// steps would leave. An unphysical state (a negative pressure has no sound
// speed) otherwise takes six guesses to the cap: 512 boxes, some of them
// unphysical, a step 83 -> 52 ms in FP64, 9.5 -> 3.3 in the mixed form.
__device__ __forceinline__ double irs_exec(const Gas<double>& G, double tol, int n_iter, const WaveSide& WL,
                                           const WaveSide& WR, double l_rho, double vl, double l_cs, double& l_f,
                                           double r_rho, double vr, double r_cs, double& r_f) {
  double p_star = 0.0, p_prev, l_fp, r_fp;
  const double du = vr - vl;
  for (int gid = 0; gid < 6; ++gid) {
    p_star = guess_p_star(G, gid, l_rho, vl, WL.p, l_cs, r_rho, vr, WR.p, r_cs);
    p_prev = p_star;
    for (int i = 1; i <= n_iter; ++i) {
      nonlinear_waves(G, WL, WR, p_star, l_f, l_fp, r_f, r_fp);
      p_star = p_prev - m_div(l_f + r_f + du, l_fp + r_fp);
      if (m_neg(p_star)) break;
      if (f64_nan(p_prev)) break;
      if (m_gt(tol, m_div(m_twice(fabs(p_star - p_prev)), p_star + p_prev))) break;
      p_prev = p_star;
    }
    if (f64_above(p_star, 0.0)) break;
  }
  if (m_neg(p_star)) p_star = 0.0;
  return p_star;
}

// rp_side_t (rhyme_riemann_problem.f90:53-56), with the pressure as a divisor
template <int D>
struct Side {
  double rho, v[D], p, cs;
  Divisor ip;
};

// rhyme_riemann_problem_w_kfan.f90:14-31
template <int D, int AX>
__device__ __noinline__ void w_kfan(const Gas<double>& G, const Side<D>& s, double dxdt, bool is_right, double* u) {
  double cs = is_right ? -s.cs : s.cs;
  const double base = G.two_gp1 + m_div(G.gm1_gp1, cs) * (s.v[AX] - dxdt);
  double prho, pp;
  m_pow2(base, G.two_gm1, G.inv_gm1_2g, prho, pp);
  double rho = s.rho * prho;
  double v[D];
#pragma unroll
  for (int a = 0; a < D; ++a) v[a] = s.v[a];
  v[AX] = G.two_gp1 * (cs + G.half_gm1 * s.v[AX] + dxdt);
  double p = s.p * pp;
  prim_vars_to_cons<D>(G, rho, v, p, u);
}

// rhyme_riemann_problem_star.f90:40-65 and rhyme_riemann_problem_sampling.f90:
// 13-47 at x/t = dxdt, for the side S of the contact that holds it (u, p: the
// star region's). The right side is the left one with the signs of its
// sound speed turned and its comparisons swapped: negation is exact, so the
// sums round alike. (The reference forms both sides' star states first; only
// the one read here is formed, with the reference's operations.)
template <int D, int AX>
__device__ __forceinline__ void rp_sample_side(const Gas<double>& G, const Side<D>& S, bool right, double us,
                                               double ps, double dxdt, double* u) {
  const double cs = right ? -S.cs : S.cs;
  const double ps_pk = m_div(ps, S.ip);
  double rho_star, inner;  // the star density and the speed that bounds the star region
  const bool shock = m_gt(ps, S.p);
  if (shock) {
    rho_star = m_div(S.rho * (G.gm1_gp1 + ps_pk), G.gm1_gp1 * ps_pk + 1.0);
    inner = S.v[AX] - cs * m_sqrt(G.gp1_2g * ps_pk + G.gm1_2g);
  } else {
    double pg, pa;
    m_pow2(ps_pk, G.g_inv, G.gm1_2g, pg, pa);
    rho_star = S.rho * pg;
    inner = us - cs * pa;
  }
  const bool star = m_gt(right ? inner : dxdt, right ? dxdt : inner);
  bool outside = shock;
  if (!star && !shock) {
    const double head = S.v[AX] - cs;
    outside = !m_gt(right ? head : dxdt, right ? dxdt : head);
  }
  if (star || outside) {
    // rhyme_riemann_problem_w_star{L,R}_{sho,fan}.f90:12-15, or the side itself
    double v[D];
#pragma unroll
    for (int a = 0; a < D; ++a) v[a] = S.v[a];
    v[AX] = star ? us : S.v[AX];
    prim_vars_to_cons<D>(G, star ? rho_star : S.rho, v, star ? ps : S.p, u);
  } else {
    w_kfan<D, AX>(G, S, dxdt, right, u);
  }
}

// The velocities across AX of the side that is sampled, from its conserved
// state q.
template <int D, int AX>
__device__ __forceinline__ void side_transverse(Side<D>& S, const double* q, const Divisor& i0) {
#pragma unroll
  for (int a = 0; a < D; ++a)
    if (a != AX) S.v[a] = m_div(q[1 + a], i0);
}

// Vacuum state W_0: prim_to_cons of w_vacuum (rho, 0.., p).
template <int D>
__device__ __forceinline__ void vacuum_state(const Gas<double>& G, const Rp<double>& rp, double* u) {
  double v[D];
#pragma unroll
  for (int a = 0; a < D; ++a) v[a] = 0.0;
  prim_vars_to_cons<D>(G, rp.vac_rho, v, rp.vac_p, u);
}

// rhyme_riemann_problem_solve.f90:17-103 sampled at x/t = dxdt. (The mixed
// sweeps' FP32 interfaces go through rp_flux_f32 instead, which sends the
// interfaces this solver handles in its vacuum branches to this one.)
template <int D, int AX>
__device__ __forceinline__ void rp_solve(const Gas<double>& G, const Rp<double>& rp, const double* l,
                                         const double* r, double dxdt, double* u) {
  Side<D> L, R;
  L.rho = fmax_ref(l[0], rp.vac_rho);
  R.rho = fmax_ref(r[0], rp.vac_rho);
  const double e_rho = rp.vac_rho_next;
  const bool l_below = m_gt(e_rho, L.rho), r_below = m_gt(e_rho, R.rho);
  const bool vacuum_right = r_below && L.rho > e_rho;
  const bool vacuum_left = l_below && R.rho > e_rho;
  const bool vacuum_both = l_below && r_below;
  const double tiny = DBL_MIN;

  if (vacuum_right) {
#pragma unroll
    for (int a = 0; a < D; ++a) L.v[a] = l[1 + a] / l[0];
    L.p = fmax_ref(pressure<D>(G, l), rp.vac_p);
    L.cs = fmax_ref(sound_speed<D>(G, l), tiny);
    double s_starl = L.v[AX] - 2.0 * L.cs / G.gm1;
    if (dxdt > s_starl) vacuum_state<D>(G, rp, u);
    else if (dxdt > L.v[AX] - L.cs) w_kfan<D, AX>(G, L, dxdt, false, u);
    else prim_vars_to_cons<D>(G, L.rho, L.v, L.p, u);
  } else if (vacuum_left) {
#pragma unroll
    for (int a = 0; a < D; ++a) R.v[a] = r[1 + a] / r[0];
    R.p = fmax_ref(pressure<D>(G, r), rp.vac_p);
    R.cs = fmax_ref(sound_speed<D>(G, r), tiny);
    double s_starr = R.v[AX] + 2.0 * R.cs / G.gm1;
    if (dxdt > R.v[AX] + R.cs) prim_vars_to_cons<D>(G, R.rho, R.v, R.p, u);
    else if (dxdt > s_starr) w_kfan<D, AX>(G, R, dxdt, true, u);
    else vacuum_state<D>(G, rp, u);
  } else if (vacuum_both) {
    vacuum_state<D>(G, rp, u);
  } else {
    // velocities across AX: only for the side sampled (side_transverse)
    const Divisor il = divisor(l[0]), ir = divisor(r[0]);
    L.v[AX] = m_div(l[1 + AX], il);
    L.p = fmax_ref(pressure<D>(G, l, il), rp.vac_p);
    L.cs = fmax_ref(sound_speed<D>(G, l, il), tiny);
    R.v[AX] = m_div(r[1 + AX], ir);
    R.p = fmax_ref(pressure<D>(G, r, ir), rp.vac_p);
    R.cs = fmax_ref(sound_speed<D>(G, r, ir), tiny);
    const double du = R.v[AX] - L.v[AX];
    const double du_crit = m_div(m_twice(L.cs + R.cs), G.by_gm1);
    if (m_gt(du, du_crit)) {  // vacuum generation
      const double s_starl = L.v[AX] - 2.0 * L.cs / G.gm1;
      const double s_starr = R.v[AX] + 2.0 * R.cs / G.gm1;
      if (dxdt > s_starr) {
        side_transverse<D, AX>(R, r, ir);
        if (dxdt > R.v[AX] + R.cs) prim_vars_to_cons<D>(G, R.rho, R.v, R.p, u);
        else w_kfan<D, AX>(G, R, dxdt, true, u);
      } else if (dxdt > s_starl) {
        vacuum_state<D>(G, rp, u);
      } else {
        side_transverse<D, AX>(L, l, il);
        if (dxdt > L.v[AX] - L.cs) w_kfan<D, AX>(G, L, dxdt, false, u);
        else prim_vars_to_cons<D>(G, L.rho, L.v, L.p, u);
      }
    } else {
      // rhyme_riemann_problem_star.f90:12-38
      double l_f = 0.0, r_f = 0.0;
      const WaveSide WL = wave_side(G, L.rho, L.p, L.cs), WR = wave_side(G, R.rho, R.p, R.cs);
      double ps = irs_exec(G, rp.tol, rp.n_iter, WL, WR, L.rho, L.v[AX], L.cs, l_f, R.rho, R.v[AX], R.cs, r_f);
      if (m_gt(rp.vac_p, ps)) ps = rp.vac_p;
      const double us = m_half((R.v[AX] + L.v[AX]) + (r_f - l_f));
      // the side of the contact that x/t = dxdt lies on
      const bool right = m_gt(dxdt, us);
      Side<D> S;
      S.rho = right ? R.rho : L.rho;
      S.v[AX] = right ? R.v[AX] : L.v[AX];
      S.p = right ? R.p : L.p;
      S.cs = right ? R.cs : L.cs;
      S.ip = right ? WR.ip : WL.ip;
      double q[D + 2];
#pragma unroll
      for (int c = 0; c < D + 2; ++c) q[c] = right ? r[c] : l[c];
      side_transverse<D, AX>(S, q, right ? ir : il);
      rp_sample_side<D, AX>(G, S, right, us, ps, dxdt, u);
    }
  }
}

// ---- the mixed form's FP32 interface flux ----------------------------------
// rhyme_riemann_problem_solve.f90:17-103 sampled at x/t = 0 (every interface
// of the sweeps) followed by rhyme_ideal_gas_flux.f90, in FP32, for the
// interfaces the FP64 solver need not redo: a density at or below the
// vacuum density on either side (every vacuum branch), vacuum generation or
// an interface within 10 % of it, a density or pressure ratio beyond 1e6,
// and an iteration that does not converge from the first guess set *need64
// instead, and the caller queues the interface for rp_solve<double>. The
// root is the FP64 form's: of the wave functions of
// rhyme_irs_nonlinear_wave_function.f90 summed, from a first guess of
// rhyme_irs_guess_p_star.f90:14-38, by an iteration of third order in place
// of rhyme_irs_exec.f90:28-39's Newton steps; then the sampled side's star
// state (rhyme_riemann_problem_star.f90:40-65) and the tests of
// rhyme_riemann_problem_sampling.f90:13-47 at x/t = 0, including the fan of
// rhyme_riemann_problem_w_kfan.f90. The FP32 arithmetic is arranged for
// fewer divisions (one reciprocal per side of rho, p and rho cs; the
// quotients of gamma from Gas; the convergence test multiplied out; the flux
// formed from the sampled primitive state instead of from its conserved
// form), which also skips the cancellation of E - |m|^2/(2 rho). Where a
// sum could fuse one product or another, or a product that is also used by
// itself, the code says which, so that every kernel that inlines it rounds
// alike. Measured with the limiter above (3-D 256^3 in a developed flow): the
// Halley steps, the series in place of log1pf, expm1f and expf, the two
// sides' sampling in one copy and the cheaper divisions took the x+y sweep
// from 968 to 866 us and the z sweep from 747 to 704 (753 and 639 since the
// step that limited_slopes describes); relative L1 error
// against FP64 over 66 runs in 1-3-D, all limiters: density 2.80e-8 ->
// 2.62e-8, energy 3.88e-8 -> 3.64e-8.
// fpp: the second derivative.
__device__ __forceinline__ void wave_f32(const Gas<float>& G, float Ak, float Bk, float c2g, float irc, float pk,
                                         float ipk, float p, float& f, float& fprime, float& fpp) {
  const float dp = p - pk;
  if (dp > 0.f) {
    const float rb = 1.f / (Bk + p);
    const float factor = sqrtf(Ak * rb);
    const float y = __fmul_rn(dp, rb);
    f = __fmul_rn(dp, factor);
    fprime = __fmul_rn(factor, 1.f - 0.5f * y);
    fpp = __fmul_rn(-factor * rb, 1.f - 0.75f * y);
  } else {
    // (p/p_k)^e - 1 as expm1(e log1p(x)), x = (p - p_k)/p_k: the same
    // quantity without the cancellation of a power near 1 (p - p_k is exact
    // there). The derivative's power follows from it:
    // (p/p_k)^(-gp1_2g) = (p/p_k)^(e - 1).
    const float x = __fmul_rn(dp, ipk);
    float E;
    if (x > -0.3f) {
      // log1p(x) = 2 atanh(s), s = x/(2 + x), |s| < 0.177, and expm1 of
      // |u| < 0.18 (e < 1/2) by their Taylor series; truncated below 1e-8
      const float s = __fdividef(x, 2.f + x), s2 = s * s;
      const float ss = s + s;
      const float t = __fmaf_rn(ss * s2, 1.f / 3.f + s2 * (1.f / 5.f + s2 * (1.f / 7.f + s2 * (1.f / 9.f))), ss);
      const float u = G.gm1_2g * t;
      E = __fmaf_rn(u * u, 0.5f + u * (1.f / 6.f + u * (1.f / 24.f + u * (1.f / 120.f + u * (1.f / 720.f)))), u);
    } else {
      E = expm1f(G.gm1_2g * log1pf(x));
    }
    const float iw = 1.f / (1.f + x);  // p_k/p
    f = __fmul_rn(c2g, E);
    fprime = __fmul_rn(irc, iw + iw * E);
    fpp = __fmul_rn(-G.gp1_2g * fprime, iw * ipk);
  }
}

template <int D, int AX>
__device__ __forceinline__ void rp_flux_f32(const Gas<float>& G, const Rp<float>& rp, const float* l,
                                            const float* r, float* f, bool* need64) {
  const float e_rho = rp.vac_rho_next;
  if (!(fmax_ref(l[0], rp.vac_rho) >= e_rho) || !(fmax_ref(r[0], rp.vac_rho) >= e_rho)) {
    *need64 = true;
    return;
  }
  // both densities above the vacuum density: the clamp of rho is inactive
  const float rl = l[0], rr = r[0];
  const float il = 1.f / rl, ir = 1.f / rr;
  float sl = 0.f, sr = 0.f;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    sl = sl + l[1 + a] * l[1 + a];
    sr = sr + r[1 + a] * r[1 + a];
  }
  const float el = l[D + 1] - 0.5f * sl * il, er = r[D + 1] - 0.5f * sr * ir;
  const float pl_raw = __fmaf_rn(el, G.gm1, el * G.gm1_lo), pr_raw = __fmaf_rn(er, G.gm1, er * G.gm1_lo);
  const float pl = fmax_ref(pl_raw, rp.vac_p), pr = fmax_ref(pr_raw, rp.vac_p);
  const float cl = fmax_ref(sqrtf(G.g * pl_raw * il), FLT_MIN);
  const float cr = fmax_ref(sqrtf(G.g * pr_raw * ir), FLT_MIN);
  const float vl = __fmul_rn(l[1 + AX], il), vr = __fmul_rn(r[1 + AX], ir);
  const float du = vr - vl;
  const float du_crit = G.two_gm1 * (cl + cr);
  const float rmin = fmin_ref(rl, rr), rmax = fmax_ref(rl, rr);
  const float pmin = fmin_ref(pl, pr), pmax = fmax_ref(pl, pr);
  if (!(du_crit - du > 0.1f * du_crit) || !(rmin * 1e6f > rmax) || !(pmin * 1e6f > pmax)) {
    *need64 = true;
    return;
  }
  const float ipl = 1.f / pl, ipr = 1.f / pr;
  const float ircl = __fdividef(il, cl), ircr = __fdividef(ir, cr);  // 1/(rho cs)
  // First guess: the linearised (PVRS) pressure where it lies near the two
  // sides' (the iteration takes it to the root in one or two steps), else
  // the two-rarefaction or two-shock value.
  float p;
  {
    const float cup = 0.25f * (rl + rr) * (cl + cr);
    const float ppv = fmax_ref(__fmaf_rn(-0.5f * du, cup, 0.5f * (pl + pr)), 0.f);
    if (pmax <= 2.f * pmin && ppv > 0.8f * pmin && ppv < 1.25f * pmax) {
      p = ppv;
    } else if (ppv < pmin) {  // two-rarefaction
      const float icl = ircl * rl, icr = ircr * rr;  // 1/cs
      const float pq = m_pow(pl * ipr, G.gm1_2g);
      const float um = __fdividef(__fmaf_rn(G.two_gm1, pq - 1.f, __fmaf_rn(pq * vl, icl, vr * icr)),
                                  __fmaf_rn(pq, icl, icr));
      const float ptl = 1.f + G.half_gm1 * (vl - um) * icl;
      const float ptr = 1.f + G.half_gm1 * (um - vr) * icr;
      p = 0.5f * __fmaf_rn(pl, m_pow(ptl, G.inv_gm1_2g), pr * m_pow(ptr, G.inv_gm1_2g));
    } else {  // two-shock
      const float gel = sqrtf(__fdividef(G.two_gp1 * il, G.gm1_gp1 * pl + ppv));
      const float ger = sqrtf(__fdividef(G.two_gp1 * ir, G.gm1_gp1 * pr + ppv));
      p = __fdividef(__fmaf_rn(gel, pl, __fmaf_rn(ger, pr, -du)), gel + ger);
    }
    p = fmax_ref(p, FLT_MIN);
  }
  // Halley's iteration from it: the wave functions' second derivatives cost
  // a few products and make it of third order, with the error of a step
  // below 0.12 of its cube (relative to p; 0.097 for gamma = 5/3, 0.103 for
  // 7/5, 0.116 for 1.1). A step below rp.tol therefore leaves an error below
  // the FP32 rounding, and the wave functions at the new p follow from their
  // Taylor series: no evaluation is spent on confirming the root. Under a
  // tolerance below FP32's resolution rp.settle asks besides that p, rounded,
  // has moved by less than the tolerance (1 otherwise: always so).
  const float Akl = G.two_gp1 * il, Bkl = __fmul_rn(G.gm1_gp1, pl), c2gl = G.two_gm1 * cl;
  const float Akr = G.two_gp1 * ir, Bkr = __fmul_rn(G.gm1_gp1, pr), c2gr = G.two_gm1 * cr;
  float fl = 0.f, fr = 0.f;
  bool conv = false;
  for (int i = 1; i <= rp.n_iter; ++i) {
    float fpl, fpr, fppl, fppr;
    wave_f32(G, Akl, Bkl, c2gl, ircl, pl, ipl, p, fl, fpl, fppl);
    wave_f32(G, Akr, Bkr, c2gr, ircr, pr, ipr, p, fr, fpr, fppr);
    const float ifp = 1.f / (fpl + fpr);
    const float newton = __fmul_rn(fl + fr + du, ifp);
    const float h = 1.f - 0.5f * newton * (fppl + fppr) * ifp;
    const float d = __fmul_rn(-newton, 1.f / fmaxf(h, 0.5f));
    const float before = p;
    p = p + d;
    if (!(p > 0.f)) break;
    if (fabsf(d) < rp.tol * p) {
      if (!(fabsf(p - before) < rp.settle * p)) continue;
      fl = __fmaf_rn(d, __fmaf_rn(0.5f * d, fppl, fpl), fl);
      fr = __fmaf_rn(d, __fmaf_rn(0.5f * d, fppr, fpr), fr);
      conv = true;
      break;
    }
  }
  if (!conv) {
    *need64 = true;
    return;
  }
  const float ps = (p < rp.vac_p) ? rp.vac_p : p;
  const float us = 0.5f * ((vr + vl) + (fr - fl));
  // the sampled side at x/t = 0: its density, normal velocity and pressure;
  // the right side is the left one with its sound speed's sign turned and the
  // comparisons with 0 swapped, so that all lanes run one copy
  float rho, vn, pp;
  const bool right = 0.f > us;
  const float k_rho = right ? rr : rl, k_v = right ? vr : vl, k_p = right ? pr : pl;
  const float k_cs = right ? -cr : cl, k_ic = right ? -(ircr * rr) : ircl * rl;  // signed cs, 1/cs
  const float ps_pk = __fmul_rn(ps, right ? ipr : ipl);
  const bool shock = ps > k_p;
  float rs, inner;  // the star density and the speed that bounds the star region
  if (shock) {
    rs = k_rho * __fdividef(G.gm1_gp1 + ps_pk, G.gm1_gp1 * ps_pk + 1.f);
    inner = k_v - k_cs * sqrtf(G.gp1_2g * ps_pk + G.gm1_2g);
  } else {
    float pg, pa;
    m_pow2(ps_pk, G.g_inv, G.gm1_2g, pg, pa);
    rs = k_rho * pg;
    inner = us - k_cs * pa;
  }
  const float head = k_v - k_cs;
  const bool star = right ? inner > 0.f : inner < 0.f;
  const bool fan = !star && !shock && (right ? head > 0.f : head < 0.f);
  rho = star ? rs : k_rho;
  vn = star ? us : k_v;
  pp = star ? ps : k_p;
  if (fan) {  // inside the rarefaction fan (w_kfan at x/t = 0)
    const float base = G.two_gp1 + G.gm1_gp1 * k_ic * k_v;
    float prho, ppw;
    m_pow2(base, G.two_gm1, G.inv_gm1_2g, prho, ppw);
    rho = k_rho * prho;
    vn = G.two_gp1 * (k_cs + G.half_gm1 * k_v);
    pp = k_p * ppw;
  }
  // the flux of the sampled primitive state
  float v[D];
  float s = 0.f;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    v[a] = (a == AX) ? vn : (right ? r[1 + a] * ir : l[1 + a] * il);
    s = s + v[a] * v[a];
  }
  const float mn = rho * vn;
  f[0] = mn;
#pragma unroll
  for (int a = 0; a < D; ++a) f[1 + a] = mn * v[a];
  f[1 + AX] = f[1 + AX] + pp;
  f[D + 1] = vn * __fmaf_rn(pp, G.g_gm1, 0.5f * rho * s);
  // a flux that is not finite: FP64's (one sum sees every component)
  float t = f[0];
#pragma unroll
  for (int c = 1; c < D + 2; ++c) t = fabsf(t) + fabsf(f[c]);
  if (!(t < 3.4e38f)) *need64 = true;
}

// Interface flux: Riemann state at x/t = 0 (dx = 0 in
// rhyme_muscl_hancock_solve_memory_intensive.f90:110-116), then calc_flux.
template <int D, int AX>
__device__ __forceinline__ void interface_flux(const Gas<double>& G, const Rp<double>& rp, const double* l,
                                               const double* r, double* f) {
  double u[D + 2];
  rp_solve<D, AX>(G, rp, l, r, 0.0, u);
  flux<D, AX>(G, u, f);
}

}  // namespace rgpu
