// box_elems.cuh -- per-element bodies of the plain FP64 box kernels.
//
// Each function processes element t of one box's index space for one pass
// (a ghost line, a cell's face states, an interface, a cell update). The
// single-box kernels (kernels_box.cu) run them over a grid-stride range; the
// batched kernels (kernels_batch.cu) run them over (box, chunk) work items of
// a box table. Both therefore execute the same arithmetic, so a box stepped
// alone and inside a batch gives bit-identical results.
#pragma once

#include "rgpu_internal.h"

namespace rgpu {

// Per-box values of the boundary and limiter modules.
struct BoxRules {
  int bc[6];
  double inflow[6][5];
  int limiter;
  double omega;
  int solver_type;
};

__host__ __device__ inline BoxRules rules_of(const DevParams& P) {
  BoxRules r;
  for (int i = 0; i < 6; ++i) {
    r.bc[i] = P.bc[i];
    for (int c = 0; c < 5; ++c) r.inflow[i][c] = P.inflow[i][c];
  }
  r.limiter = P.limiter;
  r.omega = P.omega;
  r.solver_type = P.solver_type;
  return r;
}

// Ghost lines of a box: line q of (axis, component), q = 0 .. ghost_lines - 1,
// the transverse positions in array order.
__host__ __device__ inline long long ghost_lines(int D, const Geom& g, int axis) {
  long long t = 1;
  for (int b = 0; b < D; ++b)
    if (b != axis) t *= g.n[b];
  return t;
}

// K1 element: fills the left then the right 2-cell ghost layer of one line
// in the order of rhyme_samr_bc_set_boundaries.f90:9-20; writes U and (if
// given) M. M (optional) receives the same ghost values (the other state
// buffer); Mf (optional) their FP32 images (the mirror of the mixed form),
// equal to what a fill of the mirror from its own interior would write.
// A plane holds fewer than 2^32 lines (the array would not fit otherwise),
// so the position is split in 32 bits.
template <int D, typename T>
__device__ __forceinline__ void ghost_line(const int* bc, const double (*inflow)[5], T* __restrict__ U, T* __restrict__ M, const Geom& g,
                                           int axis, int c, unsigned q, float* __restrict__ Mf) {
  const unsigned n1 = (D == 1) ? 1u : (unsigned)g.n[axis == 0 ? 1 : 0];
  unsigned i2 = 0, i1 = q;
  if constexpr (D == 3) {
    i2 = q / n1;
    i1 = q - i2 * n1;
  }
  // cell 0 of the line
  long long base = g.s[0] + (D > 1 ? g.s[1] : 0) + (D > 2 ? g.s[2] : 0);
  const int t1 = (axis == 0) ? 1 : 0, t2 = (axis == 2) ? 1 : 2;
  if constexpr (D > 1) base += (long long)(i1 + 1) * g.s[t1];
  if constexpr (D > 2) base += (long long)(i2 + 1) * g.s[t2];
  const long long sa = g.s[axis], N = g.n[axis];
  T* f = U + (long long)c * g.field;
  T* m = M ? M + (long long)c * g.field : nullptr;
  float* mf = Mf ? Mf + (long long)c * g.field : nullptr;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int type = bc[2 * axis + side];
    if (type < 1 || type > 4) continue;  // the caller fills this face
    const bool far = (type == 3) != (side == 1);  // the sources lie at the line's other end
    const long long g0 = side ? base + (N + 1) * sa : base, g1 = side ? g0 + sa : g0 - sa;
    const long long s0 = far ? base + N * sa : base + sa, s1 = far ? s0 - sa : s0 + sa;
    T v0, v1;
    if (type == 4) {  // inflow
      v0 = v1 = (T)inflow[2 * axis + side][c];
    } else {
      v0 = f[s0];
      v1 = (s1 == g0) ? v0 : f[s1];  // a periodic line of one cell: the first ghost is the second's source
      if (type == 1 && c == 1 + axis) {  // reflective: negate normal momentum
        v0 = -v0;
        v1 = -v1;
      }
    }
    f[g0] = v0;
    f[g1] = v1;
    if (m) {
      m[g0] = v0;
      m[g1] = v1;
    }
    if (mf) {
      mf[g0] = mirror_of(v0);
      mf[g1] = mirror_of(v1);
    }
  }
}

// Extents of the face (cells 0..N+1 along AX) and interface (0..N) passes.
template <int AX>
__host__ __device__ inline long long face_count(const Geom& g) {
  long long t = 1;
  for (int a = 0; a < 3; ++a) t *= (a == AX) ? g.n[a] + 2 : g.n[a];
  return t;
}
template <int AX>
__host__ __device__ inline long long iface_count(const Geom& g) {
  long long t = 1;
  for (int a = 0; a < 3; ++a) t *= (a == AX) ? g.n[a] + 1 : g.n[a];
  return t;
}

template <int D, int AX>
__device__ __forceinline__ long long pass_offset(const Geom& g, int extra, long long t) {
  int e[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) e[a] = (a == AX) ? g.n[a] + extra : g.n[a];
  int c0 = (int)(t % e[0]);
  const long long q = t / e[0];
  int c1 = (int)(q % e[1]);
  int c2 = (int)(q / e[1]);
  if (AX != 0) c0 += 1;
  if (AX != 1) c1 += 1;
  if (AX != 2) c2 += 1;
  return g.at(D, c0, c1, c2);
}

// K3a element: limited slopes and half-step face states of one cell
// (loop 1 of rhyme_muscl_hancock_solve_memory_intensive.f90:56-98).
template <int D, int AX>
__device__ __forceinline__ void faces_elem(const Gas<double>& G, const BoxRules& R,
                                           const double* __restrict__ U, const Geom& g, double hdtdx,
                                           double* __restrict__ FS, long long t) {
  const long long F = g.field;
  const long long sa = g.s[AX];
  double* ul = FS + (long long)(AX * 2 + 0) * (D + 2) * F;
  double* ur = FS + (long long)(AX * 2 + 1) * (D + 2) * F;
  const long long o = pass_offset<D, AX>(g, 2, t);
  double um[D + 2], u0[D + 2], up[D + 2], l[D + 2], r[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    const double* f = U + (long long)c * F + o;
    um[c] = f[-sa];
    u0[c] = f[0];
    up[c] = f[sa];
  }
  face_states<D, AX>(G, R.limiter, R.omega, um, u0, up, hdtdx, l, r);
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    ul[(long long)c * F + o] = l[c];
    ur[(long long)c * F + o] = r[c];
  }
}

// K3b element: exact Riemann problem at x/t = 0 and its flux for one
// interface (loop 2, :107-140).
template <int D, int AX>
__device__ __forceinline__ void flux_elem(const Gas<double>& G, const Rp<double>& rp,
                                          const double* __restrict__ FS, const Geom& g,
                                          double* __restrict__ FR, long long t) {
  const long long F = g.field;
  const long long sa = g.s[AX];
  const double* ul = FS + (long long)(AX * 2 + 0) * (D + 2) * F;
  const double* ur = FS + (long long)(AX * 2 + 1) * (D + 2) * F;
  double* fr = FR + (long long)AX * (D + 2) * F;
  const long long o = pass_offset<D, AX>(g, 1, t);
  double l[D + 2], r[D + 2], f[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    l[c] = ur[(long long)c * F + o];
    r[c] = ul[(long long)c * F + o + sa];
  }
  interface_flux<D, AX>(G, rp, l, r, f);
#pragma unroll
  for (int c = 0; c < D + 2; ++c) fr[(long long)c * F + o] = f[c];
}

// K3c element: U^{n+1} of one interior cell, U + ((X + Y) + Z) or, for the
// cpu-intensive solver, ((U + X) + Y) + Z (loop 3, :148-180;
// rhyme_muscl_hancock_solve_cpu_intensive.f90:117-136).
template <int D>
__device__ __forceinline__ void update_elem(int solver_type, const double* __restrict__ U,
                                            const double* __restrict__ FR, const Geom& g,
                                            const double* dtdx, double* __restrict__ Unew,
                                            long long t) {
  const long long n0 = g.n[0], n1 = g.n[1];
  const int i = (int)(t % n0) + 1;
  const long long q = t / n0;
  const int j = (int)(q % n1) + 1;
  const int k = (int)(q / n1) + 1;
  const long long o = g.at(D, i, j, k);
  const long long F = g.field;
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    double d[3];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const double* fr = FR + ((long long)a * (D + 2) + c) * F + o;
      d[a] = dtdx[a] * (fr[-g.s[a]] - fr[0]);
    }
    const double u = U[(long long)c * F + o];
    double out;
    if (solver_type == 1) {
      out = u;
#pragma unroll
      for (int a = 0; a < D; ++a) out = out + d[a];
    } else {
      double acc = d[0];
#pragma unroll
      for (int a = 1; a < D; ++a) acc = acc + d[a];
      out = u + acc;
    }
    Unew[(long long)c * F + o] = out;
  }
}

// Signal speed |v| + cs of one interior cell for the CFL maximum
// (rhyme_cfl_time_step.f90:77-84); sets bad for non-positive density or a
// non-finite value.
template <int D>
__device__ __forceinline__ double signal_speed_elem(const Gas<double>& G, const double* __restrict__ U,
                                                    const Geom& g, long long t, int& bad) {
  const long long n0 = g.n[0], n1 = g.n[1];
  const int i = (int)(t % n0) + 1;
  const long long q = t / n0;
  const int j = (int)(q % n1) + 1;
  const int k = (int)(q / n1) + 1;
  const long long o = g.at(D, i, j, k);
  double u[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) u[c] = U[(long long)c * g.field + o];
  double ss = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) ss = ss + u[1 + a] * u[1 + a];
  const Divisor i0 = divisor(u[0]);
  const double v = m_div(m_sqrt(ss), i0) + sound_speed<D>(G, u, i0);
  if (!(u[0] > 0.0) || !isfinite(v)) bad = 1;
  return v;
}

}  // namespace rgpu
