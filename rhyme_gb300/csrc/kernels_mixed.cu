// kernels_mixed.cu -- mixed-precision MUSCL-Hancock step.
//
// The conserved state stays FP64 in HBM (U) with an FP32 mirror (Uf), which
// the last sweep of each step writes along with U^{n+1} and its FP32 signal
// speeds, so that the next step's CFL pass only forms dt; after an upload or
// a change from outside the CFL pass writes the mirror itself.
// Each axis is one fused sweep kernel (the x and y axes of a 3-D box one
// kernel together): a CTA stages a slab of Uf (S cells along the sweep axis
// plus the 2-cell ghost/halo layer, for P pencils) in shared memory, computes
// FP32 limited slopes and half-step face states for S+2 cells, solves the S+1
// exact Riemann problems of the slab in FP32 and forms the flux difference of
// its S cells; the last sweep of a large box marches along its columns
// instead (sweep.cuh). Ghost cells come from the interior while a tile is
// staged, so a resident run fills them in memory only at its end. The flux
// differences of the axes are summed in FP32 in the reference's association
// ((X + Y) + Z), and the last sweep adds the sum to U in FP64 and writes
// U^{n+1}: one FP64 add per conserved component and cell, since on GB300 even
// FP64 adds are scarce (the conversions around it are integer operations).
//
// Interfaces that near vacuum, whose FP32 iteration does not end (under a
// tolerance below FP32's resolution: whose p does not settle), or whose FP32
// face states or flux are not finite, get a zero flux in the sweep and are appended (once, by the tile
// that owns them) to a device queue. After the last sweep one kernel redoes
// each queued interface in FP64 from U^n, which the step leaves intact
// (limited slopes and half-step face states of its two cells, exact Riemann
// problem, flux: the device code of the plain path instantiated for double),
// and applies -+ dt/dx * F to the two adjacent interior cells of U^{n+1}.
// Keeping the FP64 code out of the sweeps keeps them at 40-51 registers (it
// tripled their register count inline).
//
// The CFL maximum of the mixed path is taken in FP32 over the mirror; dt
// itself is formed in FP64.
//
// For the drop-in loop with the state in host memory, ingest_kernel takes
// each slab of an upload as it arrives (the mirror, the ghost cells of the
// other buffer, the slab's share of the CFL maximum), cfl_finish_kernel
// forms dt from that maximum, and launch_mh_solve_mixed_slab solves the box
// in slabs of rows, each with the FP64 fix-up of the entries queued so far,
// so that finished rows can be copied back while the next slab is solved.
#include <math_constants.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>

#include "../../include/rhyme_gpu.h"
#include "rgpu_internal.h"

namespace rgpu {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 152 * 32;

inline int grid_for(long long total, int block) {
  long long b = (total + block - 1) / block;
  if (b < 1) b = 1;
  if (b > kMaxBlocks) b = kMaxBlocks;
  return (int)b;
}

// U (FP64) -> Uf (FP32) over whole component blocks (ghosts included).
__global__ void __launch_bounds__(kThreads) to_f32_kernel(const double* __restrict__ U,
                                                          float* __restrict__ Uf, long long n) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    Uf[t] = mirror_of(U[t]);
}

// |v| + cs of one cell in FP32; bad marks non-positive density or a
// non-finite value.

// Interior cell t: its FP32 mirror, written to Uf from U, and its signal
// speed.
template <int D>
__device__ __forceinline__ float signal_speed_f32(const MixedParams& M, const double* __restrict__ U,
                                                  float* __restrict__ Uf, const Geom& g, long long t, int& bad) {
  const long long n0 = g.n[0], n1 = g.n[1];
  const int i = (int)(t % n0) + 1;
  const long long q = t / n0;
  const int j = (int)(q % n1) + 1;
  const int k = (int)(q / n1) + 1;
  const long long o = g.at(D, i, j, k);
  float u[D + 2];
#pragma unroll
  for (int c = 0; c < D + 2; ++c) {
    u[c] = mirror_of(U[(long long)c * g.field + o]);
    Uf[(long long)c * g.field + o] = u[c];
  }
  return speed_f32<D>(M, u, bad);
}

// Block-wide maximum and or of (m, bad), folded into *bits and *status by
// one thread.
__device__ __forceinline__ void block_fold(float m, int bad, unsigned long long* bits, int* status) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_down_sync(0xffffffffu, m, off);
    if (o > m) m = o;
    bad |= __shfl_down_sync(0xffffffffu, bad, off);
  }
  __shared__ float sm[kThreads / 32];
  __shared__ int sb[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sm[warp] = m;
    sb[warp] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kThreads / 32; ++k) {
      if (sm[k] > m) m = sm[k];
      bad |= sb[k];
    }
    atomicMax(bits, (unsigned long long)__float_as_uint(m));
    if (bad) atomicOr(status, 1);
  }
}

// The arrival of rows [e0, e1) (elements of every component block; whole
// rows of the outermost axis, ghosts included) of a box just copied into U:
// the FP32 mirror Uf of every cell is written, the ghost cells are copied
// into the other state buffer V, whose interior the next solve writes, and
// its mirror Vf, and (bits given) the FP32 signal speed of every interior
// cell (the arithmetic of cfl_f32_kernel) is folded into *bits, so that the
// CFL maximum is ready when the last row has arrived. Indexes are split in 32
// bits (a component block of 2^32 elements does not fit the GPU).
// With H the elements are read from there, page-locked host memory mapped
// for the GPU, and written to U as well: one launch per upload of a box too
// small to be sent in overlapped slabs (the host link carries SM loads as
// fast as copies; 96 boxes of 3 MB took 2.97 ms as a copy and a pass each).
template <int D>
__global__ void __launch_bounds__(kThreads)
    ingest_kernel(MixedParams M, const double* __restrict__ H, double* __restrict__ U, double* __restrict__ V,
                  float* __restrict__ Uf, float* __restrict__ Vf, Geom g, unsigned e0, unsigned e1, unsigned long long* bits, int* status) {
  const long long F = g.field;
  const unsigned E0 = (unsigned)g.n[0] + 4;  // row length along x, ghosts included
  const unsigned E1 = (unsigned)g.n[1] + 4;  // rows per plane
  float m = 0.f;
  int bad = 0;
  for (unsigned long long tt = e0 + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; tt < e1;
       tt += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned t = (unsigned)tt;
    const unsigned r = (D > 1) ? t / E0 : 0;
    const int i = (int)(t - r * E0);
    bool in = i >= 2 && i <= g.n[0] + 1;
    if constexpr (D == 2) in = in && (int)r >= 2 && (int)r <= g.n[1] + 1;
    if constexpr (D > 2) {
      const unsigned k = r / E1;
      const int j = (int)(r - k * E1);
      in = in && j >= 2 && j <= g.n[1] + 1 && (int)k >= 2 && (int)k <= g.n[2] + 1;
    }
    const double* src = H ? H : U;
    double x5[D + 2];
    float u[D + 2];
#pragma unroll
    for (int c = 0; c < D + 2; ++c) x5[c] = src[(long long)c * F + t];
#pragma unroll
    for (int c = 0; c < D + 2; ++c) {
      const double x = x5[c];
      if (H) U[(long long)c * F + t] = x;
      u[c] = mirror_of(x);
      Uf[(long long)c * F + t] = u[c];
      if (!in) {
        V[(long long)c * F + t] = x;
        Vf[(long long)c * F + t] = u[c];
      }
    }
    if (in && bits) {
      const float v = speed_f32<D>(M, u, bad);
      if (v > m) m = v;
    }
  }
  if (bits) block_fold(m, bad, bits, status);
}

// dt from a maximum folded by ingest_kernel: the last step of cfl_f32_kernel.
__global__ void cfl_finish_kernel(const unsigned long long* __restrict__ bits, double courant, double mdx,
                                  StepScratch s) {
  const float mu = __uint_as_float((unsigned int)*bits);
  const double dt = courant * mdx / (double)mu;
  *s.dt = dt;
  if (s.dt_trace) {
    const int pos = *s.trace_pos;
    if (pos >= 0 && pos < s.trace_cap) s.dt_trace[pos] = dt;
    *s.trace_pos = pos + 1;
  }
}

// FP32 mirror of the interior of U and its signal-speed maximum; the last
// block forms dt = courant * min(dx) / max in FP64 and resets the
// accumulators.
template <int D>
__global__ void __launch_bounds__(kThreads)
    cfl_f32_kernel(MixedParams M, const double* __restrict__ U, float* __restrict__ Uf, Geom g, double courant,
                   double mdx, StepScratch s) {
  const long long total = (long long)g.n[0] * g.n[1] * (long long)g.n[2];
  float m = 0.f;
  int bad = 0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const float v = signal_speed_f32<D>(M, U, Uf, g, t, bad);
    if (v > m) m = v;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_down_sync(0xffffffffu, m, off);
    if (o > m) m = o;
    bad |= __shfl_down_sync(0xffffffffu, bad, off);
  }
  __shared__ float sm[kThreads / 32];
  __shared__ int sb[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sm[warp] = m;
    sb[warp] = bad;
  }
  __syncthreads();
  if (warp == 0) {
    m = (lane < kThreads / 32) ? sm[lane] : 0.f;
    bad = (lane < kThreads / 32) ? sb[lane] : 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_down_sync(0xffffffffu, m, off);
      if (o > m) m = o;
      bad |= __shfl_down_sync(0xffffffffu, bad, off);
    }
    if (lane == 0) {
      // non-negative floats order like their bit patterns
      atomicMax(s.max_bits, (unsigned long long)__float_as_uint(m));
      if (bad) atomicOr(s.status, 1);
      __threadfence();
      const unsigned int prev = atomicAdd(s.counter, 1u);
      if (prev == gridDim.x - 1) {
        __threadfence();
        const float mu = __uint_as_float((unsigned int)atomicAdd(s.max_bits, 0ull));
        const double dt = courant * mdx / (double)mu;
        *s.dt = dt;
        if (s.dt_trace) {
          const int pos = *s.trace_pos;
          if (pos >= 0 && pos < s.trace_cap) s.dt_trace[pos] = dt;
          *s.trace_pos = pos + 1;
        }
        atomicExch(s.max_bits, 0ull);
        atomicExch(s.counter, 0u);
      }
    }
  }
}

// The CFL of a step after a carrying step: dt from the carried maximum when
// it is the current state's (no FP64 fix-up changed cells after it), else
// the pass of cfl_f32_kernel; then the carry is cleared for this step's own
// carrying sweep.
template <int D>
__global__ void __launch_bounds__(kThreads)
    cfl_carry_kernel(MixedParams M, const double* __restrict__ U, float* __restrict__ Uf, Geom g, double courant,
                     double mdx, StepScratch s, unsigned long long* carry_bits, int* carry_ok,
                     const int* __restrict__ prev_fix, int* __restrict__ this_fix) {
  step_begin();
  if (blockIdx.x == 0 && threadIdx.x == 0) *this_fix = 0;
  const bool use = *carry_ok != 0 && *prev_fix == 0;
  if (use) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const unsigned long long carried = *carry_bits;
      const float mu = __uint_as_float((unsigned int)carried);
      if (carried >> 32) atomicOr(s.status, 1);
      const double dt = courant * mdx / (double)mu;
      *s.dt = dt;
      if (s.dt_trace) {
        const int pos = *s.trace_pos;
        if (pos >= 0 && pos < s.trace_cap) s.dt_trace[pos] = dt;
        *s.trace_pos = pos + 1;
      }
      *carry_bits = 0ull;
    }
    return;
  }
  const long long total = (long long)g.n[0] * g.n[1] * (long long)g.n[2];
  float m = 0.f;
  int bad = 0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const float v = signal_speed_f32<D>(M, U, Uf, g, t, bad);
    if (v > m) m = v;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_down_sync(0xffffffffu, m, off);
    if (o > m) m = o;
    bad |= __shfl_down_sync(0xffffffffu, bad, off);
  }
  __shared__ float sm[kThreads / 32];
  __shared__ int sb[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sm[warp] = m;
    sb[warp] = bad;
  }
  __syncthreads();
  if (warp == 0) {
    m = (lane < kThreads / 32) ? sm[lane] : 0.f;
    bad = (lane < kThreads / 32) ? sb[lane] : 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_down_sync(0xffffffffu, m, off);
      if (o > m) m = o;
      bad |= __shfl_down_sync(0xffffffffu, bad, off);
    }
    if (lane == 0) {
      atomicMax(s.max_bits, (unsigned long long)__float_as_uint(m));
      if (bad) atomicOr(s.status, 1);
      __threadfence();
      const unsigned int prev = atomicAdd(s.counter, 1u);
      if (prev == gridDim.x - 1) {
        __threadfence();
        const float mu = __uint_as_float((unsigned int)atomicAdd(s.max_bits, 0ull));
        const double dt = courant * mdx / (double)mu;
        *s.dt = dt;
        if (s.dt_trace) {
          const int pos = *s.trace_pos;
          if (pos >= 0 && pos < s.trace_cap) s.dt_trace[pos] = dt;
          *s.trace_pos = pos + 1;
        }
        atomicExch(s.max_bits, 0ull);
        atomicExch(s.counter, 0u);
        *carry_bits = 0ull;
        *carry_ok = 1;
      }
    }
  }
}

// launch_carry_status: see rgpu_internal.h. The speeds' mirror is written as
// the next whole CFL pass would.
template <int D>
__global__ void __launch_bounds__(kThreads)
    carry_status_kernel(MixedParams M, const double* __restrict__ U, float* __restrict__ Uf, Geom g,
                        unsigned long long* carry_bits, const int* __restrict__ carry_ok,
                        const int* __restrict__ prev_fix, int* status) {
  if (*carry_ok != 0 && (!prev_fix || *prev_fix == 0)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (*carry_bits >> 32) atomicOr(status, 1);
      *carry_bits &= 0xffffffffull;
    }
    return;
  }
  const long long total = (long long)g.n[0] * g.n[1] * (long long)g.n[2];
  int bad = 0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x)
    signal_speed_f32<D>(M, U, Uf, g, t, bad);
  if (bad) atomicOr(status, 1);
}

// FP64 flux of the interface between cell o (index ga along AX) and cell
// o + s_AX, from U^n: face states of both cells (cells ga-1 .. ga+2, those
// beyond a face of bc type 1..4 from the interior, as the sweeps take them)
// and the exact Riemann problem at x/t = 0. bc: null where every ghost cell
// is in memory.
template <int D, int AX>
__device__ __noinline__ void redo_interface(const MixedParams& M, int limiter, double omega,
                                            const double* __restrict__ U, const Geom& g, int ga, long long o,
                                            const int* bc, const double (*inflow)[5], double hdtdx, double* f) {
  const long long F = g.field, sa = g.s[AX];
  const int N = g.n[AX];
  double w0[D + 2], w1[D + 2], w2[D + 2], w3[D + 2];
  auto cell = [&](int k, double* w) {  // cell ga + k
    const int i = ga + k;
    const int side = 2 * AX + (i < 1 ? 0 : 1);
    const int type = (bc && (i < 1 || i > N)) ? bc[side] : 0;
    const bool from = type >= 1 && type <= 4;
    const long long at = o + (long long)((from && type != 4 ? ghost_source(i, N, type) : i) - ga) * sa;
#pragma unroll
    for (int c = 0; c < D + 2; ++c) {
      w[c] = (type == 4) ? inflow[side][c] : U[(long long)c * F + at];
      if (type == 1 && c == 1 + AX) w[c] = -w[c];
    }
  };
  cell(-1, w0);
  cell(0, w1);
  cell(1, w2);
  cell(2, w3);
  // a non-finite U^n (a box the scheme has already lost) makes the FP64
  // solve iterate to its cap for a NaN result: give the NaN directly
  bool finite = true;
#pragma unroll
  for (int c = 0; c < D + 2; ++c) finite = finite && isfinite(w0[c]) && isfinite(w1[c]) && isfinite(w2[c]) && isfinite(w3[c]);
  if (!finite) {
#pragma unroll
    for (int c = 0; c < D + 2; ++c) f[c] = CUDART_NAN;
    return;
  }
  double lo[D + 2], ro[D + 2], l1[D + 2], r1[D + 2];
  face_states<D, AX>(M.G64, limiter, omega, w0, w1, w2, hdtdx, lo, ro);
  face_states<D, AX>(M.G64, limiter, omega, w1, w2, w3, hdtdx, l1, r1);
  interface_flux<D, AX>(M.G64, M.rp64, ro, l1, f);
}

template <int D>
__device__ __forceinline__ void redo_any_axis(const MixedParams& M, int limiter, double omega,
                                              const double* __restrict__ U, const Geom& g,
                                              const FallbackEntry& e, const int* bc, const double (*inflow)[5],
                                              double hdtdx, double* f) {
  const int axis = e.axis;
  if (axis == 0) redo_interface<D, 0>(M, limiter, omega, U, g, e.ga, e.o, bc, inflow, hdtdx, f);
  if constexpr (D > 1) {
    if (axis == 1) redo_interface<D, 1>(M, limiter, omega, U, g, e.ga, e.o, bc, inflow, hdtdx, f);
  }
  if constexpr (D > 2) {
    if (axis == 2) redo_interface<D, 2>(M, limiter, omega, U, g, e.ga, e.o, bc, inflow, hdtdx, f);
  }
}

// Boundary types and inflow values for the fix-up (types 0: from memory).
struct FixBC {
  int bc[6];
  double inflow[6][5];
};

// The fix-up kernels: one CTA per SM, few enough for an early launch (the
// queue is nearly always empty), of 8 warps, since a redo is a chain of
// dependent FP64 and integer instructions: a step of 512 boxes of 8..64^3
// took 3.37 ms with 4 warps, 3.30 with 8 or 16. A short queue is spread over
// the SMs, a warp of entries each.
constexpr int kFixGrid = 152, kFixBlock = 256;
__device__ __forceinline__ int fix_first() {
  return ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
}

// FP64 redo of the queued interfaces; -+ dt/dx * F applied to the adjacent
// interior cells of U^{n+1} (atomically: a cell can border two queued
// interfaces).
// Entries from *from (0 when from is null) to the queue's end: a solve in
// slabs fixes the entries of each slab after its sweeps.
template <int D>
__global__ void __launch_bounds__(kFixBlock)
    fallback_fix_kernel(MixedParams M, FallbackQueue q, Geom g, Dx dx, const double* __restrict__ dtp,
                        const double* __restrict__ U, double* __restrict__ Unew, const int* __restrict__ from,
                        const __grid_constant__ FixBC fbc) {
  step_begin();
  const int n = min(*q.n, q.cap);
  const int lo = from ? min(*from, n) : 0;
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > lo) atomicAdd(q.total, n - lo);
  const double dt = *dtp;
  const long long F = g.field;
  for (int i = lo + fix_first(); i < n; i += gridDim.x * kFixBlock) {
    const FallbackEntry e = q.e[i];
    double f[D + 2];
    redo_any_axis<D>(M, M.limiter, M.omega64, U, g, e, fbc.bc, fbc.inflow, 0.5 * dt / dx.v[e.axis], f);
    const double dtdx = dt / dx.v[e.axis];
    const long long sa = g.s[e.axis];
    const int NA = g.n[e.axis];
#pragma unroll
    for (int c = 0; c < D + 2; ++c) {
      const double corr = dtdx * f[c];
      if (e.ga >= 1) atomicAdd(&Unew[(long long)c * F + e.o], -corr);
      if (e.ga + 1 <= NA) atomicAdd(&Unew[(long long)c * F + e.o + sa], corr);
    }
  }
}

template <int D>
cudaError_t launch_fallback(const MixedParams& M, const FallbackQueue& q, const Geom& g, const Dx& dx,
                            const double* dtp, const double* U, double* Unew, cudaStream_t st,
                            const HaloBC& halo, const int* from = nullptr) {
  FixBC fbc;
  for (int i = 0; i < 6; ++i) {
    fbc.bc[i] = halo.type[i];
    for (int c = 0; c < 5; ++c) fbc.inflow[i][c] = halo.inflow64[i][c];
  }
  launch_step(fallback_fix_kernel<D>, kFixGrid, kFixBlock, st, M, q, g, dx, dtp, U, Unew, from, fbc);
  return cudaGetLastError();
}

// Batched FP32 CFL over work items (chunks of a box's cells), per box as
// cfl_carry_kernel: dt from the maximum that the box's last sweep folded,
// unless *whole is set (some box was not stepped by a batch last) or the FP64
// fix-up changed the box after that sweep (carry_ok cleared): then the pass
// over its cells, per-box maximum through atomics, the last item of a box
// forming its dt in FP64.
template <int D>
__global__ void __launch_bounds__(256)
    batch_cfl_f32_kernel(MixedParams M, double courant, const BoxDesc* __restrict__ TB,
                         const WorkItem* __restrict__ items, int n, const int* __restrict__ whole,
                         int* __restrict__ heads, int* __restrict__ queued) {
  if (blockIdx.x == 0) {  // for this step's queues
    if (threadIdx.x < kBatchHeads) heads[threadIdx.x] = 0;
    if (threadIdx.x == 0) *queued = 0;
  }
  __shared__ float sm[8];
  __shared__ int sb[8];
  const bool all = *whole != 0;
  for (int it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const BoxDesc& b = TB[w.box];
    // every thread sees the flag that the box's last item sets at its end as
    // it was before the pass (that item ends after this one's own count)
    const bool carried = !all && *(volatile int*)carry_ok_of(b) != 0;
    if (carried) {
      if (w.chunk == 0 && threadIdx.x == 0) {
        const unsigned long long folded = *carry_bits_of(b);
        const float mu = __uint_as_float((unsigned int)folded);
        if (folded >> 32) atomicOr((int*)(b.ctl + 2) + 1, 1);
        b.ctl[0] = courant * b.dx.min / (double)mu;
        *carry_bits_of(b) = 0ull;
      }
      continue;
    }
    const long long total = (long long)b.g.n[0] * b.g.n[1] * b.g.n[2];
    const long long t1 = min(total, (w.chunk + 1) * kBatchCflChunk);
    float m = 0.f;
    int bad = 0;
    for (long long t = w.chunk * kBatchCflChunk + threadIdx.x; t < t1; t += 256) {
      const float v = signal_speed_f32<D>(M, b.U, b.Uf, b.g, t, bad);
      if (v > m) m = v;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_down_sync(0xffffffffu, m, off);
      if (o > m) m = o;
      bad |= __shfl_down_sync(0xffffffffu, bad, off);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
      sm[warp] = m;
      sb[warp] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < 8; ++k) {
        if (sm[k] > m) m = sm[k];
        bad |= sb[k];
      }
      unsigned long long* max_bits = (unsigned long long*)(b.ctl + 1);
      unsigned int* counter = (unsigned int*)(b.ctl + 2);
      int* status = (int*)(b.ctl + 2) + 1;
      atomicMax(max_bits, (unsigned long long)__float_as_uint(m));
      if (bad) atomicOr(status, 1);
      __threadfence();
      if (atomicAdd(counter, 1u) == (unsigned int)(b.cfl_items - 1)) {
        __threadfence();
        const float mu = __uint_as_float((unsigned int)atomicAdd(max_bits, 0ull));
        b.ctl[0] = courant * b.dx.min / (double)mu;
        atomicExch(max_bits, 0ull);
        atomicExch(counter, 0u);
        *carry_bits_of(b) = 0ull;
        *(volatile int*)carry_ok_of(b) = 1;
      }
    }
    __syncthreads();
  }
}

// Batched FP64 fix-up: as fallback_fix_kernel, with the box of each entry.
template <int D>
__global__ void __launch_bounds__(kFixBlock)
    batch_fallback_fix_kernel(MixedParams M, FallbackQueue q, const BoxDesc* __restrict__ TB) {
  const int n = min(*q.n, q.cap);
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(q.total, n);
  for (int i = fix_first(); i < n; i += gridDim.x * kFixBlock) {
    const FallbackEntry e = q.e[i];
    const BoxDesc& b = TB[e.box];
    *carry_ok_of(b) = 0;  // the box's cells change after its last sweep: its next CFL pass is whole
    double f[D + 2];
    redo_any_axis<D>(M, b.limiter, b.omega, b.U, b.g, e, b.halo.type, b.inflow, 0.5 * b.ctl[0] / b.dx.v[e.axis], f);
    const double dtdx = b.ctl[0] / b.dx.v[e.axis];
    const long long sa = b.g.s[e.axis];
    const int NA = b.g.n[e.axis];
    const long long F = b.g.field;
#pragma unroll
    for (int c = 0; c < D + 2; ++c) {
      const double corr = dtdx * f[c];
      if (e.ga >= 1) atomicAdd(&b.V[(long long)c * F + e.o], -corr);
      if (e.ga + 1 <= NA) atomicAdd(&b.V[(long long)c * F + e.o + sa], corr);
    }
  }
}

template <int D>
cudaError_t launch_batch_fallback(const MixedParams& M, const BoxDesc* TB, const FallbackQueue& q,
                                  cudaStream_t st) {
  batch_fallback_fix_kernel<D><<<kFixGrid, kFixBlock, 0, st>>>(M, q, TB);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_to_f32(const double* U, float* Uf, long long n, cudaStream_t st) {
  to_f32_kernel<<<grid_for(n, kThreads), kThreads, 0, st>>>(U, Uf, n);
  return cudaGetLastError();
}

cudaError_t launch_cfl_mixed(const MixedParams& M, const double* U, float* Uf, const Geom& g, double courant,
                             const Dx& dx, const StepScratch& s, cudaStream_t st) {
  const long long total = (long long)g.n[0] * g.n[1] * g.n[2];
  int grid = grid_for(total, kThreads);
  if (grid > 152 * 4) grid = 152 * 4;
  switch (M.ndim) {
    case 1: cfl_f32_kernel<1><<<grid, kThreads, 0, st>>>(M, U, Uf, g, courant, dx.min, s); break;
    case 2: cfl_f32_kernel<2><<<grid, kThreads, 0, st>>>(M, U, Uf, g, courant, dx.min, s); break;
    case 3: cfl_f32_kernel<3><<<grid, kThreads, 0, st>>>(M, U, Uf, g, courant, dx.min, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_cfl_carry(const MixedParams& M, const double* U, float* Uf, const Geom& g, double courant,
                             const Dx& dx, const StepScratch& s, unsigned long long* carry_bits, int* carry_ok,
                             const int* prev_fix, int* this_fix, cudaStream_t st) {
  const long long total = (long long)g.n[0] * g.n[1] * g.n[2];
  int grid = grid_for(total, kThreads);
  if (grid > 152 * 4) grid = 152 * 4;
  switch (M.ndim) {
    case 1:
      launch_step(cfl_carry_kernel<1>, grid, kThreads, st, M, U, Uf, g, courant, dx.min, s, carry_bits, carry_ok, prev_fix, this_fix);
      break;
    case 2:
      launch_step(cfl_carry_kernel<2>, grid, kThreads, st, M, U, Uf, g, courant, dx.min, s, carry_bits, carry_ok, prev_fix, this_fix);
      break;
    case 3:
      launch_step(cfl_carry_kernel<3>, grid, kThreads, st, M, U, Uf, g, courant, dx.min, s, carry_bits, carry_ok, prev_fix, this_fix);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_carry_status(const MixedParams& M, const double* U, float* Uf, const Geom& g,
                                unsigned long long* carry_bits, const int* carry_ok, const int* prev_fix, int* status,
                                cudaStream_t st) {
  int grid = grid_for((long long)g.n[0] * g.n[1] * g.n[2], kThreads);
  if (grid > 152 * 4) grid = 152 * 4;
  switch (M.ndim) {
    case 1: carry_status_kernel<1><<<grid, kThreads, 0, st>>>(M, U, Uf, g, carry_bits, carry_ok, prev_fix, status); break;
    case 2: carry_status_kernel<2><<<grid, kThreads, 0, st>>>(M, U, Uf, g, carry_bits, carry_ok, prev_fix, status); break;
    case 3: carry_status_kernel<3><<<grid, kThreads, 0, st>>>(M, U, Uf, g, carry_bits, carry_ok, prev_fix, status); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_mh_solve_mixed(const MixedParams& M, const double* U, const float* Uf,
                                  double* Unew, float* acc, const Geom& g,
                                  const Dx& dx, const StepScratch& s, const FallbackQueue& q,
                                  const SweepPlan& plan, cudaStream_t st, const HaloBC& halo, cudaEvent_t* ev,
                                  const SweepCarry& carry, int* fused, bool queue_reset) {
  // ev (optional, 3 events): recorded after the x sweep, after the y sweep
  // and at the end (the z sweep and the FP64 fix-up); absent axes record
  // at the same point, and so do both when one kernel ran the x and y
  // sweeps (*fused, optional, is then 1).
  const int D = M.ndim;
  if (D < 1 || D > 3) return cudaErrorInvalidValue;
  cudaError_t e = queue_reset ? cudaMemsetAsync(q.n, 0, sizeof(int), st) : cudaSuccess;
  int first = 0;
  if (fused) *fused = 0;
  if (e == cudaSuccess && D == 3 && plan.fuse_xy) {
    // the x and y sweeps in one kernel where the mirror's rows allow the
    // plane's tensor copy (bit-identical to the two sweeps)
    e = launch_sweep_xy_3(M, Uf, g, dx, s.dt, acc, q, halo, st);
    if (e == cudaSuccess) {
      first = 2;
      if (fused) *fused = 1;
      if (ev) e = cudaEventRecord(ev[0], st);
      if (e == cudaSuccess && ev) e = cudaEventRecord(ev[1], st);
    } else if (e == cudaErrorNotSupported) {
      e = cudaSuccess;
    }
  }
  for (int a = first; a < D; ++a) {
    if (e == cudaSuccess)
      e = launch_sweep_axis(D, a, plan.shape[a], M, Uf, U, g, dx, s.dt, acc, Unew, q, st,
                            a == D - 1 ? carry : SweepCarry(), halo);
    if (e == cudaSuccess && ev && a < 2) e = cudaEventRecord(ev[a], st);
  }
  for (int a = D; a < 2; ++a)
    if (e == cudaSuccess && ev) e = cudaEventRecord(ev[a], st);
  if (e == cudaSuccess) {
    switch (D) {
      case 1: e = launch_fallback<1>(M, q, g, dx, s.dt, U, Unew, st, halo); break;
      case 2: e = launch_fallback<2>(M, q, g, dx, s.dt, U, Unew, st, halo); break;
      case 3: e = launch_fallback<3>(M, q, g, dx, s.dt, U, Unew, st, halo); break;
    }
  }
  if (e == cudaSuccess && ev) e = cudaEventRecord(ev[2], st);
  return e;
}

cudaError_t launch_mh_solve_mixed_slab(const MixedParams& M, const double* U, const float* Uf, double* Unew,
                                       float* acc, const Geom& g, const Dx& dx, const StepScratch& s,
                                       const FallbackQueue& q, int* done, const SweepPlan& plan, int lo, int hi,
                                       cudaStream_t st) {
  const int D = M.ndim;
  if (D < 1 || D > 3) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  for (int a = 0; a < D && e == cudaSuccess; ++a)
    e = launch_sweep_slab(D, a, plan.shape[a], M, Uf, U, g, dx, s.dt, acc, Unew, q, lo, hi, st, SweepCarry(), no_halo(),
                          true);
  if (e == cudaSuccess) {
    switch (D) {
      case 1: e = launch_fallback<1>(M, q, g, dx, s.dt, U, Unew, st, no_halo(), done); break;
      case 2: e = launch_fallback<2>(M, q, g, dx, s.dt, U, Unew, st, no_halo(), done); break;
      case 3: e = launch_fallback<3>(M, q, g, dx, s.dt, U, Unew, st, no_halo(), done); break;
    }
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(done, q.n, sizeof(int), cudaMemcpyDeviceToDevice, st);
  return e;
}

cudaError_t launch_ingest_mixed(const MixedParams& M, const double* H, double* U, double* V, float* Uf, float* Vf,
                                const Geom& g, long long e0, long long e1, unsigned long long* bits, int* status,
                                cudaStream_t st) {
  if (e1 <= e0) return cudaSuccess;
  if (e1 > 0xffffffffLL) return cudaErrorInvalidValue;
  int grid = grid_for(e1 - e0, kThreads);
  if (grid > 152 * 8) grid = 152 * 8;
  const unsigned a = (unsigned)e0, b = (unsigned)e1;
  switch (M.ndim) {
    case 1: ingest_kernel<1><<<grid, kThreads, 0, st>>>(M, H, U, V, Uf, Vf, g, a, b, bits, status); break;
    case 2: ingest_kernel<2><<<grid, kThreads, 0, st>>>(M, H, U, V, Uf, Vf, g, a, b, bits, status); break;
    case 3: ingest_kernel<3><<<grid, kThreads, 0, st>>>(M, H, U, V, Uf, Vf, g, a, b, bits, status); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_cfl_finish(const unsigned long long* bits, double courant, const Dx& dx, const StepScratch& s,
                              cudaStream_t st) {
  cfl_finish_kernel<<<1, 1, 0, st>>>(bits, courant, dx.min, s);
  return cudaGetLastError();
}

long long sweep_tile_count(int ndim, int axis, int shape, const int* n) {
  int S, P;
  sweep_shape(ndim, shape, &S, &P);
  const int bax = (ndim == 1) ? 1 : (axis == 0 ? 1 : 0);
  const int cax = (ndim == 3) ? 3 - axis - bax : 2;
  const long long nB = (bax < ndim) ? n[bax] : 1;
  const long long nC = (cax < ndim) ? n[cax] : 1;
  const long long nA = (n[axis] + S - 1) / S;
  return nA * ((nB + P - 1) / P) * nC;
}

cudaError_t launch_batch_cfl_mixed(const MixedParams& M, double courant, const BoxDesc* TB,
                                   const BatchLists& L, const FallbackQueue& q, cudaStream_t st) {
  if (!L.n_cfl) return cudaSuccess;
  const int grid = L.n_cfl < 152 * 8 ? L.n_cfl : 152 * 8;
  switch (M.ndim) {
    case 1: batch_cfl_f32_kernel<1><<<grid, 256, 0, st>>>(M, courant, TB, L.cfl, L.n_cfl, L.whole, L.heads, q.n); break;
    case 2: batch_cfl_f32_kernel<2><<<grid, 256, 0, st>>>(M, courant, TB, L.cfl, L.n_cfl, L.whole, L.heads, q.n); break;
    case 3: batch_cfl_f32_kernel<3><<<grid, 256, 0, st>>>(M, courant, TB, L.cfl, L.n_cfl, L.whole, L.heads, q.n); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// The mixed passes of one batch step after the CFL and ghost passes: the
// sweeps of every box, axis by axis (one launch per tile shape in use, each
// with its own queue head), then the FP64 fix-up of the queued interfaces.
cudaError_t launch_batch_sweeps(const MixedParams& M, const BoxDesc* TB, const BatchLists& L,
                                const FallbackQueue& q, cudaStream_t st) {
  const int D = M.ndim;
  if (D < 1 || D > 3) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  for (int a = 0; a < D; ++a)
    for (int k = 0; k < kSweepShapes; ++k)
      if (e == cudaSuccess && L.n_sweep[a][k]) {
        int* head = L.heads + kHeadSweep0 + kSweepShapes * a + k;
        e = (L.fuse_xy && a == 0)
                ? launch_batch_sweep_xy_3(k, M, TB, L.sweep[a][k], L.n_sweep[a][k], head, q, st)
                : launch_batch_sweep_axis(D, a, k, M, TB, L.sweep[a][k], L.n_sweep[a][k], head, q, st);
      }
  if (e == cudaSuccess) {
    switch (D) {
      case 1: e = launch_batch_fallback<1>(M, TB, q, st); break;
      case 2: e = launch_batch_fallback<2>(M, TB, q, st); break;
      case 3: e = launch_batch_fallback<3>(M, TB, q, st); break;
    }
  }
  return e;
}

// ---- tensor maps of the FP32 mirror (TMA staging of the sweeps) --------------
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

std::atomic<long long> g_tma_launches{0};

EncodeTiledFn encoder() {
  const char* env = getenv("RHYME_GPU_TMA");
  if (env && env[0] == '0') return nullptr;
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return (EncodeTiledFn) nullptr;
    }
    return (EncodeTiledFn)p;
  }();
  return fn;
}

}  // namespace

bool encode_mirror_map(CUtensorMap* out, const float* Uf, const Geom& g, int D, int A, int S, int P) {
  if (D < 2 || A < 0 || A >= D) return false;
  const EncodeTiledFn fn = encoder();
  if (!fn) return false;
  const long long X = g.s[1], Y = g.s[2] / g.s[1], Z = g.field / g.s[2];
  // rows (and so every stride) a multiple of 16 bytes; base 16-byte aligned
  if (X % 4 != 0 || ((uintptr_t)Uf % 16) != 0) return false;
  cuuint64_t dim[4] = {(cuuint64_t)X, (cuuint64_t)Y, (cuuint64_t)Z, (cuuint64_t)(D + 2)};
  cuuint64_t stride[3] = {(cuuint64_t)X * 4, (cuuint64_t)(X * Y) * 4, (cuuint64_t)g.field * 4};
  // the slab: S+4 cells along A; along x P pencils (A = y, z: P+4 cells from
  // an aligned start); one cell along the third axis
  cuuint32_t box[4] = {1, 1, 1, (cuuint32_t)(D + 2)};
  box[A] = (cuuint32_t)(S + 4);
  if (A == 0) {
    box[1] = (cuuint32_t)P;
  } else {
    box[0] = (cuuint32_t)(P + 4);
  }
  for (int i = 0; i < 4; ++i)
    if (box[i] > 256 || box[i] > dim[i]) return false;
  if ((box[0] * 4) % 16 != 0) return false;
  cuuint32_t estride[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void*)Uf, dim, stride, box, estride,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return false;
  g_tma_launches.fetch_add(1, std::memory_order_relaxed);
  return true;
}

bool encode_xy_map(CUtensorMap* out, const float* Uf, const Geom& g, int TX, int TY) {
  const EncodeTiledFn fn = encoder();
  if (!fn) return false;
  const long long X = g.s[1], Y = g.s[2] / g.s[1], Z = g.field / g.s[2];
  if (X % 4 != 0 || ((uintptr_t)Uf % 16) != 0) return false;
  cuuint64_t dim[4] = {(cuuint64_t)X, (cuuint64_t)Y, (cuuint64_t)Z, 5};
  cuuint64_t stride[3] = {(cuuint64_t)X * 4, (cuuint64_t)(X * Y) * 4, (cuuint64_t)g.field * 4};
  // one z plane of the tile with its 2-cell halo along x and y, every component
  cuuint32_t box[4] = {(cuuint32_t)(TX + 4), (cuuint32_t)(TY + 4), 1, 5};
  for (int i = 0; i < 4; ++i)
    if (box[i] > 256 || box[i] > dim[i]) return false;
  if ((box[0] * 4) % 16 != 0) return false;
  cuuint32_t estride[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void*)Uf, dim, stride, box, estride,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return false;
  g_tma_launches.fetch_add(1, std::memory_order_relaxed);
  return true;
}

}  // namespace rgpu

extern "C" int rhyme_gpu_tma_launches(long long* n) {
  if (!n) return RHYME_GPU_EINVAL;
  *n = rgpu::g_tma_launches.load(std::memory_order_relaxed);
  return RHYME_GPU_OK;
}

namespace rgpu {

}  // namespace rgpu
