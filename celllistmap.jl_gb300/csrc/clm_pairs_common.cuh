// What the pair map kernels share: pair-value arithmetic, operator parameters, group sums, force sums.
//
// Replaces _pairwise! and its inner loops:
//   self  src/internals/self.jl:106-184      cross src/internals/cross.jl:81-129
//   vicinal cells with projection culling    src/internals/vicinal_cells.jl:4-75,
//                                            src/internals/auxiliary_functions.jl:66-111
//   non-periodic inner loops                 src/internals/NonPeriodicCells.jl:281-352
// and the per-batch output copies + reduce_output! with on-chip reductions.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "clm_pairs_args.hpp"

namespace clm {
namespace pk {

template <class T> __device__ __forceinline__ T pos_of(const SetView<T>& S, int d, int t) {
  return d == 0 ? S.px[t] : (d == 1 ? S.py[t] : S.pz[t]);
}

// Reciprocal and reciprocal square root for pair VALUES (energies, forces), which are checked against
// tolerances, never used for pair membership or neighbour-list distances.
//  FP32: hardware approximations (rcp.approx / rsqrt.approx, a couple of ulp).
//  FP64: the hardware FP64 estimate y (rcp / rsqrt.approx.ftz.f64: the upper word's value, relative error
//        2^-20) refined by the second-order terms of a series in its residual e, which cubes the error to far
//        below FP64 rounding:
//        1/x = y / (1 - e) = y (1 + e + e^2 + ...) with e = 1 - x y;
//        1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3e^2/8 + ...) with e = 1 - x y^2.
//        Three and five FP64 instructions: GB300's FP64 pipe takes 16 cycles per warp instruction and bounds the
//        FP64 pair kernels.  rsqrt.approx.f64 without .ftz is a sequence of its own: refined, it took 11 FP64
//        slots and was within 1.7e-16 of 1/sqrt(x); this takes 5.7 and is within 1.2e-16 (3e9 values).  It takes
//        subnormal x for zero: pairs that close (1.5e-154) are evaluated apart (vrsqrt_tiny), as a test of x here costs
//        the exact histograms 1 % as a call, 8 % in line and 15 % as a predicated instruction.
__device__ __forceinline__ float vrcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float vrsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double vrcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  e = fma(e, e, e);  // e + e^2
  return fma(y, e, y);
}
__device__ __forceinline__ double vrsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  const double p = fma(0.375, e, 0.5);  // 1/2 + 3e/8
  return fma(y * e, p, y);
}
// For subnormal x, scaled by 2^108 (exactly).
__device__ __forceinline__ double vrsqrt_tiny(double x) { return 0x1p54 * rsqrt(x * 0x1p108); }
template <bool TINY, class V> __device__ __forceinline__ V vroot(V x) {
  if constexpr (TINY) return (V)vrsqrt_tiny((double)x);
  else return vrsqrt(x);
}

// a <= b and a < b for non-negative values (squared distances, the cutoff, +inf), decided on the bit
// patterns, which are ordered like the values for non-negative IEEE numbers: for FP64 an integer compare,
// which leaves the FP64 pipe (one warp instruction per 16 cycles on GB300) to arithmetic.
template <class T> __device__ __forceinline__ bool nonneg_le(T a, T b) {
  if constexpr (std::is_same<T, double>::value) return __double_as_longlong(a) <= __double_as_longlong(b);
  else return a <= b;
}
template <class T> __device__ __forceinline__ bool nonneg_lt(T a, T b) {
  if constexpr (std::is_same<T, double>::value) return __double_as_longlong(a) < __double_as_longlong(b);
  else return a < b;
}

// Operator parameter k and the LJ type tables in the precision of the pair value (no conversions per pair).
template <class V, class T> __device__ __forceinline__ V par(const PairArgs<T>& A, int k) {
  if constexpr (std::is_same<V, float>::value) return A.pf[k];
  else return (V)A.p[k];
}
// Lennard-Jones products of one eps and sigma: sigma^2, eps c12, eps c6, 12 eps c12, 6 eps c6.
template <class V, class T> __device__ __forceinline__ V ljc(const PairArgs<T>& A, int k) {
  if constexpr (std::is_same<V, float>::value) return A.ljf[k];
  else return (V)A.ljd[k];
}
template <class V, class T> __device__ __forceinline__ V eps_tab(const PairArgs<T>& A, int k) {
  if constexpr (std::is_same<V, float>::value) return A.eps_tf[k];
  else return (V)A.eps_t[k];
}
template <class V, class T> __device__ __forceinline__ V sig_tab(const PairArgs<T>& A, int k) {
  if constexpr (std::is_same<V, float>::value) return A.sig_tf[k];
  else return (V)A.sig_t[k];
}
// Per-particle weight of particle k of set x (or y when ys).
template <class V, class T> __device__ __forceinline__ V weight(const PairArgs<T>& A, bool ys, int k) {
  if constexpr (std::is_same<V, float>::value) return (ys ? A.wyf : A.wxf)[k];
  else return (V)(ys ? A.wy : A.wx)[k];
}

// Sum of `v` over the lanes of a match group (`peers`: the lanes sharing this lane's key), returned in
// the group's lowest lane.  Pairwise tree: at each step every lane at an even position of its group adds
// the value of the next remaining peer, and the lanes at odd positions drop out, so a group of g lanes
// needs ceil(log2 g) steps and the whole warp at most 5, however many groups there are.  All lanes of
// the warp call it.
template <class V> __device__ __forceinline__ V group_sum(unsigned peers, V v, int lane) {
  unsigned pos = __popc(peers & ((1u << lane) - 1u));  // position of this lane in its group
  unsigned rest = peers & ~((2u << lane) - 1u);         // peers above this lane (lane 31: none)
  if (lane == 31) rest = 0u;
  while (__any_sync(0xffffffffu, rest != 0u)) {
    const int nxt = __ffs(rest);                          // 1 + lane of the next remaining peer, 0 if none
    const V t = __shfl_sync(0xffffffffu, v, nxt > 0 ? nxt - 1 : lane);
    if (nxt > 0) v += t;
    const unsigned gone = __ballot_sync(0xffffffffu, (pos & 1u) != 0u);  // consumed by their left neighbour
    rest &= ~gone;
    pos >>= 1;
  }
  return v;
}

// Geometry of the cell being processed: the launch's own (one system) or that of the cell's system
// (batches); `cb` returns the first global cell of that system.
template <bool B, class T>
__device__ __forceinline__ const DevGeom<T>& geo_of(const PairArgs<T>& A, int li, int& cb) {
  if constexpr (B) {
    const int s = A.cell_sys[li];
    cb = A.cbase[s];
    return A.gtab[s];
  } else {
    cb = 0;
    return A.g;
  }
}

// Adds a force term to the sums of particle `idx` (set y when `ys`): one 16-byte vector atomic for FP32
// pair values, one FP64 atomic per component otherwise.
template <class T, int N, class FA>
__device__ __forceinline__ void force_add(const PairArgs<T>& A, bool ys, int idx, const FA* v) {
  if constexpr (std::is_same<FA, float>::value) {
    atomicAdd((ys ? A.f4y : A.f4x) + idx, make_float4(v[0], v[1], (N == 3) ? v[2] : 0.f, 0.f));
  } else {
    double* f = (ys ? A.fy : A.fx) + (int64_t)idx * N;
#pragma unroll
    for (int d = 0; d < N; d++) atomicAdd(f + d, (double)v[d]);
  }
}

// The part of its cell that work item r is, the cell being the rcell-th of S parts each.  The parts of a cell differ in
// size (the first stages hold the cell itself, the last are short), and a warp takes every nw-th item: in plain order a
// warp whose nw is a multiple of S would take the same part of every cell.  So the parts of a cell are turned by `step`
// (A.part_step, such that nw + step and S have no common factor) for each wave of items before it.  The neighbour list
// of 100k Float64 points at cutoff 8 (8 parts per cell, 3040 warps): map 690 -> 625 us.
__device__ __forceinline__ int part_of(int r, int rcell, int S, int nw, int step) {
  const int first = rcell * S;
  unsigned p = (unsigned)(r - first);
  if (step) p = (p + (unsigned)(first / nw) * (unsigned)step) % (unsigned)S;
  return (int)p;
}

// The reference's d2, with its separately rounded operations.
template <class T, int N> __device__ __forceinline__ T exact_d2(const T* dx) {
  T d2 = xmul(dx[0], dx[0]);
#pragma unroll
  for (int d = 1; d < N; d++) d2 = xadd(d2, xmul(dx[d], dx[d]));
  return d2;
}

// The exact test of a pair whose FP32 distance is near the cutoff: d2 <= cutoff^2, and the reference's
// projection filter above proj_lo, seen from the cell of the reference's i (the candidate's cell is `me` away;
// `same`: the particle's own cell, where the filter does not apply; swapped: the candidate is the
// reference's i).  A call: a few pairs in ten thousand come here, and its registers stay out of the sweep.
template <class T, int N>
__device__ __noinline__ bool near_cutoff(const DevGeom<T>& g, T cutoff_sqr, int3 ci, int me, bool same, bool swapped, T x0,
                                         T x1, T x2, T y0, T y1, T y2) {
  const T xi[3] = {x0, x1, x2}, xj[3] = {y0, y1, y2};
  T dx[3];
#pragma unroll
  for (int d = 0; d < N; d++) dx[d] = xsub(xi[d], xj[d]);
  const T d2 = exact_d2<T, N>(dx);
  if (!nonneg_le(d2, cutoff_sqr)) return false;
  if (!nonneg_lt(g.proj_lo, d2) || same) return true;
  const int ca[3] = {ci.x, ci.y, ci.z};
  const int cj[3] = {ci.x + (me & 255) - 128, ci.y + ((me >> 8) & 255) - 128,
                     (N == 3) ? ci.z + ((me >> 16) & 255) - 128 : 1};
  T ctr_i[3], ctr_j[3];
  cell_center<T, N>(g, ca, ctr_i);
  cell_center<T, N>(g, cj, ctr_j);
  return swapped ? projection_pass<T, N>(g, ctr_j, ctr_i, xj, xi) : projection_pass<T, N>(g, ctr_i, ctr_j, xi, xj);
}

}  // namespace pk
}  // namespace clm
