// Argument block of the cell-pair map kernel and the launch interface shared by the host code
// (clm_pairs.cu) and the translation units that instantiate the kernel (clm_pairs_f32.cu,
// clm_pairs_f64.cu, clm_pairs_batch.cu).
#pragma once
#include <cuda_runtime.h>

#include "clm_device.cuh"
#include "clm_geometry.hpp"
#include "clm_internal.hpp"

namespace clm {
namespace pk {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
// Sizes of the pair kernel.  A stage holds at most kStage candidates in shared memory as planes of
// coordinates and codes (kPad words of each plane per 32 candidates: 4 more than the candidates, so that the
// lane groups of small chunks read different banks); kQueue hits fit the queue of a neighbour-list sweep (32
// tests of every lane never give more); a warp's histogram bins hold at most kHistPairs pairs before they move
// into the block's FP64 bins.
constexpr int kStage = 256;
constexpr int kPad = 36;
constexpr int kPlane = kStage / 32 * kPad;
constexpr int kQueue = 1024;
constexpr int kHistPairs = 1024;
// blocks per SM of the round-based adjoint: Float32 handles, the split form of Float64 handles
constexpr int kAdjBlocks32 = 6, kAdjBlocks64 = 3;

template <class T> struct SetView {
  const T* px;
  const T* py;
  const T* pz;
  const float4* off;  // FP32 offsets from the cell origin; .w = particle code
  const float4* xq;   // Float32 handles: coordinates; .w = particle code
  const int* code;
  const int* cell_start;
  const int* cell_real;  // per cell: 1 when it holds a real particle
};

template <class T> struct PairArgs {
  DevGeom<T> g;
  SetView<T> X, Y;
  const int* real_list;
  const int* n_real_dev;  // number of cells with real particles (device)
  int self;
  int split;
  int op;
  int* err;
  // operator parameters
  double p[4];
  float pf[4];  // the same in FP32 (set by set_params)
  double ljd[5];  // LJ: sigma^2, eps c12, eps c6, 12 eps c12, 6 eps c6 (p = eps, sigma, c12, c6)
  float ljf[5];
  int ntypes;
  const int* tx;
  const int* ty;
  const double* eps_t;
  const double* sig_t;
  const float* eps_tf;  // the same tables in FP32 (pair values of the FP32 forms)
  const float* sig_tf;
  const T* vx;
  const T* vy;
  const T* bins;
  int nbins;
  const float* vxf;  // velocities in FP32 (pair values of the FP32 forms)
  const float* vyf;
  const double* wx;   // per-particle weights (WEIGHTED_INV_D) of x and y, and FP32 copies
  const double* wy;
  const float* wxf;
  const float* wyf;
  // outputs
  int* nl_i;
  int* nl_j;
  T* nl_d;
  unsigned long long* nl_count;
  long long nl_cap;
  // force sums in the rotated frame, added with atomics (f[i] -= df, f[j] += df for each visited pair):
  // FP32 pair values into one 16-byte record per particle, FP64 pair values into n * dim doubles
  float4* f4x;
  float4* f4y;      // cross: set y
  double* fx;
  double* fy;       // cross: set y
  double* part_e;   // per-block energy
  unsigned long long* part_c;  // per-block count
  T* part_min_d2;
  int* part_min_ij;
  unsigned long long* part_hc;  // nbins per block
  double* part_hs;              // nbins per block
  double* part_v;               // kAdjVals per block (adjoint)
  // work decomposition and batches of independent systems
  int cell_split;               // parts of a cell's particles: part p takes the chunks p, p + S, p + 2S, ... of 32
  int stage_split;              // parts of its candidates: part p takes the stages p, p + S, p + 2S, ...
  int part_step;                // turn of a cell's parts per wave of items (part_of)
  int stage;                    // candidates per stage, at most kStage (a multiple of 32)
  float hist_err;               // RHIST, Float64 exact: absolute error of the FP32 distance of cell offsets
  const DevGeom<T>* gtab;       // batch: geometry of each system
  const int* cell_sys;          // batch: system of each global cell
  const int* cbase;             // batch: first global cell of each system
  double first_edge;            // RHIST: bins[0], for the host
  float thr_tiny;               // FP32 d2 from which on the Float64 d2 is a normal number (set_params)
};

// Operator parameters in both precisions, and the line below which a pair's root may not be taken from its estimate:
// coordinates whose exact d2 is subnormal (below 2^-1022) are within 2^-960 of each other and of zero in every dimension
// that they differ in, so their FP32 distance is rounding only, some 2^-20 of a cell side; the line is far above that.
template <class T> inline void set_params(PairArgs<T>& A, const double* p) {
  for (int k = 0; k < 4; k++) {
    A.p[k] = p[k];
    A.pf[k] = (float)p[k];
  }
  auto lj = [](auto* o, const auto* q) {
    o[0] = q[1] * q[1];
    o[1] = q[0] * q[2];
    o[2] = q[0] * q[3];
    o[3] = 12 * o[1];
    o[4] = 6 * o[2];
  };
  A.thr_tiny = (float)((double)A.g.cutoff_sqr * 0x1p-30);
  lj(A.ljd, A.p);
  lj(A.ljf, A.pf);
}

enum OpKind { OPK_NL = 0, OPK_SCALAR = 1, OPK_FORCES = 2, OPK_MIN = 3, OPK_HIST = 4, OPK_ADJ = 5 };
// Maps of the round-based kernel (clm_pairs_rounds.cuh): FP32 sums (Float32 handles, the split form) that are
// given out in FP64, whose last digits depend on the order of the additions: the adjoint, histograms, forces of
// Float64 handles and the sums of batches.  k_pairs takes all other maps.
constexpr bool in_rounds(int opk, bool f64, bool split, bool batch) {
  return (!f64 || split) && (opk == OPK_ADJ || opk == OPK_HIST || (opk == OPK_FORCES && (f64 || batch)) ||
                             (opk == OPK_SCALAR && batch));
}
constexpr int kAdjVals = 13;  // energy, virial (xx yy zz xy xz yz), dU/deps[3], dU/dsigma[3]

// Dynamic shared memory of the radial-histogram kernel: block bins (FP64 sums, 64-bit counts), the bin
// edges in the handle dtype and in FP32, and per-warp bins (sums in the accumulation type, counts).
struct HistSmem {
  size_t hs, hc, bins, binf, ws, wc, total;
};
__host__ __device__ inline HistSmem hist_smem(int nb, int tsize, int fsize) {
  auto up = [](size_t v) { return (v + 15) / 16 * 16; };
  HistSmem m;
  m.hs = 0;
  m.hc = up(m.hs + 8 * (size_t)nb);
  m.bins = up(m.hc + 8 * (size_t)nb);
  m.binf = up(m.bins + (size_t)tsize * (nb + 1));
  m.ws = up(m.binf + 4 * (size_t)(nb + 1));
  m.wc = up(m.ws + (size_t)fsize * kWarps * nb);
  m.total = up(m.wc + 4 * (size_t)kWarps * nb);
  return m;
}

// Which instantiation of the kernel a launch needs.
struct LaunchSel {
  int dim;     // 2 or 3
  int opk;     // OpKind
  bool self;   // one set (self pairs) or two (cross pairs)
  bool split;  // FP32-split arithmetic
  bool batch;  // many independent systems in one launch (self pairs only)
};

// Launch on `st` with at most `grid` blocks (one resident wave); `grid` returns the blocks used.
cudaError_t launch_pairs_plain(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<float>& A);
cudaError_t launch_pairs_plain(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<double>& A);
cudaError_t launch_pairs_batch(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<float>& A);
cudaError_t launch_pairs_batch(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<double>& A);
// Resident blocks per SM of that instantiation (0 if none).
int pairs_blocks_per_sm(const LaunchSel& s, const PairArgs<float>* tag);
int pairs_blocks_per_sm(const LaunchSel& s, const PairArgs<double>* tag);

template <class T> inline SetView<T> view_of(const SetData& S) {
  SetView<T> v;
  v.px = S.px.as<T>();
  v.py = S.py.as<T>();
  v.pz = S.pz.as<T>();
  v.off = S.off.as<float4>();
  v.xq = S.xq.as<float4>();
  v.code = S.code.as<int>();
  v.cell_start = S.cell_start.as<int>();
  v.cell_real = S.cell_flags.as<int>();
  return v;
}

inline int opkind_of(int op) {
  switch (op) {
    case 1: return OPK_NL;
    case 2: case 3: case 4: case 5: case 6: case 8: return OPK_SCALAR;
    case 7: case 9: case 12: case 14: return OPK_FORCES;
    case 13: return OPK_ADJ;
    case 10: return OPK_MIN;
    case 11: return OPK_HIST;
    default: return -1;
  }
}

template <class T> inline cudaError_t launch_pairs(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<T>& A) {
  return s.batch ? launch_pairs_batch(s, grid, st, A) : launch_pairs_plain(s, grid, st, A);
}

}  // namespace pk
}  // namespace clm
