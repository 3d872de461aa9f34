// Cell-pair map kernel (self and cross pairs, operator epilogues), included by the translation units
// that instantiate it.
//
// Replaces _pairwise! and its inner loops:
//   self  src/internals/self.jl:106-184      cross src/internals/cross.jl:81-129
//   vicinal cells with projection culling    src/internals/vicinal_cells.jl:4-75,
//                                            src/internals/auxiliary_functions.jl:66-111
//   non-periodic inner loops                 src/internals/NonPeriodicCells.jl:281-352
// and the per-batch output copies + reduce_output! with on-chip reductions.
#pragma once
#include "clm_pairs_common.cuh"
#include "clm_pairs_rounds.cuh"

namespace clm {
namespace pk {

// What the adjoint needs of a Lennard-Jones pair besides its energy and force: (sigma/d)^6, the pair's
// parameters and its type class (2 types: AA = 0, AB = 1, BB = 2).
template <class V> struct LJTerm {
  V sr6 = 0, eps = 0, sig = 0;
  int cls = 0;
  template <class W> __device__ __forceinline__ void from(const LJTerm<W>& o) {
    sr6 = (V)o.sr6;
    eps = (V)o.eps;
    sig = (V)o.sig;
    cls = o.cls;
  }
};

// Per-pair energy u and g = (du/dr)/r (force contribution df = g*(x_i - x_j)).
// OPC 9: LJ forces with one eps and sigma, whose products come from the host.
// TINY: d2 is subnormal.
template <class V, int OPC, bool TINY = false, class T>
__device__ __forceinline__ void pair_value(const PairArgs<T>& A, int op, V d2, int i, int j, V& u, V& g, LJTerm<V>& lj) {
  if constexpr (OPC == 9) {
    const V r2i = vrcp(d2);
    const V sr2 = ljc<V>(A, 0) * r2i;
    const V sr6 = sr2 * sr2 * sr2;
    u = sr6 * (ljc<V>(A, 1) * sr6 - ljc<V>(A, 2));
    g = (sr6 * r2i) * (ljc<V>(A, 4) - ljc<V>(A, 3) * sr6);
    return;
  }
  switch (op) {
    case 2:  // COUNT
      u = V(1);
      g = V(0);
      break;
    case 3:  // SUM_D2
      u = d2;
      g = V(0);
      break;
    case 4:  // SUM_D
      u = d2 * vroot<TINY>(d2);
      g = V(0);
      break;
    case 5:  // SUM_INV_D
      u = vroot<TINY>(d2);
      g = V(0);
      break;
    case 6:
    case 7: {  // SOFT (c - d)^2
      V ri = vroot<TINY>(d2);
      V d = d2 * ri;
      V c = par<V>(A, 0);
      u = (c - d) * (c - d);
      g = V(-2) * (c - d) * ri;
      break;
    }
    case 8:
    case 9:
    case 13: {  // LJ eps*(c12 (s/d)^12 - c6 (s/d)^6), with s6 = (s/d)^6 taken out: s6 (eps c12 s6 - eps c6)
      V eps = par<V>(A, 0), sig = par<V>(A, 1);
      if (A.ntypes > 0) {
        int ti = A.tx[i];
        int tj = A.self ? A.tx[j] : A.ty[j];
        eps = eps_tab<V>(A, ti * A.ntypes + tj);
        sig = sig_tab<V>(A, ti * A.ntypes + tj);
        lj.cls = ti + tj;
      }
      const V e12 = eps * par<V>(A, 2), e6 = eps * par<V>(A, 3);
      const V r2i = vrcp(d2);
      const V sr2 = (sig * sig) * r2i;
      const V sr6 = sr2 * sr2 * sr2;
      u = sr6 * (e12 * sr6 - e6);
      g = (sr6 * r2i) * (V(6) * e6 - (V(12) * e12) * sr6);
      lj.sr6 = sr6;
      lj.eps = eps;
      lj.sig = sig;
      break;
    }
    case 14: {  // weighted 1/d: u = -c w_i w_j / d, g = (c w_i w_j / d^2) / d
      const V cw = par<V>(A, 0) * weight<V>(A, false, i) * weight<V>(A, A.self == 0, j);
      const V ri = vroot<TINY>(d2);
      u = -(cw * ri);
      g = cw * (ri * ri * ri);
      break;
    }
    case 12: {  // 1/d with gradient accumulation
      V ri = vroot<TINY>(d2);
      u = ri;
      g = ri * ri * ri;
      break;
    }
    default:
      u = V(0);
      g = V(0);
  }
}

// Resident blocks per SM the kernel is compiled for.  Float64 lists and histograms take 128 registers (100k points: list
// map 563 us, 620 at five blocks; histogram 47.1 ms, 48.1), Float64 forces do not gain by it (371 us, 379 at four).
template <class T, int OPK, bool SPLIT> constexpr int min_blocks() {
  if (sizeof(T) == 4) return 7;
  return !SPLIT && (OPK == OPK_NL || OPK == OPK_HIST) ? 4 : 5;
}

// Shared memory of one warp.
template <class T, bool EXACT64, bool FP64, bool NL> struct WarpSmem {
  float p[4][kPlane];              // the staged candidates: x, y, z and codes
  float4 i4[32];                   // particles of the chunk: prefilter coordinates, code in .w
  unsigned mask[kStage / 32][32];  // hits: word w of each lane's tests
  int pref[33];                    // stream position of the first copy of each stencil entry
  int delta[32];                   // its position in the cell list minus that
  int meta[32];                    // its cell's offset
  int tj[EXACT64 ? kPlane : 1];    // position of the candidate in the cell list
  T ix[3][FP64 ? 32 : 1];          // Float64 handles: the particles' coordinates
  unsigned short q[NL ? kQueue : 2];  // neighbour lists: (particle slot << 9) | plane index

  // the last stencil entry whose prefix is <= stream position e (that entry is not empty)
  __device__ __forceinline__ int entry_of(int e) const {
    int lo = 0;
#pragma unroll
    for (int st = 16; st > 0; st >>= 1)
      if (pref[lo + st] <= e) lo += st;
    return lo;
  }
};

// Pair map kernel.  CROSS: x-y pairs; otherwise self pairs.  Every pair is visited once, from the side
// the reference visits it (forward half stencil, or the full stencil with index_i < index_j for
// triclinic cells); forces add -df to the particle's sums and +df to the partner's.
//
// Each warp takes one work item: a cell, or a part of it (some of its chunks of 32 particles against some of
// the stages of its candidates; the host picks the parts so that every resident warp has work).  The cells of
// the stencil are concatenated into one candidate stream, read in stages of at most 256 candidates: every lane
// finds the cells of its stream positions, loads their 16-byte records (coordinates or cell offsets, the
// particle code in .w) and writes planes of x, y, z and codes to shared memory (offsets shifted by the cell
// displacement on the way).  Triclinic self pairs visit each pair of cells once (the forward half stencil, and
// the backward cells without real particles: sym_stencil_offset), as orthorhombic self pairs do.
//   Tests: every lane tests its particle against runs of 32 staged candidates with an FP32 distance (FMA, two
// candidates per instruction) and records those inside cutoff^2 (1 + 2^-13) in a bit mask; chunks of at most
// 16, 8 or 4 particles split the warp into 2, 4 or 8 lane groups that take different runs.
//   Sweep: the hits of a stage (all set bits of its masks, in the order particle, run, candidate) are shared out
// evenly: each lane finds its first hit by the prefix sums of the lanes' counts and then walks the masks, so
// every lane is busy whatever the particles' shares are.  A sweep applies the reference's pair rules where an
// image copy takes part, the exact test in the input dtype within 2^-13 of the cutoff, and the operator's
// epilogue.  The projection filter of the reference is evaluated only for pairs with d2 > cutoff^2 (1 - 2^-13):
// any pair further inside passes it (the projection of the separation on a unit vector cannot exceed the
// separation, and the margin covers the half cell), so skipping it elsewhere leaves the pair set unchanged.
// Neighbour lists copy the hits into a queue first, for one reservation and dense writes per sweep.
// OPC: the operator id when fixed at compile time, 0 = read from the arguments (9 only without types, 11 only with a first
// edge above the distances of subnormal squares).
template <class T, int N, int OPK, bool SPLIT, bool CROSS, bool BATCH, int OPC = 0>
__global__ void __launch_bounds__(kThreads, min_blocks<T, OPK, SPLIT>()) k_pairs(const __grid_constant__ PairArgs<T> A) {
  static_assert(!in_rounds(OPK, std::is_same<T, double>::value, SPLIT, BATCH), "a map of k_pairs_rounds");
  static_assert((OPK != OPK_HIST && OPK != OPK_ADJ) || (std::is_same<T, double>::value && !SPLIT), "FP64 sums");
  using V = T;
  using FA = typename std::conditional<std::is_same<T, double>::value && !SPLIT, double, float>::type;
  constexpr bool IS_F = (OPK == OPK_FORCES) || (OPK == OPK_ADJ);
  constexpr bool FP64 = std::is_same<T, double>::value;
  constexpr bool EXACT64 = FP64 && !SPLIT;  // pair values in FP64 from the coordinates themselves
  constexpr bool ABS_PF = !FP64;            // Float32 handles test the coordinates themselves
  // the operator may take the root of an FP64 d2: pairs too close for it (thr_tiny) are decided one by one
  constexpr bool ROOT = EXACT64 && ((OPK == OPK_SCALAR && OPC != 8) || (OPK == OPK_FORCES && OPC != 9) ||
                                    (OPK == OPK_HIST && OPC != 11));
  const DevGeom<T>& g = A.g;
  const int op = OPC ? OPC : A.op;
  using Smem = WarpSmem<T, EXACT64, FP64, OPK == OPK_NL>;
  __shared__ __align__(16) unsigned char s_warps[kWarps * sizeof(Smem)];
  // kept in registers (the compiler would recompute them from the thread index at every shared-memory access)
  int lane, at;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  const int warp = threadIdx.x >> 5;
  asm volatile("mul.lo.s32 %0, %1, %2;" : "=r"(at) : "r"(warp), "n"((int)sizeof(Smem)));
  Smem& W = *reinterpret_cast<Smem*>(s_warps + at);
  const unsigned FULL = 0xffffffffu;

  // radial histogram (dynamic shared memory, layout in hist_smem): block bins in FP64, bin edges, and
  // per-warp bins that the warp updates without atomics
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const HistSmem hl = hist_smem((OPK == OPK_HIST) ? A.nbins : 0, (int)sizeof(T), (int)sizeof(FA));
  double* s_hs = reinterpret_cast<double*>(s_dyn + hl.hs);
  unsigned long long* s_hc = reinterpret_cast<unsigned long long*>(s_dyn + hl.hc);
  T* s_bins = reinterpret_cast<T*>(s_dyn + hl.bins);
  float* s_binf = reinterpret_cast<float*>(s_dyn + hl.binf);
  FA* s_ws = reinterpret_cast<FA*>(s_dyn + hl.ws) + warp * A.nbins;
  unsigned* s_wc = reinterpret_cast<unsigned*>(s_dyn + hl.wc) + warp * A.nbins;
  __shared__ double s_red[kWarps];
  __shared__ unsigned long long s_redc[kWarps];

  const bool tri = (g.kind == TRICLINIC);
  const bool nonper = (g.kind == NONPERIODIC);
  const bool sym = tri && !CROSS;  // triclinic self pairs: each pair of cells once (sym_stencil_offset)
  const int sym_mask = sym ? -1 : 0;
  const int l = g.lcell;
  const int w = 2 * l + 1;
  const int wN = (N == 3) ? w * w * w : w * w;
  const int nf = (wN - 1) / 2;
  // entry 0 is the cell itself; then all neighbours (cross pairs), the forward and the backward half
  // (triclinic self pairs) or the forward half
  const int nent = CROSS ? wN : (sym ? 2 * nf + 1 : nf + 1);
  // offset of stencil entry kk, three biased bytes; kBack: in the backward half
  constexpr int kBack = 1 << 24;
  auto entry_meta = [&](int kk) {
    int o[3] = {0, 0, 0};
    bool back = false;
    if (kk > 0 && kk < nent) {
      if (CROSS) stencil_offset(false, l, N, kk - 1, o);
      else sym_stencil_offset(l, N, nf, kk - 1, o, &back);
    }
    return ((o[0] + 128) | ((o[1] + 128) << 8) | ((o[2] + 128) << 16)) | (back ? kBack : 0);
  };
  int meta = entry_meta(lane);  // lane k holds entry k0 + k; computed again only when there are more than 32

  if constexpr (OPK == OPK_HIST) {
    for (int b = threadIdx.x; b < A.nbins; b += kThreads) {
      s_hc[b] = 0ull;
      s_hs[b] = 0.0;
    }
    for (int b = lane; b < A.nbins; b += 32) {
      s_ws[b] = FA(0);
      s_wc[b] = 0u;
    }
    for (int b = threadIdx.x; b <= A.nbins; b += kThreads) {
      s_bins[b] = A.bins[b];
      s_binf[b] = (float)A.bins[b];
    }
    __syncthreads();
  }

  double e_tot = 0.0;  // per-lane energy (FP64); FP32 partial sums are folded in per particle chunk
  FA e_part = 0;
  FA adj[kAdjVals - 1];  // adjoint accumulators: virial (6), dU/deps (3), dU/dsigma (3)
#pragma unroll
  for (int k = 0; k < kAdjVals - 1; k++) adj[k] = FA(0);
  unsigned long long c_acc = 0;
  T best_d2 = INFINITY;
  int best_i = 0x7fffffff, best_j = 0x7fffffff;

  const int gw = blockIdx.x * kWarps + warp;
  const int nw = gridDim.x * kWarps;
  // a build that flagged an overflow left cells without copies: nothing is mapped, and the build is repeated
  const int n_real = (*A.err & kBuildFailed) ? 0 : *A.n_real_dev;
  const int SI = A.cell_split, SJ = A.stage_split;  // the host keeps cells x parts below 2^31
  const int S = SI * SJ;
  const int n_items = n_real * S;
  for (int r = gw; r < n_items; r += nw) {
    int rcell = r, part_i = 0, part_j = 0;
    if (S > 1) {
      rcell = r / S;
      part_i = part_of(r, rcell, S, nw, A.part_step);
      part_j = part_i / SI;
      part_i -= part_j * SI;
    }
    const int li = A.real_list[rcell];
    int cb = 0;  // first global cell of the system (batches)
    const DevGeom<T>& gc = geo_of<BATCH>(A, li, cb);
    int ci[3];
    cart_of_fast<N>(gc, li - cb, ci);
    const int si = A.X.cell_start[li];
    const int ni = A.X.cell_start[li + 1] - si;

    for (int ib = part_i * 32; ib < ni; ib += 32 * SI) {
      // chunk of m particles: GS = log2 of the lane groups; the lanes of one particle are adjacent, so that the
      // hits are ordered by particle
      const int m = min(32, ni - ib);
      const int GS = (m <= 4) ? 3 : (m <= 8) ? 2 : (m <= 16) ? 1 : 0;
      const int grp = lane & ((1 << GS) - 1);
      const int il = lane >> GS;
      const int ii = ib + il;
      const bool vi = ii < ni;
      float4 i4 = make_float4(0.f, 0.f, 0.f, 0.f);  // the lane's particle: prefilter coordinates and code
      if (vi) {
        i4 = (ABS_PF ? A.X.xq : A.X.off)[si + ii];
        if (!ABS_PF && grp == 0) {
#pragma unroll
          for (int d = 0; d < N; d++) W.ix[d][il] = pos_of(A.X, d, si + ii);
        }
      }
      if (grp == 0) W.i4[il] = i4;
      const int code_l = __float_as_int(i4.w);
      const bool act_i = (tri && CROSS) ? (vi && code_l >= 0) : vi;
      int stage_no = 0;  // counts the item's stages over all stencil tables: part_j takes every SJ-th

      for (int k0 = 0; k0 < nent; k0 += 32) {
        // ---- stencil table for entries k0 .. k0+31: lane k holds entry k0 + k
        if (nent > 32) meta = entry_meta(k0 + lane);
        int same_end, total;
        {
          int e_start = 0, e_cnt = 0;
          if (k0 + lane < nent) {
            int lj = 0;
            bool inr = true;
#pragma unroll
            for (int d = N - 1; d >= 0; d--) {
              const int c = ci[d] - 1 + ((meta >> (8 * d)) & 255) - 128;  // 0-based
              inr = inr && (unsigned)c < (unsigned)gc.nc[d];
              lj = lj * gc.nc[d] + c;
            }
            if (!inr) {
              atomicOr(A.err, DERR_CELL_RANGE);
            } else {
              lj += cb;
              // a backward cell holding real particles is an item of its own, which visits this pair of cells
              if (!(meta & kBack) || !A.Y.cell_real[lj]) {
                e_start = A.Y.cell_start[lj];
                e_cnt = A.Y.cell_start[lj + 1] - e_start;
              }
            }
          }
          int incl = e_cnt;
#pragma unroll
          for (int o2 = 1; o2 < 32; o2 <<= 1) {
            int y = __shfl_up_sync(FULL, incl, o2);
            if (lane >= o2) incl += y;
          }
          W.pref[lane + 1] = incl;
          if (lane == 0) W.pref[0] = 0;
          W.delta[lane] = e_start - (incl - e_cnt);
          W.meta[lane] = meta;
          total = __shfl_sync(FULL, incl, 31);
          same_end = (k0 == 0) ? __shfl_sync(FULL, incl, 0) : 0;  // stream positions of the cell itself
        }
        __syncwarp();

        // stages of equal size (rounded up to whole runs of 32)
        int sz = total;
        if (total > A.stage) {
          const int nst = (total + A.stage - 1) / A.stage;
          sz = ((total + nst - 1) / nst + 31) & ~31;
        }
        for (int w0 = 0; w0 < total; w0 += sz) {
          const int wc = min(sz, total - w0);
          if (SJ > 1) {
            const bool mine = (stage_no % SJ) == part_j;
            stage_no++;
            if (!mine) continue;
          }
          // ---- stage: records to planes, four loads of a lane in flight.  Plain loads: one bulk copy per
          // stencil cell (cp.async.bulk takes its operands from uniform registers, so a warp issues its 14
          // copies one by one) cost about 300 of the item's 3300 warp instructions against 150
          {
            const float4* rec = ABS_PF ? A.Y.xq : A.Y.off;
            constexpr int LB = 4;  // loads in flight per lane
#pragma unroll 1
            for (int kb = 0; 32 * kb < wc; kb += LB) {
              float4 rv[LB];
#pragma unroll
              for (int k = 0; k < LB; k++) {
                if (32 * (kb + k) < wc) {
                  const int e = w0 + min(32 * (kb + k) + lane, wc - 1);
                  const int lo = W.entry_of(e);
                  const int t = W.delta[lo] + e;
                  rv[k] = rec[t];
                  if constexpr (!ABS_PF) {
                    // shift the offsets by the cell displacement so that x_i - x_j ~ off_i - plane
                    const int me = W.meta[lo];
                    rv[k].x += gc.csf[0] * (float)((me & 255) - 128);
                    rv[k].y += gc.csf[1] * (float)(((me >> 8) & 255) - 128);
                    if (N == 3) rv[k].z += gc.csf[2] * (float)(((me >> 16) & 255) - 128);
                    if constexpr (EXACT64) W.tj[(kb + k) * kPad + lane] = t;
                  }
                }
              }
#pragma unroll
              for (int k = 0; k < LB; k++) {
                if (32 * (kb + k) < wc) {
                  const int p = (kb + k) * kPad + lane;
                  W.p[0][p] = rv[k].x;
                  W.p[1][p] = rv[k].y;
                  if (N == 3) W.p[2][p] = rv[k].z;
                  W.p[3][p] = rv[k].w;
                }
              }
            }
          }
          __syncwarp();

          // ---- tests: word k of a lane holds stream positions w0 + 32 ((k << GS) + grp) ..., candidate b on bit b.
          // thr carries a 2^-13 relative margin, far above the FP32 rounding of dx^2 - thr + dy^2 + dz^2, so the
          // strict comparison keeps every pair the exact test can accept.
          const int nwords = (wc + (32 << GS) - 1) >> (5 + GS);
          int hits = 0;
          for (int k = 0; k < nwords; k++) {
            const int run = (k << GS) + grp;
            unsigned mask = 0u;
            {
              const float nthr = -g.thr_hi;
              const float2 tx = make_float2(-i4.x, -i4.x), ty = make_float2(-i4.y, -i4.y);
              const float2 tz = make_float2(-i4.z, -i4.z), tt = make_float2(nthr, nthr);
              // runs past the stage's end read the last run again (their bits are dropped below)
              const int pb = min(run, (wc - 1) >> 5) * kPad;
              const float* bx = &W.p[0][pb];
#pragma unroll
              for (int b = 28; b >= 0; b -= 4) {
                const float4 X = *reinterpret_cast<const float4*>(bx + b);
                const float4 Y = *reinterpret_cast<const float4*>(bx + kPlane + b);
                float2 d = __fadd2_rn(make_float2(X.z, X.w), tx);
                float2 eh = __ffma2_rn(d, d, tt);
                d = __fadd2_rn(make_float2(X.x, X.y), tx);
                float2 el = __ffma2_rn(d, d, tt);
                d = __fadd2_rn(make_float2(Y.z, Y.w), ty);
                eh = __ffma2_rn(d, d, eh);
                d = __fadd2_rn(make_float2(Y.x, Y.y), ty);
                el = __ffma2_rn(d, d, el);
                if constexpr (N == 3) {
                  const float4 Z = *reinterpret_cast<const float4*>(bx + 2 * kPlane + b);
                  d = __fadd2_rn(make_float2(Z.z, Z.w), tz);
                  eh = __ffma2_rn(d, d, eh);
                  d = __fadd2_rn(make_float2(Z.x, Z.y), tz);
                  el = __ffma2_rn(d, d, el);
                }
                // (mask << 1) | sign bit of d2 - thr
                mask = __funnelshift_l(__float_as_uint(eh.y), mask, 1);
                mask = __funnelshift_l(__float_as_uint(eh.x), mask, 1);
                mask = __funnelshift_l(__float_as_uint(el.y), mask, 1);
                mask = __funnelshift_l(__float_as_uint(el.x), mask, 1);
              }
            }
            // Dropped: positions past the stage's end, and in the cell itself the pairs the reference does not
            // visit from this copy: the earlier slots for self pairs (each pair of the cell once), every slot for
            // an image copy in cross pairs of orthorhombic cells (the particle copy must be real there).  What
            // remains of the pair rules is in the sweep (pairs of images, and of an image and a real copy).
            const int nb = wc - 32 * run;
            if (!act_i || nb <= 0) mask = 0u;
            else if (nb < 32) mask &= (1u << nb) - 1u;
            if (w0 + 32 * (k << GS) < same_end) {  // the warp's runs of this word reach into the cell itself
              const int base = w0 + 32 * run;
              int lim = -1;  // last dropped position of the cell itself
              if (!CROSS) lim = min(ii, same_end - 1);
              else if (!tri && !nonper && code_l < 0) lim = same_end - 1;
              if (lim >= base) {
                const int nr = lim - base + 1;
                mask &= (nr >= 32) ? 0u : ~((1u << nr) - 1u);
              }
            }
            W.mask[k][lane] = mask;
            hits += __popc(mask);
          }

          // ---- what a sweep needs of one pair
          struct Pair {
            int code_i, code_j;
            float d2f, dvf[3];  // the FP32 distance (Float32 handles near the cutoff: the reference's d2)
            bool sure;          // the FP32 distance decided
            T xi[3], xj[3], dxs[3];  // coordinates and x_i - x_j (EXACT64, or Float64 handles near the cutoff)
          };
          auto idx_of = [](int code) { return code ^ (code >> 31); };  // code >= 0 ? code : ~code
          auto load_x = [&](int jp, int ie, Pair& q) {
            if constexpr (FP64) {
              int t;
              if constexpr (EXACT64) {
                t = W.tj[jp];
              } else {
                const int e = w0 + jp - ((jp / kPad) << 2);
                t = W.delta[W.entry_of(e)] + e;
              }
#pragma unroll
              for (int d = 0; d < N; d++) {
                q.xi[d] = W.ix[d][ie];
                q.xj[d] = pos_of(A.Y, d, t);
                q.dxs[d] = xsub(q.xi[d], q.xj[d]);
              }
            }
          };
          // d2 of a kept pair in FP64 for values (fused; the decision is made): EXACT64, or Float64 handles near the
          // cutoff
          auto value_d2 = [&](const Pair& q) {
            T d2 = q.dxs[0] * q.dxs[0];
#pragma unroll
            for (int d = 1; d < N; d++) d2 = fma(q.dxs[d], q.dxs[d], d2);
            return d2;
          };
          // A kept pair whose d2 is subnormal, evaluated by itself.
          auto is_tiny = [](T d2) { return d2 > T(0) && d2 < T(0x1p-1022); };
          auto tiny_pair = [&](const Pair& q) {
            const int idx_i = idx_of(q.code_i), idx_j = idx_of(q.code_j);
            const bool sw = sym && idx_j < idx_i;
            if constexpr (OPK == OPK_HIST) {
              const int b = first_edge_at_or_above(s_bins, A.nbins, xsqrt(exact_d2<T, N>(q.dxs))) - 1;
              if (b < 0 || b >= A.nbins) return;
              const T* vy = CROSS ? A.vy : A.vx;
              FA dot = 0;
#pragma unroll
              for (int a = 0; a < N; a++) {
                FA x = q.dxs[a];
                if (tri) {
                  x = 0;
#pragma unroll
                  for (int k = 0; k < N; k++) x += (FA)gc.Rinv[a][k] * q.dxs[k];
                }
                dot += (A.vx[(int64_t)idx_i * N + a] - vy[(int64_t)idx_j * N + a]) * x;
              }
              atomicAdd(&s_hc[b], 1ull);
              atomicAdd(&s_hs[b], (double)(dot * vroot<true>(value_d2(q))));
            } else {
              V u, gg;
              LJTerm<V> lv;
              pair_value<V, OPC, true>(A, op, value_d2(q), sw ? idx_j : idx_i, sw ? idx_i : idx_j, u, gg, lv);
              if (op == 2) c_acc++;
              else e_part += (FA)u;
              if constexpr (OPK == OPK_FORCES) {
                FA df[3] = {0, 0, 0}, nf[3] = {0, 0, 0};
#pragma unroll
                for (int d = 0; d < N; d++) {
                  df[d] = (FA)(gg * q.dxs[d]);
                  nf[d] = -df[d];
                }
                force_add<T, N, FA>(A, false, idx_i, nf);
                force_add<T, N, FA>(A, CROSS, idx_j, df);
              }
            }
          };
          // Whether the reference keeps the pair.  The rest of the pair rules on the codes (image: negative code
          // ~index): pairs of two images are dropped; in triclinic self pairs of a real copy and an image, the copy of
          // the lower index is the reference's i and must be real, so with r the real copy's index and m the
          // image's it is kept when r < m, that is code_i + code_j + 1 = r - m < 0.
          auto keep_pair = [&](int jp, int ie, const float4& p4, Pair& q) {
            q.code_i = __float_as_int(p4.w);
            q.code_j = __float_as_int(W.p[3][jp]);
            q.dvf[0] = p4.x - W.p[0][jp];
            q.dvf[1] = p4.y - W.p[1][jp];
            q.dvf[2] = (N == 3) ? p4.z - W.p[2][jp] : 0.f;
            q.d2f = fmaf(q.dvf[2], q.dvf[2], fmaf(q.dvf[1], q.dvf[1], q.dvf[0] * q.dvf[0]));
            if constexpr (EXACT64) load_x(jp, ie, q);
            const int drop = (q.code_i & q.code_j) | ((q.code_i ^ q.code_j) & ~(q.code_i + q.code_j + 1) & sym_mask);
            q.sure = q.d2f <= g.thr_lo && (!ROOT || q.d2f >= A.thr_tiny);
            if (drop < 0 || !q.sure) {
              if (drop < 0) return false;
              const int e = w0 + jp - ((jp / kPad) << 2);
              const int lo = W.entry_of(e);
              const bool sw = sym && idx_of(q.code_j) < idx_of(q.code_i);
              const int3 c3 = make_int3(ci[0], ci[1], ci[2]);
              if constexpr (FP64) {
                if constexpr (!EXACT64) load_x(jp, ie, q);
                const bool in = near_cutoff<T, N>(gc, g.cutoff_sqr, c3, W.meta[lo], e < same_end, sw, q.xi[0], q.xi[1],
                                                  (N == 3) ? q.xi[2] : T(0), q.xj[0], q.xj[1], (N == 3) ? q.xj[2] : T(0));
                if constexpr (ROOT) {
                  if (in && is_tiny(value_d2(q))) {
                    tiny_pair(q);
                    return false;
                  }
                }
                return in;
              } else {
                q.d2f = exact_d2<float, N>(q.dvf);
                return near_cutoff<T, N>(gc, g.cutoff_sqr, c3, W.meta[lo], e < same_end, sw, p4.x, p4.y, p4.z,
                                         W.p[0][jp], W.p[1][jp], (N == 3) ? W.p[2][jp] : 0.f);
              }
            }
            return true;
          };
          // values in FP64: always (EXACT64), never (Float32 handles), or near the cutoff (split form)
          auto in_fp64 = [&](const Pair& q) { return EXACT64 || (FP64 && !q.sure); };

          const int H = __reduce_add_sync(FULL, hits);
          if constexpr (OPK == OPK_NL) {
            // ---- queue: all words of the stage at once, or as many as fit
            const bool whole = H <= kQueue;
            int hq = hits, Hq = H;
            for (int k0w = 0, k1w; k0w < nwords; k0w = k1w) {
              k1w = nwords;
              if (!whole) {
                hq = 0;
                Hq = 0;
                for (k1w = k0w; k1w < nwords; k1w++) {
                  const int c = __popc(W.mask[k1w][lane]);
                  const int hw = __reduce_add_sync(FULL, c);
                  if (Hq + hw > kQueue) break;
                  Hq += hw;
                  hq += c;
                }
              }
              {
                int incl = hq;
#pragma unroll
                for (int o2 = 1; o2 < 32; o2 <<= 1) {
                  int y = __shfl_up_sync(FULL, incl, o2);
                  if (lane >= o2) incl += y;
                }
                unsigned short* qp = &W.q[incl - hq];
                for (int k = k0w; k < k1w; k++) {
                  unsigned mm = W.mask[k][lane];
                  const int ent0 = (il << 9) + ((k << GS) + grp) * kPad;
                  while (mm) {
                    const int b = 31 - __clz(mm);
                    mm ^= 1u << b;
                    *qp++ = (unsigned short)(ent0 + b);
                  }
                }
              }
              __syncwarp();
              // The queue is first reduced to the pairs the reference keeps (in place: an entry moves to an
              // earlier or its own slot), so that one atomic per sweep
              // reserves their places in the list: an atomic on one address takes 0.67 ns on GB300 wherever it
              // comes from, and one per 32 entries took half of the list's time (674 us for 1.07e7 Float64 pairs)
              int kept = 0;
              for (int t0 = 0; t0 < Hq; t0 += 32) {
                const int t = t0 + lane;
                bool keep = t < Hq;
                int ent = 0;
                if (keep) {
                  ent = W.q[t];
                  Pair q;
                  keep = keep_pair(ent & 511, ent >> 9, W.i4[ent >> 9], q);
                }
                const unsigned bal = __ballot_sync(FULL, keep);
                __syncwarp();  // every lane has read its entry (a ballot orders no memory)
                if (keep) W.q[kept + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)ent;
                kept += __popc(bal);
                __syncwarp();
              }
              if constexpr (BATCH) c_acc += (lane == 0) ? (unsigned long long)kept : 0ull;  // pairs per system
              unsigned long long first = 0;
              if (lane == 0 && kept) first = atomicAdd(A.nl_count, (unsigned long long)kept);
              first = __shfl_sync(FULL, first, 0);
              for (int t = lane; t < kept; t += 32) {
                const int ent = W.q[t];
                const int jp = ent & 511, ie = ent >> 9;
                const float4 p4 = W.i4[ie];
                const int idx_i = idx_of(__float_as_int(p4.w)), idx_j = idx_of(__float_as_int(W.p[3][jp]));
                const bool sw = sym && idx_j < idx_i;
                T dval;
                const float dvf[3] = {p4.x - W.p[0][jp], p4.y - W.p[1][jp], (N == 3) ? p4.z - W.p[2][jp] : 0.f};
                const float d2f = fmaf(dvf[2], dvf[2], fmaf(dvf[1], dvf[1], dvf[0] * dvf[0]));
                if constexpr (!FP64) {
                  dval = xsqrt(exact_d2<float, N>(dvf));
                } else if (SPLIT && d2f <= g.thr_lo) {
                  dval = (T)sqrtf(d2f);
                } else {
                  Pair q;
                  load_x(jp, ie, q);
                  dval = xsqrt(exact_d2<T, N>(q.dxs));
                }
                const unsigned long long pos = first + t;
                if ((long long)pos < A.nl_cap) {
                  A.nl_i[pos] = sw ? idx_j : idx_i;
                  A.nl_j[pos] = sw ? idx_i : idx_j;
                  A.nl_d[pos] = dval;
                }
              }
              __syncwarp();
            }
          } else {
            // ---- sweep: lane t takes the hits t per .. t per + per - 1
            __syncwarp();  // the masks of all lanes are written (reductions and shuffles order no memory)
            const int per = (H + 31) >> 5;
            const int first = lane * per;
            int left = min(per, H - first);  // this lane's hits (<= 0: none)
            int own, wd = 0;                 // the test lane and word the next hit is in
            unsigned bits = 0u;              // that word's hits not taken yet
            {
              int incl = hits;
#pragma unroll
              for (int o2 = 1; o2 < 32; o2 <<= 1) {
                int y = __shfl_up_sync(FULL, incl, o2);
                if (lane >= o2) incl += y;
              }
              const int excl = incl - hits;
              own = 0;  // the last lane whose prefix is <= first: it has hits when first < H
#pragma unroll
              for (int st = 16; st > 0; st >>= 1) {
                const int v = __shfl_sync(FULL, excl, own + st);
                if (v <= first) own += st;
              }
              int skip = first - __shfl_sync(FULL, excl, own);
              if (left > 0) {
                bits = W.mask[0][own];
                for (int c; skip >= (c = __popc(bits));) {
                  skip -= c;
                  bits = W.mask[++wd][own];
                }
                for (; skip > 0; skip--) bits ^= 0x80000000u >> __clz(bits);
              }
            }
            int ie = own >> GS;  // the particle slot of the next hit
            float4 p4 = W.i4[ie];
            int jb = ((wd << GS) + (own & ((1 << GS) - 1))) * kPad;  // plane index of the word's bit 0
            FA acc[3] = {0, 0, 0};  // IS_F: the particle's share of the hits taken so far
            // the next hit's plane index; moves to the next word (and particle) with hits when this one is done
            auto next_hit = [&]() {
              if (bits == 0u) {
                do {
                  if (++wd == nwords) {
                    wd = 0;
                    own++;
                  }
                  bits = W.mask[wd][own];
                } while (bits == 0u);
                jb = ((wd << GS) + (own & ((1 << GS) - 1))) * kPad;
                if ((own >> GS) != ie) {
                  if constexpr (IS_F) {
                    force_add<T, N, FA>(A, false, idx_of(__float_as_int(p4.w)), acc);
#pragma unroll
                    for (int d = 0; d < N; d++) acc[d] = FA(0);
                  }
                  ie = own >> GS;
                  p4 = W.i4[ie];
                }
              }
              const int b = 31 - __clz(bits);
              bits ^= 1u << b;
              return jb + b;
            };

            if constexpr (IS_F) {
              const bool any = left > 0;
              for (; left > 0; left--) {
                Pair q;
                const int jp = next_hit();
                if (keep_pair(jp, ie, p4, q)) {
                  const int idx_i = idx_of(q.code_i), idx_j = idx_of(q.code_j);
                  const bool sw = sym && idx_j < idx_i;
                  const int oi = sw ? idx_j : idx_i, oj = sw ? idx_i : idx_j;
                  FA uu, gg;
                  FA dv[3] = {0, 0, 0}, df[3] = {0, 0, 0};
                  LJTerm<FA> lj;
                  if (in_fp64(q)) {
                    V uv, gv;
                    LJTerm<V> lv;
                    pair_value<V, OPC>(A, op, value_d2(q), oi, oj, uv, gv, lv);
                    uu = (FA)uv;
                    gg = (FA)gv;
                    lj.from(lv);
#pragma unroll
                    for (int d = 0; d < N; d++) dv[d] = (FA)q.dxs[d];
                  } else {
                    float uf, gf;
                    LJTerm<float> lv;
                    pair_value<float, OPC>(A, op, q.d2f, oi, oj, uf, gf, lv);
                    uu = (FA)uf;
                    gg = (FA)gf;
                    lj.from(lv);
#pragma unroll
                    for (int d = 0; d < N; d++) dv[d] = (FA)q.dvf[d];
                  }
#pragma unroll
                  for (int d = 0; d < N; d++) df[d] = gg * dv[d];
                  if constexpr (OPK == OPK_ADJ) {
                    // virial W += g dx dx^T (g = u'(r)/r), and the parameter derivatives of the LJ term
                    adj[0] += df[0] * dv[0];
                    adj[1] += df[1] * dv[1];
                    adj[2] += df[2] * dv[2];
                    adj[3] += df[0] * dv[1];
                    adj[4] += df[0] * dv[2];
                    adj[5] += df[1] * dv[2];
                    const FA c12 = par<FA>(A, 2), c6 = par<FA>(A, 3);
                    const FA ue = lj.sr6 * (c12 * lj.sr6 - c6);  // u / eps
                    const FA dsg = lj.eps * lj.sr6 * (FA(12) * c12 * lj.sr6 - FA(6) * c6) * vrcp(lj.sig);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                      adj[6 + k] += (lj.cls == k) ? ue : FA(0);
                      adj[9 + k] += (lj.cls == k) ? dsg : FA(0);
                    }
                  }
#pragma unroll
                  for (int d = 0; d < N; d++) acc[d] -= df[d];
                  e_part += uu;
                  force_add<T, N, FA>(A, CROSS, idx_j, df);  // the partner's share
                }
              }
              if (any) force_add<T, N, FA>(A, false, idx_of(__float_as_int(p4.w)), acc);
            } else if constexpr (OPK == OPK_SCALAR) {
              for (; left > 0; left--) {
                Pair q;
                const int jp = next_hit();
                if (keep_pair(jp, ie, p4, q)) {
                  const int idx_i = idx_of(q.code_i), idx_j = idx_of(q.code_j);
                  const bool sw = sym && idx_j < idx_i;
                  const int oi = sw ? idx_j : idx_i, oj = sw ? idx_i : idx_j;
                  if (op == 2) {
                    c_acc++;
                  } else if (in_fp64(q)) {
                    V uu, gg;
                    LJTerm<V> lv;
                    pair_value<V, OPC>(A, op, value_d2(q), oi, oj, uu, gg, lv);
                    e_part += (FA)uu;
                  } else {
                    float uu, gg;
                    LJTerm<float> lv;
                    pair_value<float, OPC>(A, op, q.d2f, oi, oj, uu, gg, lv);
                    e_part += (FA)uu;
                  }
                }
              }
            } else if constexpr (OPK == OPK_MIN) {
              for (; left > 0; left--) {
                Pair q;
                const int jp = next_hit();
                if (keep_pair(jp, ie, p4, q)) {
                  const int idx_i = idx_of(q.code_i), idx_j = idx_of(q.code_j);
                  const bool sw = sym && idx_j < idx_i;
                  const int oi = sw ? idx_j : idx_i, oj = sw ? idx_i : idx_j;
                  T dd2;
                  if constexpr (!FP64) dd2 = exact_d2<float, N>(q.dvf);
                  else dd2 = in_fp64(q) ? exact_d2<T, N>(q.dxs) : (T)q.d2f;
                  if (nonneg_lt(dd2, best_d2) ||
                      (!nonneg_lt(best_d2, dd2) && (oi < best_i || (oi == best_i && oj < best_j)))) {
                    best_d2 = dd2;
                    best_i = oi;
                    best_j = oj;
                  }
                }
              }
            } else if constexpr (OPK == OPK_HIST) {
              int room = kHistPairs / 32;  // sweeps before the warp's bins move on
              for (int t = 0; t < per; t++) {
                int hb = -1;   // bin of this lane's pair (-1: none)
                FA hv = 0;     // its accumulator term
                if (t < left) {
                  Pair q;
                  const int jp = next_hit();
                  if (keep_pair(jp, ie, p4, q)) {
                    const int idx_i = idx_of(q.code_i), idx_j = idx_of(q.code_j);
                    // the bin from the FP32 distance, decided again from the IEEE distance of the reference's d2 when
                    // an edge lies within 2^-12 and the error of the FP32 distance of cell offsets of it
                    bool exact_r = !q.sure;
                    int b = -1;
                    if (q.sure) {
                      const float rf = sqrtf(q.d2f);
                      const int lo = first_edge_at_or_above(s_binf, A.nbins, rf);
                      b = lo - 1;
                      exact_r = near_edge(s_binf, A.nbins, lo, rf, A.hist_err);
                    }
                    if (exact_r) b = first_edge_at_or_above(s_bins, A.nbins, xsqrt(exact_d2<T, N>(q.dxs))) - 1;
                    if (b >= 0 && b < A.nbins) {
                      FA dv[3] = {0, 0, 0};
#pragma unroll
                      for (int d = 0; d < N; d++) dv[d] = q.dxs[d];
                      if (tri) {
                        FA rv[3];
#pragma unroll
                        for (int a = 0; a < N; a++) {
                          FA s = 0;
#pragma unroll
                          for (int k = 0; k < N; k++) s += (FA)gc.Rinv[a][k] * dv[k];
                          rv[a] = s;
                        }
#pragma unroll
                        for (int a = 0; a < N; a++) dv[a] = rv[a];
                      }
                      FA dot = 0;
                      const T* vy = CROSS ? A.vy : A.vx;
#pragma unroll
                      for (int d = 0; d < N; d++)
                        dot += (A.vx[(int64_t)idx_i * N + d] - vy[(int64_t)idx_j * N + d]) * dv[d];
                      hv = dot * vrsqrt(value_d2(q));
                      hb = b;
                    }
                  }
                }
                // lanes holding the same bin are summed by a tree over their group; the group's first lane
                // then updates the warp's own bin (groups have distinct bins: no atomics)
                if (__any_sync(FULL, hb >= 0)) {
                  const unsigned peers = __match_any_sync(FULL, hb);
                  const FA v = group_sum(peers, hv, lane);
                  if (hb >= 0 && lane == __ffs(peers) - 1) {
                    s_ws[hb] += v;
                    s_wc[hb] += (unsigned)__popc(peers);
                  }
                  __syncwarp();
                }
                if (--room == 0 || t == per - 1) {
                  // move the warp's bins (at most kHistPairs pairs) into the block's FP64 bins
                  room = kHistPairs / 32;
                  for (int b = lane; b < A.nbins; b += 32) {
                    const unsigned c = s_wc[b];
                    if (c) {
                      atomicAdd(&s_hc[b], (unsigned long long)c);
                      atomicAdd(&s_hs[b], (double)s_ws[b]);
                      s_wc[b] = 0u;
                      s_ws[b] = FA(0);
                    }
                  }
                  __syncwarp();
                }
              }
            }
          }
          __syncwarp();  // the next stage overwrites the planes and masks
        }
        __syncwarp();  // the next table overwrites this one
      }
      e_tot += (double)e_part;
      e_part = 0;
      __syncwarp();  // the next chunk's particles overwrite s_i4
    }
    if constexpr (BATCH) {
      // per work item partials, reduced per system in a fixed order afterwards
      double e = e_tot;
      unsigned long long c = c_acc;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        e += __shfl_xor_sync(FULL, e, s);
        c += __shfl_xor_sync(FULL, c, s);
      }
      if (lane == 0) {
        A.part_e[r] = e;
        A.part_c[r] = c;
      }
      e_tot = 0.0;
      c_acc = 0;
    }
  }
  if constexpr (BATCH) return;

  // ---------------- block reductions to per-block partials
  if constexpr (OPK == OPK_SCALAR || OPK == OPK_FORCES) {
    double e = e_tot;
    unsigned long long c = c_acc;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      e += __shfl_xor_sync(FULL, e, s);
      c += __shfl_xor_sync(FULL, c, s);
    }
    if (lane == 0) {
      s_red[warp] = e;
      s_redc[warp] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double es = 0;
      unsigned long long cs = 0;
      for (int k = 0; k < kWarps; k++) {
        es += s_red[k];
        cs += s_redc[k];
      }
      A.part_e[blockIdx.x] = es;
      A.part_c[blockIdx.x] = cs;
    }
  } else if constexpr (OPK == OPK_ADJ) {
    __shared__ double s_adj[kWarps][kAdjVals];
    double v[kAdjVals];
    v[0] = e_tot;
#pragma unroll
    for (int k = 1; k < kAdjVals; k++) v[k] = (double)adj[k - 1];
#pragma unroll
    for (int k = 0; k < kAdjVals; k++) {
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v[k] += __shfl_xor_sync(FULL, v[k], s);
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < kAdjVals; k++) s_adj[warp][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < kAdjVals) {
      double acc = 0;
      for (int w = 0; w < kWarps; w++) acc += s_adj[w][threadIdx.x];
      A.part_v[(int64_t)blockIdx.x * kAdjVals + threadIdx.x] = acc;
    }
  } else if constexpr (OPK == OPK_MIN) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      T od = __shfl_xor_sync(FULL, best_d2, s);
      int oi_ = __shfl_xor_sync(FULL, best_i, s);
      int oj_ = __shfl_xor_sync(FULL, best_j, s);
      if (od < best_d2 || (od == best_d2 && (oi_ < best_i || (oi_ == best_i && oj_ < best_j)))) {
        best_d2 = od;
        best_i = oi_;
        best_j = oj_;
      }
    }
    __shared__ T s_md[kWarps];
    __shared__ int s_mi[kWarps], s_mj[kWarps];
    if (lane == 0) {
      s_md[warp] = best_d2;
      s_mi[warp] = best_i;
      s_mj[warp] = best_j;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      T bd = s_md[0];
      int bi = s_mi[0], bj = s_mj[0];
      for (int k = 1; k < kWarps; k++) {
        if (s_md[k] < bd || (s_md[k] == bd && (s_mi[k] < bi || (s_mi[k] == bi && s_mj[k] < bj)))) {
          bd = s_md[k];
          bi = s_mi[k];
          bj = s_mj[k];
        }
      }
      A.part_min_d2[blockIdx.x] = bd;
      A.part_min_ij[2 * blockIdx.x] = bi;
      A.part_min_ij[2 * blockIdx.x + 1] = bj;
    }
  } else if constexpr (OPK == OPK_HIST) {
    __syncthreads();
    for (int b = threadIdx.x; b < A.nbins; b += kThreads) {
      A.part_hc[(int64_t)blockIdx.x * A.nbins + b] = s_hc[b];
      A.part_hs[(int64_t)blockIdx.x * A.nbins + b] = s_hs[b];
    }
  }
}

// Resident blocks per SM of a kernel (0 if none).
template <class K> int blocks_per_sm(K kernel, size_t dyn) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, dyn) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm;
}

// One wave of resident blocks (the warps loop over cells): grid = min(cells/warps, SMs x blocks per SM).
inline int resident_grid(int want, int per_sm) {
  static const int sms = [] {
    int n = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, n);
  }();
  return std::max(1, std::min(want, std::max(1, per_sm) * sms));
}

// The smallest step with no common factor of n + step and parts.
inline int coprime_step(int n, int parts) {
  for (int step = 0;; step++) {
    int a = n + step, b = parts;
    while (b) {
      const int t = a % b;
      a = b;
      b = t;
    }
    if (a == 1) return step;
  }
}

template <class T, int N, int OPK, bool SPLIT, bool CROSS, bool BATCH = false, int OPC = 0>
cudaError_t launch_k(int& grid, cudaStream_t st, const PairArgs<T>& A) {
  using FA = typename std::conditional<std::is_same<T, double>::value && !SPLIT, double, float>::type;
  void (*k)(const PairArgs<T>);
  if constexpr (in_rounds(OPK, sizeof(T) == 8, SPLIT, BATCH)) k = rounds::k_pairs_rounds<T, N, OPK, SPLIT, CROSS, BATCH, OPC>;
  else k = k_pairs<T, N, OPK, SPLIT, CROSS, BATCH, OPC>;
  size_t dyn = 0;
  int per_sm = 0;
  if constexpr (OPK == OPK_HIST) {
    dyn = hist_smem(A.nbins, (int)sizeof(T), (int)sizeof(FA)).total;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    per_sm = blocks_per_sm(k, dyn);
  } else {
    static const int resident = blocks_per_sm(k, 0);  // asked once: the query costs the host a few us
    per_sm = resident;
    // the adjoint's FP32 sums run over all items of a lane: the same warps get the same items whatever the occupancy
    if (OPK == OPK_ADJ && in_rounds(OPK, sizeof(T) == 8, SPLIT, BATCH))
      per_sm = std::min(per_sm, sizeof(T) == 4 ? kAdjBlocks32 : kAdjBlocks64);
  }
  grid = resident_grid(grid, per_sm);
  // turned parts (part_of), except where the order of the sums has to stay
  const int parts = A.cell_split * A.stage_split;
  if (!BATCH && parts > 1 && !in_rounds(OPK, sizeof(T) == 8, SPLIT, BATCH)) {
    PairArgs<T> B = A;
    B.part_step = coprime_step(grid * kWarps, parts);
    k<<<grid, kThreads, dyn, st>>>(B);
  } else {
    k<<<grid, kThreads, dyn, st>>>(A);
  }
  return cudaGetLastError();
}

// The potentials of the force and energy maps are known at compile time: the sweep's switch over the operators costs it
// 4 to 12 % (100k points at cutoff 8, soft potential: forces 631 -> 602 us, energy 397 -> 369, split energy 141 -> 125,
// split forces 274 -> 242).  Each is another set of kernels to compile, so the other operators, and Lennard-Jones forces
// with type tables, take the switch.
template <class T, int N, bool SPLIT, bool CROSS>
cudaError_t launch_s(int opk, int& grid, cudaStream_t st, const PairArgs<T>& A) {
  switch (opk) {
    case OPK_NL: return launch_k<T, N, OPK_NL, SPLIT, CROSS>(grid, st, A);
    case OPK_SCALAR:
      if (A.op == 6) return launch_k<T, N, OPK_SCALAR, SPLIT, CROSS, false, 6>(grid, st, A);
      if (A.op == 8) return launch_k<T, N, OPK_SCALAR, SPLIT, CROSS, false, 8>(grid, st, A);
      return launch_k<T, N, OPK_SCALAR, SPLIT, CROSS>(grid, st, A);
    case OPK_FORCES:
      if (A.op == 9 && A.ntypes == 0) return launch_k<T, N, OPK_FORCES, SPLIT, CROSS, false, 9>(grid, st, A);
      if (A.op == 7) return launch_k<T, N, OPK_FORCES, SPLIT, CROSS, false, 7>(grid, st, A);
      return launch_k<T, N, OPK_FORCES, SPLIT, CROSS>(grid, st, A);
    case OPK_MIN: return launch_k<T, N, OPK_MIN, SPLIT, CROSS>(grid, st, A);
    case OPK_HIST:
      // pairs too close for the root's estimate are below such a first edge: no test for them (2D 1.4 %, 3D 0.3 %)
      if constexpr (!in_rounds(OPK_HIST, sizeof(T) == 8, SPLIT, false))
        if (A.first_edge >= 0x1p-510) return launch_k<T, N, OPK_HIST, SPLIT, CROSS, false, 11>(grid, st, A);
      return launch_k<T, N, OPK_HIST, SPLIT, CROSS>(grid, st, A);
    case OPK_ADJ:
      if constexpr (!CROSS) return launch_k<T, N, OPK_ADJ, SPLIT, false, false, 13>(grid, st, A);
      return cudaErrorInvalidValue;
  }
  return cudaErrorInvalidValue;
}

// Plain launches of one dtype: every operator kind, self and cross pairs, exact and split forms.
template <class T>
cudaError_t launch_plain_t(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<T>& A) {
  if constexpr (std::is_same<T, float>::value) {
    // Float32 inputs: the split form is the exact form (the input arithmetic is FP32 already)
    if (s.dim == 3) return s.self ? launch_s<T, 3, false, false>(s.opk, grid, st, A) : launch_s<T, 3, false, true>(s.opk, grid, st, A);
    return s.self ? launch_s<T, 2, false, false>(s.opk, grid, st, A) : launch_s<T, 2, false, true>(s.opk, grid, st, A);
  } else {
    if (s.dim == 3) {
      if (s.self) return s.split ? launch_s<T, 3, true, false>(s.opk, grid, st, A) : launch_s<T, 3, false, false>(s.opk, grid, st, A);
      return s.split ? launch_s<T, 3, true, true>(s.opk, grid, st, A) : launch_s<T, 3, false, true>(s.opk, grid, st, A);
    }
    if (s.self) return s.split ? launch_s<T, 2, true, false>(s.opk, grid, st, A) : launch_s<T, 2, false, false>(s.opk, grid, st, A);
    return s.split ? launch_s<T, 2, true, true>(s.opk, grid, st, A) : launch_s<T, 2, false, true>(s.opk, grid, st, A);
  }
}

// Batched launches: self pairs of many systems; neighbour lists, scalar reductions and forces.
template <class T, int N, bool SPLIT>
cudaError_t launch_b(int opk, int& grid, cudaStream_t st, const PairArgs<T>& A) {
  switch (opk) {
    case OPK_NL: return launch_k<T, N, OPK_NL, SPLIT, false, true>(grid, st, A);
    case OPK_SCALAR:
      if (A.op == 6) return launch_k<T, N, OPK_SCALAR, SPLIT, false, true, 6>(grid, st, A);
      if (A.op == 8) return launch_k<T, N, OPK_SCALAR, SPLIT, false, true, 8>(grid, st, A);
      return launch_k<T, N, OPK_SCALAR, SPLIT, false, true>(grid, st, A);
    case OPK_FORCES:
      if (A.op == 7) return launch_k<T, N, OPK_FORCES, SPLIT, false, true, 7>(grid, st, A);
      return launch_k<T, N, OPK_FORCES, SPLIT, false, true>(grid, st, A);
  }
  return cudaErrorInvalidValue;
}

template <class T>
cudaError_t launch_batch_t(const LaunchSel& s, int& grid, cudaStream_t st, const PairArgs<T>& A) {
  if (!s.self) return cudaErrorInvalidValue;
  if constexpr (std::is_same<T, float>::value) {
    return s.dim == 3 ? launch_b<T, 3, false>(s.opk, grid, st, A) : launch_b<T, 2, false>(s.opk, grid, st, A);
  } else {
    if (s.dim == 3) return s.split ? launch_b<T, 3, true>(s.opk, grid, st, A) : launch_b<T, 3, false>(s.opk, grid, st, A);
    return s.split ? launch_b<T, 2, true>(s.opk, grid, st, A) : launch_b<T, 2, false>(s.opk, grid, st, A);
  }
}

// Occupancy of the scalar and min-distance instantiations (the allocation-free entry point sizes its
// partials with it).  Float32 handles have no split instantiation (their split form is the exact one).
template <class T, int N, int OPK, bool SPLIT, bool CROSS> int occupancy_once() {
  static const int n = blocks_per_sm(k_pairs<T, N, OPK, SPLIT, CROSS, false>, 0);
  return n;
}
template <class T, int N, int OPK> int occupancy_pick(bool split, bool self) {
  if constexpr (!std::is_same<T, float>::value) {
    if (split) return self ? occupancy_once<T, N, OPK, true, false>() : occupancy_once<T, N, OPK, true, true>();
  }
  return self ? occupancy_once<T, N, OPK, false, false>() : occupancy_once<T, N, OPK, false, true>();
}

template <class T>
int occupancy_t(const LaunchSel& s) {
  if (s.opk == OPK_SCALAR)
    return s.dim == 3 ? occupancy_pick<T, 3, OPK_SCALAR>(s.split, s.self) : occupancy_pick<T, 2, OPK_SCALAR>(s.split, s.self);
  if (s.opk == OPK_MIN)
    return s.dim == 3 ? occupancy_pick<T, 3, OPK_MIN>(s.split, s.self) : occupancy_pick<T, 2, OPK_MIN>(s.split, s.self);
  return 0;
}

}  // namespace pk
}  // namespace clm
