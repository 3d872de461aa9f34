// Pair map kernel that works through its candidates in rounds, for the sums that are taken in FP32 and given
// out in FP64: forces of the split form, the adjoint and histograms of Float32 handles and of the split form,
// and the sums of FP32 batches.  Their last digits depend on the order of the FP32 additions (split-form forces
// of 100,000 points differ by 5e-7 between the two kernels' orders, each 5e-7 from 64-bit sums), which is this
// kernel's; k_pairs, which is faster, takes every other map.
#pragma once
#include "clm_pairs_common.cuh"

namespace clm {
namespace pk {
namespace rounds {

constexpr int kWindow = 128;                  // candidates staged at a time
constexpr int kWPlane = kWindow / 32 * kPad;  // words of one plane

// Shared memory of one warp.
template <class T, bool FP64, bool IS_F> struct RoundSmem {
  float p[4][kWPlane];             // the staged candidates: x, y, z and codes
  float4 i4[32];                   // particles of the chunk: prefilter coordinates, code in .w
  int pref[33];                    // stream position of the first copy of each stencil entry
  int delta[32];                   // its position in the cell list minus that
  int meta[32];                    // its cell's offset
  unsigned img[kWindow / 32];      // image copies among the candidates of each run
  unsigned short q[1024];          // compacted hits: (particle slot << 8) | plane index, 0x8000 marks
  T ix[3][FP64 ? 32 : 1];          // Float64 handles: the particles' coordinates
  float f[3][IS_F ? 32 : 1];       // force sums of the particles

  // the last stencil entry whose prefix is <= stream position e (that entry is not empty)
  __device__ __forceinline__ int entry_of(int e) const {
    int lo = 0;
#pragma unroll
    for (int st = 16; st > 0; st >>= 1)
      if (pref[lo + st] <= e) lo += st;
    return lo;
  }
};

// Per-pair energy u and g = (du/dr)/r (force contribution df = g*(x_i - x_j)).
template <class V, class T>
__device__ __forceinline__ void pair_value(const PairArgs<T>& A, int op, V d2, int i, int j, V& u, V& g) {
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
      u = d2 * vrsqrt(d2);
      g = V(0);
      break;
    case 5:  // SUM_INV_D
      u = vrsqrt(d2);
      g = V(0);
      break;
    case 6:
    case 7: {  // SOFT (c - d)^2
      V ri = vrsqrt(d2);
      V d = d2 * ri;
      V c = par<V>(A, 0);
      u = (c - d) * (c - d);
      g = V(-2) * (c - d) * ri;
      break;
    }
    case 8:
    case 9:
    case 13: {  // LJ eps*(c12 (s/d)^12 - c6 (s/d)^6)
      V eps = par<V>(A, 0), sig = par<V>(A, 1);
      if (A.ntypes > 0) {
        int ti = A.tx[i];
        int tj = A.self ? A.tx[j] : A.ty[j];
        eps = eps_tab<V>(A, ti * A.ntypes + tj);
        sig = sig_tab<V>(A, ti * A.ntypes + tj);
      }
      V c12 = par<V>(A, 2), c6 = par<V>(A, 3);
      V r2i = vrcp(d2);
      V sr2 = (sig * sig) * r2i;
      V sr6 = sr2 * sr2 * sr2;
      V sr12 = sr6 * sr6;
      u = eps * (c12 * sr12 - c6 * sr6);
      g = eps * (V(-12) * c12 * sr12 + V(6) * c6 * sr6) * r2i;
      break;
    }
    case 14: {  // weighted 1/d: u = -c w_i w_j / d, g = (c w_i w_j / d^2) / d
      const V cw = par<V>(A, 0) * weight<V>(A, false, i) * weight<V>(A, A.self == 0, j);
      const V ri = vrsqrt(d2);
      u = -(cw * ri);
      g = cw * (ri * ri * ri);
      break;
    }
    case 12: {  // 1/d with gradient accumulation
      V ri = vrsqrt(d2);
      u = ri;
      g = ri * ri * ri;
      break;
    }
    default:
      u = V(0);
      g = V(0);
  }
}

// Work items, stencil and pair rules as in k_pairs; a part of a cell takes interleaved chunks of its particles
// (LP = 32, 16 or 8 in a chunk, the other lanes being 2 or 4 groups that share the candidates).  Windows of 128
// candidates are staged as planes, and each round tests 32 candidates per lane (candidate b of lane group k is
// the round's b G + k), compacts the hits into a queue ordered by particle and sweeps over it: every lane takes a
// contiguous run, the particle's share of a force staying in registers along the run, then in shared memory
// until the chunk ends, the partner's going out pair by pair.  Pairs within 2^-13 of the cutoff are marked in
// the sweep and decided exactly in a second one, made only when a lane marked one.
// Issue and latency bound it.  Against the same rounds with bulk copies into double-buffered windows, scalar tests and
// shared-memory addresses recomputed from the thread index at each access: adjoint of 200k Float32 particles 154 us
// (165), split forces of 100k points at cutoff 8 242 us (274).  More items per cell or six resident blocks would take
// the latter to 190 us, but the FP32 additions then come in another order.
template <class T, int N, int OPK, bool SPLIT, bool CROSS, bool BATCH, int OPC = 0>
__global__ void __launch_bounds__(kThreads, (sizeof(T) == 4) ? 6 : 5)
    k_pairs_rounds(const __grid_constant__ PairArgs<T> A) {
  using V = T;
  static_assert(std::is_same<T, float>::value || SPLIT, "FP32 sums");
  constexpr bool IS_F = (OPK == OPK_FORCES) || (OPK == OPK_ADJ);
  constexpr bool FP64 = std::is_same<T, double>::value;
  constexpr bool ABS_PF = !FP64;  // Float32 handles test the coordinates themselves
  const DevGeom<T>& g = A.g;
  const int op = OPC ? OPC : A.op;
  using Smem = RoundSmem<T, FP64, IS_F>;
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
  const HistSmem hl = hist_smem((OPK == OPK_HIST) ? A.nbins : 0, (int)sizeof(T), (int)sizeof(float));
  double* s_hs = reinterpret_cast<double*>(s_dyn + hl.hs);
  unsigned long long* s_hc = reinterpret_cast<unsigned long long*>(s_dyn + hl.hc);
  T* s_bins = reinterpret_cast<T*>(s_dyn + hl.bins);
  float* s_binf = reinterpret_cast<float*>(s_dyn + hl.binf);
  float* s_ws = reinterpret_cast<float*>(s_dyn + hl.ws) + warp * A.nbins;
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
  const int nent = CROSS ? wN : (sym ? 2 * nf + 1 : nf + 1);
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
      s_ws[b] = 0.f;
      s_wc[b] = 0u;
    }
    for (int b = threadIdx.x; b <= A.nbins; b += kThreads) {
      s_bins[b] = A.bins[b];
      s_binf[b] = (float)A.bins[b];
    }
    __syncthreads();
  }

  double e_tot = 0.0;  // per-lane energy (FP64); FP32 partial sums are folded in per particle chunk
  float e_part = 0.f;
  float adj[kAdjVals - 1];  // adjoint accumulators: virial (6), dU/deps (3), dU/dsigma (3)
#pragma unroll
  for (int k = 0; k < kAdjVals - 1; k++) adj[k] = 0.f;
  unsigned long long c_acc = 0;

  const int gw = blockIdx.x * kWarps + warp;
  const int nw = gridDim.x * kWarps;
  // a build that flagged an overflow left cells without copies: nothing is mapped, and the build is repeated
  const int n_real = (*A.err & kBuildFailed) ? 0 : *A.n_real_dev;
  const int S = A.cell_split;  // the host keeps cells x parts below 2^31
  const int n_items = n_real * S;
  for (int r = gw; r < n_items; r += nw) {
    int rcell = r, part = 0;
    if (S > 1) {
      rcell = r / S;
      part = r - rcell * S;
    }
    const int li = A.real_list[rcell];
    int cb = 0;  // first global cell of the system (batches)
    const DevGeom<T>& gc = geo_of<BATCH>(A, li, cb);
    int ci[3];
    cart_of_fast<N>(gc, li - cb, ci);
    const int si = A.X.cell_start[li];
    const int ni = A.X.cell_start[li + 1] - si;
    const int GS = (ni <= 8) ? 2 : ((ni <= 16) ? 1 : 0);  // log2 of the lane groups
    const int LP = 32 >> GS;
    const int grp = lane & ((1 << GS) - 1);  // the lanes of one particle are adjacent
    const int il = lane >> GS;
    const int JR = 32 << GS;  // candidates per round

    for (int ib = part * LP; ib < ni; ib += LP * S) {
      const int ii = ib + il;
      const bool vi = ii < ni;
      float4 i4 = make_float4(0.f, 0.f, 0.f, 0.f);  // the lane's particle: prefilter coordinates and code
      if (vi) i4 = (ABS_PF ? A.X.xq : A.X.off)[si + ii];
      if (grp == 0) {
        W.i4[il] = i4;
#pragma unroll
        for (int d = 0; d < N; d++) {
          if (FP64 && vi) W.ix[d][il] = pos_of(A.X, d, si + ii);
          if constexpr (IS_F) W.f[d][il] = 0.f;
        }
      }
      const int code_l = __float_as_int(i4.w);
      const bool act_i = (tri && CROSS) ? (vi && code_l >= 0) : vi;

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

        for (int w0 = 0; w0 < total; w0 += kWindow) {
          const int wc = min(kWindow, total - w0);
          // ---- stage the window as planes: candidate q of the window goes to candidate b of its run
          {
            const float4* rec = ABS_PF ? A.Y.xq : A.Y.off;
            if (lane < kWindow / 32) W.img[lane] = 0u;
            __syncwarp();
            float4 rv[kWindow / 32];
#pragma unroll
            for (int k = 0; k < kWindow / 32; k++) {
              if (32 * k < wc) {
                const int e = w0 + min(32 * k + lane, wc - 1);
                const int lo = W.entry_of(e);
                rv[k] = rec[W.delta[lo] + e];
                if constexpr (!ABS_PF) {
                  // shift the offsets by the cell displacement so that x_i - x_j ~ off_i - plane
                  const int me = W.meta[lo];
                  rv[k].x += gc.csf[0] * (float)((me & 255) - 128);
                  rv[k].y += gc.csf[1] * (float)(((me >> 8) & 255) - 128);
                  rv[k].z += gc.csf[2] * (float)(((me >> 16) & 255) - 128);
                }
              }
            }
#pragma unroll
            for (int k = 0; k < kWindow / 32; k++) {
              if (32 * k < wc) {
                const int qq = 32 * k + lane, in = qq & (JR - 1);
                const int run = ((qq >> (5 + GS)) << GS) + (in & ((1 << GS) - 1)), b = in >> GS;
                const int p = run * kPad + b;
                W.p[0][p] = rv[k].x;
                W.p[1][p] = rv[k].y;
                if (N == 3) W.p[2][p] = rv[k].z;
                W.p[3][p] = rv[k].w;
                if (__float_as_int(rv[k].w) < 0) atomicOr(&W.img[run], 1u << b);
              }
            }
          }
          __syncwarp();
          for (int rb = 0; rb < wc; rb += JR) {
            const int cntr = min(JR, wc - rb);
            const int run = ((rb >> (5 + GS)) << GS) + grp;
            // ---- tests: a test passes when d2 - thr is negative.  thr carries a 2^-13 relative margin, far above
            // the FP32 rounding of dx^2 - thr + dy^2 + dz^2, so the strict comparison keeps every pair the
            // exact test can accept.
            unsigned mask = 0u;
            {
              const float nthr = -g.thr_hi;
              const float2 tx = make_float2(-i4.x, -i4.x), ty = make_float2(-i4.y, -i4.y);
              const float2 tz = make_float2(-i4.z, -i4.z), tt = make_float2(nthr, nthr);
              const float* bx = &W.p[0][run * kPad];
#pragma unroll
              for (int b = 28; b >= 0; b -= 4) {
                const float4 X = *reinterpret_cast<const float4*>(bx + b);
                const float4 Y = *reinterpret_cast<const float4*>(bx + kWPlane + b);
                float2 d = __fadd2_rn(make_float2(X.z, X.w), tx);
                float2 eh = __ffma2_rn(d, d, tt);
                d = __fadd2_rn(make_float2(X.x, X.y), tx);
                float2 el = __ffma2_rn(d, d, tt);
                d = __fadd2_rn(make_float2(Y.z, Y.w), ty);
                eh = __ffma2_rn(d, d, eh);
                d = __fadd2_rn(make_float2(Y.x, Y.y), ty);
                el = __ffma2_rn(d, d, el);
                if constexpr (N == 3) {
                  const float4 Z = *reinterpret_cast<const float4*>(bx + 2 * kWPlane + b);
                  d = __fadd2_rn(make_float2(Z.z, Z.w), tz);
                  eh = __ffma2_rn(d, d, eh);
                  d = __fadd2_rn(make_float2(Z.x, Z.y), tz);
                  el = __ffma2_rn(d, d, el);
                }
                mask = __funnelshift_l(__float_as_uint(eh.y), mask, 1);  // (mask << 1) | sign bit
                mask = __funnelshift_l(__float_as_uint(eh.x), mask, 1);
                mask = __funnelshift_l(__float_as_uint(el.y), mask, 1);
                mask = __funnelshift_l(__float_as_uint(el.x), mask, 1);
              }
            }
            {
              // bit b is stream position base + b G.  Dropped: positions past the window's end (stale
              // records), pairs of two images (never the reference's), and in the cell itself the pairs the
              // reference does not visit from this copy: the earlier slots for self pairs (each pair of the cell
              // once), every slot for an image copy in cross pairs of orthorhombic cells (the particle copy must be
              // real there).  What remains of the pair rules is in the sweep (triclinic self pairs of a real copy
              // and an image).
              const int base = w0 + rb + grp;
              const int nb = (cntr - grp + (1 << GS) - 1) >> GS;
              if (!act_i || nb <= 0) mask = 0u;
              else if (nb < 32) mask &= (1u << nb) - 1u;
              if (code_l < 0) mask &= ~W.img[run];
              int lim = -1;  // last dropped position of the cell itself
              if (!CROSS) lim = min(ii, same_end - 1);
              else if (!tri && !nonper && code_l < 0) lim = same_end - 1;
              if (lim >= base) {
                const int nr = ((lim - base) >> GS) + 1;
                mask &= (nr >= 32) ? 0u : ~((1u << nr) - 1u);
              }
            }
            // ---- queue: the hits of all lanes
            int H;
            {
              const int nh = __popc(mask);
              int incl = nh;
#pragma unroll
              for (int o2 = 1; o2 < 32; o2 <<= 1) {
                int y = __shfl_up_sync(FULL, incl, o2);
                if (lane >= o2) incl += y;
              }
              H = __shfl_sync(FULL, incl, 31);
              unsigned short* qp = &W.q[incl - nh];
              const int ent0 = (il << 8) | (run * kPad);  // the plane index is below 256 - 32
              for (unsigned m = mask; m;) {
                const int b = __ffs(m) - 1;
                m &= m - 1u;
                *qp++ = (unsigned short)(ent0 + b);
              }
            }
            __syncwarp();
            const int per = (H + 31) >> 5;
            const int qbeg = lane * per;
            bool marked = false;
            auto sweep = [&](auto rare_c) {
              constexpr bool RARE = decltype(rare_c)::value;
              int cur = -1;  // the particle slot of this lane's run (its data below, its force sums in acc)
              float4 p4 = make_float4(0.f, 0.f, 0.f, 0.f);
              float acc[3] = {0.f, 0.f, 0.f};
              for (int t = 0; t < per; t++) {
                const int qi = qbeg + t;
                const bool has = qi < H;
                bool live = has;  // the entry is evaluated in this sweep
                int jp = 0, ie = (cur < 0) ? 0 : cur;
                if (has) {
                  const int ent = W.q[qi];
                  ie = (ent >> 8) & 31;
                  jp = ent & 255;
                  if constexpr (RARE) live = (ent & 0x8000) != 0;
                }
                // `cur` follows every queue entry (hit or not), so the lanes holding a particle are exactly the
                // lanes whose runs cover its entries: adjacent, and only the last one moves past it inside its
                // run; no other lane updates that particle's sums during the loop
                if (has && ie != cur) {
                  if constexpr (IS_F) {
                    if (cur >= 0) {
#pragma unroll
                      for (int d = 0; d < N; d++) W.f[d][cur] += acc[d];
                    }
#pragma unroll
                    for (int d = 0; d < N; d++) acc[d] = 0.f;
                  }
                  cur = ie;
                  p4 = W.i4[ie];
                }
                const int code_i = __float_as_int(p4.w);
                const int idx_i = code_i ^ (code_i >> 31);
                bool hit = false, sure = false;
                int idx_j = 0;
                int oi = 0, oj = 0;  // the pair as the reference orients it (i, j)
                float d2f = 0.f;
                float dvf[3] = {0.f, 0.f, 0.f};
                T d2 = 0;
                T dxs[3] = {0, 0, 0};  // x_i - x_j of the exact test, reused by the force epilogues
                auto load_x = [&](T* xi, T* xj) {
                  if constexpr (FP64) {
                    const int run_q = jp / kPad;
                    const int e = w0 + ((run_q >> GS) << (5 + GS)) + ((jp - run_q * kPad) << GS) + (run_q & ((1 << GS) - 1));
                    const int tj = W.delta[W.entry_of(e)] + e;
#pragma unroll
                    for (int d = 0; d < N; d++) {
                      xi[d] = W.ix[d][ie];
                      xj[d] = pos_of(A.Y, d, tj);
                    }
                  }
                };
                if (live) {
                  const int code_j = __float_as_int(W.p[3][jp]);
                  idx_j = code_j ^ (code_j >> 31);
                  // the rest of the pair rules: in triclinic self pairs of a real copy and an image, the copy of
                  // the lower index is the reference's i and must be real (see k_pairs)
                  const bool cand = ((code_i ^ code_j) & ~(code_i + code_j + 1) & sym_mask) >= 0;
                  const bool sw = sym && idx_j < idx_i;
                  oi = sw ? idx_j : idx_i;
                  oj = sw ? idx_i : idx_j;
                  if (cand) {
                    dvf[0] = p4.x - W.p[0][jp];
                    dvf[1] = p4.y - W.p[1][jp];
                    dvf[2] = (N == 3) ? p4.z - W.p[2][jp] : 0.f;
                    d2f = fmaf(dvf[2], dvf[2], fmaf(dvf[1], dvf[1], dvf[0] * dvf[0]));
                    if constexpr (!RARE) {
                      // well inside the cutoff the FP32 value decides; the others are marked for the second sweep
                      if (d2f <= g.thr_lo) {
                        hit = true;
                        sure = true;
                      } else {
                        W.q[qi] = (unsigned short)(W.q[qi] | 0x8000u);
                        marked = true;
                      }
                    } else {
                      T xi[3] = {0, 0, 0}, xj[3] = {0, 0, 0};
                      if constexpr (FP64) {
                        load_x(xi, xj);
                      } else {
                        xi[0] = p4.x, xi[1] = p4.y, xi[2] = p4.z;
#pragma unroll
                        for (int d = 0; d < N; d++) xj[d] = W.p[d][jp];
                      }
#pragma unroll
                      for (int d = 0; d < N; d++) dxs[d] = xsub(xi[d], xj[d]);
                      d2 = exact_d2<T, N>(dxs);
                      const int run_q = jp / kPad;
                      const int e = w0 + ((run_q >> GS) << (5 + GS)) + ((jp - run_q * kPad) << GS) + (run_q & ((1 << GS) - 1));
                      hit = near_cutoff<T, N>(gc, g.cutoff_sqr, make_int3(ci[0], ci[1], ci[2]),
                                              W.meta[W.entry_of(e)], e < same_end, sw, xi[0], xi[1], xi[2], xj[0], xj[1],
                                              xj[2]);
                    }
                  }
                }
                // ---------------- operator epilogues
                if constexpr (OPK == OPK_SCALAR) {
                  if (hit) {
                    if (op == 2) {
                      c_acc++;
                    } else if (sure) {
                      float uu, gg;
                      pair_value<float, T>(A, op, d2f, oi, oj, uu, gg);
                      e_part += uu;
                    } else {
                      V uu, gg;
                      pair_value<V, T>(A, op, (V)d2, oi, oj, uu, gg);
                      e_part += (float)uu;
                    }
                  }
                } else if constexpr (IS_F) {
                  if (hit) {
                    float uu, gg;
                    float df[3] = {0.f, 0.f, 0.f};
                    float dv[3] = {0.f, 0.f, 0.f};
                    if (sure) {
                      pair_value<float, T>(A, op, d2f, oi, oj, uu, gg);
#pragma unroll
                      for (int d = 0; d < N; d++) dv[d] = dvf[d];
                    } else {
                      V uv, gv;
                      pair_value<V, T>(A, op, (V)d2, oi, oj, uv, gv);
                      uu = (float)uv;
                      gg = (float)gv;
#pragma unroll
                      for (int d = 0; d < N; d++) dv[d] = (float)dxs[d];
                    }
#pragma unroll
                    for (int d = 0; d < N; d++) df[d] = gg * dv[d];
                    if constexpr (OPK == OPK_ADJ) {
                      // virial W += g dx dx^T (g = u'(r)/r), and the parameter derivatives of the LJ term
                      adj[0] += gg * dv[0] * dv[0];
                      adj[1] += gg * dv[1] * dv[1];
                      adj[2] += gg * dv[2] * dv[2];
                      adj[3] += gg * dv[0] * dv[1];
                      adj[4] += gg * dv[0] * dv[2];
                      adj[5] += gg * dv[1] * dv[2];
                      float eps = par<float>(A, 0), sig = par<float>(A, 1);
                      int cls = 0;
                      if (A.ntypes > 0) {
                        const int ti = A.tx[oi], tj = A.tx[oj];
                        eps = eps_tab<float>(A, ti * A.ntypes + tj);
                        sig = sig_tab<float>(A, ti * A.ntypes + tj);
                        cls = ti + tj;  // 2 types: AA = 0, AB = 1, BB = 2
                      }
                      const float c12 = par<float>(A, 2), c6 = par<float>(A, 3);
                      const float dd2 = sure ? d2f : (float)d2;
                      const float sr2 = sig * sig * vrcp(dd2);
                      const float sr6 = sr2 * sr2 * sr2;
                      const float sr12 = sr6 * sr6;
                      const float lj = c12 * sr12 - c6 * sr6;
                      const float dsg = eps * (12.f * c12 * sr12 - 6.f * c6 * sr6) * vrcp(sig);
#pragma unroll
                      for (int k = 0; k < 3; k++) {
                        adj[6 + k] += (cls == k) ? lj : 0.f;
                        adj[9 + k] += (cls == k) ? dsg : 0.f;
                      }
                    }
#pragma unroll
                    for (int d = 0; d < N; d++) acc[d] -= df[d];
                    e_part += uu;
                    force_add<T, N, float>(A, CROSS, idx_j, df);  // the partner's share
                  }
                } else if constexpr (OPK == OPK_HIST) {
                  int hb = -1;     // bin of this lane's pair (-1: none)
                  float hv = 0.f;  // its accumulator term
                  if (hit) {
                    bool exact_r = !sure;
                    float rfl = 0.f;  // the distance in FP32 for the pair value
                    int b = -1;
                    if (sure) {
                      rfl = sqrtf(d2f);
                      const int lo = first_edge_at_or_above(s_binf, A.nbins, rfl);
                      b = lo - 1;
                      if (near_edge(s_binf, A.nbins, lo, rfl)) exact_r = true;  // an edge within 2^-12: decide exactly
                    }
                    if (exact_r) {
                      T e2 = d2;  // the exact test's d2 (not sure), or recomputed near a bin edge
                      if (sure) {
                        T dx[3];
                        if constexpr (FP64) {
                          T xi[3], xj[3];
                          load_x(xi, xj);
#pragma unroll
                          for (int d = 0; d < N; d++) dx[d] = xsub(xi[d], xj[d]);
                        } else {
#pragma unroll
                          for (int d = 0; d < N; d++) dx[d] = dvf[d];
                        }
                        e2 = exact_d2<T, N>(dx);
                      }
                      const T rr = xsqrt(e2);
                      rfl = (float)rr;
                      b = first_edge_at_or_above(s_bins, A.nbins, rr) - 1;
                    }
                    if (b >= 0 && b < A.nbins) {
                      float dv[3] = {0.f, 0.f, 0.f};
#pragma unroll
                      for (int d = 0; d < N; d++) dv[d] = sure ? dvf[d] : (float)dxs[d];
                      if (tri) {
                        float rv[3];
#pragma unroll
                        for (int a = 0; a < N; a++) {
                          float s = 0.f;
#pragma unroll
                          for (int k = 0; k < N; k++) s += (float)gc.Rinv[a][k] * dv[k];
                          rv[a] = s;
                        }
#pragma unroll
                        for (int a = 0; a < N; a++) dv[a] = rv[a];
                      }
                      float dot = 0.f;
                      // velocities converted once by the host code
                      const float* vy = CROSS ? A.vyf : A.vxf;
#pragma unroll
                      for (int d = 0; d < N; d++)
                        dot += (A.vxf[(int64_t)idx_i * N + d] - vy[(int64_t)idx_j * N + d]) * dv[d];
                      hv = dot * vrcp(rfl);
                      hb = b;
                    }
                  }
                  // lanes holding the same bin are summed by a tree over their group; the group's first lane
                  // then updates the warp's own bin (groups have distinct bins: no atomics)
                  if (__any_sync(FULL, hb >= 0)) {
                    const unsigned peers = __match_any_sync(FULL, hb);
                    const float v = group_sum(peers, hv, lane);
                    if (hb >= 0 && lane == __ffs(peers) - 1) {
                      s_ws[hb] += v;
                      s_wc[hb] += (unsigned)__popc(peers);
                    }
                    __syncwarp();
                  }
                }
              }
              if constexpr (IS_F) {
                // lanes ending on the same particle are adjacent: sum each run of equal `cur` into its first
                // lane, which alone adds it to the particle's sums
                __syncwarp();
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                  const int co = __shfl_down_sync(FULL, cur, off);
                  float t[3];
#pragma unroll
                  for (int d = 0; d < N; d++) t[d] = __shfl_down_sync(FULL, acc[d], off);
                  if (lane + off < 32 && co == cur) {
#pragma unroll
                    for (int d = 0; d < N; d++) acc[d] += t[d];
                  }
                }
                const int cprev = __shfl_up_sync(FULL, cur, 1);
                if (cur >= 0 && (lane == 0 || cprev != cur)) {
#pragma unroll
                  for (int d = 0; d < N; d++) W.f[d][cur] += acc[d];
                }
              }
            };
            sweep(std::false_type());
            if (__any_sync(FULL, marked)) {
              __syncwarp();
              sweep(std::true_type());
            }
            if constexpr (OPK == OPK_HIST) {
              // move the warp's bins (at most 1024 pairs of this round) into the block's FP64 bins
              __syncwarp();
              for (int b = lane; b < A.nbins; b += 32) {
                const unsigned c = s_wc[b];
                if (c) {
                  atomicAdd(&s_hc[b], (unsigned long long)c);
                  atomicAdd(&s_hs[b], (double)s_ws[b]);
                  s_wc[b] = 0u;
                  s_ws[b] = 0.f;
                }
              }
            }
            __syncwarp();
          }
        }
        __syncwarp();  // the next table overwrites this one
      }
      e_tot += (double)e_part;
      e_part = 0.f;
      if constexpr (IS_F) {
        __syncwarp();
        float f[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < N; d++) f[d] = W.f[d][il];
        if (grp == 0 && vi && (f[0] != 0.f || f[1] != 0.f || f[2] != 0.f))
          force_add<T, N, float>(A, false, code_l ^ (code_l >> 31), f);
      }
      __syncwarp();  // the next chunk's particles overwrite W.i4
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
  } else if constexpr (OPK == OPK_HIST) {
    __syncthreads();
    for (int b = threadIdx.x; b < A.nbins; b += kThreads) {
      A.part_hc[(int64_t)blockIdx.x * A.nbins + b] = s_hc[b];
      A.part_hs[(int64_t)blockIdx.x * A.nbins + b] = s_hs[b];
    }
  }
}


}  // namespace rounds
}  // namespace pk
}  // namespace clm
