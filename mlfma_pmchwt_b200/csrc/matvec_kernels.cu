// The PMCHWT MLFMA matvec on the GPU, FP64 (the `ax` closure of
// Code/MLFMM.cpp:189-368). J and M currents share the tree and the tables,
// so every stage processes both (6 complex components per direction) in one
// pass over the tables; media k1 and k2 run as separate launches.
//
//   agg      leaf aggregation           Code/ProcessMLFMM.h:33-56   (mexp)
//   up       interpolation + shift up   Code/ProcessMLFMM.h:61-107  (m2m)
//   m2l      translation over the interaction list   Code/ProcessMLFMM.h:112-147
//   l2l      the parent's incoming pattern, shifted and anterpolated onto
//            the child grid, added                    Code/ProcessMLFMM.h:152-202
//   near     the near-field rows, written once per unknown   Code/MLFMM.cpp:353-366
//   leaf     receive-pattern testing of both media, added    Code/MLFMM.cpp:285-351
// Every stage writes its output before anything accumulates into it (l2l adds
// onto the Bm that m2l of the same level has just written), so no clearing
// pass (Code/ProcessMLFMM.h:14-28) is needed.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <tuple>
#include <type_traits>
#include <utility>

#include "agg_tc.hpp"
#include "bulk.cuh"
#include "cplx.cuh"
#include "plan.hpp"
#include "solver.hpp"

namespace mlfma {

namespace {

constexpr int kThreads = 128;

// Aggregation: thread per (leaf box, direction), J and M from one pattern
// load. The box's currents are staged in shared memory (in the storage type)
// and the next RWGs' patterns are always in flight, so the loop waits for
// no index. HBM-bound (245,760 unknowns: 4.8 GB). One B200, both media, against
// the loop that read each RWG's index, then its currents: FP64 at 245,760 unknowns
// 0.94 -> 0.85 ms, at 7,260 70 -> 50 us, complex64 at 61,440 202 -> 140 us.
constexpr int kAggRwgs = 48;  // RWGs of a box staged at a time (a multiple of the RWGs in flight)

template <class C>
__global__ void __launch_bounds__(kThreads, sizeof(C) == 16 ? 6 : 8) agg_kernel(const C* __restrict__ Vs, const int* __restrict__ leaf_ptr,
                                                       const int* __restrict__ leaf_rwg,
                                                       const double2* __restrict__ x, int N, int K,
                                                       C* __restrict__ S) {
  constexpr int kFlight = sizeof(C) == 16 ? 2 : 4;
  __shared__ C xs[kAggRwgs][2];
  const int kk = blockIdx.y * blockDim.x + threadIdx.x;
  const int b = blockIdx.x;
  const int r0 = leaf_ptr[b], nb = leaf_ptr[b + 1] - r0;
  const C* V = Vs + static_cast<size_t>(r0) * 3 * K + min(kk, K - 1);
  C next[kFlight][3];
  auto fetch = [&](int r) {
#pragma unroll
    for (int u = 0; u < kFlight; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        next[u][c] = r + u < nb ? __ldg(V + (static_cast<size_t>(r + u) * 3 + c) * K) : Cx<C>::zero();
  };
  fetch(0);
  C acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = Cx<C>::zero();
  for (int s0 = 0; s0 < nb; s0 += kAggRwgs) {
    const int n = min(kAggRwgs, nb - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * n; i += blockDim.x)
      xs[i >> 1][i & 1] = Cx<C>::from(__ldg(x + (i & 1) * N + __ldg(leaf_rwg + r0 + s0 + (i >> 1))));
    __syncthreads();
#pragma unroll 1
    for (int r = 0; r < n; r += kFlight) {
      C v[kFlight][3];
#pragma unroll
      for (int u = 0; u < kFlight; ++u)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[u][c] = next[u][c];
      fetch(s0 + r + kFlight);
#pragma unroll
      for (int u = 0; u < kFlight; ++u)
        if (r + u < n) {
          const C xJ = xs[r + u][0], xM = xs[r + u][1];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            acc[c] = cfma(v[u][c], xJ, acc[c]);
            acc[3 + c] = cfma(v[u][c], xM, acc[3 + c]);
          }
        }
    }
  }
  if (kk >= K) return;
  C* out = S + static_cast<size_t>(b) * 6 * K + kk;
#pragma unroll
  for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * K] = acc[c];
}

struct AggBoxArg {
  const double2* Vs[2];  // radiation patterns per medium [N][3][K] (leaf order)
  double2* S[2];         // leaf-level patterns per medium [Bleaf][6][K]
  int K[2];
  const int* leaf_ptr;
  const int* leaf_rwg;
  const double2* x;
  int N;
};

// Aggregation, CTA per (leaf box, medium): the box's radiation patterns are
// one contiguous block [n_b][3K] in leaf order, streamed by threads over its
// 3K entries, two columns per thread (J components land at S[b][0..2], M at
// S[b][3..5]). The box's currents are staged in shared memory first (boxes
// of more than kAggStage RWGs read them from global memory).
constexpr int kAggStage = 64;

__global__ void __launch_bounds__(kThreads) agg_box_kernel(AggBoxArg a) {
  __shared__ double2 sx[2][kAggStage];
  const int b = blockIdx.x, m = blockIdx.y;
  const int K3 = 3 * a.K[m];
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  const bool staged = nb <= kAggStage;
  if (staged)
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
      const int id = a.leaf_rwg[r0 + i];
      sx[0][i] = a.x[id];
      sx[1][i] = a.x[a.N + id];
    }
  __syncthreads();
  const double2* V = a.Vs[m] + static_cast<size_t>(r0) * K3;
  double2* out = a.S[m] + static_cast<size_t>(b) * 2 * K3;
  for (int e0 = threadIdx.x; e0 < K3; e0 += 2 * blockDim.x) {
    const int e1 = e0 + blockDim.x;
    const bool two = e1 < K3;
    double2 aJ0 = c2(0.0, 0.0), aM0 = c2(0.0, 0.0), aJ1 = c2(0.0, 0.0), aM1 = c2(0.0, 0.0);
    const double2* v = V + e0;
#pragma unroll 4
    for (int r = 0; r < nb; ++r, v += K3) {
      double2 xJ, xM;
      if (staged) {
        xJ = sx[0][r];
        xM = sx[1][r];
      } else {
        const int id = __ldg(a.leaf_rwg + r0 + r);
        xJ = __ldg(a.x + id);
        xM = __ldg(a.x + a.N + id);
      }
      const double2 s0 = __ldg(v);
      const double2 s1 = two ? __ldg(v + blockDim.x) : c2(0.0, 0.0);
      aJ0 = cfma(s0, xJ, aJ0);
      aM0 = cfma(s0, xM, aM0);
      aJ1 = cfma(s1, xJ, aJ1);
      aM1 = cfma(s1, xM, aM1);
    }
    out[e0] = aJ0;
    out[K3 + e0] = aM0;
    if (two) {
      out[e1] = aJ1;
      out[K3 + e1] = aM1;
    }
  }
}

template <class C>
struct Up2Arg {
  const C* Sc;   // child level patterns [Bc][6][Kc]
  C* Sp;         // parent level patterns [Bp][6][Kp]
  const int* child_begin;
  const int* octant;  // of child boxes
  const int4* row;    // per pair of parent theta rows: its 4 child rows
  const double2* w;   // [4] per pair: weights in the two parent rows
  const int* pidx;
  const double* lp;
  const C* ph_up;
  int Kp, nthp, nphp, Kc;
  long long slot_c = 0, slot_p = 0;  // element strides between right-hand-side slots (grid.z = 6 x slots)
};

// Interpolation (m2m), a thread per (parent box, pair of parent theta rows,
// parent phi column, component): the two rows' stencils lie on at most 4
// child rows (a parent's grid is finer than its children's, so neighbouring
// rows' stencils are at most one child row apart), and 12 loads serve two
// outputs where 9 taps per output are 18; each child row is interpolated in phi
// once, then in theta, times the child's shift phase, summed over the children.
// Loads address from the child's uniform base by 32-bit offsets. kSlots: grid.z =
// 6 x slots with the slot offsets of the batched tree; the single apply
// instantiates without them. kT: threads per CTA.
// Bound by L1 throughput (85 % of its data pipe in complex64): a gather of 32
// phi taps straddles lines. One B200, interpolation of all levels and both media,
// against a thread per output over its 9 taps: FP64 at 245,760 unknowns 1.34 ->
// 1.05 ms, 16 slots of complex64 at 61,440 3.36 -> 3.07 ms. The occupancy bounds
// are the measured best (FP64 96, complex64 72 registers; 64 spill). In
// complex64 the phi and theta weights are rounded one by one where the 9 taps
// had their products rounded, but an output meets fewer roundings: its error is
// 0.84 to 0.97 of the 9 taps' over 78 pairs of levels of 24 bodies (5.3e-8 to
// 5.9e-8 against 5.9e-8 to 6.3e-8).
template <class C, bool kSlots, int kT>
__global__ void __launch_bounds__(kT, (sizeof(C) == 16 ? 640 : 896) / kT) up2_kernel(const __grid_constant__ Up2Arg<C> a) {
  using R = typename Cx<C>::real;
  const int q = blockIdx.y * kT + threadIdx.x;
  const int b = blockIdx.x;
  const int slot = kSlots ? blockIdx.z / 6 : 0;
  const int c = blockIdx.z - 6 * slot;
  if (q >= ((a.nthp + 1) >> 1) * a.nphp) return;
  const int tp = q / a.nphp, p = q - tp * a.nphp;
  const bool two = 2 * tp + 1 < a.nthp;
  unsigned at[3];
  R wp[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    at[j] = __ldg(a.pidx + 3 * p + j);
    wp[j] = static_cast<R>(__ldg(a.lp + 3 * p + j));
  }
  const int4 r4 = __ldg(a.row + tp);
  const unsigned row[4] = {static_cast<unsigned>(r4.x), static_cast<unsigned>(r4.y), static_cast<unsigned>(r4.z),
                           static_cast<unsigned>(r4.w)};
  R w0[4], w1[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const double2 w = __ldg(a.w + 4 * tp + r);
    w0[r] = static_cast<R>(w.x);
    w1[r] = static_cast<R>(w.y);
  }
  const unsigned kk = 2u * tp * a.nphp + p;
  C acc0 = Cx<C>::zero(), acc1 = Cx<C>::zero();
  const C* const Sl = kSlots ? a.Sc + slot * a.slot_c : a.Sc;
  const int c1 = a.child_begin[b + 1];
  for (int ch = a.child_begin[b]; ch < c1; ++ch) {
    const C* sc = Sl + (static_cast<size_t>(ch) * 6 + c) * a.Kc;
    const C* ph = a.ph_up + static_cast<size_t>(a.octant[ch]) * a.Kp;
    C s[4][3];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 3; ++j) s[r][j] = __ldg(sc + (row[r] + at[j]));
    const C e0 = __ldg(ph + kk), e1 = __ldg(ph + (two ? kk + a.nphp : kk));
    C v0 = Cx<C>::zero(), v1 = Cx<C>::zero();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const C f = cfmas(wp[2], s[r][2], cfmas(wp[1], s[r][1], cscale(s[r][0], wp[0])));
      v0 = cfmas(w0[r], f, v0);
      v1 = cfmas(w1[r], f, v1);
    }
    acc0 = cfma(e0, v0, acc0);
    acc1 = cfma(e1, v1, acc1);
  }
  C* out = (kSlots ? a.Sp + slot * a.slot_p : a.Sp) + (static_cast<size_t>(b) * 6 + c) * a.Kp + kk;
  out[0] = acc0;
  if (two) out[a.nphp] = acc1;
}

// grid: (parent boxes, tiles of t (row pair, phi column)s, zdim = 6 components x slots)
template <class C, bool kSlots>
void launch_up2(int t, int boxes, int zdim, const Up2Arg<C>& a, cudaStream_t s) {
  const dim3 g(boxes, (((a.nthp + 1) / 2) * a.nphp + t - 1) / t, zdim);
  if (t == 64)
    up2_kernel<C, kSlots, 64><<<g, 64, 0, s>>>(a);
  else if (t == 256)
    up2_kernel<C, kSlots, 256><<<g, 256, 0, s>>>(a);
  else
    up2_kernel<C, kSlots, 128><<<g, 128, 0, s>>>(a);
}

struct UpArg {
  const double2* Sc;   // child level patterns [Bc][6][Kc]
  double2* Sp;         // parent level patterns [Bp][6][Kp]
  const int* child_begin;
  const int* octant;   // of child boxes
  const int* tidx;
  const double* lt;
  const int* pidx;
  const double* lp;
  const double2* ph_up;
  int Kp, nphp, Kc, nphc;
};

// Interpolation (m2m), one thread per (parent box, parent direction) for all
// 6 components: the stencil (3 theta x 3 phi taps and weights) and the
// child's shift phase are loaded once per child and applied to the 6
// component rows, 54 independent loads per child in flight.
__global__ void __launch_bounds__(kThreads) up6_kernel(UpArg a) {
  const int kk = blockIdx.y * blockDim.x + threadIdx.x;
  const int b = blockIdx.x;
  if (kk >= a.Kp) return;
  const int t = kk / a.nphp, p = kk - t * a.nphp;
  int ti[3], pi[3];
  double wt[3], wp[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    ti[i] = __ldg(a.tidx + 3 * t + i) * a.nphc;
    wt[i] = __ldg(a.lt + 3 * t + i);
    pi[i] = __ldg(a.pidx + 3 * p + i);
    wp[i] = __ldg(a.lp + 3 * p + i);
  }
  double2 acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = c2(0.0, 0.0);
  const int c1 = a.child_begin[b + 1];
  for (int ch = a.child_begin[b]; ch < c1; ++ch) {
    const double2 e = __ldg(a.ph_up + a.octant[ch] * a.Kp + kk);
    const double2* sc = a.Sc + static_cast<size_t>(ch) * 6 * a.Kc;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const double2* sr = sc + static_cast<size_t>(c) * a.Kc;
      double2 v = c2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) v = cfmas(wt[i] * wp[j], __ldg(sr + ti[i] + pi[j]), v);
      acc[c] = cfma(e, v, acc[c]);
    }
  }
  double2* out = a.Sp + static_cast<size_t>(b) * 6 * a.Kp + kk;
#pragma unroll
  for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * a.Kp] = acc[c];
}

// Interpolation (m2m), separable in registers: thread per (parent box, band
// of kUpColBand parent theta rows, component, parent phi column). For each
// child it interpolates in phi each child theta row the band needs (3 taps;
// kept in the thread's own shared-memory slots, so no barrier), then forms
// the band's parent directions from 3 theta taps each, times the child's
// shift phase, accumulated over the children. About 5.5 loads per output
// against 10 for the 9-tap gather.
template <class C>
struct UpColArg {
  const C* Sc;
  C* Sp;
  const int* child_begin;
  const int* octant;
  const int* pidx;
  const double* lp;
  const double* lt;
  const int* row_ptr;  // per band: the child theta rows it needs
  const int* row;
  const int* tpos;     // [nthp][3]: band row of each theta tap
  const C* ph_up;
  int nthp, nphp, nphc, Kc;
};

template <class C>
__global__ void __launch_bounds__(kThreads) up_col_kernel(UpColArg<C> a) {
  using R = typename Cx<C>::real;
  __shared__ C rv[kUpColRows][kThreads];
  const int P = blockIdx.x, bi = blockIdx.y;
  const int q = blockIdx.z * blockDim.x + threadIdx.x;
  if (q >= 6 * a.nphp) return;
  const int c = q / a.nphp, p = q - c * a.nphp;
  const int t0 = bi * kUpColBand, nt = min(kUpColBand, a.nthp - t0);
  const int r0 = a.row_ptr[bi], nr = a.row_ptr[bi + 1] - r0;
  int pj[3];
  R wp[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    pj[j] = __ldg(a.pidx + 3 * p + j);
    wp[j] = static_cast<R>(__ldg(a.lp + 3 * p + j));
  }
  int tp[kUpColBand][3];
  R wt[kUpColBand][3];
#pragma unroll
  for (int t = 0; t < kUpColBand; ++t)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const bool in = t < nt;
      tp[t][i] = in ? __ldg(a.tpos + 3 * (t0 + t) + i) : 0;
      wt[t][i] = in ? static_cast<R>(__ldg(a.lt + 3 * (t0 + t) + i)) : R(0);
    }
  int rowoff[kUpColRows];
#pragma unroll
  for (int r = 0; r < kUpColRows; ++r) rowoff[r] = r < nr ? __ldg(a.row + r0 + r) * a.nphc : 0;
  C acc[kUpColBand];
#pragma unroll
  for (int t = 0; t < kUpColBand; ++t) acc[t] = Cx<C>::zero();
  const int Kp = a.nthp * a.nphp;
  C(*mine)[kThreads] = rv;
  const int me = threadIdx.x;
  const int c1 = a.child_begin[P + 1];
  for (int ch = a.child_begin[P]; ch < c1; ++ch) {
    const C* sc = a.Sc + (static_cast<size_t>(ch) * 6 + c) * a.Kc;
#pragma unroll
    for (int r = 0; r < kUpColRows; ++r) {
      if (r < nr) {
        const C* srow = sc + rowoff[r];
        C v = cscale(__ldg(srow + pj[0]), wp[0]);
        v = cfmas(wp[1], __ldg(srow + pj[1]), v);
        v = cfmas(wp[2], __ldg(srow + pj[2]), v);
        mine[r][me] = v;
      }
    }
    const C* ph = a.ph_up + a.octant[ch] * Kp + t0 * a.nphp + p;
#pragma unroll
    for (int t = 0; t < kUpColBand; ++t) {
      if (t < nt) {
        C v = cscale(mine[tp[t][0]][me], wt[t][0]);
        v = cfmas(wt[t][1], mine[tp[t][1]][me], v);
        v = cfmas(wt[t][2], mine[tp[t][2]][me], v);
        acc[t] = cfma(__ldg(ph + t * a.nphp), v, acc[t]);
      }
    }
  }
  C* out = a.Sp + (static_cast<size_t>(P) * 6 + c) * Kp + t0 * a.nphp + p;
#pragma unroll
  for (int t = 0; t < kUpColBand; ++t)
    if (t < nt) out[t * a.nphp] = acc[t];
}

struct UpSepArg {
  const double2* Sc;   // child level patterns [Bc][6][Kc]
  double2* Sp;         // parent level patterns [Bp][6][Kp]
  const int* child_begin;
  const int* octant;   // of child boxes
  const int* pidx;     // [nphp][3] into the child phi grid
  const double* lp;
  const double* lt;    // [nthp][3]
  const int* row_ptr;  // per band: child theta rows it needs
  const int* row;
  const int* tpos;     // [nthp][3]: band row of each theta tap
  const double2* ph_up;
  int nthp, nphp, nphc, Kc, R;
};

// Interpolation (m2m), separable: CTA per (parent box, component, band of R
// parent theta rows). For each child, the phi interpolation of the child
// rows the band needs goes to shared memory (3 taps), then each parent
// direction takes its 3 theta taps from there, times the child's shift
// phase, accumulated over the children in registers. The reference's 9-tap
// weight is the product of the two 1-D weights (Code/AlgoMLFMM.h:347-351).
__global__ void __launch_bounds__(256) up_sep_kernel(UpSepArg a) {
  __shared__ double2 T[kUpBandEntries];
  const int P = blockIdx.x, c = blockIdx.y, bi = blockIdx.z;
  const int t0 = bi * a.R;
  const int nout = min(a.R, a.nthp - t0) * a.nphp;
  const int r0 = a.row_ptr[bi], nr = a.row_ptr[bi + 1] - r0;
  const int Kp = a.nthp * a.nphp;
  constexpr int kPer = kUpBandOut / 256;
  double2 acc[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) acc[q] = c2(0.0, 0.0);
  const int ch1 = a.child_begin[P + 1];
  for (int ch = a.child_begin[P]; ch < ch1; ++ch) {
    const double2* sc = a.Sc + (static_cast<size_t>(ch) * 6 + c) * a.Kc;
    __syncthreads();
    for (int e = threadIdx.x; e < nr * a.nphp; e += blockDim.x) {
      const int r = e / a.nphp, p = e - r * a.nphp;
      const double2* srow = sc + __ldg(a.row + r0 + r) * a.nphc;
      double2 v = cscale(__ldg(srow + __ldg(a.pidx + 3 * p)), __ldg(a.lp + 3 * p));
      v = cfmas(__ldg(a.lp + 3 * p + 1), __ldg(srow + __ldg(a.pidx + 3 * p + 1)), v);
      v = cfmas(__ldg(a.lp + 3 * p + 2), __ldg(srow + __ldg(a.pidx + 3 * p + 2)), v);
      T[e] = v;
    }
    __syncthreads();
    const double2* ph = a.ph_up + a.octant[ch] * Kp + t0 * a.nphp;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int e = threadIdx.x + q * 256;
      if (e < nout) {
        const int r = e / a.nphp, p = e - r * a.nphp;
        const int t = t0 + r;
        double2 v = cscale(T[__ldg(a.tpos + 3 * t) * a.nphp + p], __ldg(a.lt + 3 * t));
        v = cfmas(__ldg(a.lt + 3 * t + 1), T[__ldg(a.tpos + 3 * t + 1) * a.nphp + p], v);
        v = cfmas(__ldg(a.lt + 3 * t + 2), T[__ldg(a.tpos + 3 * t + 2) * a.nphp + p], v);
        acc[q] = cfma(__ldg(ph + e), v, acc[q]);
      }
    }
  }
  double2* out = a.Sp + (static_cast<size_t>(P) * 6 + c) * Kp + t0 * a.nphp;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int e = threadIdx.x + q * 256;
    if (e < nout) out[e] = acc[q];
  }
}

struct M2lArg {
  const double2* S;     // this level's aggregated patterns
  double2* Bm;          // this level's incoming patterns (written)
  const int* far_ptr;
  const int* far_idx;
  const int* far_off;
  const int* off2vec;
  const double2* tfw;
  int K;
};

// Translation (m2l): one thread per (box, direction); the 6 components of
// each interaction-list source are applied with one transfer-factor load.
// Writes Bm (no accumulation into an earlier value).
__global__ void __launch_bounds__(kThreads) m2l_kernel(M2lArg a) {
  const int kk = blockIdx.y * blockDim.x + threadIdx.x;
  const int b = blockIdx.x;
  if (kk >= a.K) return;
  double2 acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = c2(0.0, 0.0);
  const int e1 = a.far_ptr[b + 1];
  for (int e = a.far_ptr[b]; e < e1; ++e) {
    const int s = a.far_idx[e];
    const double2 tf = a.tfw[static_cast<size_t>(a.off2vec[a.far_off[e]]) * a.K + kk];
    const double2* src = a.S + static_cast<size_t>(s) * 6 * a.K + kk;
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = cfma(tf, src[static_cast<size_t>(c) * a.K], acc[c]);
  }
  double2* out = a.Bm + static_cast<size_t>(b) * 6 * a.K + kk;
#pragma unroll
  for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * a.K] = acc[c];
}

struct M2lTileArg {
  const double2* S;
  double2* Bm;
  const int* child_begin;  // parent level: range of children (the targets)
  const int* usrc_ptr;     // per parent: union of its children's interaction sources
  const int* usrc;
  const int* coord;        // [3 * B] integer box coordinates at this level
  const int* off2vec;
  const double2* tfw;
  int K;
};

constexpr int kTileDirs = 32;   // directions per CTA (one per lane)
constexpr int kTileWarps = 8;   // one warp per child slot of the parent
constexpr int kTileBatch = 14;  // sources staged per round (static shared memory < 48 KB)

// Translation by sibling groups: one CTA per (parent box, 32-direction
// chunk), one warp per child. The union of the children's interaction
// sources (children of the parent's 27-neighbourhood) is staged through
// shared memory in batches, so each source pattern crosses L2 once per
// sibling group instead of once per target. Each warp then applies the
// sources that interact with its child (Chebyshev distance >= 2 in box
// units), in the same ascending source order as m2l_kernel.
__global__ void __launch_bounds__(kTileDirs * kTileWarps) m2l_tile_kernel(M2lTileArg a) {
  __shared__ double2 sS[kTileBatch][6][kTileDirs];
  __shared__ int sSrc[kTileBatch][4];  // x, y, z, box
  __shared__ int sVec[343];
  const int P = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int kk = blockIdx.y * kTileDirs + lane;
  for (int i = threadIdx.x; i < 343; i += blockDim.x) sVec[i] = a.off2vec[i];
  const int c0 = a.child_begin[P], nc = a.child_begin[P + 1] - c0;
  const int t = c0 + w;
  const bool active = w < nc;
  int tx = 0, ty = 0, tz = 0;
  if (active) {
    tx = a.coord[3 * t];
    ty = a.coord[3 * t + 1];
    tz = a.coord[3 * t + 2];
  }
  double2 acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = c2(0.0, 0.0);
  const int u0 = a.usrc_ptr[P], nu = a.usrc_ptr[P + 1] - u0;
  for (int base = 0; base < nu; base += kTileBatch) {
    const int nb = min(kTileBatch, nu - base);
    __syncthreads();
    if (threadIdx.x < nb) {
      const int sb = a.usrc[u0 + base + threadIdx.x];
      sSrc[threadIdx.x][0] = a.coord[3 * sb];
      sSrc[threadIdx.x][1] = a.coord[3 * sb + 1];
      sSrc[threadIdx.x][2] = a.coord[3 * sb + 2];
      sSrc[threadIdx.x][3] = sb;
    }
    // stage nb sources x 6 components x 32 directions (one 512-byte row per warp load)
    for (int row = w; row < nb * 6; row += kTileWarps) {
      const int j = row / 6, c = row - 6 * j;
      const int sb = a.usrc[u0 + base + j];
      sS[j][c][lane] = kk < a.K ? a.S[(static_cast<size_t>(sb) * 6 + c) * a.K + kk] : c2(0.0, 0.0);
    }
    __syncthreads();
    if (active && kk < a.K) {
      for (int j = 0; j < nb; ++j) {
        const int dx = tx - sSrc[j][0], dy = ty - sSrc[j][1], dz = tz - sSrc[j][2];
        if (max(abs(dx), max(abs(dy), abs(dz))) < 2) continue;  // near: not translated
        const int v = sVec[(dx + 3) * 49 + (dy + 3) * 7 + (dz + 3)];
        const double2 tf = __ldg(a.tfw + static_cast<size_t>(v) * a.K + kk);
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[c] = cfma(tf, sS[j][c][lane], acc[c]);
      }
    }
  }
  if (active && kk < a.K) {
    double2* out = a.Bm + static_cast<size_t>(t) * 6 * a.K + kk;
#pragma unroll
    for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * a.K] = acc[c];
  }
}

// Translation by octant registers, all levels of one medium in one launch.
// A CTA takes one parent box and 64 directions; thread (direction, half,
// group) keeps the incoming patterns of 4 of the parent's 8 octant children
// (group 0: octants 0-3, group 1: 4-7) for the J (half 0) or M (half 1)
// components in registers. The union of the children's interaction-list
// sources is staged in shared memory; each source pattern is loaded once per
// thread (the next one prefetched) and applied to every child of the group
// whose list holds it (octant mask), with that child's transfer factor.
constexpr int kM2lDirs = 64;
constexpr int kM2lThreads = 4 * kM2lDirs;
constexpr int kM2lMaxSeg = 14;  // levels 2..15
constexpr int kM2lStage = 512;  // union entries staged per round

struct M2lSeg {
  const double2* S;
  double2* Bm;
  const double2* tfw;
  const int* off2vec;
  const int* ufar_ptr;
  const int* ufar;
  const int* upack;
  const int* child_begin;  // parent level
  const int* octant;       // this level
  int K, nchunk, cta_begin;
};
struct M2lOctArg {
  M2lSeg seg[kM2lMaxSeg];
  int nseg;
};

__global__ void __launch_bounds__(kM2lThreads, 2) m2l_oct_kernel(const __grid_constant__ M2lOctArg a) {
  __shared__ int sVec[343];
  __shared__ int sChild[8];
  __shared__ int sSrc[kM2lStage];
  __shared__ int sPack[kM2lStage];
  int si = 0;
  while (si + 1 < a.nseg && static_cast<int>(blockIdx.x) >= a.seg[si + 1].cta_begin) ++si;
  const M2lSeg& g = a.seg[si];
  const int local = blockIdx.x - g.cta_begin;
  const int P = local / g.nchunk;
  const int k = (local - P * g.nchunk) * kM2lDirs + (threadIdx.x & (kM2lDirs - 1));
  const int h = (threadIdx.x / kM2lDirs) & 1;   // J or M
  const int grp = threadIdx.x / (2 * kM2lDirs);  // octants 4 grp .. 4 grp + 3
  const int K = g.K;
  const bool live = k < K;
  const int kq = live ? k : K - 1;
  for (int i = threadIdx.x; i < 343; i += blockDim.x) sVec[i] = g.off2vec[i];
  if (threadIdx.x < 8) sChild[threadIdx.x] = -1;
  __syncthreads();
  const int c0 = g.child_begin[P], c1 = g.child_begin[P + 1];
  if (threadIdx.x < c1 - c0) sChild[g.octant[c0 + threadIdx.x]] = c0 + threadIdx.x;
  double2 acc[4][3];
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[o][c] = c2(0.0, 0.0);
  const double2* Sbase = g.S + static_cast<size_t>(3 * h) * K + kq;
  const int u0 = g.ufar_ptr[P], nu = g.ufar_ptr[P + 1] - u0;
  for (int base = 0; base < nu; base += kM2lStage) {
    const int nb = min(kM2lStage, nu - base);
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
      sSrc[i] = g.ufar[u0 + base + i];
      sPack[i] = g.upack[u0 + base + i];
    }
    __syncthreads();
    const double2* src = Sbase + static_cast<size_t>(sSrc[0]) * 6 * K;
    double2 n0 = __ldg(src), n1 = __ldg(src + K), n2 = __ldg(src + 2 * K);
    for (int j = 0; j < nb; ++j) {
      const double2 s0 = n0, s1 = n1, s2 = n2;
      if (j + 1 < nb) {
        src = Sbase + static_cast<size_t>(sSrc[j + 1]) * 6 * K;
        n0 = __ldg(src);
        n1 = __ldg(src + K);
        n2 = __ldg(src + 2 * K);
      }
      const int pk = sPack[j];
      const int enc0 = pk & 511;
      const int mask = (pk >> (9 + 4 * grp)) & 15;
      double2 tf[4];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int oo = 4 * grp + o;
        const int v = sVec[enc0 + (oo & 1) * 49 + ((oo >> 1) & 1) * 7 + (oo >> 2)];
        tf[o] = (mask >> o) & 1 ? __ldg(g.tfw + static_cast<size_t>(max(v, 0)) * K + kq) : c2(0.0, 0.0);
      }
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        if ((mask >> o) & 1) {
          acc[o][0] = cfma(tf[o], s0, acc[o][0]);
          acc[o][1] = cfma(tf[o], s1, acc[o][1]);
          acc[o][2] = cfma(tf[o], s2, acc[o][2]);
        }
      }
    }
  }
  __syncthreads();
  if (!live) return;
#pragma unroll
  for (int o = 0; o < 4; ++o) {
    const int t = sChild[4 * grp + o];
    if (t >= 0) {
      double2* out = g.Bm + (static_cast<size_t>(t) * 6 + 3 * h) * K + k;
      out[0] = acc[o][0];
      out[static_cast<size_t>(K)] = acc[o][1];
      out[2 * static_cast<size_t>(K)] = acc[o][2];
    }
  }
}

// Translation, warp per box: a CTA takes 8 Morton-consecutive boxes (one
// warp each) and 32 directions; every level of a medium in one launch. Each
// lane accumulates its box's 6 components over the box's interaction list,
// with one transfer-factor load per entry. Neighbouring boxes' lists hold
// largely the same sources in the same (ascending) order, so the 8 warps
// read the same source patterns at about the same time and L1 serves the
// repeats.
constexpr int kWarpBoxes = 8;

template <class C>
struct M2lWarpSeg {
  const C* S;
  C* Bm;
  const C* tfw;
  const int* far_ptr;
  const int* far_idx;
  const int* far_vec;
  int B, K, nchunk, cta_begin;
};
template <class C>
struct M2lWarpArg {
  M2lWarpSeg<C> seg[kM2lMaxSeg];
  int nseg;
};

template <class C>
__global__ void __launch_bounds__(32 * kWarpBoxes) m2l_warp_kernel(const __grid_constant__ M2lWarpArg<C> a) {
  int si = 0;
  while (si + 1 < a.nseg && static_cast<int>(blockIdx.x) >= a.seg[si + 1].cta_begin) ++si;
  const M2lWarpSeg<C>& g = a.seg[si];
  const int local = blockIdx.x - g.cta_begin;
  const int grp = local / g.nchunk;
  const int b = grp * kWarpBoxes + (threadIdx.x >> 5);
  const int k = (local - grp * g.nchunk) * 32 + (threadIdx.x & 31);
  const int K = g.K;
  if (b >= g.B || k >= K) return;
  C acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = Cx<C>::zero();
  const int e1 = g.far_ptr[b + 1];
  int e = g.far_ptr[b];
  for (; e + 1 < e1; e += 2) {
    const int s0 = __ldg(g.far_idx + e), s1 = __ldg(g.far_idx + e + 1);
    const C t0 = __ldg(g.tfw + static_cast<size_t>(__ldg(g.far_vec + e)) * K + k);
    const C t1 = __ldg(g.tfw + static_cast<size_t>(__ldg(g.far_vec + e + 1)) * K + k);
    const C* p0 = g.S + static_cast<size_t>(s0) * 6 * K + k;
    const C* p1 = g.S + static_cast<size_t>(s1) * 6 * K + k;
    C v0[6], v1[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      v0[c] = __ldg(p0 + static_cast<size_t>(c) * K);
      v1[c] = __ldg(p1 + static_cast<size_t>(c) * K);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = cfma(t1, v1[c], cfma(t0, v0[c], acc[c]));
  }
  if (e < e1) {
    const int s0 = __ldg(g.far_idx + e);
    const C t0 = __ldg(g.tfw + static_cast<size_t>(__ldg(g.far_vec + e)) * K + k);
    const C* p0 = g.S + static_cast<size_t>(s0) * 6 * K + k;
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = cfma(t0, __ldg(p0 + static_cast<size_t>(c) * K), acc[c]);
  }
  C* out = g.Bm + static_cast<size_t>(b) * 6 * K + k;
#pragma unroll
  for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * K] = acc[c];
}

struct L2lArg {
  double2* Bm;           // child level (accumulated into)
  const double2* Bp;     // parent level
  const int* parent;     // of child boxes
  const int* octant;     // of child boxes
  const double2* ph_dn;  // parent level table [8][Kp]
  const int* tr_ptr;     // child direction -> (parent direction, weight)
  const int* tr_kp;
  const double* tr_w;
  int K, Kp;
};

// Anterpolation (l2l): one thread per (child box, child direction,
// component) adds the parent's incoming pattern, shifted to the child centre
// and interpolated transposed onto the child grid.
__global__ void __launch_bounds__(kThreads) l2l_kernel(L2lArg a) {
  const int kk = blockIdx.y * blockDim.x + threadIdx.x;
  const int b = blockIdx.x;
  const int c = blockIdx.z;
  if (kk >= a.K) return;
  const double2* ph = a.ph_dn + a.octant[b] * a.Kp;
  const double2* bp = a.Bp + (static_cast<size_t>(a.parent[b]) * 6 + c) * a.Kp;
  double2 acc = c2(0.0, 0.0);
  const int t1 = a.tr_ptr[kk + 1];
  for (int e = a.tr_ptr[kk]; e < t1; ++e) {
    const int kp = __ldg(a.tr_kp + e);
    acc = cfma(cscale(__ldg(ph + kp), __ldg(a.tr_w + e)), __ldg(bp + kp), acc);
  }
  double2* out = a.Bm + (static_cast<size_t>(b) * 6 + c) * a.K + kk;
  *out = cadd(*out, acc);
}

// Translation, warp per box pair: a CTA takes 4 pairs of Morton-consecutive
// boxes (2g, 2g+1; mostly siblings) and 32 directions. A lane walks the
// pair's merged, source-ordered interaction lists: each source pattern is
// loaded once and applied to whichever of the two boxes lists it, with that
// box's transfer factor. Each box sums its sources in ascending order (kSplit: each
// warp's every kW-th entry in that order, then the warps).
constexpr int kPairWarps = 4;

template <class C>
struct M2lPairSeg {
  const C* S;
  C* Bm;
  const C* tfw;
  const int* pair_ptr;
  const int* pair_src;
  const int2* pair_vec;
  int B, K, nchunk, cta_begin;
  long long slot_S = 0, slot_B = 0;  // element strides between right-hand-side slots (grid.y = slots)
};
template <class C>
struct M2lPairArg {
  M2lPairSeg<C> seg[kM2lMaxSeg];
  int nseg;
};

// kSlots: the slot offsets of the batched tree (grid.y = slot); the single
// apply instantiates without them.
// kW: box pairs (warps) per CTA.
// Off: the type of byte offsets into a level's arrays; with 32 bits (arrays
// below 4 GB) the 6 components share one offset and their base pointers are
// uniform, which takes a quarter of the instructions off the loop.
// FP64 is bound by latency and L1 (96 registers, five CTAs per SM), complex64
// by instruction issue (74 % active before, half of it multiply-adds). One B200,
// translation of all levels and both media: FP64 at 245,760 unknowns 2.27 ->
// 2.05 ms, 16 slots of complex64 at 61,440 5.38 -> 4.24 ms. Two directions per
// lane (16-byte loads) in complex64: 4.45 ms, too few warps.
template <class C, class Off>
__device__ __forceinline__ C load_at(const C* base, Off byte) {
  return __ldg(reinterpret_cast<const C*>(reinterpret_cast<const char*>(base) + byte));
}

// kSplit: the CTA's warps share one pair, each walking every kW-th entry, and
// meet in shared memory (see kSplitWarps).
template <class C, bool kSlots, int kW, class Off, bool kSplit>
__global__ void __launch_bounds__(32 * kW, (sizeof(C) == 16 ? 640 : 1024) / (32 * kW))
    m2l_pair_kernel(const __grid_constant__ M2lPairArg<C> a) {
  int si = 0;
  while (si + 1 < a.nseg && static_cast<int>(blockIdx.x) >= a.seg[si + 1].cta_begin) ++si;
  const M2lPairSeg<C>& g = a.seg[si];
  const int local = blockIdx.x - g.cta_begin;
  const int grp = local / g.nchunk;
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pg = kSplit ? grp : grp * kW + wp;
  const int K = g.K;
  const int k0 = (local - grp * g.nchunk) * 32 + lane;
  if (!kSplit && (2 * pg >= g.B || k0 >= K)) return;
  const int k = kSplit ? min(k0, K - 1) : k0;
  constexpr int kStep = kSplit ? kW : 1;
  const C* const Sl = kSlots ? g.S + blockIdx.y * g.slot_S : g.S;
  C* const Bl = kSlots ? g.Bm + blockIdx.y * g.slot_B : g.Bm;
  C a0[6], a1[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) a0[c] = a1[c] = Cx<C>::zero();
  // The next entry's source and factor rows are read one entry ahead, and an
  // entry's 6 pattern and up to 2 factor values are requested together: one
  // memory latency per entry instead of three (indices, then the patterns and
  // the first box's factor, then the second's behind its branch).
  const int e1 = g.pair_ptr[pg + 1];
  int e = g.pair_ptr[pg] + (kSplit ? wp : 0);
  int src = e < e1 ? __ldg(g.pair_src + e) : 0;
  int2 v = e < e1 ? __ldg(g.pair_vec + e) : make_int2(-1, -1);
  const Off row = static_cast<Off>(K) * static_cast<Off>(sizeof(C)), at = static_cast<Off>(k) * static_cast<Off>(sizeof(C));
  while (e < e1) {
    const Off o = static_cast<Off>(src) * (6 * row) + at;
    C sv[6], t0, t1;
#pragma unroll
    for (int c = 0; c < 6; ++c) sv[c] = load_at(Sl + static_cast<size_t>(c) * K, o);
    const bool in0 = v.x >= 0, in1 = v.y >= 0;
    if (in0) t0 = load_at(g.tfw, static_cast<Off>(v.x) * row + at);
    if (in1) t1 = load_at(g.tfw, static_cast<Off>(v.y) * row + at);
    if ((e += kStep) < e1) {
      src = __ldg(g.pair_src + e);
      v = __ldg(g.pair_vec + e);
    }
    if (in0) {
#pragma unroll
      for (int c = 0; c < 6; ++c) a0[c] = cfma(t0, sv[c], a0[c]);
    }
    if (in1) {
#pragma unroll
      for (int c = 0; c < 6; ++c) a1[c] = cfma(t1, sv[c], a1[c]);
    }
  }
  if constexpr (kSplit) {
    static_assert(12 % kW == 0, "every warp adds up as many components");
    __shared__ C part[kW][12][32];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      part[wp][c][lane] = a0[c];
      part[wp][6 + c][lane] = a1[c];
    }
    __syncthreads();
    if (k0 >= K) return;
#pragma unroll
    for (int i = 0; i < 12 / kW; ++i) {
      const int c = wp * (12 / kW) + i, box = 2 * pg + c / 6;
      C v = part[0][c][lane];
#pragma unroll
      for (int q = 1; q < kW; ++q) v = cadd(v, part[q][c][lane]);
      if (box < g.B) Bl[(static_cast<size_t>(box) * 6 + c % 6) * K + k] = v;
    }
    return;
  }
  C* out0 = Bl + static_cast<size_t>(2 * pg) * 6 * K + k;
#pragma unroll
  for (int c = 0; c < 6; ++c) out0[static_cast<size_t>(c) * K] = a0[c];
  if (2 * pg + 1 < g.B) {
    C* out1 = Bl + static_cast<size_t>(2 * pg + 1) * 6 * K + k;
#pragma unroll
    for (int c = 0; c < 6; ++c) out1[static_cast<size_t>(c) * K] = a1[c];
  }
}

// The same walk with each pair's J and M halves on two warps: a CTA of 8
// warps takes 4 pairs x {J, M}; a lane keeps 3 components of both boxes
// (half the registers of m2l_pair_kernel, twice the resident warps), and
// the transfer factors the two halves both load come from L1.
template <class C>
__global__ void __launch_bounds__(64 * kPairWarps) m2l_pairh_kernel(const __grid_constant__ M2lPairArg<C> a) {
  int si = 0;
  while (si + 1 < a.nseg && static_cast<int>(blockIdx.x) >= a.seg[si + 1].cta_begin) ++si;
  const M2lPairSeg<C>& g = a.seg[si];
  const int local = blockIdx.x - g.cta_begin;
  const int grp = local / g.nchunk;
  const int w = threadIdx.x >> 5;
  const int pg = grp * kPairWarps + (w >> 1), h = w & 1;
  const int k = (local - grp * g.nchunk) * 32 + (threadIdx.x & 31);
  const int K = g.K;
  if (2 * pg >= g.B || k >= K) return;
  C a0[3], a1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) a0[c] = a1[c] = Cx<C>::zero();
  const int e1 = g.pair_ptr[pg + 1];
  for (int e = g.pair_ptr[pg]; e < e1; ++e) {
    const int src = __ldg(g.pair_src + e);
    const int2 v = __ldg(g.pair_vec + e);
    const C* p = g.S + (static_cast<size_t>(src) * 6 + 3 * h) * K + k;
    C sv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) sv[c] = __ldg(p + static_cast<size_t>(c) * K);
    if (v.x >= 0) {
      const C t = __ldg(g.tfw + static_cast<size_t>(v.x) * K + k);
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = cfma(t, sv[c], a0[c]);
    }
    if (v.y >= 0) {
      const C t = __ldg(g.tfw + static_cast<size_t>(v.y) * K + k);
#pragma unroll
      for (int c = 0; c < 3; ++c) a1[c] = cfma(t, sv[c], a1[c]);
    }
  }
  C* out0 = g.Bm + (static_cast<size_t>(2 * pg) * 6 + 3 * h) * K + k;
#pragma unroll
  for (int c = 0; c < 3; ++c) out0[static_cast<size_t>(c) * K] = a0[c];
  if (2 * pg + 1 < g.B) {
    C* out1 = g.Bm + (static_cast<size_t>(2 * pg + 1) * 6 + 3 * h) * K + k;
#pragma unroll
    for (int c = 0; c < 3; ++c) out1[static_cast<size_t>(c) * K] = a1[c];
  }
}

// Tile shapes chosen at run time (tuning keys "m2l.pair_warps", "up.threads").
inline int pair_warps(const Plan& P) { return 2 << P.tuning.m2l_pair_warps; }
inline int up_threads(const Plan& P) { return 64 << P.tuning.up_threads; }

// FP64 launches of fewer warps than this (5 per SM) share each pair's list among
// the warps of a CTA: a warp walks ~70 entries at ~0.3 us each with nothing beside
// it, so both translations of a plan of 56 boxes took 23 us, and take 9.5 split
// (apply at 960 unknowns 54.5 -> 41.7 us alone, 27.3 -> 24.6 among others). With
// the line at 10 or 20 warps per SM the kernels of an apply at 7,260 unknowns
// shorten too (204 -> 159 and 124 us in all), but the apply does not (231 -> 234
// and 239 us). Complex64 stays unsplit: its batched form sums whole lists, and a
// slot equals the single apply to rounding of identical operations.
constexpr int kSplitWarps = 148 * 5;

template <class C, bool kSlots, class Off>
void launch_m2l_pair_as(int w, bool split, dim3 grid, const M2lPairArg<C>& a, cudaStream_t st) {
  if constexpr (!kSlots && sizeof(C) == 16) {
    if (split) {
      m2l_pair_kernel<C, false, kPairWarps, Off, true><<<grid, 32 * kPairWarps, 0, st>>>(a);
      return;
    }
  }
  if (w == 2)
    m2l_pair_kernel<C, kSlots, 2, Off, false><<<grid, 64, 0, st>>>(a);
  else if (w == 8)
    m2l_pair_kernel<C, kSlots, 8, Off, false><<<grid, 256, 0, st>>>(a);
  else
    m2l_pair_kernel<C, kSlots, 4, Off, false><<<grid, 128, 0, st>>>(a);
}

// The segments of `a` (cta_begin set here) for `slots` right-hand-side slots.
template <class C, bool kSlots>
void launch_m2l_pair(const Plan& P, M2lPairArg<C>& a, int slots, cudaStream_t st) {
  bool small = true;  // every level's patterns and factors within 32-bit byte offsets
  long long warps = 0;
  for (int i = 0; i < a.nseg; ++i) {
    const size_t row = sizeof(C) * static_cast<size_t>(a.seg[i].K);
    small = small && row * 6 * static_cast<size_t>(a.seg[i].B) < (1ull << 32) && row * 343 < (1ull << 32);
    warps += static_cast<long long>((a.seg[i].B + 1) / 2) * a.seg[i].nchunk;
  }
  const bool split = sizeof(C) == 16 && warps < kSplitWarps;
  const int w = pair_warps(P), per = split ? 1 : w;
  int ctas = 0;
  for (int i = 0; i < a.nseg; ++i) {
    a.seg[i].cta_begin = ctas;
    ctas += (((a.seg[i].B + 1) / 2 + per - 1) / per) * a.seg[i].nchunk;
  }
  if (small)
    launch_m2l_pair_as<C, kSlots, uint32_t>(w, split, dim3(ctas, slots), a, st);
  else
    launch_m2l_pair_as<C, kSlots, size_t>(w, split, dim3(ctas, slots), a, st);
}

// Translation with staged sources: a CTA takes a group of 8 Morton-
// consecutive boxes and 32 directions. The group's interaction lists are
// merged into one source-ordered union whose entries carry the transfer-
// factor row of each member that lists the source. A producer warp stages,
// per union entry, the source's 6 pattern rows (one tiled TMA copy of a
// 6-row box) and the listed members' transfer-factor rows (two tile::gather4
// copies of 4 rows each) for 32 directions into a ring of shared-memory
// stages, completing on the stage's mbarrier, kGrpStages entries ahead of the
// arithmetic. kGrpBoxes / kBW compute warps, one direction per lane, apply
// every staged entry to their kBW boxes from shared memory only: no compute
// warp waits on a global load. A source pattern crosses L2 once per group
// instead of once per box pair. Each box still sums its sources in ascending
// order.
constexpr int kGrpBoxes = 8;
constexpr int kGrpDirs = 32;
constexpr int kGrpStages = 6;
constexpr int kGrpRows = 6 + kGrpBoxes;  // staged rows per entry: 6 pattern components, 8 transfer factors
constexpr int kGrpMaxSeg = 8;            // levels per launch

template <class C>
struct M2lGrpSeg {
  CUtensorMap smap;  // the level's patterns as rows [B * 6][2K] of scalars, box 2 * kGrpDirs x 6
  const C* S;
  const C* tfw;
  C* Bm;
  const int* grp_ptr;
  const int* grp_src;
  const int4* grp_code;
  int B, K, G, nchunk, cta_begin;
};
template <class C>
struct M2lGrpArg {
  M2lGrpSeg<C> seg[kGrpMaxSeg];
  int nseg;
  int* status;
};

template <class C>
constexpr size_t grp_smem_bytes() {
  return static_cast<size_t>(kGrpStages) * kGrpRows * kGrpDirs * sizeof(C) + kGrpStages * sizeof(int4) +
         2 * kGrpStages * sizeof(uint64_t);
}

__device__ __forceinline__ int grp_field(const int4& w, int j) {
  const int v = (j >> 1) == 0 ? w.x : (j >> 1) == 1 ? w.y : (j >> 1) == 2 ? w.z : w.w;
  return (j & 1) ? (v >> 16) : static_cast<int>(static_cast<short>(v & 0xffff));
}

template <class C, int kBW, bool kTmaS>
__global__ void __launch_bounds__(32 * (kGrpBoxes / kBW + 1)) m2l_grp_kernel(const __grid_constant__ M2lGrpArg<C> a) {
  constexpr int kCW = kGrpBoxes / kBW;  // compute warps; warp kCW is the producer
  constexpr uint32_t kRowBytes = kGrpDirs * sizeof(C);
  extern __shared__ __align__(128) unsigned char smem[];
  C* stage = reinterpret_cast<C*>(smem);  // [kGrpStages][kGrpRows][kGrpDirs]
  int4* codes = reinterpret_cast<int4*>(smem + static_cast<size_t>(kGrpStages) * kGrpRows * kRowBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(codes + kGrpStages);
  uint64_t* empty = full + kGrpStages;

  int si = 0;
  while (si + 1 < a.nseg && static_cast<int>(blockIdx.x) >= a.seg[si + 1].cta_begin) ++si;
  const M2lGrpSeg<C>& g = a.seg[si];
  const int local = blockIdx.x - g.cta_begin;
  const int chunk = local / g.G, grp = local - chunk * g.G;
  const int k0 = chunk * kGrpDirs;
  const int nk = min(kGrpDirs, g.K - k0);
  const int e0 = g.grp_ptr[grp], n = g.grp_ptr[grp + 1] - e0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (status_now(a.status) != 0) return;  // an earlier wait ran out: the output is void anyway
  if (threadIdx.x == 0) {
    for (int i = 0; i < kGrpStages; ++i) {
      mbar_init(full + i, 33);  // the producer's 32 lanes after their copies, and lane 0 with the codes
      mbar_init(empty + i, kCW);
    }
    mbar_init_fence();
  }
  __syncthreads();

  if (warp == kCW) {  // producer
    if (kTmaS && lane == 0) tma_prefetch_map(&g.smap);
    bool ok = true;
    int i = 0;
    for (int base = 0; base < n && ok; base += 32) {
      int src = 0;
      int4 cd = make_int4(-1, -1, -1, -1);
      if (base + lane < n) {
        src = __ldg(g.grp_src + e0 + base + lane);
        cd = __ldg(g.grp_code + e0 + base + lane);
      }
      const int cnt = min(32, n - base);
      for (int j = 0; j < cnt; ++j, ++i) {
        const int sj = __shfl_sync(0xffffffffu, src, j);
        const int4 cj = make_int4(__shfl_sync(0xffffffffu, cd.x, j), __shfl_sync(0xffffffffu, cd.y, j),
                                  __shfl_sync(0xffffffffu, cd.z, j), __shfl_sync(0xffffffffu, cd.w, j));
        const int st = i % kGrpStages;
        const bool waited =
            i < kGrpStages || mbar_wait(empty + st, ((i / kGrpStages) - 1) & 1, a.status, true, kStatusM2lGrp);
        if (!__all_sync(0xffffffffu, waited)) {
          ok = false;
          break;
        }
        C* dst = stage + st * kGrpRows * kGrpDirs;
        if (lane == 0) {  // the codes, released to the compute warps by this arrival
          codes[st] = cj;
          if (kTmaS) {
            mbar_arrive_expect_tx(full + st, 6 * kRowBytes);
            tma_load_2d(dst, &g.smap, 2 * k0, 6 * sj, full + st);
          } else {
            mbar_arrive(full + st);
          }
        }
        if (lane < nk) {
          if (!kTmaS) {
            const C* p = g.S + static_cast<size_t>(sj) * 6 * g.K + k0 + lane;
#pragma unroll
            for (int c = 0; c < 6; ++c) cp_async_ca<sizeof(C)>(dst + c * kGrpDirs + lane, p + static_cast<size_t>(c) * g.K);
          }
#pragma unroll
          for (int b = 0; b < kGrpBoxes; ++b) {
            const int code = grp_field(cj, b);
            if (code >= 0)
              cp_async_ca<sizeof(C)>(dst + (6 + b) * kGrpDirs + lane, g.tfw + static_cast<size_t>(code) * g.K + k0 + lane);
          }
        }
        cp_async_arrive(full + st);
      }
    }
    // the copies still in flight land before the producer leaves, so that the
    // CTA never ends (a compute warp may give up after a failed wait) with a
    // copy into its shared memory outstanding
    if (lane == 0)
      for (int q = max(0, i - kGrpStages); q < i; ++q)
        mbar_wait(full + q % kGrpStages, (q / kGrpStages) & 1, a.status, false, kStatusM2lGrp);
    return;
  }

  const int k = k0 + lane;
  C acc[kBW][6];
#pragma unroll
  for (int j = 0; j < kBW; ++j)
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[j][c] = Cx<C>::zero();
  bool ok = true;
  for (int i = 0; i < n; ++i) {
    const int st = i % kGrpStages;
    if (!mbar_wait(full + st, (i / kGrpStages) & 1, a.status, true, kStatusM2lGrp)) {
      ok = false;
      break;
    }
    const int4 cw = codes[st];
    const C* sp = stage + st * kGrpRows * kGrpDirs + lane;
    unsigned mask = 0;  // this warp's boxes that list the source (warp-uniform)
#pragma unroll
    for (int j = 0; j < kBW; ++j) mask |= (grp_field(cw, warp * kBW + j) >= 0 ? 1u : 0u) << j;
    if (mask != 0) {
      C sv[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) sv[c] = sp[c * kGrpDirs];
#pragma unroll
      for (int j = 0; j < kBW; ++j) {
        if (mask & (1u << j)) {
          const C t = sp[(6 + warp * kBW + j) * kGrpDirs];
#pragma unroll
          for (int c = 0; c < 6; ++c) acc[j][c] = cfma(t, sv[c], acc[j][c]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + st);
  }
  if (!ok || lane >= nk) return;
#pragma unroll
  for (int j = 0; j < kBW; ++j) {
    const int b = grp * kGrpBoxes + warp * kBW + j;
    if (b < g.B) {
      C* out = g.Bm + static_cast<size_t>(b) * 6 * g.K + k;
#pragma unroll
      for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * g.K] = acc[j][c];
    }
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    MLFMA_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || p == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// A 2-D tensor map over rows of K complex values (2K scalars each) with a
// box of 2 * kGrpDirs scalars by box_rows rows.
template <class C>
CUtensorMap rows_tensor_map(const C* base, int K, long long rows, int box_rows) {
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (static_cast<size_t>(K) * sizeof(C)) % 16 != 0)
    throw std::runtime_error("tensor map: rows not 16-byte aligned");
  CUtensorMap m;
  const cuuint64_t dims[2] = {2ull * static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * sizeof(C)};
  const cuuint32_t box[2] = {2 * kGrpDirs, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = tensor_map_encoder()(
      &m, sizeof(C) == 16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
      const_cast<C*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed: " + std::to_string(r));
  return m;
}

// Segments (levels lo..hi) of staged-group translation launches, at most
// kGrpMaxSeg levels per launch. tf_at(l) gives the level's transfer-factor
// table and row count.
template <class C, class SAt, class BAt, class TfAt>
void launch_m2l_grp(Plan& P, int lo, int hi, int bw, bool tma_s, SAt S_at, BAt B_at, TfAt tf_at, cudaStream_t s) {
  static_assert(grp_smem_bytes<double2>() <= 48 * 1024, "staged translation needs the opt-in shared memory size");
  constexpr size_t smem = grp_smem_bytes<C>();
  for (int l0 = lo; l0 <= hi; l0 += kGrpMaxSeg) {
    M2lGrpArg<C> a{};
    a.status = P.d_status;
    int ctas = 0;
    for (int l = l0; l <= std::min(hi, l0 + kGrpMaxSeg - 1); ++l) {
      const auto tf = tf_at(l);  // (table, rows, K)
      M2lGrpSeg<C>& g = a.seg[a.nseg++];
      if (tma_s) g.smap = rows_tensor_map<C>(S_at(l), std::get<2>(tf), 6LL * P.lv[l].B, 6);
      g.S = S_at(l);
      g.tfw = std::get<0>(tf);
      g.Bm = B_at(l);
      g.grp_ptr = P.lv[l].grp_ptr;
      g.grp_src = P.lv[l].grp_src;
      g.grp_code = P.lv[l].grp_code;
      g.B = P.lv[l].B;
      g.K = std::get<2>(tf);
      g.G = (P.lv[l].B + kGrpBoxes - 1) / kGrpBoxes;
      g.nchunk = (g.K + kGrpDirs - 1) / kGrpDirs;
      g.cta_begin = ctas;
      ctas += g.G * g.nchunk;
    }
    if (tma_s)
      m2l_grp_kernel<C, 4, true><<<ctas, 32 * (kGrpBoxes / 4 + 1), smem, s>>>(a);
    else if (bw == 4)
      m2l_grp_kernel<C, 4, false><<<ctas, 32 * (kGrpBoxes / 4 + 1), smem, s>>>(a);
    else
      m2l_grp_kernel<C, 2, false><<<ctas, 32 * (kGrpBoxes / 2 + 1), smem, s>>>(a);
    MLFMA_CUDA(cudaGetLastError());
  }
}

template <class C>
struct L2lSepArg {
  C* Bm;                 // child level (accumulated into)
  const C* Bp;     // parent level
  const int* parent;     // of child boxes
  const int* octant;     // of child boxes
  const C* ph_dn;        // parent level table [8][Kp]
  const int* th_ptr;     // pairs of child theta rows: groups of two taps (MediumLevel::th2_*)
  const int2* th_row;
  const double2* th_w;
  const int* ph_ptr;     // child phi columns: groups of two taps (MediumLevel::ph2_*)
  const int2* ph_src;
  const double2* ph_w;
  int ntc, npc, ntp, npp;
  long long slot_c = 0, slot_p = 0;  // element strides between right-hand-side slots (grid.z = slots)
};

constexpr int kL2lBand = 2944;     // band entries in shared memory (46 KiB), all 6 components

// child theta rows per band of the separable anterpolation
__host__ __device__ __forceinline__ int l2l_band_rows(int ntc, int npp) {
  return max(1, min(ntc, kL2lBand / (6 * npp)));
}

// CTAs per child box: one per band on levels with few boxes (so that the
// level fills the GPU), else one CTA walks all the bands of its box.
constexpr int kL2lSplitBoxes = 1024;
inline int l2l_grid_y(int boxes, int ntc, int npp) {
  const int nband = (ntc + l2l_band_rows(ntc, npp) - 1) / l2l_band_rows(ntc, npp);
  return boxes < kL2lSplitBoxes ? nband : 1;
}

// Anterpolation (l2l), separable: a CTA per child box (and, on levels with few
// boxes, per band of child theta rows) does all 6 components. The parent's
// incoming pattern is shifted to the child centre and spread onto the child
// grid by the transposed theta interpolation (into a shared-memory band of
// child rows x parent phi columns x 6 components), then by the transposed phi
// interpolation, and added to the child's Bm. The reference's 9-tap weight of
// a (parent, child) direction pair is the product of the two 1-D weights used
// here (Code/AlgoMLFMM.h:347-351).
// A thread's unit is 3 components (J or M): in theta, one parent column of two
// neighbouring child rows, whose taps overlap (5.3 parent rows instead of 8),
// two taps at a time, so that 8 independent loads are in flight; in phi, one
// child direction, its old values requested before the taps are summed.
// kSlots: grid.z = slots with the slot offsets of the batched tree; the single
// apply instantiates without them.
template <class C, bool kSlots = false>
__global__ void __launch_bounds__(256, sizeof(C) == 16 ? 3 : 4) l2l_sep_kernel(const __grid_constant__ L2lSepArg<C> a) {
  using R = typename Cx<C>::real;
  __shared__ C band[kL2lBand];
  const int b = blockIdx.x;
  const int band_rows = l2l_band_rows(a.ntc, a.npp);
  const unsigned Kp = a.ntp * a.npp, Kc = a.ntc * a.npc;
  const C* ph = a.ph_dn + static_cast<size_t>(a.octant[b]) * Kp;
  const C* bp = (kSlots ? a.Bp + blockIdx.z * a.slot_p : a.Bp) + static_cast<size_t>(a.parent[b]) * 6 * Kp;
  C* out = (kSlots ? a.Bm + blockIdx.z * a.slot_c : a.Bm) + static_cast<size_t>(b) * 6 * Kc;
  for (int tc0 = blockIdx.y * band_rows; tc0 < a.ntc; tc0 += gridDim.y * band_rows) {
    const int rows = min(band_rows, a.ntc - tc0);
    const int stride = rows * a.npp;  // of a component in the band
    const int q0 = tc0 >> 1, nq = ((tc0 + rows - 1) >> 1) - q0 + 1;  // row pairs
    const int half = nq * a.npp;
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * half; e += blockDim.x) {
      const int h = e >= half, ee = e - h * half;
      const int q = ee / a.npp, pp = ee - q * a.npp;
      C v0[3], v1[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v0[c] = v1[c] = Cx<C>::zero();
      const C* bh = bp + h * 3 * Kp;
      const int g1 = __ldg(a.th_ptr + q0 + q + 1);
      for (int g = __ldg(a.th_ptr + q0 + q); g < g1; ++g) {
        const int2 r = __ldg(a.th_row + g);
        const double2 wa = __ldg(a.th_w + 2 * g), wb = __ldg(a.th_w + 2 * g + 1);
        const unsigned ka = r.x + pp, kb = r.y + pp;
        const C ea = __ldg(ph + ka), eb = __ldg(ph + kb);
        C sa[3], sb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sa[c] = __ldg(bh + (c * Kp + ka));
          sb[c] = __ldg(bh + (c * Kp + kb));
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C fa = cmul(ea, sa[c]), fb = cmul(eb, sb[c]);
          v0[c] = cfmas(static_cast<R>(wb.x), fb, cfmas(static_cast<R>(wa.x), fa, v0[c]));
          v1[c] = cfmas(static_cast<R>(wb.y), fb, cfmas(static_cast<R>(wa.y), fa, v1[c]));
        }
      }
      const int r0 = 2 * (q0 + q) - tc0;  // band row of the pair's first child row (-1: before the band)
      C* o = band + 3 * h * stride + r0 * a.npp + pp;
      if (r0 >= 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c * stride] = v0[c];
      if (r0 + 1 < rows)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c * stride + a.npp] = v1[c];
    }
    __syncthreads();
    const int nout = rows * a.npc;
    for (int e = threadIdx.x; e < 2 * nout; e += blockDim.x) {
      const int h = e >= nout, ee = e - h * nout;
      const int r = ee / a.npc, pc = ee - r * a.npc;
      C* o = out + (h * 3 * Kc + static_cast<unsigned>(tc0 * a.npc + ee));
      C v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = o[c * Kc];
      const C* src = band + 3 * h * stride + r * a.npp;
      const int g1 = __ldg(a.ph_ptr + pc + 1);
      for (int g = __ldg(a.ph_ptr + pc); g < g1; ++g) {
        const int2 t = __ldg(a.ph_src + g);
        const double2 w = __ldg(a.ph_w + g);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          v[c] = cfmas(static_cast<R>(w.y), src[c * stride + t.y], cfmas(static_cast<R>(w.x), src[c * stride + t.x], v[c]));
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) o[c * Kc] = v[c];
    }
  }
}

template <class C>
struct LeafArg {
  const C* Vf[2];
  const C* Bm[2];
  const double* khat[2];
  int K[2];
  const int* leaf_rwg;
  const int* leaf_ptr;
  double2* w;
  int N;
  C c1, c2, etai, ietai;
};

template <class C>
__device__ __forceinline__ C warp_sum(C v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// Far-field testing of both media, added to the near-field product already in
// w. With c and e of a medium (c1, 1 or c2, etai),
//   w_J += c sum over directions of Vf . (e B_J - khat x B_M),
//   w_M += c sum over directions of Vf . (khat x B_J + B_M / e),
// because ((-khat) x Vf) . B = Vf . (khat x B) (Code/MLFMM.cpp:285-351). CTA per
// (leaf box, kLeafRows RWGs); its warps take every fourth 32 directions of
// both media, form the bracketed vectors from the box's B in registers, once
// for all the CTA's RWGs, and meet in shared memory at the end.
// HBM-bound: the receive patterns are read once (245,760 unknowns: 4.35 GB,
// 0.65 ms). One B200, this kernel and the near-field product before it against
// one warp per RWG for both: FP64 at 245,760 unknowns 0.98 + 0.28 against 1.29
// ms, at 7,260 40 + 12 against 56 us, complex64 at 61,440 149 + 54 against 217
// us. With 2, 3, 4 and 6 RWGs per CTA the FP64 kernel takes 1.44, 1.11, 1.22 and
// 1.07 ms; with the vectors staged in shared memory for 24 RWGs, 1.37 ms.
constexpr int kLeafRows = 5;
constexpr int kLeafWarps = 4;

template <class C>
__global__ void __launch_bounds__(32 * kLeafWarps, sizeof(C) == 16 ? 3 : 5)
    leaf_rows_kernel(const __grid_constant__ LeafArg<C> a) {
  using R = typename Cx<C>::real;
  __shared__ C red[kLeafWarps][2 * kLeafRows];
  const int b = blockIdx.x;
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  const int t0 = blockIdx.y * kLeafRows;
  if (t0 >= nb) return;
  const int nt = min(kLeafRows, nb - t0);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int n0 = (a.K[0] + 31) / 32, n = n0 + (a.K[1] + 31) / 32;
  C acc[2 * kLeafRows];
#pragma unroll
  for (int i = 0; i < 2 * kLeafRows; ++i) acc[i] = Cx<C>::zero();
  bool second = false;  // the sums are in units of c2 instead of c1
  for (int i = wp; i < n; i += kLeafWarps) {
    const int m = i >= n0, K = a.K[m], k = (i - m * n0) * 32 + lane;
    if (m && !second) {
      const C q = cdiv(a.c1, a.c2);
#pragma unroll
      for (int j = 0; j < 2 * kLeafRows; ++j) acc[j] = cmul(acc[j], q);
      second = true;
    }
    if (k >= K) continue;
    const C* V = a.Vf[m] + (static_cast<size_t>(r0 + t0) * 3) * K + k;
    const C* B = a.Bm[m] + static_cast<size_t>(b) * 6 * K + k;
    C v[kLeafRows][3], f[6];
    R kh[3];
#pragma unroll
    for (int u = 0; u < kLeafRows; ++u)
      if (u < nt)
#pragma unroll
        for (int q = 0; q < 3; ++q) v[u][q] = __ldg(V + (u * 3 + q) * K);
#pragma unroll
    for (int c = 0; c < 6; ++c) f[c] = __ldg(B + c * K);
#pragma unroll
    for (int c = 0; c < 3; ++c) kh[c] = static_cast<R>(__ldg(a.khat[m] + c * K + k));
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
      const C xJ = csub(cscale(f[q2], kh[q1]), cscale(f[q1], kh[q2]));  // khat x B_J
      const C xM = csub(cscale(f[3 + q2], kh[q1]), cscale(f[3 + q1], kh[q2]));
      const C dJ = csub(m ? cmul(a.etai, f[q]) : f[q], xM);
      const C dM = cadd(m ? cmul(a.ietai, f[3 + q]) : f[3 + q], xJ);
#pragma unroll
      for (int u = 0; u < kLeafRows; ++u)
        if (u < nt) {
          acc[2 * u] = cfma(v[u][q], dJ, acc[2 * u]);
          acc[2 * u + 1] = cfma(v[u][q], dM, acc[2 * u + 1]);
        }
    }
  }
  const C c = second ? a.c2 : a.c1;
#pragma unroll
  for (int j = 0; j < 2 * kLeafRows; ++j) {
    const C s = warp_sum(acc[j]);
    if (lane == 0) red[wp][j] = cmul(c, s);
  }
  __syncthreads();
  if (threadIdx.x < 2 * nt) {
    C s = red[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < kLeafWarps; ++q) s = cadd(s, red[q][threadIdx.x]);
    double2* w = a.w + (threadIdx.x & 1) * a.N + a.leaf_rwg[r0 + t0 + (threadIdx.x >> 1)];
    *w = cadd(*w, Cx<C>::to64(s));
  }
}

template <class C>
void launch_leaf(const Plan& P, LeafArg<C>& a, cudaStream_t s) {
  a.ietai = cdiv(Cx<C>::from(c2(1.0, 0.0)), a.etai);
  const dim3 grid(P.lv[P.maxL].B, (P.max_leaf_rwgs + kLeafRows - 1) / kLeafRows);
  leaf_rows_kernel<C><<<grid, 32 * kLeafWarps, 0, s>>>(a);
}

// Leaf-level pattern arrays of a tree pass: the plan's own, or one RHS slot
// of a batched apply. Levels above the leaf always use the plan's arrays.
struct LeafView {
  const double2* S;
  double2* B;
};

const double2* level_S(const Plan& P, int m, int l, const LeafView& v) { return l == P.maxL ? v.S : P.ml[m][l].S; }
double2* level_B(const Plan& P, int m, int l, const LeafView& v) { return l == P.maxL ? v.B : P.ml[m][l].Bm; }

// Interpolation up the tree (levels L-1 .. 2) of medium m.
void launch_up(Plan& P, int m, const LeafView& v, cudaStream_t s) {
  const int L = P.maxL;
  for (int l = L - 1; l >= 2; --l) {
    const MediumLevel& pm = P.ml[m][l];
    const MediumLevel& cm = P.ml[m][l + 1];
    const double2* Sc = level_S(P, m, l + 1, v);
    if (P.tuning.up_variant == 3 && pm.up4_row_ptr) {
      UpColArg<double2> a{Sc,     pm.S,           P.lv[l].child_begin, P.lv[l + 1].octant, pm.pidx, pm.lp,
                          pm.lt,  pm.up4_row_ptr, pm.up4_row,          pm.up4_tpos,        pm.ph_up, pm.nth,
                          pm.nph, cm.nph,         cm.K};
      up_col_kernel<double2>
          <<<dim3(P.lv[l].B, pm.up4_nband, (6 * pm.nph + kThreads - 1) / kThreads), kThreads, 0, s>>>(a);
    } else if (P.tuning.up_variant == 2) {
      UpArg a{Sc, pm.S, P.lv[l].child_begin, P.lv[l + 1].octant, pm.tidx, pm.lt, pm.pidx, pm.lp,
              pm.ph_up, pm.K, pm.nph, cm.K, cm.nph};
      up6_kernel<<<dim3(P.lv[l].B, (pm.K + kThreads - 1) / kThreads), kThreads, 0, s>>>(a);
    } else if (P.tuning.up_variant == 1 && pm.up_rows > 0) {
      UpSepArg a{Sc,    pm.S,     P.lv[l].child_begin, P.lv[l + 1].octant, pm.pidx,
                 pm.lp, pm.lt,    pm.up_row_ptr,       pm.up_row,          pm.up_tpos,
                 pm.ph_up, pm.nth, pm.nph,             cm.nph,             cm.K,
                 pm.up_rows};
      up_sep_kernel<<<dim3(P.lv[l].B, 6, pm.up_nband), 256, 0, s>>>(a);
    } else {
      const Up2Arg<double2> a{Sc,      pm.S,  P.lv[l].child_begin, P.lv[l + 1].octant, pm.up2_row, pm.up2_w, pm.pidx, pm.lp,
                              pm.ph_up, pm.K, pm.nth,              pm.nph,             cm.K};
      launch_up2<double2, false>(up_threads(P), P.lv[l].B, 6, a, s);
    }
  }
}

// Translations of levels lo..hi of medium m (independent of each other).
void launch_m2l(Plan& P, int m, const LeafView& v, cudaStream_t s, int lo, int hi) {
  if (lo > hi) return;
  if (P.tuning.m2l_variant >= 6 && P.tuning.m2l_variant <= 8) {
    launch_m2l_grp<double2>(
        P, lo, hi, P.tuning.m2l_variant == 6 ? 2 : 4, P.tuning.m2l_variant == 8,
        [&](int l) { return level_S(P, m, l, v); },
        [&](int l) { return level_B(P, m, l, v); },
        [&](int l) {
          return std::make_tuple(static_cast<const double2*>(P.ml[m][l].tfw), P.ml[m][l].nvec, P.ml[m][l].K);
        },
        s);
    return;
  }
  if (P.tuning.m2l_variant == 4 || P.tuning.m2l_variant == 5) {
    if (hi - lo + 1 > kM2lMaxSeg) throw std::runtime_error("m2l: more levels than one launch takes");
    M2lPairArg<double2> a{};
    int ctas = 0;
    for (int l = lo; l <= hi; ++l) {
      const MediumLevel& cm = P.ml[m][l];
      M2lPairSeg<double2>& g = a.seg[a.nseg++];
      g = M2lPairSeg<double2>{level_S(P, m, l, v), level_B(P, m, l, v), cm.tfw, P.lv[l].pair_ptr, P.lv[l].pair_src,
                              P.lv[l].pair_vec,    P.lv[l].B,           cm.K,   (cm.K + 31) / 32,  ctas};
      const int G = (P.lv[l].B + 1) / 2;
      ctas += ((G + kPairWarps - 1) / kPairWarps) * g.nchunk;
    }
    if (P.tuning.m2l_variant == 5)
      m2l_pairh_kernel<double2><<<ctas, 64 * kPairWarps, 0, s>>>(a);
    else
      launch_m2l_pair<double2, false>(P, a, 1, s);
    return;
  }
  if (P.tuning.m2l_variant == 3) {
    if (hi - lo + 1 > kM2lMaxSeg) throw std::runtime_error("m2l: more levels than one launch takes");
    M2lWarpArg<double2> a{};
    int ctas = 0;
    for (int l = lo; l <= hi; ++l) {
      const MediumLevel& cm = P.ml[m][l];
      M2lWarpSeg<double2>& g = a.seg[a.nseg++];
      g = M2lWarpSeg<double2>{level_S(P, m, l, v), level_B(P, m, l, v), cm.tfw, P.lv[l].far_ptr, P.lv[l].far_idx,
                     P.lv[l].far_vec, P.lv[l].B, cm.K, (cm.K + 31) / 32, ctas};
      ctas += ((P.lv[l].B + kWarpBoxes - 1) / kWarpBoxes) * g.nchunk;
    }
    m2l_warp_kernel<double2><<<ctas, 32 * kWarpBoxes, 0, s>>>(a);
    return;
  }
  if (P.tuning.m2l_variant == 2) {
    if (hi - lo + 1 > kM2lMaxSeg) throw std::runtime_error("m2l: more levels than one launch takes");
    M2lOctArg a{};
    int ctas = 0;
    for (int l = lo; l <= hi; ++l) {
      const MediumLevel& cm = P.ml[m][l];
      M2lSeg& g = a.seg[a.nseg++];
      g = M2lSeg{level_S(P, m, l, v), level_B(P, m, l, v), cm.tfw, cm.off2vec, P.lv[l].ufar_ptr, P.lv[l].ufar,
                 P.lv[l].upack, P.lv[l - 1].child_begin, P.lv[l].octant, cm.K, (cm.K + kM2lDirs - 1) / kM2lDirs,
                 ctas};
      ctas += P.lv[l - 1].B * g.nchunk;
    }
    m2l_oct_kernel<<<ctas, kM2lThreads, 0, s>>>(a);
    return;
  }
  for (int l = lo; l <= hi; ++l) {
    const MediumLevel& cm = P.ml[m][l];
    if (P.tuning.m2l_variant == 1) {
      M2lTileArg a{level_S(P, m, l, v), level_B(P, m, l, v), P.lv[l - 1].child_begin, P.lv[l].usrc_ptr,
                   P.lv[l].usrc,        P.lv[l].coord,       cm.off2vec,              cm.tfw,
                   cm.K};
      dim3 gd(P.lv[l - 1].B, (cm.K + kTileDirs - 1) / kTileDirs);
      m2l_tile_kernel<<<gd, kTileDirs * kTileWarps, 0, s>>>(a);
    } else {
      M2lArg a{level_S(P, m, l, v), level_B(P, m, l, v), P.lv[l].far_ptr, P.lv[l].far_idx, P.lv[l].far_off,
               cm.off2vec,          cm.tfw,              cm.K};
      dim3 gd(P.lv[l].B, (cm.K + kThreads - 1) / kThreads);
      m2l_kernel<<<gd, kThreads, 0, s>>>(a);
    }
  }
}

// Anterpolation down the tree: level l receives level l-1 once that is final.
void launch_l2l(Plan& P, int m, const LeafView& v, cudaStream_t s) {
  const int L = P.maxL;
  for (int l = 3; l <= L; ++l) {
    const MediumLevel& cm = P.ml[m][l];
    const MediumLevel& pm = P.ml[m][l - 1];
    double2* Bc = level_B(P, m, l, v);
    if (P.tuning.l2l_variant == 1 && 6 * pm.nph <= kL2lBand) {
      L2lSepArg<double2> b{Bc,         pm.Bm,    P.lv[l].parent, P.lv[l].octant, pm.ph_dn, cm.th2_ptr,
                  cm.th2_row, cm.th2_w, cm.ph2_ptr,     cm.ph2_src,     cm.ph2_w, cm.nth,
                  cm.nph,     pm.nth,   pm.nph};
      l2l_sep_kernel<double2><<<dim3(P.lv[l].B, l2l_grid_y(P.lv[l].B, cm.nth, pm.nph)), 256, 0, s>>>(b);
    } else {
      L2lArg b{Bc, pm.Bm, P.lv[l].parent, P.lv[l].octant, pm.ph_dn, cm.tr_ptr, cm.tr_kp, cm.tr_w, cm.K, pm.K};
      dim3 gl(P.lv[l].B, (cm.K + kThreads - 1) / kThreads, 6);
      l2l_kernel<<<gl, kThreads, 0, s>>>(b);
    }
  }
}

template <class Arg>
void fill_leaf_common(const Plan& P, Arg& a) {
  using C = std::remove_reference_t<decltype(a.c1)>;
  a.leaf_rwg = P.d_leaf_rwg;
  a.leaf_ptr = P.d_leaf_ptr;
  a.N = P.N;
  const cplx c1 = P.k1 * P.k1 / (16.0 * kPi * kPi);
  const cplx c2v = P.k2 * P.k2 / (16.0 * kPi * kPi);
  a.c1 = Cx<C>::from(c2(c1.real(), c1.imag()));
  a.c2 = Cx<C>::from(c2(c2v.real(), c2v.imag()));
  a.etai = Cx<C>::from(c2(P.etai.real(), P.etai.imag()));
}

// Medium 1's tree passes go to the plan's second stream, forked from and
// joined back into s; with stage profiling on, both media stay on s so that
// the stage events bracket one medium at a time.
struct MediumStreams {
  Plan& P;
  cudaStream_t s;
  bool two;
  MediumStreams(Plan& P_, cudaStream_t s_, bool concurrent) : P(P_), s(s_), two(concurrent && P_.stream2) {
    if (two) {
      MLFMA_CUDA(cudaEventRecord(P.ev_fork, s));
      MLFMA_CUDA(cudaStreamWaitEvent(P.stream2, P.ev_fork, 0));
    }
  }
  cudaStream_t of(int m) const { return two && m == 1 ? P.stream2 : s; }
  void join() {
    if (two) {
      MLFMA_CUDA(cudaEventRecord(P.ev_join, P.stream2));
      MLFMA_CUDA(cudaStreamWaitEvent(s, P.ev_join, 0));
      two = false;
    }
  }
};

// The near-field product needs only x and writes w, to which the leaf kernel
// adds: with leaf variant 1 it starts at the beginning of the apply on its own
// stream, else it runs before the leaf kernel on the caller's.
struct NearAhead {
  Plan& P;
  cudaStream_t s;
  bool own;
  const double2* x;
  double2* w;
  int prec;
  NearAhead(Plan& P_, cudaStream_t s_, bool own_, const double2* x_, double2* w_, int prec_)
      : P(P_), s(s_), own(own_), x(x_), w(w_), prec(prec_) {
    if (!own) return;
    MLFMA_CUDA(cudaEventRecord(P.ev_start, s));
    MLFMA_CUDA(cudaStreamWaitEvent(P.stream_near, P.ev_start, 0));
    near_apply(P, x, w, P.stream_near, prec);
    MLFMA_CUDA(cudaEventRecord(P.ev_near, P.stream_near));
  }
  void join() {
    if (own)
      MLFMA_CUDA(cudaStreamWaitEvent(s, P.ev_near, 0));
    else
      near_apply(P, x, w, s, prec);
  }
};

cudaEvent_t* profiler_events(Plan& P, cudaStream_t s) {
  if (!P.prof.on) return nullptr;
  if (P.prof.used == P.prof.sets.size()) {
    if (P.prof.sets.size() >= 4096) throw std::runtime_error("stage profiler: read it at least every 4096 applies");
    std::array<cudaEvent_t, StageProfiler::kEvents> set{};
    for (auto& e : set) MLFMA_CUDA(cudaEventCreate(&e));
    P.prof.sets.push_back(set);
  }
  cudaEvent_t* ev = P.prof.sets[P.prof.used++].data();
  MLFMA_CUDA(cudaEventRecord(ev[0], s));
  return ev;
}

// The tree passes of medium m with fixed kernel choices (interpolation 0,
// translation 4, anterpolation 1) for either storage type; leafS / leafB are
// the leaf-level arrays (the plan's own or one batch slot). With a leaf
// stream sx, the leaf level's translation runs there after the aggregation
// (ev_agg) while the interpolation climbs the tree on s; s waits for it
// (ev_leaf) before the anterpolation chain.
template <class C>
void tree_pass_fixed(Plan& P, int m, C* leafS, C* leafB, cudaStream_t s, cudaStream_t sx = nullptr,
                     cudaEvent_t ev_agg = nullptr, cudaEvent_t ev_leaf = nullptr) {
  const int L = P.maxL;
  auto S_at = [&](int l) -> C* { return l == L ? leafS : Store<C>::S(P.ml[m][l]); };
  auto B_at = [&](int l) -> C* { return l == L ? leafB : Store<C>::Bm(P.ml[m][l]); };
  auto translate = [&](int lo, int hi, cudaStream_t st) {
    if (lo > hi) return;
    if (P.tuning.m2l_variant >= 6 && P.tuning.m2l_variant <= 8) {
      launch_m2l_grp<C>(
          P, lo, hi, P.tuning.m2l_variant == 6 ? 2 : 4, P.tuning.m2l_variant == 8, S_at, B_at,
          [&](int l) {
            return std::make_tuple(static_cast<const C*>(Store<C>::tfw(P.ml[m][l])), P.ml[m][l].nvec, P.ml[m][l].K);
          },
          st);
      return;
    }
    if (hi - lo + 1 > kM2lMaxSeg) throw std::runtime_error("m2l: more levels than one launch takes");
    M2lPairArg<C> t{};
    for (int l = lo; l <= hi; ++l) {
      const MediumLevel& cm = P.ml[m][l];
      M2lPairSeg<C>& g = t.seg[t.nseg++];
      g = M2lPairSeg<C>{S_at(l),          B_at(l),   Store<C>::tfw(cm), P.lv[l].pair_ptr, P.lv[l].pair_src,
                        P.lv[l].pair_vec, P.lv[l].B, cm.K,              (cm.K + 31) / 32, 0};
    }
    launch_m2l_pair<C, false>(P, t, 1, st);
  };
  if (sx) {
    MLFMA_CUDA(cudaEventRecord(ev_agg, s));
    MLFMA_CUDA(cudaStreamWaitEvent(sx, ev_agg, 0));
    translate(L, L, sx);
    MLFMA_CUDA(cudaEventRecord(ev_leaf, sx));
  }
  for (int l = L - 1; l >= 2; --l) {
    const MediumLevel& pm = P.ml[m][l];
    const MediumLevel& cm = P.ml[m][l + 1];
    const Up2Arg<C> a{S_at(l + 1), S_at(l), P.lv[l].child_begin, P.lv[l + 1].octant, pm.up2_row, pm.up2_w, pm.pidx, pm.lp,
                      Store<C>::ph_up(pm), pm.K, pm.nth, pm.nph, cm.K};
    launch_up2<C, false>(up_threads(P), P.lv[l].B, 6, a, s);
  }
  if (sx) {
    translate(2, L - 1, s);
    MLFMA_CUDA(cudaStreamWaitEvent(s, ev_leaf, 0));
  } else {
    translate(2, L, s);
  }
  for (int l = 3; l <= L; ++l) {
    const MediumLevel& cm = P.ml[m][l];
    const MediumLevel& pm = P.ml[m][l - 1];
    if (6 * pm.nph > kL2lBand) throw std::runtime_error("anterpolation band: phi grid too large for this precision");
    L2lSepArg<C> b{B_at(l),    B_at(l - 1), P.lv[l].parent, P.lv[l].octant, Store<C>::ph_dn(pm), cm.th2_ptr,
                   cm.th2_row, cm.th2_w,    cm.ph2_ptr,     cm.ph2_src,     cm.ph2_w,            cm.nth,
                   cm.nph,     pm.nth,      pm.nph};
    l2l_sep_kernel<C><<<dim3(P.lv[l].B, l2l_grid_y(P.lv[l].B, cm.nth, pm.nph)), 256, 0, s>>>(b);
  }
}

// The tree passes of medium m for rn right-hand-side slots at once (mixed
// plans): every level's interpolation, translation and anterpolation is one
// launch over all slots of the slot-major arrays btS / btB (the slot is a grid
// dimension), with the kernels of tree_pass_fixed. The leaf level's
// translation runs on sx beside the interpolation chain, as there.
void tree_pass_slots(Plan& P, int m, int rn, cudaStream_t s, cudaStream_t sx, cudaEvent_t ev_agg,
                     cudaEvent_t ev_leaf) {
  using C = float2;
  const int L = P.maxL;
  if (P.btS[m][2] == nullptr) throw std::runtime_error("batched apply: slots of the upper levels not reserved");
  auto stride = [&](int l) { return static_cast<long long>(P.lv[l].B) * 6 * P.ml[m][l].K; };
  auto translate = [&](int lo, int hi, cudaStream_t st) {
    if (lo > hi) return;
    if (hi - lo + 1 > kM2lMaxSeg) throw std::runtime_error("m2l: more levels than one launch takes");
    M2lPairArg<C> t{};
    for (int l = lo; l <= hi; ++l) {
      const MediumLevel& cm = P.ml[m][l];
      M2lPairSeg<C>& g = t.seg[t.nseg++];
      g = M2lPairSeg<C>{P.btS[m][l],      P.btB[m][l], cm.tfw32,          P.lv[l].pair_ptr, P.lv[l].pair_src,
                        P.lv[l].pair_vec, P.lv[l].B,   cm.K,              (cm.K + 31) / 32, 0,
                        stride(l),        stride(l)};
    }
    launch_m2l_pair<C, true>(P, t, rn, st);
    MLFMA_CUDA(cudaGetLastError());
  };
  MLFMA_CUDA(cudaEventRecord(ev_agg, s));
  MLFMA_CUDA(cudaStreamWaitEvent(sx, ev_agg, 0));
  translate(L, L, sx);
  MLFMA_CUDA(cudaEventRecord(ev_leaf, sx));
  for (int l = L - 1; l >= 2; --l) {
    const MediumLevel& pm = P.ml[m][l];
    const MediumLevel& cm = P.ml[m][l + 1];
    const Up2Arg<C> a{P.btS[m][l + 1], P.btS[m][l], P.lv[l].child_begin, P.lv[l + 1].octant, pm.up2_row, pm.up2_w,
                      pm.pidx,         pm.lp,       pm.ph_up32,          pm.K,               pm.nth,     pm.nph,
                      cm.K,            stride(l + 1), stride(l)};
    launch_up2<C, true>(up_threads(P), P.lv[l].B, 6 * rn, a, s);
  }
  translate(2, L - 1, s);
  MLFMA_CUDA(cudaStreamWaitEvent(s, ev_leaf, 0));
  for (int l = 3; l <= L; ++l) {
    const MediumLevel& cm = P.ml[m][l];
    const MediumLevel& pm = P.ml[m][l - 1];
    if (6 * pm.nph > kL2lBand) throw std::runtime_error("anterpolation band: phi grid too large for this precision");
    L2lSepArg<C> b{P.btB[m][l], P.btB[m][l - 1], P.lv[l].parent, P.lv[l].octant, pm.ph_dn32, cm.th2_ptr,
                   cm.th2_row,  cm.th2_w,        cm.ph2_ptr,     cm.ph2_src,     cm.ph2_w,   cm.nth,
                   cm.nph,      pm.nth,          pm.nph,         stride(l),      stride(l - 1)};
    l2l_sep_kernel<C, true><<<dim3(P.lv[l].B, l2l_grid_y(P.lv[l].B, cm.nth, pm.nph), rn), 256, 0, s>>>(b);
  }
  MLFMA_CUDA(cudaGetLastError());
}

template <class C>
void apply_fixed(Plan& P, const double2* x, double2* w, cudaStream_t s) {
  const int L = P.maxL;
  LeafArg<C> a{};
  NearAhead near(P, s, P.tuning.leaf_variant == 1, x, w, std::is_same<C, float2>::value ? 1 : 0);
  MediumStreams ms(P, s, true);
  for (int m = 0; m < 2; ++m) {
    const cudaStream_t sm = ms.of(m);
    const MediumLevel& leaf = P.ml[m][L];
    agg_kernel<C><<<dim3(P.lv[L].B, (leaf.K + kThreads - 1) / kThreads), kThreads, 0, sm>>>(
        Store<C>::Vs(P, m), P.d_leaf_ptr, P.d_leaf_rwg, x, P.N, leaf.K, Store<C>::S(leaf));
    tree_pass_fixed<C>(P, m, Store<C>::S(leaf), Store<C>::Bm(leaf), sm, P.stream_leaf[m], P.ev_agg[m], P.ev_leaf[m]);
    a.Vf[m] = Store<C>::Vf(P, m);
    a.Bm[m] = Store<C>::Bm(leaf);
    a.khat[m] = leaf.khat;
    a.K[m] = leaf.K;
  }
  ms.join();
  near.join();
  fill_leaf_common(P, a);
  a.w = w;
  launch_leaf(P, a, s);
  MLFMA_CUDA(cudaGetLastError());
}

// The batched complex64 apply: leaf stages of leaf_batch.cu (or, with
// batch_tc.variant 1, of agg_tc.cu), tree passes over all slots or slot by
// slot, near-field rows by the tiled product.
void apply_batch_slots(Plan& P, int R, const double2* X, long long ldx, double2* W, long long ldw, cudaStream_t s) {
  using C = float2;
  const int L = P.maxL;
  if (P.bS32[0].empty()) throw std::runtime_error("batched apply: slots not reserved");
  for (int g0 = 0; g0 < R; g0 += kBatchSlots) {
    const int rn = std::min(kBatchSlots, R - g0);
    AggTcArg ag{};
    LeafTcArg lf{};
    for (int m = 0; m < 2; ++m) {
      ag.Vs[m] = reinterpret_cast<const float*>(P.d_Vs32[m]);
      lf.Vf[m] = P.d_Vf32[m];
      lf.khat[m] = P.ml[m][L].khat;
      ag.K[m] = lf.K[m] = P.ml[m][L].K;
      for (int j = 0; j < rn; ++j) {
        ag.S[m][j] = P.bS32[m][j];
        lf.Bm[m][j] = P.bB32[m][j];
      }
    }
    ag.leaf_ptr = lf.leaf_ptr = P.d_leaf_ptr;
    ag.leaf_rwg = lf.leaf_rwg = P.d_leaf_rwg;
    ag.X = X + g0 * ldx;
    ag.ldx = ldx;
    ag.N = lf.N = P.N;
    ag.R = lf.R = rn;
    ag.kmax = (P.max_leaf_rwgs + 7) & ~7;
    ag.status = lf.status = P.d_status;
    lf.W = W + g0 * ldw;
    lf.ldw = ldw;
    LeafArg<C> common{};
    fill_leaf_common(P, common);
    lf.c1 = common.c1;
    lf.c2 = common.c2;
    lf.etai = common.etai;
    const bool tensor_cores = P.tuning.batch_tc == 1 && agg_tc_supported(P, rn);
    if (tensor_cores)
      launch_agg_tc(P, ag, s);
    else
      launch_agg_slots(P, ag, s);
    {
      MediumStreams ms(P, s, true);
      if (P.tuning.batch_tree == 1) {
        for (int m = 0; m < 2; ++m)
          tree_pass_slots(P, m, rn, ms.of(m), P.stream_leaf[m], P.ev_agg[m], P.ev_leaf[m]);
      } else {
        for (int j = 0; j < rn; ++j)
          for (int m = 0; m < 2; ++m) tree_pass_fixed<C>(P, m, P.bS32[m][j], P.bB32[m][j], ms.of(m));
      }
      ms.join();
    }
    // near-field rows first (writing w), then the far field (adding)
    near_apply_batch(P, rn, ag.X, ldx, lf.W, ldw, P.d_pack, s);
    if (tensor_cores)
      launch_leaf_tc(P, lf, s);
    else
      launch_leaf_slots(P, lf, s);
  }
}

}  // namespace

void apply_direct(Plan& P, const double2* x, double2* w, cudaStream_t s) {
  const int L = P.maxL;
  cudaEvent_t* ev = profiler_events(P, s);
  NearAhead near(P, s, P.tuning.leaf_variant == 1 && ev == nullptr, x, w, 0);
  if (P.tuning.agg_variant == 1) {  // both media in one launch, timed as medium 1's aggregation
    AggBoxArg a{};
    for (int m = 0; m < 2; ++m) {
      a.Vs[m] = P.d_Vs[m];
      a.S[m] = P.ml[m][L].S;
      a.K[m] = P.ml[m][L].K;
    }
    a.leaf_ptr = P.d_leaf_ptr;
    a.leaf_rwg = P.d_leaf_rwg;
    a.x = x;
    a.N = P.N;
    agg_box_kernel<<<dim3(P.lv[L].B, 2), kThreads, 0, s>>>(a);
  }
  MediumStreams ms(P, s, ev == nullptr);
  for (int m = 0; m < 2; ++m) {
    const cudaStream_t sm = ms.of(m);
    const MediumLevel& leaf = P.ml[m][L];
    if (P.tuning.agg_variant == 0) {
      dim3 g(P.lv[L].B, (leaf.K + kThreads - 1) / kThreads);
      agg_kernel<double2><<<g, kThreads, 0, sm>>>(P.d_Vs[m], P.d_leaf_ptr, P.d_leaf_rwg, x, P.N, leaf.K, leaf.S);
    }
    if (ev) MLFMA_CUDA(cudaEventRecord(ev[1 + 4 * m], s));
    const LeafView v{leaf.S, leaf.Bm};
    if (ev) {  // one stage after the other, for the stage events
      launch_up(P, m, v, s);
      MLFMA_CUDA(cudaEventRecord(ev[2 + 4 * m], s));
      launch_m2l(P, m, v, s, L, L);  // the launches of the other branch: their sizes choose the sums' order
      launch_m2l(P, m, v, s, 2, L - 1);
      MLFMA_CUDA(cudaEventRecord(ev[3 + 4 * m], s));
      launch_l2l(P, m, v, s);
      MLFMA_CUDA(cudaEventRecord(ev[4 + 4 * m], s));
      continue;
    }
    // The leaf level's translation needs only the aggregation: it runs on a
    // stream of its own while the interpolation climbs the tree; the
    // anterpolation chain starts once both are done.
    const cudaStream_t sx = P.stream_leaf[m];
    MLFMA_CUDA(cudaEventRecord(P.ev_agg[m], sm));
    MLFMA_CUDA(cudaStreamWaitEvent(sx, P.ev_agg[m], 0));
    launch_m2l(P, m, v, sx, L, L);
    MLFMA_CUDA(cudaEventRecord(P.ev_leaf[m], sx));
    launch_up(P, m, v, sm);
    launch_m2l(P, m, v, sm, 2, L - 1);
    MLFMA_CUDA(cudaStreamWaitEvent(sm, P.ev_leaf[m], 0));
    launch_l2l(P, m, v, sm);
  }
  ms.join();
  LeafArg<double2> a{};
  for (int m = 0; m < 2; ++m) {
    a.Vf[m] = P.d_Vf[m];
    a.Bm[m] = P.ml[m][L].Bm;
    a.khat[m] = P.ml[m][L].khat;
    a.K[m] = P.ml[m][L].K;
  }
  fill_leaf_common(P, a);
  a.w = w;
  near.join();
  launch_leaf(P, a, s);
  MLFMA_CUDA(cudaGetLastError());
  if (ev) MLFMA_CUDA(cudaEventRecord(ev[9], s));
}

// The default of batch_tree: up to this size of a slot's tree arrays every level
// runs once for all slots (1), above it the slots run one after another (0). A
// launch over all slots of a large tree fills the GPU by itself, so the
// interpolation (bound by L1), the leaf translation (instruction issue) and the
// anterpolation (latency) of both media follow one another; the launches of
// single slots overlap: at 16 x 61,440 unknowns 13.9 ms of kernels in 11.2 ms,
// against 12.0 in 11.7. One B200, 16 slots, all at once / one after another:
// 15,360 unknowns (58 MB) 2.43 / 2.74 ms, 24,000 (104 MB) 4.50 / 4.57, 34,560
// (129 MB) 5.69 / 5.59, 61,440 (271 MB) 11.73 / 11.21, 121,500 (539 MB) 24.20 /
// 23.10; at 2 and 4 slots the sides change at the same size.
constexpr size_t kSlotGridBytes = size_t{116} << 20;
int default_batch_tree(const Plan& P) {
  size_t n = 0;
  for (int m = 0; m < 2; ++m)
    for (int l = 2; l <= P.maxL; ++l) n += static_cast<size_t>(P.lv[l].B) * 12 * P.ml[m][l].K * sizeof(float2);
  return n <= kSlotGridBytes ? 1 : 0;
}

void reserve_batch_staging(Plan& P) {
  if (P.xb_cap > 0) return;
  P.d_xb = P.alloc<double2>(static_cast<size_t>(kBatchSlots) * 2 * P.N);
  P.d_wb = P.alloc<double2>(static_cast<size_t>(kBatchSlots) * 2 * P.N);
  P.xb_cap = kBatchSlots;
}

void reserve_batch(Plan& P) {
  const int L = P.maxL;
  if (P.precision != 1) return;
  const bool leaf = P.bS32[0].empty();
  const bool upper = P.tuning.batch_tree == 1 && L > 2 && P.btS[0][2] == nullptr;
  if (!leaf && !upper) return;
  // slot-major per level, and with the leaf level the near-field product's
  // packed inputs, in one allocation
  const int lo = upper ? 2 : L, hi = leaf ? L : L - 1;
  auto count = [&](int m, int l) { return static_cast<size_t>(P.lv[l].B) * 6 * P.ml[m][l].K; };
  size_t total = leaf ? near_pack_values(P) : 0;
  for (int m = 0; m < 2; ++m)
    for (int l = lo; l <= hi; ++l) total += 2 * kBatchSlots * count(m, l);
  float2* p = P.alloc<float2>(total);
  for (int m = 0; m < 2; ++m) {
    for (int l = lo; l <= hi; ++l) {
      P.btS[m][l] = p;
      P.btB[m][l] = p + kBatchSlots * count(m, l);
      p += 2 * kBatchSlots * count(m, l);
    }
    for (int j = 0; leaf && j < kBatchSlots; ++j) {
      P.bS32[m].push_back(P.btS[m][L] + j * count(m, L));
      P.bB32[m].push_back(P.btB[m][L] + j * count(m, L));
    }
  }
  if (leaf) P.d_pack = p;
}

// FP64: one captured apply per row. Sharing the leaf tables among rows saves
// traffic but its kernels were slower than the single apply's, whose media and
// leaf translation also overlap: 3 rows at 10,140 unknowns 1.02 ms shared, 0.88 ms
// row by row; 7.4 against 6.7 ms per row at 245,760 unknowns.
void apply_batch_device(Plan& P, int R, const double2* X, long long ldx, double2* W, long long ldw, cudaStream_t s) {
  struct Unprofiled {  // the stage profiler covers single applies only
    bool& on;
    const bool was;
    explicit Unprofiled(bool& o) : on(o), was(o) { on = false; }
    ~Unprofiled() { on = was; }
  } quiet(P.prof.on);
  for (int j = 0; j < R; ++j) apply_device(P, X + j * ldx, W + j * ldw, s);
}

// Replays the captured apply of (stream, precision), capturing it on first
// use. The graph reads and writes the plan's staging vectors d_gx / d_gw, so
// that one graph serves every (x, w) pair: x is copied in and w out around
// the replay (two device copies of 2N complex values, microseconds against
// the apply), and a solver whose Krylov vectors change every iteration does
// not capture a graph per vector. Launches directly while stage profiling,
// inside another capture, or on the legacy default stream.
template <class F>
void apply_graphed(Plan& P, const double2* x, double2* w, cudaStream_t s, int precision, F&& launch) {
  if (!P.tuning.graph || P.prof.on || s == nullptr) return launch(x, w);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  MLFMA_CUDA(cudaStreamIsCapturing(s, &cs));
  if (cs != cudaStreamCaptureStatusNone) return launch(x, w);
  const size_t bytes = 2 * static_cast<size_t>(P.N) * sizeof(double2);
  if (P.d_gx == nullptr) {
    P.d_gx = P.alloc<double2>(2 * static_cast<size_t>(P.N));
    P.d_gw = P.alloc<double2>(2 * static_cast<size_t>(P.N));
  }
  cudaGraphExec_t exec = nullptr;
  for (const ApplyGraph& g : P.graphs)
    if (g.s == s && g.precision == precision) exec = g.exec;
  if (exec == nullptr && P.graphs.size() >= kMaxApplyGraphs) return launch(x, w);
  if (x != P.d_gx) MLFMA_CUDA(cudaMemcpyAsync(P.d_gx, x, bytes, cudaMemcpyDeviceToDevice, s));
  if (exec == nullptr) {
    MLFMA_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    try {
      launch(P.d_gx, P.d_gw);
    } catch (...) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(s, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    cudaGraph_t graph = nullptr;
    MLFMA_CUDA(cudaStreamEndCapture(s, &graph));
    const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    MLFMA_CUDA(e);
    P.graphs.push_back(ApplyGraph{s, precision, exec});
  }
  MLFMA_CUDA(cudaGraphLaunch(exec, s));
  if (w != P.d_gw) MLFMA_CUDA(cudaMemcpyAsync(w, P.d_gw, bytes, cudaMemcpyDeviceToDevice, s));
}

void apply_device(Plan& P, const double2* x, double2* w, cudaStream_t s) {
  apply_graphed(P, x, w, s, 0, [&](const double2* xx, double2* ww) { apply_direct(P, xx, ww, s); });
}

void clear_graphs(Plan& P) {
  for (auto& g : P.graphs) cudaGraphExecDestroy(g.exec);
  P.graphs.clear();
}

void apply_mixed_device(Plan& P, const double2* x, double2* w, cudaStream_t s) {
  if (P.precision != 1) throw std::invalid_argument("plan was not created with mixed precision");
  apply_graphed(P, x, w, s, 1, [&](const double2* xx, double2* ww) { apply_fixed<float2>(P, xx, ww, s); });
}

void apply_batch_mixed_device(Plan& P, int R, const double2* X, long long ldx, double2* W, long long ldw,
                              cudaStream_t s) {
  if (P.precision != 1) throw std::invalid_argument("plan was not created with mixed precision");
  apply_batch_slots(P, R, X, ldx, W, ldw, s);
}

}  // namespace mlfma

namespace mlfma {
// Sums the recorded stage times (ms) since the last read: out[0] aggregation,
// out[1] interpolation up, out[2] translation, out[3] anterpolation down,
// out[4] leaf testing + near field. Returns the number of applies covered.
int read_stage_times(Plan& P, double out[kStages]) {
  for (int i = 0; i < kStages; ++i) out[i] = 0.0;
  const int n = static_cast<int>(P.prof.used);
  for (int a = 0; a < n; ++a) {
    auto& e = P.prof.sets[a];
    MLFMA_CUDA(cudaEventSynchronize(e[StageProfiler::kEvents - 1]));
    float t[StageProfiler::kEvents - 1];
    for (int i = 0; i + 1 < StageProfiler::kEvents; ++i) MLFMA_CUDA(cudaEventElapsedTime(&t[i], e[i], e[i + 1]));
    for (int m = 0; m < 2; ++m)
      for (int k = 0; k < 4; ++k) out[k] += t[4 * m + k];
    out[4] += t[8];
  }
  P.prof.used = 0;
  return n;
}
}  // namespace mlfma
