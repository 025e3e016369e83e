// Length-n complex128 vector kernels of the Krylov solvers (internal linkage:
// one copy per including file): Gram-Schmidt projections against a block of
// basis vectors, updates, norms, and the small GMRES of the near-field
// preconditioner, whose state stays on the device.
//
// Every kernel works on a set of lockstep positions (grid.y; one for a single
// solve). A reduction is one launch: each block writes its partial sums, and
// the last block of a position to finish adds them up in block order, so
// results do not depend on scheduling.
//
// Bound: latency, not bandwidth (the basis of a solve is L2-resident at up
// to ~100,000 unknowns and a pass over 16 vectors of 34,560 complex values
// takes ~1 us), so what counts is the number of dependent launches and the
// serial code between them. Twice-classical Gram-Schmidt is one launch for
// short vectors (gs_cluster_kernel) and three for others: coefficients,
// projection fused with the coefficients of the second pass (each thread still
// holds the updated rows), second projection fused with the norm.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <complex>
#include <vector>

#include "bulk.cuh"
#include "cplx.cuh"
#include "plan.hpp"
#include "reduce.cuh"

namespace mlfma {
namespace blas1 {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 8;       // basis vectors per pass of the dot products
constexpr int kMaxBasis = 64;  // largest basis a projection may use
constexpr int kLdp = kMaxBasis;
constexpr int kLdh = 2 * kMaxBasis + 2;  // reduced values of a position: both passes' coefficients, ||w||^2

// One operand of a batched kernel: the vector of lockstep position a lives at
// p + (by_sys ? sys[a] : a) * stride + off.
struct VecRef {
  double2* p;
  long long stride, off;
  int by_sys;
  __device__ __forceinline__ double2* at(int a, const int* sys) const {
    return p + (by_sys ? sys[a] : a) * stride + off;
  }
};

// Complex Givens rotation as MGMRES builds and applies it (Code/GMRES.h:22-48).
inline void givens_make(std::complex<double> a, std::complex<double> b, std::complex<double>& c,
                        std::complex<double>& s) {
  const double eps = 1e-16;
  if (std::abs(b) < eps) {
    c = 1.0;
    s = 0.0;
  } else if (std::abs(a) < eps) {
    c = 0.0;
    s = 1.0;
  } else {
    const double r = std::sqrt(std::real(a * std::conj(a) + b * std::conj(b)));
    c = a / r;
    s = b / r;
  }
}
inline void givens_apply(std::complex<double>& x, std::complex<double>& y, std::complex<double> c,
                         std::complex<double> s) {
  const std::complex<double> t = std::conj(c) * x + std::conj(s) * y;
  y = -s * x + c * y;
  x = t;
}

// Upper-triangular solve of the rotated least-squares system (Code/GMRES.h:165-182).
inline void back_substitute(const std::vector<std::complex<double>>& H, int ld,
                            const std::vector<std::complex<double>>& s, int m,
                            std::vector<std::complex<double>>& y) {
  const double eps = 1e-16;
  y.assign(m, std::complex<double>(0.0));
  for (int i = m - 1; i >= 0; --i) {
    y[i] = s[i];
    for (int j = i + 1; j < m; ++j) y[i] -= H[i + j * ld] * y[j];
    if (std::abs(H[i + i * ld]) > eps)
      y[i] /= H[i + i * ld];
    else
      y[i] = std::complex<double>(0.0);
  }
}

// The same rotations on the device, for the inner GMRES steps that run
// without a host round trip.
__device__ __forceinline__ double2 dconj(double2 a) { return c2(a.x, -a.y); }
__device__ inline void dgivens_make(double2 a, double2 b, double2& c, double2& s) {
  const double eps = 1e-16;
  if (sqrt(b.x * b.x + b.y * b.y) < eps) {
    c = c2(1.0, 0.0);
    s = c2(0.0, 0.0);
  } else if (sqrt(a.x * a.x + a.y * a.y) < eps) {
    c = c2(0.0, 0.0);
    s = c2(1.0, 0.0);
  } else {
    const double r = sqrt(a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y);
    c = c2(a.x / r, a.y / r);
    s = c2(b.x / r, b.y / r);
  }
}
__device__ inline void dgivens_apply(double2& x, double2& y, double2 c, double2 s) {
  const double2 t = cadd(cmul(dconj(c), x), cmul(dconj(s), y));
  y = cadd(cmul(c2(-s.x, -s.y), x), cmul(c, y));
  x = t;
}

// Device state of the preconditioner's inner GMRES for every lockstep
// position. Basis vector j is kept unscaled (the vector after its two
// projections); vs[j] is its scale, 0 after a breakdown, applied wherever
// the vector is used.
struct Inner {
  double2* H;    // [R][inner][ld], rotated columns
  double2* cs;   // [R][inner]
  double2* sn;   // [R][inner]
  double2* g;    // [R][ld] rotated right-hand side
  double2* y;    // [R][ld] coefficients of the unscaled basis vectors in the solution
  double* vs;    // [R][ld]
  double* beta;  // [R]
  int* done;     // [R] breakdown
  int* m;        // [R] columns in use
  int ld, inner;
  static size_t bytes(int R, int inner) {
    const size_t ld = inner + 1;
    return static_cast<size_t>(R) * (sizeof(double2) * (ld * inner + 2 * inner + 2 * ld) +
                                     sizeof(double) * (ld + 1) + 2 * sizeof(int));
  }
  static Inner carve(void* base, int R, int inner) {
    const size_t Rz = R, ld = inner + 1;
    Inner I{};
    I.ld = inner + 1;
    I.inner = inner;
    I.H = static_cast<double2*>(base);
    I.cs = I.H + Rz * ld * inner;
    I.sn = I.cs + Rz * inner;
    I.g = I.sn + Rz * inner;
    I.y = I.g + Rz * ld;
    I.vs = reinterpret_cast<double*>(I.y + Rz * ld);
    I.beta = I.vs + Rz * ld;
    I.done = reinterpret_cast<int*>(I.beta + Rz);
    I.m = I.done + Rz;
    return I;
  }
};

// What the last block of a position does once the squared norm is known.
enum Finish {
  kFinishNone,
  kFinishBegin,  // inner GMRES: beta, the scale of v, an empty system
  kFinishStep,   // inner GMRES: column j of H, its rotations, the scale of the next vector;
                 // after the last step the solution of the triangular system
};

// Sums 8 values over the warp; value q ends up in the lanes with (lane >> 2)
// & 7 == q (bit-reversed halves: 9 shuffles of a complex value instead of 40).
__device__ __forceinline__ double2 warp_sum8(double2 (&v)[kTile]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4, o = 16; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double2 give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, o);
      v[i].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, o);
    }
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    v[0].x += __shfl_xor_sync(0xffffffffu, v[0].x, o);
    v[0].y += __shfl_xor_sync(0xffffffffu, v[0].y, o);
  }
  return v[0];
}

// Warp 0 of the last block, position a: inner GMRES state from ||v||^2.
__device__ __forceinline__ void inner_begin(const Inner& I, int a, double norm2) {
  const int lane = threadIdx.x & 31;
  const double beta = sqrt(norm2);
  for (int i = lane; i < I.ld; i += 32) I.g[static_cast<long long>(a) * I.ld + i] = c2(i == 0 ? beta : 0.0, 0.0);
  if (lane == 0) {
    I.beta[a] = beta;
    I.vs[static_cast<long long>(a) * I.ld] = beta > 0.0 ? 1.0 / beta : 0.0;
    I.done[a] = 0;
    I.m[a] = 0;
  }
}

// Warp 0 of the last block, position a: column j of H from both passes'
// coefficients h[i] + h[kMaxBasis + i] and hn = ||u||; its rotations; the
// scale of basis vector j + 1 (0 after a breakdown). The operands come in
// parallel into shared memory (sm: 3 * kMaxBasis values); one lane then runs
// the serial chain of rotations. After the last step, the triangular system
// R y = g, column by column over the lanes (Code/GMRES.h:165-182), y times
// each basis vector's scale.
__device__ __forceinline__ void inner_step(const Inner& I, int a, int j, const double2* h, double norm2,
                                           double2* sm) {
  const int lane = threadIdx.x & 31;
  double2* H = I.H + static_cast<long long>(a) * I.inner * I.ld;
  double2* Hj = H + static_cast<long long>(j) * I.ld;
  double2* cs = I.cs + static_cast<long long>(a) * I.inner;
  double2* sn = I.sn + static_cast<long long>(a) * I.inner;
  double2* g = I.g + static_cast<long long>(a) * I.ld;
  double* vs = I.vs + static_cast<long long>(a) * I.ld;
  const int done = I.done[a];
  int m = I.m[a];
  if (done) {
    if (lane == 0) vs[j + 1] = 0.0;
  } else {
    double2 *col = sm, *c = sm + kMaxBasis, *s = sm + 2 * kMaxBasis;
    for (int i = lane; i <= j; i += 32) {
      col[i] = cadd(__ldcg(h + i), __ldcg(h + kMaxBasis + i));
      if (i < j) {
        c[i] = cs[i];
        s[i] = sn[i];
      }
    }
    __syncwarp();
    if (lane == 0) {
      const double hn = sqrt(norm2);
      double2 x = col[0];
      for (int i = 0; i < j; ++i) {
        double2 y = col[i + 1];
        dgivens_apply(x, y, c[i], s[i]);
        col[i] = x;
        x = y;
      }
      double2 y = c2(hn, 0.0);
      I.m[a] = j + 1;
      if (hn < 1e-14 * I.beta[a]) {
        I.done[a] = 1;
        vs[j + 1] = 0.0;
      } else {
        vs[j + 1] = 1.0 / hn;
        double2 cj, sj;
        dgivens_make(x, y, cj, sj);
        dgivens_apply(x, y, cj, sj);
        cs[j] = cj;
        sn[j] = sj;
        double2 g0 = g[j], g1 = g[j + 1];
        dgivens_apply(g0, g1, cj, sj);
        g[j] = g0;
        g[j + 1] = g1;
        y = c2(0.0, 0.0);
      }
      col[j] = x;
      Hj[j + 1] = y;
    }
    __syncwarp();
    for (int i = lane; i <= j; i += 32) Hj[i] = col[i];
    m = j + 1;
    __syncwarp();
  }
  if (j + 1 < I.inner) return;
  const double eps = 1e-16;
  double2 g0 = lane < m ? g[lane] : c2(0.0, 0.0), g1 = lane + 32 < m ? g[lane + 32] : c2(0.0, 0.0);
  double2* y = I.y + static_cast<long long>(a) * I.ld;
  double2 n0 = c2(0.0, 0.0), n1 = c2(0.0, 0.0);  // column i of R, the next one in flight
  auto column = [&](int i, double2& p, double2& q) {
    p = i >= 0 && lane <= i ? H[static_cast<long long>(i) * I.ld + lane] : c2(0.0, 0.0);
    q = i >= 0 && lane + 32 <= i ? H[static_cast<long long>(i) * I.ld + lane + 32] : c2(0.0, 0.0);
  };
  column(m - 1, n0, n1);
  for (int i = m - 1; i >= 0; --i) {
    const double2 r0 = n0, r1 = n1;
    column(i - 1, n0, n1);
    const double2 gs = i < 32 ? g0 : g1, rs = i < 32 ? r0 : r1;
    const double2 gi = c2(__shfl_sync(0xffffffffu, gs.x, i & 31), __shfl_sync(0xffffffffu, gs.y, i & 31));
    const double2 ri = c2(__shfl_sync(0xffffffffu, rs.x, i & 31), __shfl_sync(0xffffffffu, rs.y, i & 31));
    const double2 yi = sqrt(ri.x * ri.x + ri.y * ri.y) > eps ? cdiv(gi, ri) : c2(0.0, 0.0);
    if (lane < i) g0 = csub(g0, cmul(r0, yi));
    if (lane + 32 < i) g1 = csub(g1, cmul(r1, yi));
    if (lane == 0) y[i] = cscale(yi, vs[i]);
  }
  for (int i = m + lane; i < I.inner; i += 32) y[i] = c2(0.0, 0.0);
}

// A complex64 copy of the vector worked on, for the lockstep near-field
// product: the positions in groups of sys, and per RWG the (J, M) pairs of a
// group side by side, [group][RWG][position][J, M]. Null: none.
struct Pack {
  float2* p;
  int sys;
};

struct GsArg {
  VecRef V, w;           // basis (vector j at V + j * n) and the vector worked on
  VecRef b;              // Norm: subtracted from, r = b - w written to w (has_b)
  VecRef copy;           // Norm: w copied here (has_copy)
  int has_b, has_copy;
  const int* sys;
  long long n;
  int nv;
  const double* vs;      // scales of the basis vectors [a * ldvs + j]; null: 1
  int ldvs;
  const double2* hin;    // coefficients to remove [a * kLdh + j]
  double2* hout;         // dot products [a * kLdh + j], or the squared norm [a * kLdh]
  const double2* hbase;  // Finish: both passes' coefficients [a * kLdh]
  double2* part;         // [a][kLdp][blocks] block partials
  unsigned* count;       // [a] blocks done
  Inner inner;
  int step;
  int cached;            // gs_cluster_kernel: basis vectors in shared memory
  Pack pack;
};

// The packed copy's slot of row i of position a
__device__ __forceinline__ void pack_row(const Pack& p, long long n, int a, long long i, double2 v) {
  const long long half = n / 2, id = i < half ? i : i - half;
  p.p[(((a / p.sys) * half + id) * p.sys + a % p.sys) * 2 + (i >= half)] = Cx<float2>::from(v);
}

// E rows of each operand per thread and chunk. kProject: w -= sum_j hin_j V_j.
// kDots: the dot products conj(V_j) . w of the (updated) w; else its squared
// norm. A thread keeps its updated rows in registers between the two parts.
template <int E, bool kProject, bool kDots, int kFin>
static __global__ void __launch_bounds__(kThreads) gs_kernel(const __grid_constant__ GsArg g) {
  __shared__ double2 hs[kMaxBasis];
  __shared__ double2 ws[kWarps][kMaxBasis];
  __shared__ bool last;
  const int a = blockIdx.y, nblk = gridDim.x;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const long long n = g.n;
  const int nv = g.nv;
  const double2* __restrict__ V = kProject || kDots ? g.V.at(a, g.sys) : nullptr;
  double2* w = g.w.at(a, g.sys);
  const double2* bb = !kProject && !kDots && g.has_b ? g.b.at(a, g.sys) : nullptr;
  double2* cp = !kProject && !kDots && g.has_copy ? g.copy.at(a, g.sys) : nullptr;
  if (kProject) {
    for (int j = threadIdx.x; j < nv; j += kThreads) {
      const double2 h = g.hin[static_cast<long long>(a) * kLdh + j];
      hs[j] = g.vs ? cscale(h, g.vs[static_cast<long long>(a) * g.ldvs + j]) : h;
    }
  }
  if (kDots)
    for (int j = lane; j < nv; j += 32) ws[wp][j] = c2(0.0, 0.0);
  __syncthreads();
  double2 nrm = c2(0.0, 0.0);
  for (long long base = static_cast<long long>(blockIdx.x) * (kThreads * E); base < n;
       base += static_cast<long long>(nblk) * (kThreads * E)) {
    double2 wi[E];
    long long at[E];
    bool in[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const long long i = base + e * kThreads + threadIdx.x;
      in[e] = i < n;
      at[e] = in[e] ? i : 0;
      wi[e] = in[e] ? w[i] : c2(0.0, 0.0);
    }
    if (kProject) {
#pragma unroll 4
      for (int j = 0; j < nv; ++j) {
        const double2* Vj = V + j * n;
        const double2 hj = hs[j];
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (in[e]) wi[e] = csub(wi[e], cmul(hj, __ldg(Vj + at[e])));
      }
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (in[e]) w[at[e]] = wi[e];
    }
    if (kDots) {
      for (int j0 = 0; j0 < nv; j0 += kTile) {
        double2 acc[kTile];
#pragma unroll
        for (int q = 0; q < kTile; ++q) {
          acc[q] = c2(0.0, 0.0);
          if (j0 + q < nv) {
            const double2* Vj = V + (j0 + q) * n;
#pragma unroll
            for (int e = 0; e < E; ++e) {
              const double2 v = in[e] ? __ldg(Vj + at[e]) : c2(0.0, 0.0);
              acc[q].x = fma(v.x, wi[e].x, fma(v.y, wi[e].y, acc[q].x));
              acc[q].y = fma(v.x, wi[e].y, fma(-v.y, wi[e].x, acc[q].y));
            }
          }
        }
        const double2 t = warp_sum8(acc);
        const int q = lane >> 2;
        if ((lane & 3) == 0 && j0 + q < nv) ws[wp][j0 + q] = cadd(ws[wp][j0 + q], t);
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (in[e]) {
          if (bb) {
            wi[e] = csub(bb[at[e]], wi[e]);
            w[at[e]] = wi[e];
          }
          if (cp) cp[at[e]] = wi[e];
          if (kFin != kFinishNone && g.pack.p) pack_row(g.pack, n, a, at[e], wi[e]);
          nrm.x = fma(wi[e].x, wi[e].x, fma(wi[e].y, wi[e].y, nrm.x));
        }
    }
  }
  if (!kDots) {
    nrm = warp_sum2(nrm);
    if (lane == 0) ws[wp][0] = nrm;
  }
  __syncthreads();
  const int np = kDots ? nv : 1;
  double2* part = g.part + static_cast<long long>(a) * kLdp * nblk;
  for (int j = threadIdx.x; j < np; j += kThreads) {
    double2 t = ws[0][j];
#pragma unroll
    for (int q = 1; q < kWarps; ++q) t = cadd(t, ws[q][j]);
    part[static_cast<long long>(j) * nblk + blockIdx.x] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(g.count + a, 1u) == static_cast<unsigned>(nblk) - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) g.count[a] = 0;
  double norm2 = 0.0;
  for (int j = wp; j < np; j += kWarps) {
    double2 t = c2(0.0, 0.0);
    for (int q = lane; q < nblk; q += 32) t = cadd(t, __ldcg(part + static_cast<long long>(j) * nblk + q));
    t = warp_sum2(t);
    if (kDots && g.vs) t = cscale(t, g.vs[static_cast<long long>(a) * g.ldvs + j]);
    if (lane == 0) g.hout[static_cast<long long>(a) * kLdh + j] = t;
    norm2 = t.x;
  }
  if (wp != 0 || kDots) return;
  if (kFin == kFinishBegin) inner_begin(g.inner, a, norm2);
  if (kFin == kFinishStep)
    inner_step(g.inner, a, g.step, g.hbase + static_cast<long long>(a) * kLdh, norm2, &ws[0][0]);
}

// Both Gram-Schmidt passes, the norm and the inner step in one launch: a
// cluster of kClBlocks blocks per position, E rows per thread, which stay in
// registers from the first dot product to the last projection. The blocks'
// sums meet through distributed shared memory, every block adding them up in
// the same order. A block first fetches its rows of as many basis vectors as
// its shared memory holds (all loads at once), and the four passes read those.
// Bound: latency (launch, three cluster barriers, the serial rotations). At
// 3,840 unknowns and 15 vectors 14.6 us for 29.7 in three launches of
// gs_kernel; 19.0 with 88 KB of shared memory, 22.6 without.
// Where the line lies (solves with 16 inner steps, ms, gs_kernel -> clusters):
//   n = 2,160:  1 system 11.8 -> 10.3, 8: 15.6 -> 14.4, 12: 19.2 -> 18.0, 16: 20.3 -> 21.6
//   n = 15,360: 1 system 32.9 -> 30.5, 8: 67.9 -> 65.6, 12: 97.5 -> 95.6, 16: 116.9 -> 117.5
//   n = 24,000 (4 rows per thread): 38.4 -> 38.9, 8: 103.3 -> 102.9
//   n = 34,560 (8 rows): 30.5 -> 32.0 (16 SMs read the basis four times)
// so up to two rows per thread and 12 positions. With 200 KB of shared memory
// 7 clusters fit at once, with 88 KB (two blocks per SM) 14: 8 systems took two
// turns with the former, 27.8 us at 15,360 unknowns, 23.0 with the latter.
constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClBlocks = 16;  // the non-portable size: a GPC's worth of SMs
constexpr int kClRows = 2;     // rows per thread at most
constexpr int kClMaxPositions = 12;
constexpr int kClCache = 200 << 10;  // bytes of the basis in shared memory, up to
constexpr int kClWide = 7;           // this many positions
constexpr int kClCacheMany = 88 << 10;

template <int E, bool kStep>
static __global__ void __launch_bounds__(kClThreads, 2) gs_cluster_kernel(const __grid_constant__ GsArg g) {
  __shared__ double2 hs[kMaxBasis];
  __shared__ double2 ws[kClWarps][kMaxBasis];
  __shared__ double2 part[2][kMaxBasis];
  __shared__ double2 pn;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int a = blockIdx.y, rank = blockIdx.x;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int n = static_cast<int>(g.n), nv = g.nv;
  const double2* __restrict__ V = g.V.at(a, g.sys);
  double2* w = g.w.at(a, g.sys);
  double2* hout = g.hout + static_cast<long long>(a) * kLdh;
  const double* vs = g.vs ? g.vs + static_cast<long long>(a) * g.ldvs : nullptr;
  const int i0 = rank * kClThreads + threadIdx.x;
  auto row = [&](int e) { return i0 + e * (kClBlocks * kClThreads); };
  extern __shared__ __align__(16) unsigned char gs_smem[];
  double2* mine = reinterpret_cast<double2*>(gs_smem) + threadIdx.x;  // own rows of the first nc basis vectors
  const int nc = g.cached;
  for (int j = 0; j < nc; ++j)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool take = row(e) < n;
      cp_async16_or_zero(mine + (j * E + e) * kClThreads, V + (take ? j * g.n + row(e) : 0), take);
    }
  cp_async_commit();
  double2 wi[E];
#pragma unroll
  for (int e = 0; e < E; ++e) wi[e] = row(e) < n ? w[row(e)] : c2(0.0, 0.0);
  cp_async_wait<0>();
  auto dots = [&](int pass) {
    for (int j0 = 0; j0 < nv; j0 += kTile) {
      double2 acc[kTile];
#pragma unroll
      for (int q = 0; q < kTile; ++q) {
        acc[q] = c2(0.0, 0.0);
        if (j0 + q < nv) {
          const bool cached = j0 + q < nc;
          const double2 *Vj = V + (j0 + q) * g.n, *own = mine + (j0 + q) * E * kClThreads;
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const double2 v = cached ? own[e * kClThreads] : row(e) < n ? __ldg(Vj + row(e)) : c2(0.0, 0.0);
            acc[q].x = fma(v.x, wi[e].x, fma(v.y, wi[e].y, acc[q].x));
            acc[q].y = fma(v.x, wi[e].y, fma(-v.y, wi[e].x, acc[q].y));
          }
        }
      }
      const double2 t = warp_sum8(acc);
      const int q = lane >> 2;
      if ((lane & 3) == 0 && j0 + q < nv) ws[wp][j0 + q] = t;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < nv; j += kClThreads) {
      double2 t = ws[0][j];
#pragma unroll
      for (int q = 1; q < kClWarps; ++q) t = cadd(t, ws[q][j]);
      part[pass][j] = t;
    }
    cl.sync();
    for (int j = wp; j < nv; j += kClWarps) {
      double2 t = lane < kClBlocks ? *cl.map_shared_rank(&part[pass][j], lane) : c2(0.0, 0.0);
      t = warp_sum2(t);
      if (lane == 0) {
        const double sc = vs ? vs[j] : 1.0;
        t = cscale(t, sc);
        if (rank == 0) hout[pass * kMaxBasis + j] = t;
        hs[j] = cscale(t, sc);
      }
    }
    __syncthreads();
  };
  auto project = [&] {
#pragma unroll 4
    for (int j = 0; j < nc; ++j) {
      const double2 hj = hs[j];
#pragma unroll
      for (int e = 0; e < E; ++e) wi[e] = csub(wi[e], cmul(hj, mine[(j * E + e) * kClThreads]));
    }
#pragma unroll 4
    for (int j = nc; j < nv; ++j) {
      const double2* Vj = V + j * g.n;
      const double2 hj = hs[j];
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (row(e) < n) wi[e] = csub(wi[e], cmul(hj, __ldg(Vj + row(e))));
    }
  };
  dots(0);
  project();
  dots(1);
  project();
  double2 nrm = c2(0.0, 0.0);
#pragma unroll
  for (int e = 0; e < E; ++e)
    if (row(e) < n) {
      w[row(e)] = wi[e];
      if (kStep && g.pack.p) pack_row(g.pack, g.n, a, row(e), wi[e]);
      nrm.x = fma(wi[e].x, wi[e].x, fma(wi[e].y, wi[e].y, nrm.x));
    }
  nrm = block_sum(nrm, &ws[0][0]);
  if (threadIdx.x == 0) pn = nrm;
  cl.sync();
  if (rank == 0 && wp == 0)
    nrm = warp_sum2(lane < kClBlocks ? *cl.map_shared_rank(&pn, lane) : c2(0.0, 0.0));
  cl.sync();  // no block leaves before its sum is read
  if (rank != 0 || wp != 0) return;
  if (lane == 0) hout[2 * kMaxBasis] = nrm;
  if (kStep) inner_step(g.inner, a, g.step, hout, nrm.x, &ws[0][0]);
}

// dst = alpha[a] * src
static __global__ void __launch_bounds__(kThreads) scale_kernel(VecRef src, VecRef dst, const int* sys, long long n,
                                                                const double* alpha) {
  const int a = blockIdx.y;
  const double2* s = src.at(a, sys);
  double2* d = dst.at(a, sys);
  const double al = alpha[a];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    d[i] = cscale(s[i], al);
}

// dst = al * src (one vector, the factor from the host)
static __global__ void __launch_bounds__(kThreads) scale1_kernel(const double2* src, double al, double2* dst,
                                                                 long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = cscale(src[i], al);
}

// x (+)= sum_{j < m[a]} V_j y[a * ldy + j]  (mfix columns when m is null)
static __global__ void __launch_bounds__(kThreads) combine_kernel(VecRef V, VecRef x, const int* sys, long long n,
                                                                  const int* m, int mfix, const double2* y, int ldy,
                                                                  int accumulate) {
  __shared__ double2 ys[kMaxBasis];
  const int a = blockIdx.y;
  const int ma = m ? m[a] : mfix;
  const double2* __restrict__ Vb = V.at(a, sys);
  double2* xb = x.at(a, sys);
  for (int j = threadIdx.x; j < ma; j += blockDim.x) ys[j] = y[(long long)a * ldy + j];
  __syncthreads();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double2 xi = accumulate ? xb[i] : c2(0.0, 0.0);
#pragma unroll 4
    for (int j = 0; j < ma; ++j) xi = cfma(ys[j], __ldg(Vb + j * n + i), xi);
    xb[i] = xi;
  }
}

// dst = src (gather into / scatter out of the contiguous staging block)
static __global__ void __launch_bounds__(kThreads) copy_kernel(VecRef src, VecRef dst, const int* sys, long long n) {
  const int a = blockIdx.y;
  const double2* s = src.at(a, sys);
  double2* d = dst.at(a, sys);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    d[i] = s[i];
}

// Blocks of the reductions: E rows per thread (1, 2 or 4) so that the
// positions together give at most four blocks per SM where one row each
// would give more, and at most kMaxBlocks in all (each then walks chunks).
// 592 resident blocks of 256 threads fill the 148 SMs; fewer rows per thread
// than that leaves SMs idle, more blocks only lengthen the last block's sum.
constexpr int kFill = 592;
constexpr int kMaxBlocks = 1184;
struct Split {
  int E, nblk;
};
inline Split split(long long n, int Ra) {
  const long long one = (n + kThreads - 1) / kThreads;
  const int E = one * Ra <= kFill ? 1 : one * Ra <= 2 * kFill ? 2 : 4;
  const long long nb = (one + E - 1) / E;
  return {E, static_cast<int>(std::max(1LL, std::min<long long>(nb, std::max(1, kMaxBlocks / Ra))))};
}
// partials one reduction over up to R positions may need (values)
inline size_t part_count(long long n, int R) {
  size_t most = 0;
  for (int Ra = 1; Ra <= R; ++Ra) most = std::max(most, static_cast<size_t>(Ra) * split(n, Ra).nblk);
  return most * kLdp;
}

template <bool kProject, bool kDots, int kFin>
inline void launch_gs(const GsArg& g, int Ra, cudaStream_t s) {
  const Split sp = split(g.n, Ra);
  const dim3 grid(sp.nblk, Ra);
  if (sp.E == 1)
    gs_kernel<1, kProject, kDots, kFin><<<grid, kThreads, 0, s>>>(g);
  else if (sp.E == 2)
    gs_kernel<2, kProject, kDots, kFin><<<grid, kThreads, 0, s>>>(g);
  else
    gs_kernel<4, kProject, kDots, kFin><<<grid, kThreads, 0, s>>>(g);
}

template <bool kStep>
inline void launch_gs_cluster(GsArg g, int Ra, cudaStream_t s) {
  auto go = [&](auto* kernel, int E) {
    MLFMA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    MLFMA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClCache));
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {kClBlocks, 1, 1};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClBlocks, Ra);
    cfg.blockDim = dim3(kClThreads);
    const int vec = 16 * kClThreads * E;
    g.cached = std::min(g.nv, (Ra <= kClWide ? kClCache : kClCacheMany) / vec);
    cfg.dynamicSmemBytes = static_cast<size_t>(g.cached) * vec;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    MLFMA_CUDA(cudaLaunchKernelEx(&cfg, kernel, g));
  };
  const long long rows = (g.n + kClBlocks * kClThreads - 1) / (kClBlocks * kClThreads);
  if (rows <= 1)
    go(gs_cluster_kernel<1, kStep>, 1);
  else
    go(gs_cluster_kernel<kClRows, kStep>, kClRows);
}

// Whether the current device can hold a cluster of kClBlocks blocks (a whole
// B200 can; a partition of one may not).
inline bool clusters_fit() {
  auto* kernel = gs_cluster_kernel<kClRows, true>;
  MLFMA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  MLFMA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClCache));
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {kClBlocks, 1, 1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kClBlocks);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = kClCache;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return fit > 0;
}

// Device work arrays owned by one solve.
struct Work {
  std::vector<void*> owned;
  ~Work() {
    for (void* p : owned) cudaFree(p);
  }
  double2* get(size_t count) {
    void* p = nullptr;
    MLFMA_CUDA(cudaMalloc(&p, (count ? count : 1) * sizeof(double2)));
    owned.push_back(p);
    return static_cast<double2*>(p);
  }
};

// The work arrays of one solve from the plan's arena (at most `values` complex
// values, pieces rounded up to 256 bytes included): a driver allocation costs
// milliseconds, and a solve at 34,560 unknowns made 20 of them, 4.5 of its 38
// ms. The block stays with the plan for its next solve, up to the arena's
// bound.
struct ArenaWork {
  Plan& P;
  ArenaWork(Plan& P_, size_t values) : P(P_) { P.arena.reserve(values * sizeof(double2)); }
  ~ArenaWork() {
    if (P.arena.cap > Plan::SolveArena::kKeepBytes) P.arena.release();
  }
  ArenaWork(const ArenaWork&) = delete;
  double2* get(size_t count) { return static_cast<double2*>(P.arena.get((count ? count : 1) * sizeof(double2))); }
};

// Launches of the vector steps on one stream for up to R positions.
struct Vec {
  cudaStream_t s;
  long long n;
  double2* part;    // [part_count(n, R)]
  unsigned* count;  // [R], zero
  double2* h;       // [R][kLdh] reduced values
  bool clusters;    // the device takes clusters of kClBlocks blocks (clusters_fit)

  dim3 grid(int Ra) const {
    return dim3(static_cast<unsigned>(std::max(1LL, std::min<long long>((n + kThreads - 1) / kThreads,
                                                                        std::max(1, 2 * kMaxBlocks / Ra)))), Ra);
  }
  GsArg base(const int* sys) const {
    GsArg g{};
    g.sys = sys;
    g.n = n;
    g.part = part;
    g.count = count;
    g.hout = h;
    return g;
  }
  // squared norms of the operand (or of b - w, written to w) at h[a * kLdh]
  void norms(int Ra, const int* sys, VecRef w) {
    GsArg g = base(sys);
    g.w = w;
    launch_gs<false, false, kFinishNone>(g, Ra, s);
  }
  void residuals(int Ra, const int* sys, VecRef w, VecRef b) {
    GsArg g = base(sys);
    g.w = w;
    g.b = b;
    g.has_b = 1;
    launch_gs<false, false, kFinishNone>(g, Ra, s);
  }
  // Classical Gram-Schmidt twice of w against V[0..nv): per position a,
  // h[a * kLdh + j] and h[a * kLdh + kMaxBasis + j] the passes' coefficients,
  // h[a * kLdh + 2 kMaxBasis] = ||w||^2 after them. With an inner GMRES, the
  // basis is scaled by inner->vs and its step nv - 1 follows the norm.
  void orthogonalise(int Ra, const int* sys, VecRef V, VecRef w, int nv, const Inner* inner = nullptr,
                     Pack pack = {}) {
    GsArg g = base(sys);
    g.V = V;
    g.w = w;
    g.nv = nv;
    if (inner) {
      g.vs = inner->vs;
      g.ldvs = inner->ld;
      g.inner = *inner;
      g.step = nv - 1;
      g.hbase = h;
    }
    if (clusters && Ra <= kClMaxPositions && n <= kClBlocks * kClThreads * kClRows) {
      g.pack = pack;
      if (inner)
        launch_gs_cluster<true>(g, Ra, s);
      else
        launch_gs_cluster<false>(g, Ra, s);
      return;
    }
    launch_gs<false, true, kFinishNone>(g, Ra, s);
    g.hin = h;
    g.hout = h + kMaxBasis;
    launch_gs<true, true, kFinishNone>(g, Ra, s);
    g.hin = h + kMaxBasis;
    g.hout = h + 2 * kMaxBasis;
    g.pack = pack;
    if (inner)
      launch_gs<true, false, kFinishStep>(g, Ra, s);
    else
      launch_gs<true, false, kFinishNone>(g, Ra, s);
  }
  // Start of the inner GMRES: v copied into basis vector 0, its norm and scale
  void inner_start(int Ra, const int* sys, VecRef v, VecRef q0, const Inner& inner, Pack pack = {}) {
    GsArg g = base(sys);
    g.w = v;
    g.copy = q0;
    g.has_copy = 1;
    g.inner = inner;
    g.pack = pack;
    launch_gs<false, false, kFinishBegin>(g, Ra, s);
  }
  void scale(int Ra, const int* sys, VecRef src, VecRef dst, const double* alpha) {
    scale_kernel<<<grid(Ra), kThreads, 0, s>>>(src, dst, sys, n, alpha);
  }
  void scale(const double2* src, double al, double2* dst) {
    scale1_kernel<<<grid(1), kThreads, 0, s>>>(src, al, dst, n);
  }
  void combine(int Ra, const int* sys, VecRef V, VecRef x, const int* m, int mfix, const double2* y, int ldy,
               bool accumulate) {
    combine_kernel<<<grid(Ra), kThreads, 0, s>>>(V, x, sys, n, m, mfix, y, ldy, accumulate ? 1 : 0);
  }
  void copy(int Ra, const int* sys, VecRef src, VecRef dst) {
    copy_kernel<<<grid(Ra), kThreads, 0, s>>>(src, dst, sys, n);
  }
};

// One system's vector steps with their results on the host.
struct Ops : Vec {
  static VecRef ref(const double2* p) { return VecRef{const_cast<double2*>(p), 0, 0, 0}; }
  double read_norm() {
    std::complex<double> o;
    MLFMA_CUDA(cudaMemcpyAsync(&o, h, sizeof(double2), cudaMemcpyDeviceToHost, s));
    MLFMA_CUDA(cudaStreamSynchronize(s));
    return std::sqrt(o.real());
  }
  // ||v||
  double norm(const double2* v) {
    norms(1, nullptr, ref(v));
    return read_norm();
  }
  // w = b - w, returns ||w||
  double residual(const double2* b, double2* w) {
    residuals(1, nullptr, ref(w), ref(b));
    return read_norm();
  }
  // hcol[j] = sum of both passes' coefficients, returns ||w|| after projection
  double orthogonalise_host(const double2* V, int nv, double2* w, std::vector<std::complex<double>>& hcol) {
    orthogonalise(1, nullptr, ref(V), ref(w), nv);
    std::complex<double> buf[kLdh];
    MLFMA_CUDA(cudaMemcpyAsync(buf, h, sizeof(buf), cudaMemcpyDeviceToHost, s));
    MLFMA_CUDA(cudaStreamSynchronize(s));
    hcol.resize(nv);
    for (int j = 0; j < nv; ++j) hcol[j] = buf[j] + buf[kMaxBasis + j];
    return std::sqrt(buf[2 * kMaxBasis].real());
  }
};
template <class W>
inline Ops make_ops(W& g, cudaStream_t s, long long n) {
  Ops o{};
  o.s = s;
  o.n = n;
  o.part = g.get(part_count(n, 1));
  o.h = g.get(kLdh);
  o.clusters = clusters_fit();
  o.count = reinterpret_cast<unsigned*>(g.get(1));
  MLFMA_CUDA(cudaMemsetAsync(o.count, 0, sizeof(double2), s));
  return o;
}

}  // namespace blas1
}  // namespace mlfma
