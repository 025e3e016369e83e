// Lockstep multi-right-hand-side FGMRES: R independent systems A x_q = b_q
// (one per plane-wave incidence, say) iterate together, so each Arnoldi
// step costs one batched operator apply (in complex64 the leaf patterns are
// read once per 16 right-hand sides and the near-field entries once per 8, in
// FP64 the rows are applied in turn, matvec_kernels.cu) and one batched
// near-field product per inner step, and every Gram-Schmidt / update step is
// one launch over all active systems (three past the clusters' range, blas1.cuh). The outer Arnoldi step
// takes one host sync (its Givens rotations and convergence test are on the
// host); the preconditioner's inner steps keep their small GMRES state on
// the device and take none.
// Per system the iteration is exactly fgmres_solve's (fgmres.cu): the
// reference's restarted GMRES (Code/GMRES.h:65-217) with CGS2 Arnoldi,
// complex Givens rotations, true residual per cycle and its divergence
// abort, optionally right-preconditioned by inner GMRES steps on Z_near.
// A system leaves the lockstep set when it converges, breaks down or runs
// out of iterations; the others go on.
#include <algorithm>
#include <chrono>
#include <complex>
#include <vector>

#include "blas1.cuh"
#include "bulk.cuh"
#include "cplx.cuh"
#include "plan.hpp"
#include "learned.hpp"
#include "solver.hpp"

namespace mlfma {

namespace {

using C = std::complex<double>;
using blas1::VecRef;

// w_a = Z_near x_a for every position, in complex64.
struct NearBatchArg {
  const int* leaf_rwg;
  const int* leaf_ptr;
  const int* near_sptr;
  const int* near_src;
  const long long* near_zoff;
  const float2* near_z;
  VecRef w;
  const int* sys;
  const double* xscale;  // factor of position a's x at xscale[a * lds]; null: 1
  int lds;
  int N, R;
};

// One CTA per (leaf box, 32 / G rows, 2G systems), a small dense product: a
// lane holds one row and two systems (J and M: 4 sums), a warp all of the
// CTA's rows and systems over a quarter of the box's sources, so no value is
// reduced across lanes. The entries (128 (row, source) pairs at a time) and
// the sources' values, which the Gram-Schmidt kernels leave packed per RWG in
// complex64 (blas1::Pack), stream through a two-stage ring per warp
// (cp.async): one chunk is in flight while one is multiplied, and no warp
// waits for another but for the sum of the quarters at the end. Sums of four
// sources, of a chunk and of the whole quarter: a row's large entries (its own
// triangles') then meet few roundings, as in a sum over 32 lanes. (One running
// sum made the 16-slot batched apply's error 1.7e-7 instead of 1.0e-7.)
// FP32-bound at 8 systems (2.2 M pairs: 7.5 us at the FP32 rate, 52 MB of
// entries 8 us); measured 28 us, 33 with three stages (fewer CTAs per SM). With a lane per source and the sources
// staged for the whole CTA first (10 warps per SM, each waiting for its
// loads, 320 shuffles per pair of rows) the product took 92 us there; with a
// CTA for all rows of a box 56 us, waiting for the fullest boxes.
constexpr int kNearWarps = 4;
constexpr int kNearStages = 2;

template <int G>
struct NearTile {
  static constexpr int kSys = 2 * G, kRows = 32 / G, kSrc = 128 / kRows;
  static constexpr int kZs = 3 * kSrc + 2;  // row pitch of a stage: 16-byte rows in different banks
  static constexpr int kOut = kRows * kSys;
  struct __align__(16) Stage {
    float2 z[kRows * kZs];
    float4 x[kSrc * kSys];  // (J, M) per (source, system)
  };
  Stage ring[kNearWarps][kNearStages];
  float4 red[kNearWarps][kOut];
};

template <int G>
__global__ void __launch_bounds__(32 * kNearWarps) near_batch_tile_kernel(NearBatchArg a,
                                                                          const float4* __restrict__ packed) {
  using T = NearTile<G>;
  constexpr int kSys = T::kSys, kRows = T::kRows, kSrc = T::kSrc, kZs = T::kZs, kOut = T::kOut;
  extern __shared__ __align__(16) unsigned char near_smem[];
  T& sm = *reinterpret_cast<T*>(near_smem);
  const int b = blockIdx.x;
  const int t0 = blockIdx.z * kRows;  // first row of this CTA
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  if (t0 >= nb) return;
  const int p0 = blockIdx.y * kSys, pn = min(kSys, a.R - p0);
  const int s0 = a.near_sptr[b], ns = a.near_sptr[b + 1] - s0, pitch = near_pitch(ns);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  typename T::Stage* ring = sm.ring[wp];
  const float2* Z = a.near_z + a.near_zoff[b];
  const float4* X = packed + static_cast<long long>(blockIdx.y) * a.N * kSys;
  const int nchunk = (ns + kSrc - 1) / kSrc;
  const int nc = nchunk > wp ? (nchunk - wp + kNearWarps - 1) / kNearWarps : 0;  // this warp's chunks
  auto source = [&](int it) {  // lane q's source of the warp's chunk it
    const int c = wp + it * kNearWarps;
    return it < nc ? __ldg(a.near_src + s0 + min(c * kSrc + (lane % kSrc), ns - 1)) : 0;
  };
  int ids = source(0);
  auto stage = [&](int it) {
    if (it < nc) {
      const int c = wp + it * kNearWarps;
      typename T::Stage& st = ring[it % kNearStages];
#pragma unroll
      for (int i = 0; i < 6; ++i) {  // pairs of sources of one plane of one row
        constexpr int kPairs = kSrc / 2;
        const int e = 32 * i + lane, row = e / (3 * kPairs), plane = e / kPairs - 3 * row, pr = e % kPairs;
        const int gr = t0 + row, src = c * kSrc + 2 * pr;
        const bool take = gr < nb && src < pitch;
        cp_async16_or_zero(&st.z[row * kZs + plane * kSrc + 2 * pr],
                           Z + (take ? (3LL * gr + plane) * pitch + src : 0), take);
      }
#pragma unroll
      for (int i = 0; i < (kSrc * kSys + 31) / 32; ++i) {
        const int e = 32 * i + lane;
        const int id = __shfl_sync(0xffffffffu, ids, (e / kSys) % kSrc);
        if (e < kSrc * kSys) cp_async_ca<16>(&st.x[e], X + static_cast<long long>(id) * kSys + e % kSys);
      }
    }
    cp_async_commit();
    ids = source(it + 1);
  };
#pragma unroll
  for (int i = 0; i + 1 < kNearStages; ++i) stage(i);
  const int row = lane / G, g = lane - row * G;
  float2 aJ[2], aM[2];
  aJ[0] = aJ[1] = aM[0] = aM[1] = make_float2(0.f, 0.f);
  for (int it = 0; it < nc; ++it) {
    stage(it + kNearStages - 1);
    cp_async_wait<kNearStages - 1>();
    __syncwarp();
    const float2* z = ring[it % kNearStages].z + row * kZs;
    const float4* x = ring[it % kNearStages].x + 2 * g;
    float2 cJ[2], cM[2], sJ[2], sM[2];  // the chunk's sums, and those of the four sources under way
    cJ[0] = cJ[1] = cM[0] = cM[1] = sJ[0] = sJ[1] = sM[0] = sM[1] = make_float2(0.f, 0.f);
    auto add = [&](int q, float2 z11, float2 z12, float2 z22) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 v = x[q * kSys + j];
        const float2 J = make_float2(v.x, v.y), M = make_float2(v.z, v.w), nJ = make_float2(-v.x, -v.y);
        sJ[j] = cfma(z11, J, cfma(z12, M, sJ[j]));
        sM[j] = cfma(z22, M, cfma(z12, nJ, sM[j]));
      }
    };
    auto carry = [&](float2(&tJ)[2], float2(&tM)[2], float2(&fJ)[2], float2(&fM)[2]) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        tJ[j] = cadd(tJ[j], fJ[j]);
        tM[j] = cadd(tM[j], fM[j]);
        fJ[j] = fM[j] = make_float2(0.f, 0.f);
      }
    };
    const int kn = min(kSrc, ns - (wp + it * kNearWarps) * kSrc);
    if (kn == kSrc) {
#pragma unroll
      for (int q = 0; q < kSrc; q += 4) {
#pragma unroll
        for (int u = q; u < q + 4; u += 2) {
          const float4 z11 = *reinterpret_cast<const float4*>(z + u);
          const float4 z12 = *reinterpret_cast<const float4*>(z + kSrc + u);
          const float4 z22 = *reinterpret_cast<const float4*>(z + 2 * kSrc + u);
          add(u, make_float2(z11.x, z11.y), make_float2(z12.x, z12.y), make_float2(z22.x, z22.y));
          add(u + 1, make_float2(z11.z, z11.w), make_float2(z12.z, z12.w), make_float2(z22.z, z22.w));
        }
        carry(cJ, cM, sJ, sM);
      }
    } else {
      for (int q = 0; q < kn; ++q) {
        add(q, z[q], z[kSrc + q], z[2 * kSrc + q]);
        if ((q & 3) == 3 || q + 1 == kn) carry(cJ, cM, sJ, sM);
      }
    }
    carry(aJ, aM, cJ, cM);
    __syncwarp();
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    sm.red[wp][row * kSys + 2 * g + j] = make_float4(aJ[j].x, aJ[j].y, aM[j].x, aM[j].y);
  __syncthreads();
  for (int o = threadIdx.x; o < kOut; o += 32 * kNearWarps) {
    const int rr = t0 + o / kSys, j = o % kSys;
    if (rr < nb && j < pn) {
      float4 v = sm.red[0][o];
#pragma unroll
      for (int q = 1; q < kNearWarps; ++q) {
        const float4 u = sm.red[q][o];
        v = make_float4(v.x + u.x, v.y + u.y, v.z + u.z, v.w + u.w);
      }
      const double sc = a.xscale ? a.xscale[static_cast<long long>(p0 + j) * a.lds] : 1.0;
      double2* w = a.w.at(p0 + j, a.sys);
      const int id = a.leaf_rwg[r0 + rr];
      w[id] = c2(sc * v.x, sc * v.y);
      w[a.N + id] = c2(sc * v.z, sc * v.w);
    }
  }
  cp_async_wait<0>();
}

// Systems per CTA: 8 from 5 systems on, 4 for 3 or 4, else 2 (lanes without
// a system would multiply zeros).
inline int near_tile_groups(int Ra) { return Ra > 4 ? 4 : Ra > 2 ? 2 : 1; }

void launch_near_tile(const Plan& P, const NearBatchArg& a, const void* packed, cudaStream_t s) {
  const int G = near_tile_groups(a.R);
  const dim3 grid(static_cast<int>(P.h_near_sptr.size()) - 1, (a.R + 2 * G - 1) / (2 * G),
                  (P.max_leaf_rwgs * G + 31) / 32);
  auto go = [&](auto* f, size_t smem) {
    // (a constant: set to the same value by every call of every thread)
    MLFMA_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    f<<<grid, 32 * kNearWarps, smem, s>>>(a, static_cast<const float4*>(packed));
  };
  if (G == 4)
    go(near_batch_tile_kernel<4>, sizeof(NearTile<4>));
  else if (G == 2)
    go(near_batch_tile_kernel<2>, sizeof(NearTile<2>));
  else
    go(near_batch_tile_kernel<1>, sizeof(NearTile<1>));
  MLFMA_CUDA(cudaGetLastError());
}

// The rows of X into packed complex64 groups (blas1::Pack)
__global__ void pack_kernel(const double2* X, long long ldx, long long n, blas1::Pack p) {
  const int a = blockIdx.y;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    blas1::pack_row(p, n, a, i, X[a * ldx + i]);
}

// The batched vector steps on one stream with their results on the host, for
// up to R positions.
struct BatchOps : blas1::Vec {
  Plan* P;           // its device status is read at every host sync
  double* alpha;     // [R]
  int* mdev;         // [R]
  double2* ydev;     // [R][kMaxBasis]
  std::vector<C> hbuf;

  void fetch(int Ra) {
    hbuf.resize(static_cast<size_t>(Ra) * blas1::kLdh);
    MLFMA_CUDA(cudaMemcpyAsync(hbuf.data(), h, hbuf.size() * sizeof(double2), cudaMemcpyDeviceToHost, s));
    fetch_device_status(*P, s);
    MLFMA_CUDA(cudaStreamSynchronize(s));
    raise_device_status(*P);
  }
  // norms of the operand for Ra positions, or of w = b - w
  std::vector<double> norms_host(int Ra, const int* sys, VecRef w, const VecRef* b = nullptr) {
    if (b)
      residuals(Ra, sys, w, *b);
    else
      norms(Ra, sys, w);
    fetch(Ra);
    std::vector<double> out(Ra);
    for (int a = 0; a < Ra; ++a) out[a] = std::sqrt(hbuf[static_cast<size_t>(a) * blas1::kLdh].real());
    return out;
  }
  // CGS2 of w_a against V_a[0..nv): hcol[a][j] and ||w_a|| after projection
  void orthogonalise_host(int Ra, const int* sys, VecRef V, VecRef w, int nv, std::vector<std::vector<C>>& hcol,
                          std::vector<double>& hn) {
    orthogonalise(Ra, sys, V, w, nv);
    fetch(Ra);
    hcol.assign(Ra, std::vector<C>(nv));
    hn.assign(Ra, 0.0);
    for (int a = 0; a < Ra; ++a) {
      const C* hp = hbuf.data() + static_cast<size_t>(a) * blas1::kLdh;
      for (int j = 0; j < nv; ++j) hcol[a][j] = hp[j] + hp[blas1::kMaxBasis + j];
      hn[a] = std::sqrt(hp[2 * blas1::kMaxBasis].real());
    }
  }
  void scale_host(int Ra, const int* sys, VecRef src, VecRef dst, const std::vector<double>& al) {
    MLFMA_CUDA(cudaMemcpyAsync(alpha, al.data(), Ra * sizeof(double), cudaMemcpyHostToDevice, s));
    scale(Ra, sys, src, dst, alpha);
  }
  void combine_host(int Ra, const int* sys, VecRef V, VecRef x, const std::vector<std::vector<C>>& y, bool acc) {
    std::vector<int> m(Ra);
    std::vector<C> yy(static_cast<size_t>(Ra) * blas1::kMaxBasis, C(0.0));
    for (int a = 0; a < Ra; ++a) {
      m[a] = static_cast<int>(y[a].size());
      std::copy(y[a].begin(), y[a].end(), yy.begin() + static_cast<size_t>(a) * blas1::kMaxBasis);
    }
    MLFMA_CUDA(cudaMemcpyAsync(mdev, m.data(), Ra * sizeof(int), cudaMemcpyHostToDevice, s));
    MLFMA_CUDA(cudaMemcpyAsync(ydev, yy.data(), yy.size() * sizeof(double2), cudaMemcpyHostToDevice, s));
    combine(Ra, sys, V, x, mdev, 0, ydev, blas1::kMaxBasis, acc);
  }
};

}  // namespace

void near_apply_batch(Plan& P, int R, const double2* X, long long ldx, double2* W, long long ldw, float2* packed,
                      cudaStream_t s) {
  const long long n = 2LL * P.N;
  const blas1::Pack p{packed, 2 * near_tile_groups(R)};
  pack_kernel<<<dim3(static_cast<unsigned>(std::min<long long>((n + 255) / 256, 1184)), R), 256, 0, s>>>(X, ldx, n, p);
  const NearBatchArg a{P.d_leaf_rwg, P.d_leaf_ptr,         P.d_near_sptr, P.d_near_src, P.d_near_zoff,
                       P.d_near_z32, VecRef{W, ldw, 0, 0}, nullptr,       nullptr,      0,
                       P.N,          R};
  launch_near_tile(P, a, packed, s);
}

std::vector<char> fgmres_batch_solve(Plan& P, int R, double* xh, const double* rhs, int itr_max, int mr, double tol_abs,
                        double tol_rel, int inner_its, std::vector<SolveStats>& st,
                        std::vector<std::vector<double>>& hist, double& seconds, int prec) {
  if (R < 1) throw std::invalid_argument("R must be positive");
  if (prec == 1 && P.precision != 1) throw std::invalid_argument("plan was not created with mixed precision");
  if (mr < 1 || mr + 1 > blas1::kMaxBasis) throw std::invalid_argument("mr must be in 1..63");
  if (inner_its < 0 || inner_its + 1 > blas1::kMaxBasis) throw std::invalid_argument("inner_its must be in 0..63");
  const auto t0 = std::chrono::steady_clock::now();
  MLFMA_CUDA(cudaSetDevice(P.device));
  reserve_batch(P);
  cudaStream_t s = P.stream;
  const long long n = 2LL * P.N;
  const long long vs = static_cast<long long>(mr + 1) * n;       // per-system basis stride
  const long long zs = static_cast<long long>(mr) * n;
  const long long qs = static_cast<long long>(inner_its + 1) * n;
  const int G = std::min(R, kBatchSlots);  // staging rows: one batched apply at a time
  const size_t Rz = static_cast<size_t>(R);
  // work arrays (counts of complex128 values), in one block of the plan's
  // arena: no allocation when the last call's block is large enough
  enum { kX, kB, kR, kV, kZ, kQ, kXs, kWs, kPart, kCount, kH, kAlpha, kM, kY, kSys, kInner, kPack, kN };
  const size_t cnt[kN] = {Rz * n, Rz * n, Rz * n, Rz * vs, inner_its > 0 ? Rz * zs : 0, inner_its > 0 ? Rz * qs : 0,
                          static_cast<size_t>(G) * n, static_cast<size_t>(G) * n, blas1::part_count(n, R), Rz,
                          Rz * blas1::kLdh, Rz, Rz, Rz * blas1::kMaxBasis, Rz,
                          inner_its > 0 ? blas1::Inner::bytes(R, inner_its) / sizeof(double2) + 1 : 0,
                          // complex64 values of 2N unknowns for whole groups of positions
                          inner_its > 0 ? (Rz + 7) / 8 * 8 * n / 2 : 0};
  size_t work_bytes = 0;
  for (size_t c : cnt) work_bytes += (c * sizeof(double2) + 255) & ~size_t(255);
  P.arena.reserve(work_bytes);
  double2* wk[kN];
  for (int i = 0; i < kN; ++i) wk[i] = cnt[i] ? static_cast<double2*>(P.arena.get(cnt[i] * sizeof(double2))) : nullptr;
  double2 *x = wk[kX], *b = wk[kB], *r = wk[kR], *V = wk[kV], *Zd = wk[kZ], *Q = wk[kQ], *Xs = wk[kXs], *Ws = wk[kWs];
  BatchOps ops{};
  ops.s = s;
  ops.n = n;
  ops.part = wk[kPart];
  ops.count = reinterpret_cast<unsigned*>(wk[kCount]);
  ops.h = wk[kH];
  ops.clusters = blas1::clusters_fit();
  ops.P = &P;
  ops.alpha = reinterpret_cast<double*>(wk[kAlpha]);
  ops.mdev = reinterpret_cast<int*>(wk[kM]);
  ops.ydev = wk[kY];
  int* sysd = reinterpret_cast<int*>(wk[kSys]);
  // inner GMRES state on the device (one row per lockstep position)
  blas1::Inner ib{};
  if (inner_its > 0) ib = blas1::Inner::carve(wk[kInner], R, inner_its);
  MLFMA_CUDA(cudaMemsetAsync(ops.count, 0, Rz * sizeof(double2), s));
  MLFMA_CUDA(cudaMemsetAsync(P.d_status, 0, sizeof(int), s));
  MLFMA_CUDA(cudaMemcpyAsync(x, xh, static_cast<size_t>(R) * n * sizeof(double2), cudaMemcpyHostToDevice, s));
  MLFMA_CUDA(cudaMemcpyAsync(b, rhs, static_cast<size_t>(R) * n * sizeof(double2), cudaMemcpyHostToDevice, s));
  st.assign(R, SolveStats());
  hist.assign(R, {});

  auto set_sys = [&](const std::vector<int>& list) {
    MLFMA_CUDA(cudaMemcpyAsync(sysd, list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  };
  auto sysref = [](double2* p, long long stride, long long off) { return VecRef{p, stride, off, 1}; };
  auto posref = [&](double2* p) { return VecRef{p, n, 0, 0}; };
  // out_q (offset off within its system block of stride stride) = A in_q,
  // in groups of G through the staging rows; list = systems
  auto batched_apply = [&](const std::vector<int>& list, VecRef in, VecRef out) {
    for (size_t g0 = 0; g0 < list.size(); g0 += G) {
      const int rn = static_cast<int>(std::min<size_t>(G, list.size() - g0));
      std::vector<int> part(list.begin() + g0, list.begin() + g0 + rn);
      set_sys(part);
      ops.copy(rn, sysd, in, posref(Xs));
      if (prec == 1) {
        apply_batch_mixed_device(P, rn, Xs, n, Ws, n, s);
      } else {
        for (int j = 0; j < rn; ++j) apply_device(P, Xs + static_cast<long long>(j) * n, Ws + static_cast<long long>(j) * n, s);
      }
      ops.copy(rn, sysd, posref(Ws), out);
      for (int q : part) st[q].matvecs++;
    }
  };
  // true residuals r_q = b_q - A x_q, returns ||r_q|| per listed system
  auto true_residuals = [&](const std::vector<int>& list) {
    batched_apply(list, sysref(x, n, 0), sysref(r, n, 0));
    set_sys(list);
    const int Ra = static_cast<int>(list.size());
    // r holds A x: r = b - r in place
    const VecRef br = sysref(b, n, 0);
    return ops.norms_host(Ra, sysd, sysref(r, n, 0), &br);
  };
  auto packed = [&](int Ra) { return blas1::Pack{reinterpret_cast<float2*>(wk[kPack]), 2 * near_tile_groups(Ra)}; };
  // z_q = (inner_its GMRES steps on Z_near from zero) applied to v_q, q in
  // list: every step is two launches (four past the clusters' range), and the
  // host waits for none of them
  auto precondition_steps = [&](int Ra) {
    for (int j = 0; j < inner_its; ++j) {
      // the preconditioner's near field is the complex64 copy at either precision
      NearBatchArg na{P.d_leaf_rwg,  P.d_leaf_ptr,              P.d_near_sptr, P.d_near_src, P.d_near_zoff,
                      P.d_near_z32,  sysref(Q, qs, (j + 1) * n), sysd,          ib.vs + j,    ib.ld,
                      P.N,           Ra};
      launch_near_tile(P, na, wk[kPack], s);
      ops.orthogonalise(Ra, sysd, sysref(Q, qs, 0), sysref(Q, qs, (j + 1) * n), j + 1, &ib, packed(Ra));
    }
    MLFMA_CUDA(cudaGetLastError());
  };
  // With apply.graph 1 the launches of the inner steps are captured once as a
  // CUDA graph on the inner basis (v copied into it, z combined out of it) and
  // replayed at every outer step; the graph is captured again only when the
  // number of iterating systems changes (the system list itself is read from
  // the device at replay).
  cudaGraphExec_t pexec = nullptr;
  int pexec_ra = 0;
  struct GraphGuard {
    cudaGraphExec_t& e;
    ~GraphGuard() {
      if (e) cudaGraphExecDestroy(e);
    }
  } pguard{pexec};
  auto precondition = [&](const std::vector<int>& list, long long voff, long long zoff) {
    const int Ra = static_cast<int>(list.size());
    set_sys(list);
    for (int q : list) st[q].near_products += inner_its;
    ops.inner_start(Ra, sysd, sysref(V, vs, voff), sysref(Q, qs, 0), ib, packed(Ra));
    if (P.tuning.graph != 1) {
      precondition_steps(Ra);
    } else {
      if (pexec != nullptr && pexec_ra != Ra) {
        MLFMA_CUDA(cudaGraphExecDestroy(pexec));
        pexec = nullptr;
      }
      if (pexec == nullptr) {
        MLFMA_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        try {
          precondition_steps(Ra);
        } catch (...) {
          cudaGraph_t gr = nullptr;
          cudaStreamEndCapture(s, &gr);
          if (gr) cudaGraphDestroy(gr);
          throw;
        }
        cudaGraph_t gr = nullptr;
        MLFMA_CUDA(cudaStreamEndCapture(s, &gr));
        const cudaError_t e = cudaGraphInstantiate(&pexec, gr, 0);
        cudaGraphDestroy(gr);
        MLFMA_CUDA(e);
        pexec_ra = Ra;
      }
      MLFMA_CUDA(cudaGraphLaunch(pexec, s));
    }
    ops.combine(Ra, sysd, sysref(Q, qs, 0), sysref(Zd, zs, zoff), ib.m, 0, ib.y, ib.ld, false);
    // a learned correction of each z, when a network is attached to the plan
    if (const __nv_bfloat16* wl = lp_attached(P))
      for (int q : list) lp_forward(P, wl, V + q * vs + voff, Zd + q * zs + zoff, Zd + q * zs + zoff, false, s);
  };

  const double eps = 1e-16;
  std::vector<int> all(R);
  for (int q = 0; q < R; ++q) all[q] = q;
  // initial residuals: r = b without an apply for the systems that start from zero
  std::vector<int> from_x;
  for (int q = 0; q < R; ++q) {
    const double* xq = xh + 2 * q * n;
    if (std::any_of(xq, xq + 2 * n, [](double v) { return v != 0.0; }))
      from_x.push_back(q);
    else
      MLFMA_CUDA(cudaMemsetAsync(r + q * n, 0, n * sizeof(double2), s));
  }
  if (!from_x.empty()) batched_apply(from_x, sysref(x, n, 0), sysref(r, n, 0));
  set_sys(all);
  const VecRef b_all = sysref(b, n, 0);
  std::vector<double> rnorm = ops.norms_host(R, sysd, sysref(r, n, 0), &b_all);
  std::vector<double> bnorm = ops.norms_host(R, sysd, b_all);
  std::vector<double> error(R);
  std::vector<char> conv(R, 0);
  std::vector<int> live, total(R, 0);
  for (int q = 0; q < R; ++q) {
    if (bnorm[q] < eps) bnorm[q] = 1.0;
    error[q] = rnorm[q] / bnorm[q];
    st[q].rel_residual = error[q];
    if (error[q] < tol_rel || error[q] < tol_abs)
      conv[q] = 1;
    else
      live.push_back(q);
  }
  const int ld = mr + 1;
  std::vector<std::vector<C>> H(R), cs(R), sn(R), sv(R);
  std::vector<int> k_used(R, 0);
  for (int cycle = 1; !live.empty(); ++cycle) {
    // start of a cycle for every live system
    set_sys(live);
    {
      std::vector<double> inv(live.size());
      for (size_t a = 0; a < live.size(); ++a) inv[a] = 1.0 / rnorm[live[a]];
      ops.scale_host(static_cast<int>(live.size()), sysd, sysref(r, n, 0), sysref(V, vs, 0), inv);
    }
    for (int q : live) {
      st[q].restarts = cycle;
      H[q].assign(static_cast<size_t>(ld) * mr, C(0.0));
      cs[q].assign(mr, C(0.0));
      sn[q].assign(mr, C(0.0));
      sv[q].assign(mr + 1, C(0.0));
      sv[q][0] = rnorm[q];
      k_used[q] = 0;
    }
    std::vector<int> act = live;  // systems still stepping in this cycle
    for (int k = 0; k < mr && !act.empty(); ++k) {
      std::vector<int> step;
      for (int q : act)
        if (total[q] < itr_max) step.push_back(q);
      if (step.empty()) break;
      for (int q : step) {
        ++total[q];
        k_used[q] = k + 1;
      }
      VecRef zk = inner_its > 0 ? sysref(Zd, zs, k * n) : sysref(V, vs, k * n);
      if (inner_its > 0) precondition(step, k * n, k * n);
      // w_q = A z_q into the next basis slot, then CGS2 against V_q[0..k]
      batched_apply(step, zk, sysref(V, vs, (k + 1) * n));
      set_sys(step);
      const int Ra = static_cast<int>(step.size());
      std::vector<std::vector<C>> hcol;
      std::vector<double> hn;
      ops.orthogonalise_host(Ra, sysd, sysref(V, vs, 0), sysref(V, vs, (k + 1) * n), k + 1, hcol, hn);
      std::vector<double> sc(Ra, 1.0);
      std::vector<int> next;
      for (int a = 0; a < Ra; ++a) {
        const int q = step[a];
        std::vector<C>& Hq = H[q];
        for (int j = 0; j <= k; ++j) Hq[j + static_cast<size_t>(k) * ld] = hcol[a][j];
        Hq[k + 1 + static_cast<size_t>(k) * ld] = hn[a];
        if (hn[a] < eps * rnorm[q]) continue;  // breakdown: this cycle ends for q
        sc[a] = 1.0 / hn[a];
        for (int j = 0; j < k; ++j) blas1::givens_apply(Hq[j + k * ld], Hq[j + 1 + k * ld], cs[q][j], sn[q][j]);
        blas1::givens_make(Hq[k + k * ld], Hq[k + 1 + k * ld], cs[q][k], sn[q][k]);
        blas1::givens_apply(Hq[k + k * ld], Hq[k + 1 + k * ld], cs[q][k], sn[q][k]);
        Hq[k + 1 + k * ld] = C(0.0);
        blas1::givens_apply(sv[q][k], sv[q][k + 1], cs[q][k], sn[q][k]);
        error[q] = std::abs(sv[q][k + 1]) / bnorm[q];
        hist[q].push_back(error[q]);
        if (!(error[q] < tol_rel || error[q] < tol_abs)) next.push_back(q);
      }
      ops.scale_host(Ra, sysd, sysref(V, vs, (k + 1) * n), sysref(V, vs, (k + 1) * n), sc);
      act = next;
    }
    // update x_q with the cycle's least-squares solution, then true residuals
    set_sys(live);
    std::vector<std::vector<C>> y(live.size());
    for (size_t a = 0; a < live.size(); ++a) {
      const int q = live[a];
      blas1::back_substitute(H[q], ld, sv[q], std::min(k_used[q], mr), y[a]);
    }
    ops.combine_host(static_cast<int>(live.size()), sysd, inner_its > 0 ? sysref(Zd, zs, 0) : sysref(V, vs, 0),
                sysref(x, n, 0), y, true);
    const std::vector<double> rn = true_residuals(live);
    std::vector<int> keep;
    for (size_t a = 0; a < live.size(); ++a) {
      const int q = live[a];
      rnorm[q] = rn[a];
      error[q] = rn[a] / bnorm[q];
      st[q].iterations = total[q];
      st[q].rel_residual = error[q];
      if (error[q] < tol_rel || error[q] < tol_abs) {
        conv[q] = 1;
        continue;
      }
      if (total[q] >= itr_max) continue;
      if (error[q] > 100.0 * tol_rel && cycle > 8 && error[q] > 1000.0 * tol_rel) continue;  // divergence abort
      keep.push_back(q);
    }
    live = keep;
  }
  MLFMA_CUDA(cudaMemcpyAsync(xh, x, static_cast<size_t>(R) * n * sizeof(double2), cudaMemcpyDeviceToHost, s));
  fetch_device_status(P, s);
  MLFMA_CUDA(cudaStreamSynchronize(s));
  raise_device_status(P);
  if (P.arena.cap > Plan::SolveArena::kKeepBytes) P.arena.release();
  seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  for (int q = 0; q < R; ++q) {
    st[q].seconds = seconds;
    if (!conv[q]) st[q].iterations = total[q];
  }
  return std::vector<char>(conv);
}

}  // namespace mlfma
