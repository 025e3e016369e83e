// Lockstep multi-right-hand-side FGMRES: R independent systems A x_q = b_q
// (one per plane-wave incidence, say) iterate together, so each Arnoldi
// step costs one batched operator apply (leaf patterns and near-field
// entries read once per group of right-hand sides, matvec_kernels.cu) and
// one batched near-field product per inner step, and every Gram-Schmidt /
// update step is one launch over all active systems. The outer Arnoldi step
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
#include "cplx.cuh"
#include "plan.hpp"
#include "learned.hpp"
#include "solver.hpp"

namespace mlfma {

namespace {

using C = std::complex<double>;
using blas1::VecRef;

// w_a = Z_near x_a for every position (warp per RWG, 4 right-hand sides per
// warp): the near-field rows of the plan, read once per group of four.
template <class Z>
struct NearBatchArg {
  const int* leaf_rwg;
  const int* rwg_box;
  const int* leaf_ptr;
  const int* near_sptr;
  const int* near_src;
  const long long* near_zoff;
  const Z* near_z;
  VecRef x, w;
  const int* sys;
  const double* xscale;  // factor of position a's x at xscale[a * lds]
  int lds;
  int N, R;
};

constexpr int kNearRB = 4;

template <class Z>
__global__ void __launch_bounds__(128) near_batch_kernel(NearBatchArg<Z> a) {
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (r >= a.N) return;
  const int p0 = blockIdx.y * kNearRB, pn = min(kNearRB, a.R - p0);
  const int id = a.leaf_rwg[r];
  const int b = a.rwg_box[id];
  const int s0 = a.near_sptr[b], ns = a.near_sptr[b + 1] - s0;
  const int tl = r - a.leaf_ptr[b];
  const Z* Zr = a.near_z + 3 * (a.near_zoff[b] + static_cast<long long>(tl) * ns);
  Z nJ[kNearRB], nM[kNearRB];
  const double2* xs[kNearRB];
  double sc[kNearRB];
#pragma unroll
  for (int j = 0; j < kNearRB; ++j) {
    nJ[j] = nM[j] = Cx<Z>::zero();
    xs[j] = j < pn ? a.x.at(p0 + j, a.sys) : nullptr;
    sc[j] = j < pn ? a.xscale[static_cast<long long>(p0 + j) * a.lds] : 0.0;
  }
  for (int q = lane; q < ns; q += 32) {
    const int src = a.near_src[s0 + q];
    const Z z11 = Zr[3 * q], z12 = Zr[3 * q + 1], z22 = Zr[3 * q + 2];
#pragma unroll
    for (int j = 0; j < kNearRB; ++j) {
      if (j < pn) {
        const Z xJ = Cx<Z>::from(cscale(xs[j][src], sc[j])), xM = Cx<Z>::from(cscale(xs[j][a.N + src], sc[j]));
        nJ[j] = cfma(z11, xJ, cfma(z12, xM, nJ[j]));
        nM[j] = cfma(z22, xM, csub(nM[j], cmul(z12, xJ)));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kNearRB; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nJ[j].x += __shfl_xor_sync(0xffffffffu, nJ[j].x, o);
      nJ[j].y += __shfl_xor_sync(0xffffffffu, nJ[j].y, o);
      nM[j].x += __shfl_xor_sync(0xffffffffu, nM[j].x, o);
      nM[j].y += __shfl_xor_sync(0xffffffffu, nM[j].y, o);
    }
    if (lane == 0 && j < pn) {
      double2* w = a.w.at(p0 + j, a.sys);
      w[id] = Cx<Z>::to64(nJ[j]);
      w[a.N + id] = Cx<Z>::to64(nM[j]);
    }
  }
}

// The same products with one CTA per (leaf box, group of kNearBoxRB systems):
// the box's source values are staged once in shared memory ([system][J, M]
// [source]) and read there by every target row of the box, instead of each
// row gathering them again from the vectors. Each row's sums are formed in
// near_batch_kernel's order (lane-strided sources, then the warp shuffle),
// so the results are identical.
constexpr int kNearBoxRB = 8;
constexpr size_t kNearBoxSmemMax = 160 * 1024;

template <class Z>
__global__ void __launch_bounds__(128) near_batch_box_kernel(NearBatchArg<Z> a) {
  extern __shared__ __align__(16) unsigned char near_smem[];
  Z* xsm = reinterpret_cast<Z*>(near_smem);
  __shared__ const double2* xbase[kNearBoxRB];
  __shared__ double xsc[kNearBoxRB];
  const int b = blockIdx.x;
  const int p0 = blockIdx.y * kNearBoxRB, pn = min(kNearBoxRB, a.R - p0);
  const int s0 = a.near_sptr[b], ns = a.near_sptr[b + 1] - s0;
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  if (threadIdx.x < pn) {
    xbase[threadIdx.x] = a.x.at(p0 + threadIdx.x, a.sys);
    xsc[threadIdx.x] = a.xscale[static_cast<long long>(p0 + threadIdx.x) * a.lds];
  }
  __syncthreads();
  // one source per thread, the values of 4 systems in flight at once
  constexpr int kStage = 4;
  for (int q = threadIdx.x; q < ns; q += blockDim.x) {
    const int src = a.near_src[s0 + q];
#pragma unroll
    for (int j0 = 0; j0 < kNearBoxRB; j0 += kStage) {
      double2 vJ[kStage], vM[kStage];
#pragma unroll
      for (int j = 0; j < kStage; ++j)
        if (j0 + j < pn) {
          vJ[j] = xbase[j0 + j][src];
          vM[j] = xbase[j0 + j][a.N + src];
        }
#pragma unroll
      for (int j = 0; j < kStage; ++j)
        if (j0 + j < pn) {
          xsm[(2 * (j0 + j)) * ns + q] = Cx<Z>::from(cscale(vJ[j], xsc[j0 + j]));
          xsm[(2 * (j0 + j) + 1) * ns + q] = Cx<Z>::from(cscale(vM[j], xsc[j0 + j]));
        }
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int nw = blockDim.x / 32;
  // each warp takes two target rows at a time (tl and tl + nw): every
  // staged source value read from shared memory serves both rows, and the
  // two rows' near-field loads are in flight together. Each row's sums are
  // formed in the same order as with one row per pass.
  for (int tl = threadIdx.x >> 5; tl < nb; tl += 2 * nw) {
    const int tl2 = tl + nw;
    const bool two = tl2 < nb;
    const Z* Zr = a.near_z + 3 * (a.near_zoff[b] + static_cast<long long>(tl) * ns);
    const Z* Zr2 = a.near_z + 3 * (a.near_zoff[b] + static_cast<long long>(two ? tl2 : tl) * ns);
    Z nJ[kNearBoxRB], nM[kNearBoxRB], nJ2[kNearBoxRB], nM2[kNearBoxRB];
#pragma unroll
    for (int j = 0; j < kNearBoxRB; ++j) nJ[j] = nM[j] = nJ2[j] = nM2[j] = Cx<Z>::zero();
    for (int q = lane; q < ns; q += 32) {
      const Z z11 = Zr[3 * q], z12 = Zr[3 * q + 1], z22 = Zr[3 * q + 2];
      const Z y11 = Zr2[3 * q], y12 = Zr2[3 * q + 1], y22 = Zr2[3 * q + 2];
#pragma unroll
      for (int j = 0; j < kNearBoxRB; ++j) {
        if (j < pn) {
          const Z xJ = xsm[(2 * j) * ns + q], xM = xsm[(2 * j + 1) * ns + q];
          nJ[j] = cfma(z11, xJ, cfma(z12, xM, nJ[j]));
          nM[j] = cfma(z22, xM, csub(nM[j], cmul(z12, xJ)));
          nJ2[j] = cfma(y11, xJ, cfma(y12, xM, nJ2[j]));
          nM2[j] = cfma(y22, xM, csub(nM2[j], cmul(y12, xJ)));
        }
      }
    }
    const int id = a.leaf_rwg[r0 + tl];
    const int id2 = a.leaf_rwg[r0 + (two ? tl2 : tl)];
#pragma unroll
    for (int j = 0; j < kNearBoxRB; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        nJ[j].x += __shfl_xor_sync(0xffffffffu, nJ[j].x, o);
        nJ[j].y += __shfl_xor_sync(0xffffffffu, nJ[j].y, o);
        nM[j].x += __shfl_xor_sync(0xffffffffu, nM[j].x, o);
        nM[j].y += __shfl_xor_sync(0xffffffffu, nM[j].y, o);
        nJ2[j].x += __shfl_xor_sync(0xffffffffu, nJ2[j].x, o);
        nJ2[j].y += __shfl_xor_sync(0xffffffffu, nJ2[j].y, o);
        nM2[j].x += __shfl_xor_sync(0xffffffffu, nM2[j].x, o);
        nM2[j].y += __shfl_xor_sync(0xffffffffu, nM2[j].y, o);
      }
      if (lane == 0 && j < pn) {
        double2* w = a.w.at(p0 + j, a.sys);
        w[id] = Cx<Z>::to64(nJ[j]);
        w[a.N + id] = Cx<Z>::to64(nM[j]);
        if (two) {
          w[id2] = Cx<Z>::to64(nJ2[j]);
          w[a.N + id2] = Cx<Z>::to64(nM2[j]);
        }
      }
    }
  }
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

std::vector<char> fgmres_batch_solve(Plan& P, int R, double* xh, const double* rhs, int itr_max, int mr, double tol_abs,
                        double tol_rel, int inner_its, std::vector<SolveStats>& st,
                        std::vector<std::vector<double>>& hist, double& seconds, int prec) {
  if (R < 1) throw std::invalid_argument("R must be positive");
  if (prec == 1 && P.precision != 1) throw std::invalid_argument("plan was not created with mixed precision");
  if (mr < 1 || mr + 1 > blas1::kMaxBasis) throw std::invalid_argument("mr must be in 1..63");
  if (inner_its < 0 || inner_its + 1 > blas1::kMaxBasis) throw std::invalid_argument("inner_its must be in 0..63");
  const auto t0 = std::chrono::steady_clock::now();
  MLFMA_CUDA(cudaSetDevice(P.device));
  reserve_batch(P, R, false);
  cudaStream_t s = P.stream;
  const long long n = 2LL * P.N;
  const long long vs = static_cast<long long>(mr + 1) * n;       // per-system basis stride
  const long long zs = static_cast<long long>(mr) * n;
  const long long qs = static_cast<long long>(inner_its + 1) * n;
  const int G = std::min(R, kBatchSlots);  // staging rows: one batched apply at a time
  const size_t Rz = static_cast<size_t>(R);
  // work arrays (counts of complex128 values), in one block of the plan's
  // arena: no allocation when the last call's block is large enough
  enum { kX, kB, kR, kV, kZ, kQ, kXs, kWs, kPart, kCount, kH, kAlpha, kM, kY, kSys, kInner, kN };
  const size_t cnt[kN] = {Rz * n, Rz * n, Rz * n, Rz * vs, inner_its > 0 ? Rz * zs : 0, inner_its > 0 ? Rz * qs : 0,
                          static_cast<size_t>(G) * n, static_cast<size_t>(G) * n, blas1::part_count(n, R), Rz,
                          Rz * blas1::kLdh, Rz, Rz, Rz * blas1::kMaxBasis, Rz,
                          inner_its > 0 ? blas1::Inner::bytes(R, inner_its) / sizeof(double2) + 1 : 0};
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
        // FP64: one captured apply per row is faster than the batched apply
        // (whose FP64 leaf kernels run on the CUDA cores: 7.4 against 6.7 ms
        // per right-hand side at 245,760 unknowns)
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
  // the box-staged near-field kernel's shared memory: the largest source list
  const int nleaf = static_cast<int>(P.h_near_sptr.size()) - 1;
  int ns_max = 0;
  for (int bx = 0; bx < nleaf; ++bx) ns_max = std::max(ns_max, P.h_near_sptr[bx + 1] - P.h_near_sptr[bx]);
  const size_t box_smem = static_cast<size_t>(2 * kNearBoxRB) * ns_max * sizeof(float2);
  // The shared-memory limit is set to the same largest value on every call:
  // solves of several plans from several host threads then never lower it
  // under another's launch.
  if (inner_its > 0 && box_smem <= kNearBoxSmemMax)
    MLFMA_CUDA(cudaFuncSetAttribute(near_batch_box_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(kNearBoxSmemMax)));
  // z_q = (inner_its GMRES steps on Z_near from zero) applied to v_q, q in
  // list: every step is four launches, the host waits for none of them
  auto precondition_steps = [&](int Ra) {
    for (int j = 0; j < inner_its; ++j) {
      // the preconditioner's near field is the complex64 copy at either precision
      NearBatchArg<float2> na{P.d_leaf_rwg,  P.d_rwg_leafbox,      P.d_leaf_ptr,
                              P.d_near_sptr, P.d_near_src,         P.d_near_zoff,
                              P.d_near_z32,  sysref(Q, qs, j * n), sysref(Q, qs, (j + 1) * n),
                              sysd,          ib.vs + j,            ib.ld,
                              P.N,           Ra};
      if (box_smem <= kNearBoxSmemMax) {
        const dim3 ng(nleaf, (Ra + kNearBoxRB - 1) / kNearBoxRB);
        near_batch_box_kernel<float2><<<ng, 128, box_smem, s>>>(na);
      } else {
        const dim3 ng((P.N + 3) / 4, (Ra + kNearRB - 1) / kNearRB);
        near_batch_kernel<float2><<<ng, 128, 0, s>>>(na);
      }
      ops.orthogonalise(Ra, sysd, sysref(Q, qs, 0), sysref(Q, qs, (j + 1) * n), j + 1, &ib);
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
    ops.inner_start(Ra, sysd, sysref(V, vs, voff), sysref(Q, qs, 0), ib);
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
