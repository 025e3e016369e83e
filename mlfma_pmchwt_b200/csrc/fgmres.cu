// Flexible GMRES with a near-field preconditioner.
//
// The right preconditioner of the MLFMA system A x = b is an approximate
// solve with the near-field part of A alone (the same Z_near rows the matvec
// uses, Code/Zmartix.h:541-643): a fixed number of GMRES steps from zero on
// Z_near z = v. Because that inner solve changes from one outer step to the
// next, the outer iteration is flexible GMRES (Saad 1993): it keeps the
// preconditioned directions Z and updates x = x0 + Z y. The outer loop keeps
// MGMRES's arguments, stopping rule, true residual per cycle and divergence
// abort (Code/GMRES.h:65-217). With inner_its = 0 the preconditioner is the
// identity and the iteration is the reference's GMRES.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <complex>

#include "blas1.cuh"
#include "learned.hpp"
#include "solver.hpp"

namespace mlfma {

namespace {

using C = std::complex<double>;

template <class Z>
struct NearArg {
  const int* leaf_rwg;
  const int* rwg_box;
  const int* leaf_ptr;
  const int* near_sptr;
  const int* near_src;
  const long long* near_zoff;
  const Z* near_z;
  const double2* x;
  const double* xscale;  // device factor applied to x; null: 1
  double2* w;
  int N;
};

// w = Z_near (xscale x): rows t and N + t of the near field, a warp per RWG; the
// entries and the arithmetic in the storage type Z (complex128 or complex64).
// x is scaled in FP64 as it is read. (near_by_rows: where this kernel is used.)
template <class Z>
__global__ void __launch_bounds__(128) near_row_kernel(NearArg<Z> a) {
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (r >= a.N) return;
  const int id = a.leaf_rwg[r];
  const int b = a.rwg_box[id];
  const int s0 = a.near_sptr[b], ns = a.near_sptr[b + 1] - s0, pitch = near_pitch(ns);
  const Z* Zr = a.near_z + a.near_zoff[b] + 3LL * (r - a.leaf_ptr[b]) * pitch;
  const double sc = a.xscale ? *a.xscale : 1.0;
  Z nJ = Cx<Z>::zero(), nM = Cx<Z>::zero();
  for (int j = lane; j < ns; j += 32) {
    const int s = a.near_src[s0 + j];
    const Z xJ = Cx<Z>::from(cscale(a.x[s], sc)), xM = Cx<Z>::from(cscale(a.x[a.N + s], sc));
    const Z z11 = Zr[j], z12 = Zr[pitch + j], z22 = Zr[2 * pitch + j];
    nJ = cfma(z11, xJ, cfma(z12, xM, nJ));
    nM = cfma(z22, xM, csub(nM, cmul(z12, xJ)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nJ.x += __shfl_xor_sync(0xffffffffu, nJ.x, o);
    nJ.y += __shfl_xor_sync(0xffffffffu, nJ.y, o);
    nM.x += __shfl_xor_sync(0xffffffffu, nM.x, o);
    nM.y += __shfl_xor_sync(0xffffffffu, nM.y, o);
  }
  if (lane == 0) {
    a.w[id] = Cx<Z>::to64(nJ);
    a.w[a.N + id] = Cx<Z>::to64(nM);
  }
}

// The same product with a CTA per (leaf box, 8 rows): the box's source values are
// gathered into shared memory (in the storage type, a row of J and a row of M; a
// list longer than kPiece piece by piece, kPieces), where the CTA's rows read
// them; the entries load 16 bytes per lane, one source in complex128 and two in
// complex64, for the two rows of a warp, always one step ahead of the arithmetic
// (the first before the sources are gathered).
// HBM- or L2-bound (each entry is read once): 4.35 M pairs in complex64 are
// 104 MB, 16 us; measured 26 us. A warp per row that gathered its sources
// from the vectors, with the three values of a pair side by side, took 31 us
// there; a CTA for all rows of a box 34 us, waiting for the fullest boxes.
// Pieces of 48 KB keep four CTAs on an SM: lists of up to 3,718 sources (15,360
// unknowns, FP64) take 155 us, 427 when staged whole. The loop over pieces takes
// the registers of the second step in flight (complex64, lists of up to 2,350
// sources: 77 us without it, 119 with it), so shorter lists go without.
constexpr int kNearThreads = 128;
constexpr int kNearRows = 2;
constexpr int kNearCtaRows = kNearRows * kNearThreads / 32;
template <class Z>
constexpr int kNearPiece = 48 * 1024 / (2 * sizeof(Z));  // sources staged at a time: 1,536 or 3,072

template <class Z>
struct alignas(16) NearVec {
  static constexpr int kPer = 16 / sizeof(Z);
  Z v[kPer];
};

template <class Z, bool kPieces>
__global__ void __launch_bounds__(kNearThreads) near_box_kernel(NearArg<Z> a) {
  using Vec = NearVec<Z>;
  extern __shared__ __align__(16) unsigned char near_stage[];
  const int b = blockIdx.x;
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  if (static_cast<int>(blockIdx.y) * kNearCtaRows >= nb) return;
  const int s0 = a.near_sptr[b], ns = a.near_sptr[b + 1] - s0, pitch = near_pitch(ns);
  const int lane = threadIdx.x & 31;
  const int t0 = blockIdx.y * kNearCtaRows + (threadIdx.x >> 5) * kNearRows;
  const int nrow = min(kNearRows, nb - t0);  // of this warp
  const Z* rows = a.near_z + a.near_zoff[b] + 3LL * t0 * pitch;
  Vec z[2][kNearRows][3];
  auto fetch = [&](int q, Vec(&f)[kNearRows][3]) {
#pragma unroll
    for (int u = 0; u < kNearRows; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (u < nrow && q < pitch) v = __ldg(reinterpret_cast<const uint4*>(rows + (3LL * u + c) * pitch + q));
        *reinterpret_cast<uint4*>(&f[u][c]) = v;
      }
  };
  int q = lane * Vec::kPer;
  fetch(q, z[0]);
  constexpr int kPiece = kNearPiece<Z>;
  Z* xJ = reinterpret_cast<Z*>(near_stage);
  Z* xM = xJ + min(pitch, kPiece);
  const double sc = a.xscale ? *a.xscale : 1.0;
  auto gather = [&](int p0) {
    const int n = min(kPiece, pitch - p0);
#pragma unroll 2
    for (int i = threadIdx.x; i < n; i += kNearThreads) {
      double2 J = c2(0.0, 0.0), M = c2(0.0, 0.0);
      if (p0 + i < ns) {
        const int s = a.near_src[s0 + p0 + i];
        J = a.x[s];
        M = a.x[a.N + s];
      }
      xJ[i] = Cx<Z>::from(cscale(J, sc));
      xM[i] = Cx<Z>::from(cscale(M, sc));
    }
    __syncthreads();
  };
  Z nJ[kNearRows], nM[kNearRows];
#pragma unroll
  for (int u = 0; u < kNearRows; ++u) nJ[u] = nM[u] = Cx<Z>::zero();
  auto add = [&](int at, int p0, const Vec(&f)[kNearRows][3]) {
    if (at >= pitch) return;
    const Vec J = *reinterpret_cast<const Vec*>(xJ + (at - p0)), M = *reinterpret_cast<const Vec*>(xM + (at - p0));
#pragma unroll
    for (int u = 0; u < kNearRows; ++u)
#pragma unroll
      for (int i = 0; i < Vec::kPer; ++i) {
        nJ[u] = cfma(f[u][0].v[i], J.v[i], cfma(f[u][1].v[i], M.v[i], nJ[u]));
        nM[u] = cfma(f[u][2].v[i], M.v[i], csub(nM[u], cmul(f[u][1].v[i], J.v[i])));
      }
  };
  constexpr int kStep = 32 * Vec::kPer;
  static_assert(kPiece % (2 * kStep) == 0, "a piece ends with a step");
  for (int p0 = 0; p0 < (kPieces ? pitch : 1); p0 += kPiece) {
    if (p0 > 0) __syncthreads();
    gather(p0);
    for (int base = p0; base < (kPieces ? min(pitch, p0 + kPiece) : pitch); base += 2 * kStep, q += 2 * kStep) {
      fetch(q + kStep, z[1]);
      add(q, p0, z[0]);
      fetch(q + 2 * kStep, z[0]);
      add(q + kStep, p0, z[1]);
    }
  }
#pragma unroll
  for (int u = 0; u < kNearRows; ++u) {
    if (u >= nrow) break;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nJ[u].x += __shfl_xor_sync(0xffffffffu, nJ[u].x, o);
      nJ[u].y += __shfl_xor_sync(0xffffffffu, nJ[u].y, o);
      nM[u].x += __shfl_xor_sync(0xffffffffu, nM[u].x, o);
      nM[u].y += __shfl_xor_sync(0xffffffffu, nM[u].y, o);
    }
    if (lane == 0) {
      const int id = a.leaf_rwg[r0 + t0 + u];
      a.w[id] = Cx<Z>::to64(nJ[u]);
      a.w[a.N + id] = Cx<Z>::to64(nM[u]);
    }
  }
}

// Row by row where it is faster (one B200, us, row kernel / box kernel):
// boxes of a few RWGs, whose CTAs leave most of their warps idle, once there
// are more of them than CTAs fit at once: complex64 at 61,440 unknowns 3.7 RWGs
// per box 18 / 26, 6.7 22 / 26, 9.3 32 / 33, at 15,360 6.7 7.8 / 8.4, 7.7 9.3 /
// 8.3, at 3,840 (505 boxes) 3.8 3.6 / 3.6; FP64 at 15,360 4.4 7.6 / 10.1, 6.7
// 8.9 / 10.1, 7.7 10.6 / 10.4, 13.7 13.7 / 12.3;
// and in FP64 entries that outgrow L2, whose loads a row's 9 warps per scheduler
// keep in flight better: 61,440 unknowns (380 MB) 72 / 78, 245,760 (1.5 GB) 268 /
// 298, but 15,360 (88 MB) 17.9 / 16.3; up to lists whose gathering by every row
// costs more: 1,264 sources (61,440 unknowns) 292 / 300, 2,018 137 / 134, 2,424
// 188 / 155.
template <class Z>
bool near_by_rows(const Plan& P) {
  const double boxes = static_cast<double>(P.h_near_sptr.size() - 1), pairs = static_cast<double>(P.near_pairs);
  if (boxes > 4 * 148 && P.N < 7 * boxes) return true;
  return sizeof(Z) == 16 && 3 * sizeof(Z) * pairs > 126e6 && pairs < 1600.0 * P.N;
}

template <class Z>
void launch_near(const Plan& P, const NearArg<Z>& a, cudaStream_t s) {
  if (near_by_rows<Z>(P)) {
    near_row_kernel<Z><<<(P.N + 3) / 4, 128, 0, s>>>(a);
    return;
  }
  const size_t smem = 2 * sizeof(Z) * static_cast<size_t>(std::min(near_pitch(P.max_near_sources), kNearPiece<Z>));
  const dim3 grid(static_cast<int>(P.h_near_sptr.size()) - 1, (P.max_leaf_rwgs + kNearCtaRows - 1) / kNearCtaRows);
  if (P.max_near_sources > kNearPiece<Z>)
    near_box_kernel<Z, true><<<grid, kNearThreads, smem, s>>>(a);
  else
    near_box_kernel<Z, false><<<grid, kNearThreads, smem, s>>>(a);
}

}  // namespace

namespace {

void near_apply_scaled(Plan& P, const double2* x, const double* xscale, double2* w, cudaStream_t s, int prec) {
  if (prec == 1) {
    if (P.d_near_z32 == nullptr) throw std::invalid_argument("plan holds no complex64 near field");
    NearArg<float2> a{P.d_leaf_rwg,  P.d_rwg_leafbox, P.d_leaf_ptr, P.d_near_sptr, P.d_near_src, P.d_near_zoff,
                      P.d_near_z32,  x,               xscale,       w,             P.N};
    launch_near(P, a, s);
  } else {
    NearArg<double2> a{P.d_leaf_rwg, P.d_rwg_leafbox, P.d_leaf_ptr, P.d_near_sptr, P.d_near_src, P.d_near_zoff,
                       P.d_near_z,   x,               xscale,       w,             P.N};
    launch_near(P, a, s);
  }
  MLFMA_CUDA(cudaGetLastError());
}

}  // namespace

void near_apply(Plan& P, const double2* x, double2* w, cudaStream_t s, int prec) {
  near_apply_scaled(P, x, nullptr, w, s, prec);
}

namespace {

// z = approximate solution of Z_near z = v by inner_its GMRES steps from
// zero, with the complex64 copy of Z_near (the outer flexible GMRES admits
// any preconditioner; its operator and residuals stay at the solve's
// precision). The inner Hessenberg matrix, rotations and triangular solve
// stay on the GPU: the inner steps run without a host round trip, as two or
// four launches each (near-field product, then the one or three of the
// Gram-Schmidt, the last with the step's rotations). Buffers come from the
// caller's Work; the reduction scratch is the caller's Ops.
struct NearPrecond {
  Plan& P;
  cudaStream_t s;
  long long n;
  int inner_its;
  blas1::Ops ops;
  double2* Q = nullptr;  // [inner_its + 1][n], unscaled basis
  blas1::Inner in{};
  template <class W>
  NearPrecond(Plan& P_, cudaStream_t s_, int inner, W& g, const blas1::Ops& o)
      : P(P_), s(s_), n(2LL * P_.N), inner_its(inner), ops(o) {
    if (inner_its <= 0) return;
    Q = g.get(static_cast<size_t>(inner_its + 1) * n);
    in = blas1::Inner::carve(g.get(blas1::Inner::bytes(1, inner_its) / sizeof(double2) + 1), 1, inner_its);
  }
  // v into the basis, then the steps, which read and write this object's own
  // arrays only (one captured graph serves every v and z), then z
  void begin(const double2* v) { ops.inner_start(1, nullptr, ops.ref(v), ops.ref(Q), in); }
  void steps() {
    for (int j = 0; j < inner_its; ++j) {
      double2* u = Q + static_cast<long long>(j + 1) * n;
      near_apply_scaled(P, Q + static_cast<long long>(j) * n, in.vs + j, u, s, 1);
      ops.orthogonalise(1, nullptr, ops.ref(Q), ops.ref(u), j + 1, &in);
    }
  }
  void end(double2* z) {
    ops.combine(1, nullptr, ops.ref(Q), ops.ref(z), nullptr, inner_its, in.y, 0, false);
    MLFMA_CUDA(cudaGetLastError());
  }
  void launch(const double2* v, double2* z) {
    begin(v);
    steps();
    end(z);
  }
};

}  // namespace

void near_precondition(Plan& P, int inner_its, const double2* v, double2* z, cudaStream_t s) {
  if (inner_its < 1 || inner_its + 1 > blas1::kMaxBasis) throw std::invalid_argument("inner_its must be in 1..63");
  MLFMA_CUDA(cudaSetDevice(P.device));
  blas1::Work g;
  const blas1::Ops ops = blas1::make_ops(g, s, 2LL * P.N);
  NearPrecond np(P, s, inner_its, g, ops);
  np.launch(v, z);
  MLFMA_CUDA(cudaStreamSynchronize(s));  // the work arrays are freed on return
}

bool fgmres_solve(Plan& P, double* xh, const double* rhs, int itr_max, int mr, double tol_abs, double tol_rel,
                  int inner_its, SolveStats& st, std::vector<double>& history, int prec) {
  if (prec == 1 && P.precision != 1) throw std::invalid_argument("plan was not created with mixed precision");
  auto op_apply = [&](const double2* in, double2* out, cudaStream_t s) {
    if (prec == 1)
      apply_mixed_device(P, in, out, s);
    else
      apply_device(P, in, out, s);
  };
  if (mr < 1 || mr + 1 > blas1::kMaxBasis) throw std::invalid_argument("mr must be in 1..63");
  if (inner_its < 0 || inner_its + 1 > blas1::kMaxBasis) throw std::invalid_argument("inner_its must be in 0..63");
  const auto t0 = std::chrono::steady_clock::now();
  MLFMA_CUDA(cudaSetDevice(P.device));
  cudaStream_t s = P.stream;
  const long long n = 2LL * P.N;
  blas1::ArenaWork g(P, (4 + (mr + 1) + (inner_its > 0 ? mr + inner_its + 1 : 0)) * static_cast<size_t>(n) +
                            blas1::part_count(n, 1) + blas1::kMaxBasis + blas1::kLdh +
                            blas1::Inner::bytes(1, inner_its) / sizeof(double2) + 1024);
  double2* x = g.get(n);
  double2* b = g.get(n);
  double2* r = g.get(n);
  double2* w = g.get(n);
  double2* V = g.get(static_cast<size_t>(mr + 1) * n);
  double2* Zd = inner_its > 0 ? g.get(static_cast<size_t>(mr) * n) : V;
  double2* y = g.get(blas1::kMaxBasis);
  blas1::Ops ops = blas1::make_ops(g, s, n);
  MLFMA_CUDA(cudaMemcpyAsync(x, xh, n * sizeof(double2), cudaMemcpyHostToDevice, s));
  MLFMA_CUDA(cudaMemcpyAsync(b, rhs, n * sizeof(double2), cudaMemcpyHostToDevice, s));
  st = SolveStats();
  history.clear();
  std::vector<C> hcol;

  auto true_residual = [&]() {
    op_apply(x, r, s);
    st.matvecs++;
    return ops.residual(b, r);
  };
  auto finish = [&](bool ok, double err) {
    MLFMA_CUDA(cudaMemcpyAsync(xh, x, n * sizeof(double2), cudaMemcpyDeviceToHost, s));
    MLFMA_CUDA(cudaStreamSynchronize(s));
    st.rel_residual = err;
    st.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return ok;
  };
  NearPrecond np(P, s, inner_its, g, ops);
  // The preconditioner's two or four launches per inner step are captured once per
  // solve as a CUDA graph on the preconditioner's own arrays: the same graph
  // serves every basis vector. A learned correction of z, when a network is
  // attached to the plan, follows it.
  cudaGraphExec_t pgraph = nullptr;
  struct GraphGuard {
    cudaGraphExec_t& e;
    ~GraphGuard() {
      if (e) cudaGraphExecDestroy(e);
    }
  } pguard{pgraph};
  auto precondition = [&](const double2* v, double2* z) {
    st.near_products += inner_its;
    np.begin(v);
    if (!P.tuning.graph) {
      np.steps();
    } else {
      if (pgraph == nullptr) {
        MLFMA_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        try {
          np.steps();
        } catch (...) {
          cudaGraph_t gr = nullptr;
          cudaStreamEndCapture(s, &gr);
          if (gr) cudaGraphDestroy(gr);
          throw;
        }
        cudaGraph_t gr = nullptr;
        MLFMA_CUDA(cudaStreamEndCapture(s, &gr));
        const cudaError_t e = cudaGraphInstantiate(&pgraph, gr, 0);
        cudaGraphDestroy(gr);
        MLFMA_CUDA(e);
      }
      MLFMA_CUDA(cudaGraphLaunch(pgraph, s));
    }
    np.end(z);
    if (const __nv_bfloat16* wl = lp_attached(P)) lp_forward(P, wl, v, z, z, false, s);
  };

  const double eps = 1e-16;
  // a zero initial guess has r = b without an apply
  const bool from_zero = std::all_of(xh, xh + 2 * n, [](double v) { return v == 0.0; });
  double rnorm;
  if (from_zero) {
    MLFMA_CUDA(cudaMemcpyAsync(r, b, n * sizeof(double2), cudaMemcpyDeviceToDevice, s));
    rnorm = ops.norm(b);
  } else {
    rnorm = true_residual();
  }
  double bnorm = ops.norm(b);
  if (bnorm < eps) bnorm = 1.0;
  double error = rnorm / bnorm;
  if (error < tol_rel || error < tol_abs) return finish(true, error);

  const int ld = mr + 1;
  std::vector<C> H(static_cast<size_t>(ld) * mr), cs(mr), sn(mr), sv(mr + 1), yy;
  int total = 0;
  for (int cycle = 1; cycle <= itr_max; ++cycle) {
    st.restarts = cycle;
    ops.scale(r, 1.0 / rnorm, V);
    std::fill(sv.begin(), sv.end(), C(0.0));
    sv[0] = rnorm;
    std::fill(H.begin(), H.end(), C(0.0));
    int k_used = 0;
    for (int k = 0; k < mr; ++k) {
      if (total >= itr_max) break;
      ++total;
      k_used = k + 1;
      const double2* vk = V + static_cast<long long>(k) * n;
      double2* zk = Zd + static_cast<long long>(k) * n;
      if (inner_its > 0) precondition(vk, zk);
      op_apply(zk, w, s);
      st.matvecs++;
      const double h_next = ops.orthogonalise_host(V, k + 1, w, hcol);
      for (int j = 0; j <= k; ++j) H[j + static_cast<size_t>(k) * ld] = hcol[j];
      H[k + 1 + static_cast<size_t>(k) * ld] = h_next;
      if (h_next < eps * rnorm) break;
      ops.scale(w, 1.0 / h_next, V + static_cast<long long>(k + 1) * n);
      for (int j = 0; j < k; ++j) blas1::givens_apply(H[j + k * ld], H[j + 1 + k * ld], cs[j], sn[j]);
      blas1::givens_make(H[k + k * ld], H[k + 1 + k * ld], cs[k], sn[k]);
      blas1::givens_apply(H[k + k * ld], H[k + 1 + k * ld], cs[k], sn[k]);
      H[k + 1 + k * ld] = C(0.0);
      blas1::givens_apply(sv[k], sv[k + 1], cs[k], sn[k]);
      error = std::abs(sv[k + 1]) / bnorm;
      history.push_back(error);
      if (error < tol_rel || error < tol_abs) break;
    }
    const int m = std::min(k_used, mr);
    blas1::back_substitute(H, ld, sv, m, yy);
    if (m > 0) {
      MLFMA_CUDA(cudaMemcpyAsync(y, yy.data(), m * sizeof(double2), cudaMemcpyHostToDevice, s));
      ops.combine(1, nullptr, ops.ref(Zd), ops.ref(x), nullptr, m, y, 0, true);
    }
    rnorm = true_residual();
    error = rnorm / bnorm;
    st.iterations = total;
    if (error < tol_rel || error < tol_abs) return finish(true, error);
    if (total >= itr_max) return finish(false, error);
    if (error > 100.0 * tol_rel && cycle > 8 && error > 1000.0 * tol_rel) return finish(false, error);
  }
  st.iterations = total;
  return finish(false, error);
}

}  // namespace mlfma
