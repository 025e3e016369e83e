// Many incidences at once: the plane-wave excitation of R incidences
// (RHS::computeV_PMCHWT, Code/Vm.h:150-203, with the incident vectors of
// EMSource::initPW, Code/EMSource.cpp:34-72) and the far field of R current
// vectors, bistatic (Code/RCS.h:116-192 per solution and angle, the
// dual-static study Code/RCS.h:345-425) or monostatic (each solution seen
// from its own backscatter angle, the mono-static loop Code/RCS.h:436-494).
//
// The reference runs these once per incidence inside its study loops; here
// one launch covers a chunk of incidences. The incidence and angle tables
// travel in the kernel parameters (read at launch), so the entry points
// allocate nothing and accept pageable or pinned host tables alike.
// Quadrature points are formed once per (RWG, point) and reused for every
// incidence of a chunk.
#include <cooperative_groups.h>

#include <cmath>
#include <stdexcept>
#include <type_traits>

#include "cplx.cuh"
#include "reduce.cuh"
#include "solver.hpp"

namespace mlfma {
namespace {

constexpr int kRhsChunk = 128;   // incidences per excitation launch (9 KB of parameters)
constexpr int kRhsTile = 8;      // incidences per thread (grid.y tiles)
constexpr int kFarChunk = 512;   // angles per far-field launch (12 KB of parameters)
constexpr int kFarAngles = 4;    // angles and
constexpr int kFarSols = 32;     // solutions per cluster of the bistatic far field
constexpr int kFarRwgs = 256;    // RWGs whose moments a block stages at a time,
constexpr int kFarFew = 64;      // of a body whose RWGs would leave blocks of a cluster without any
constexpr int kFarFewSols = 4;   // solutions of a block that forms the moments it sums
constexpr int kFarSlices = 8;    // blocks of a cluster, each with a slice of the RWGs
constexpr int kFarThreads = 512;

struct Geo {
  const double* xyz;
  const int* face_v;
  const int* fpos;
  const int* fneg;
  const int* vpos;
  const int* vneg;
  const double* len;
  int nq, N;
  int skew;  // the barycentric coordinates of some point do not add up to 1
  double l1[16], l2[16], l3[16], w[16];
  double2 k1;
};

Geo geo(const Plan& P) {
  Geo g{};
  g.xyz = P.d_xyz;
  g.face_v = P.d_face_v;
  g.fpos = P.d_rwg_fpos;
  g.fneg = P.d_rwg_fneg;
  g.vpos = P.d_rwg_vpos;
  g.vneg = P.d_rwg_vneg;
  g.len = P.d_rwg_len;
  g.nq = P.quad.n;
  g.N = P.N;
  for (int i = 0; i < P.quad.n; ++i) {
    g.l1[i] = P.quad.l1[i];
    g.l2[i] = P.quad.l2[i];
    g.l3[i] = P.quad.l3[i];
    g.w[i] = P.quad.w[i];
    // the rules are tabulated to 15 digits (sums within 1.1e-15 of 1), the
    // centroid of the rules of 1 and 4 points to 12 (1e-12)
    if (std::abs(1.0 - g.l1[i] - g.l2[i] - g.l3[i]) > 4e-15) g.skew = 1;
  }
  g.k1 = make_double2(P.k1.real(), P.k1.imag());
  return g;
}

__device__ __forceinline__ void load3(const double* p, double* o) {
  o[0] = p[0];
  o[1] = p[1];
  o[2] = p[2];
}

// Quadrature point i of side `side` (0: T+, 1: T-) of RWG m: position p and
// the RWG vector rho (p - free vertex on T+, free vertex - p on T-).
__device__ __forceinline__ void rwg_point(const Geo& g, int m, int side, int i, double p[3], double rho[3]) {
  const int f = side ? g.fneg[m] : g.fpos[m];
  const double* A = &g.xyz[3 * g.face_v[3 * f]];
  const double* B = &g.xyz[3 * g.face_v[3 * f + 1]];
  const double* Cc = &g.xyz[3 * g.face_v[3 * f + 2]];
  const double* fv = &g.xyz[3 * (side ? g.vneg[m] : g.vpos[m])];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    p[c] = g.l1[i] * A[c] + g.l2[i] * B[c] + g.l3[i] * Cc[c];
    rho[c] = side ? fv[c] - p[c] : p[c] - fv[c];
  }
}

struct RhsBatchArg {
  Geo g;
  double inc[kRhsChunk][9];  // per incidence: kinc, einc, hinc
  int R;
  double2* V;                // [R][2N] for this chunk
};

// thread per RWG, kRhsTile incidences (blockIdx.y tile): V[r][m], V[r][N + m]
__global__ void __launch_bounds__(128) rhs_batch_kernel(const __grid_constant__ RhsBatchArg a) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int r0 = blockIdx.y * kRhsTile;
  const Geo& g = a.g;
  if (m >= g.N) return;
  const int nr = min(kRhsTile, a.R - r0);
  const double lm = g.len[m];
  double2 ve[kRhsTile], vh[kRhsTile];
#pragma unroll
  for (int q = 0; q < kRhsTile; ++q) ve[q] = vh[q] = c2(0.0, 0.0);
  for (int i = 0; i < g.nq; ++i) {
    for (int side = 0; side < 2; ++side) {
      double p[3], rho[3];
      rwg_point(g, m, side, i, p, rho);
      const double wl = lm * g.w[i];
#pragma unroll
      for (int q = 0; q < kRhsTile; ++q) {
        if (q < nr) {
          const double* d = a.inc[r0 + q];
          const double2 e = cexp_mjkt(g.k1, d[0] * p[0] + d[1] * p[1] + d[2] * p[2]);
          const double de = d[3] * rho[0] + d[4] * rho[1] + d[5] * rho[2];
          const double dh = d[6] * rho[0] + d[7] * rho[1] + d[8] * rho[2];
          ve[q] = cadd(ve[q], cscale(e, wl * de));
          vh[q] = cadd(vh[q], cscale(e, wl * dh));
        }
      }
    }
  }
  const size_t n = 2 * static_cast<size_t>(g.N);
#pragma unroll
  for (int q = 0; q < kRhsTile; ++q)
    if (q < nr) {
      a.V[(r0 + q) * n + m] = ve[q];
      a.V[(r0 + q) * n + g.N + m] = vh[q];
    }
}

// sin and cos of |x| <= 1 by their Taylor series (the first terms left out
// are below 1e-17 and 5e-19)
__device__ __forceinline__ void sincos_series(double x, double* sn, double* cs) {
  const double z = x * x;
  double s = 1.0 / 355687428096000.0, c = -1.0 / 6402373705728000.0;
  s = fma(s, z, -1.0 / 1307674368000.0);
  c = fma(c, z, 1.0 / 20922789888000.0);
  s = fma(s, z, 1.0 / 6227020800.0);
  c = fma(c, z, -1.0 / 87178291200.0);
  s = fma(s, z, -1.0 / 39916800.0);
  c = fma(c, z, 1.0 / 479001600.0);
  s = fma(s, z, 1.0 / 362880.0);
  c = fma(c, z, -1.0 / 3628800.0);
  s = fma(s, z, -1.0 / 5040.0);
  c = fma(c, z, 1.0 / 40320.0);
  s = fma(s, z, 1.0 / 120.0);
  c = fma(c, z, -1.0 / 720.0);
  s = fma(s, z, -1.0 / 6.0);
  c = fma(c, z, 1.0 / 24.0);
  c = fma(c, z, -0.5);
  *sn = fma(s * z, x, x);
  *cs = fma(c, z, 1.0);
}

// An orthonormal basis u, v of the plane across the unit vector r, u x v = r
__device__ __forceinline__ void transverse(const double r[3], double u[3], double v[3]) {
  const bool z = fabs(r[2]) < 0.9;
  u[0] = z ? -r[1] : 0.0;
  u[1] = z ? r[0] : -r[2];
  u[2] = z ? 0.0 : r[1];
  const double q = 1.0 / sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  for (int c = 0; c < 3; ++c) u[c] *= q;
  v[0] = r[1] * u[2] - r[2] * u[1];
  v[1] = r[2] * u[0] - r[0] * u[2];
  v[2] = r[0] * u[1] - r[1] * u[0];
}

// The far-field moment A = sum l w rho e^{+j k1 r.p} of RWG m along u and v.
// The reference's factors (Code/RCS.h:140-170) follow from it: sum l w (I - r r)
// rho e = Au u + Av v and sum l w (r x rho) e = Au v - Av u.
// Per triangle, with the phase of its centroid taken out: the moments of the
// three barycentric coordinates, M_j = sum_q w l_j e^{j k1 r.(p - centroid)},
// then rho = sum_j l_j (v_j - v_free). Phases up to 1 rad from the centroid
// (vertices within 0.16 wavelengths) and a real k1 take the series instead
// of a sine, a cosine and an exponential per point: 7 points cost a third.
// All of that needs coordinates that add up to 1: with the 1e-12 that 12-digit
// centroids miss, p and rho would be off by 1e-12 times the distance from the
// origin.
__device__ __forceinline__ void far_moment_vertices(const Geo& g, int m, const double r[3], const double u[3],
                                                    const double v[3], double2& Au, double2& Av) {
  Au = Av = c2(0.0, 0.0);
  const double ln = g.len[m];
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const int f = side ? g.fneg[m] : g.fpos[m];
    const double* fv = &g.xyz[3 * (side ? g.vneg[m] : g.vpos[m])];
    double X[3][3], d[3], tc = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) load3(&g.xyz[3 * g.face_v[3 * f + j]], X[j]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double ctr = (X[0][c] + X[1][c] + X[2][c]) * (1.0 / 3.0);
      tc = fma(r[c], ctr, tc);
#pragma unroll
      for (int j = 0; j < 3; ++j) d[j] = fma(r[c], X[j][c] - ctr, c == 0 ? 0.0 : d[j]);
    }
    const double2 e0 = cexp(make_double2(-g.k1.y * tc, g.k1.x * tc));
    double2 M[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) M[j] = c2(0.0, 0.0);
    if (g.k1.y == 0.0 && fabs(g.k1.x) * fmax(fabs(d[0]), fmax(fabs(d[1]), fabs(d[2]))) <= 1.0) {
#pragma unroll
      for (int j = 0; j < 3; ++j) d[j] *= g.k1.x;
      for (int i = 0; i < g.nq; ++i) {
        double sn, cs;
        sincos_series(g.l1[i] * d[0] + g.l2[i] * d[1] + g.l3[i] * d[2], &sn, &cs);
        sn *= g.w[i];
        cs *= g.w[i];
        M[0] = cadd(M[0], c2(cs * g.l1[i], sn * g.l1[i]));
        M[1] = cadd(M[1], c2(cs * g.l2[i], sn * g.l2[i]));
        M[2] = cadd(M[2], c2(cs * g.l3[i], sn * g.l3[i]));
      }
    } else {
      for (int i = 0; i < g.nq; ++i) {
        const double t = g.l1[i] * d[0] + g.l2[i] * d[1] + g.l3[i] * d[2];
        const double2 e = cscale(cexp(make_double2(-g.k1.y * t, g.k1.x * t)), g.w[i]);
        M[0] = cadd(M[0], cscale(e, g.l1[i]));
        M[1] = cadd(M[1], cscale(e, g.l2[i]));
        M[2] = cadd(M[2], cscale(e, g.l3[i]));
      }
    }
    const double2 e = cscale(e0, side ? -ln : ln);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double q[3] = {X[j][0] - fv[0], X[j][1] - fv[1], X[j][2] - fv[2]};
      const double2 t = cmul(e, M[j]);
      Au = cfmas(q[0] * u[0] + q[1] * u[1] + q[2] * u[2], t, Au);
      Av = cfmas(q[0] * v[0] + q[1] * v[1] + q[2] * v[2], t, Av);
    }
  }
}

// The moment point by point, as the rule gives the points.
__device__ __forceinline__ void far_moment_points(const Geo& g, int m, const double r[3], const double u[3],
                                                  const double v[3], double2& Au, double2& Av) {
  Au = Av = c2(0.0, 0.0);
  const double ln = g.len[m];
  for (int i = 0; i < g.nq; ++i) {
    for (int side = 0; side < 2; ++side) {
      double p[3], rho[3];
      rwg_point(g, m, side, i, p, rho);
      const double t = p[0] * r[0] + p[1] * r[1] + p[2] * r[2];
      const double2 e = cscale(cexp(make_double2(-g.k1.y * t, g.k1.x * t)), ln * g.w[i]);
      Au = cfmas(rho[0] * u[0] + rho[1] * u[1] + rho[2] * u[2], e, Au);
      Av = cfmas(rho[0] * v[0] + rho[1] * v[1] + rho[2] * v[2], e, Av);
    }
  }
}

// kSkew: a rule whose coordinates miss 1 (it has at most four points)
template <bool kSkew>
__device__ __forceinline__ void far_moment(const Geo& g, int m, const double r[3], const double u[3],
                                           const double v[3], double2& Au, double2& Av) {
  if constexpr (kSkew)
    far_moment_points(g, m, r, u, v, Au, Av);
  else
    far_moment_vertices(g, m, r, u, v, Au, Av);
}

struct FarBatchArg {
  Geo g;
  double dir[kFarChunk][3];
  int n_angles, angle0, n_total_angles, R;
  const double2* I;  // [R][2N]
  double2* out;      // [R][n_total_angles][3]
};

// E = -j k1 (F_M . I_M - F_J . I_J), bistatic: cluster of kFarSlices blocks per
// (kFarAngles angles, kFarSols solutions), each block over a slice of the RWGs.
// A block forms the moments of kFarRwgs RWGs at its angles once, in shared
// memory, for all its solutions; a warp then sums 2 solutions x 4 angles
// over 32 RWGs at a time (with 8 pairs of solutions or fewer, 2 angles or 1).
// The blocks' sums meet in distributed shared memory, in rank order. A sum's
// order is the same whatever else is in the call, so a solution's field is too.
// FP64-bound: 361 angles x 32 solutions x 30,720 RWGs are ~0.35 ms of moments
// and 0.31 ms of sums at the FP64 rate. With a block per (angle, 4
// solutions), which formed the factors once per 4 solutions from 14 sincos
// and exp each, that call took 12.3 ms; now 1.7 ms (alone). Few solutions: with
// warps that shared the RWGs of a pair instead of its angles, 361 angles at
// 3,840 unknowns took 115 us for one solution and 142 for 16, now 101 and 129;
// at 61,440 unknowns 1,056 and 1,385, now 1,078 and 1,357.
template <bool kSkew, int kRwgs>
__global__ void __cluster_dims__(1, 1, kFarSlices) __launch_bounds__(kFarThreads, 1)
    far_batch_kernel(const __grid_constant__ FarBatchArg a) {
  __shared__ double2 A[kFarAngles][2][kRwgs];
  __shared__ double2 sums[kFarSols * kFarAngles * 2];
  const Geo& g = a.g;
  const int ang0 = blockIdx.x * kFarAngles, na = min(kFarAngles, a.n_angles - ang0);
  const int r0 = blockIdx.y * kFarSols, nr = min(kFarSols, a.R - r0);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  constexpr int kW = kFarThreads / 32;
  const int npair = (nr + 1) / 2;
  const int per = 4 * npair <= kW ? 1 : 2 * npair <= kW ? 2 : kFarAngles;  // angles of a warp
  const int pair = wp % npair, t0 = wp / npair * per;
  const bool working = t0 < kFarAngles;
  const bool two = 2 * pair + 1 < nr;
  const size_t n = 2 * static_cast<size_t>(g.N);
  const double2* I0 = a.I + (r0 + 2 * pair) * n;
  const double2* I1 = two ? I0 + n : I0;
  double2 acc[2][kFarAngles][2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int t = 0; t < kFarAngles; ++t) acc[q][t][0] = acc[q][t][1] = c2(0.0, 0.0);
  auto add = [&](int m0, auto angles) {
    constexpr int kA = decltype(angles)::value, kAhead = kRwgs == kFarRwgs ? 8 / kA : 2;
    const int first = kA == kFarAngles ? 0 : t0;
#pragma unroll kAhead
    for (int c = 0; c < kRwgs / 32; ++c) {
      const int q = 32 * c + lane, m = min(m0 + q, g.N - 1);  // moments beyond N are zero
      const double2 J0 = __ldg(I0 + m), M0 = __ldg(I0 + g.N + m);
      const double2 J1 = __ldg(I1 + m), M1 = __ldg(I1 + g.N + m);
#pragma unroll
      for (int t = 0; t < kA; ++t) {
        const double2 u = A[first + t][0][q], v = A[first + t][1][q], mu = cneg(u), mv = cneg(v);
        acc[0][t][0] = cfma(mv, M0, cfma(mu, J0, acc[0][t][0]));
        acc[0][t][1] = cfma(u, M0, cfma(mv, J0, acc[0][t][1]));
        acc[1][t][0] = cfma(mv, M1, cfma(mu, J1, acc[1][t][0]));
        acc[1][t][1] = cfma(u, M1, cfma(mv, J1, acc[1][t][1]));
      }
    }
  };
  const int tiles = (g.N + kRwgs - 1) / kRwgs;
  for (int tile = blockIdx.z; tile < tiles; tile += kFarSlices) {
    const int m0 = tile * kRwgs;
    __syncthreads();
    {
      const int q = threadIdx.x & (kRwgs - 1), m = m0 + q;
#pragma unroll 1
      for (int t = threadIdx.x / kRwgs; t < kFarAngles; t += kFarThreads / kRwgs) {
        double2 Au = c2(0.0, 0.0), Av = c2(0.0, 0.0);
        if (m < g.N && t < na) {
          double u[3], v[3];
          transverse(a.dir[ang0 + t], u, v);
          far_moment<kSkew>(g, m, a.dir[ang0 + t], u, v, Au, Av);
        }
        A[t][0][q] = Au;
        A[t][1][q] = Av;
      }
    }
    __syncthreads();
    if (!working) continue;
    if (per == 1)
      add(m0, std::integral_constant<int, 1>{});
    else if (per == 2)
      add(m0, std::integral_constant<int, 2>{});
    else
      add(m0, std::integral_constant<int, kFarAngles>{});
  }
  __syncthreads();
  double2* red = &A[0][0][0];  // [kW][2 x kFarAngles x 2]
  constexpr int kPer = 2 * kFarAngles * 2;
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int t = 0; t < kFarAngles; ++t)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (t >= per) continue;
        const double2 v = blas1::warp_sum2(acc[q][t][c]);
        if (lane == 0) red[wp * kPer + (q * kFarAngles + t) * 2 + c] = v;
      }
  __syncthreads();
  for (int i = threadIdx.x; i < npair * kPer; i += kFarThreads) {
    const int p = i / kPer, e = i - p * kPer, t = e / 2 % kFarAngles;
    sums[i] = red[(t / per * npair + p) * kPer + e - 2 * (t - t % per)];
  }
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (cl.block_rank() == 0) {
    const double2 coeff = c2(g.k1.y, -g.k1.x);  // -j k1
    for (int i = threadIdx.x; i < nr * na; i += kFarThreads) {
      const int rr = i / na, t = i - rr * na;
      double2 su = c2(0.0, 0.0), sv = c2(0.0, 0.0);
      for (int q = 0; q < kFarSlices; ++q) {
        const double2* o = cl.map_shared_rank(&sums[0], q) + (rr / 2) * kPer + ((rr & 1) * kFarAngles + t) * 2;
        su = cadd(su, o[0]);
        sv = cadd(sv, o[1]);
      }
      double u[3], v[3];
      transverse(a.dir[ang0 + t], u, v);
      double2* out = a.out + ((r0 + rr) * static_cast<size_t>(a.n_total_angles) + a.angle0 + ang0 + t) * 3;
#pragma unroll
      for (int c = 0; c < 3; ++c) out[c] = cmul(coeff, cadd(cscale(su, u[c]), cscale(sv, v[c])));
    }
  }
  cl.sync();  // the other blocks' sums stay until rank 0 has read them
}

// The same sums for up to kS solutions with a block per angle and a warp for each
// slice: a lane forms the moments it sums, so nothing is staged and no warp waits
// for another until the end. Same order, same bits as far_batch_kernel, which
// shares a moment among more solutions but holds an SM's 16 warps in step.
template <bool kSkew, int kRwgs, int kS>
__global__ void __launch_bounds__(32 * kFarSlices, 2) far_few_kernel(const __grid_constant__ FarBatchArg a) {
  __shared__ double2 red[kFarSlices][kS][2];
  const Geo& g = a.g;
  const int r0 = blockIdx.y * kS, nr = min(kS, a.R - r0);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const size_t n = 2 * static_cast<size_t>(g.N);
  const double* r = a.dir[blockIdx.x];
  double u[3], v[3];
  transverse(r, u, v);
  double2 acc[kS][2];
#pragma unroll
  for (int s = 0; s < kS; ++s) acc[s][0] = acc[s][1] = c2(0.0, 0.0);
  for (int tile = wp; tile * kRwgs < g.N; tile += kFarSlices) {
#pragma unroll 1
    for (int c = 0; c < kRwgs / 32; ++c) {
      const int m = tile * kRwgs + 32 * c + lane;
      if (m >= g.N) break;
      double2 Au, Av;
      far_moment<kSkew>(g, m, r, u, v, Au, Av);
      const double2 mu = cneg(Au), mv = cneg(Av);
#pragma unroll
      for (int s = 0; s < kS; ++s) {
        if (s >= nr) break;
        const double2 J = __ldg(a.I + (r0 + s) * n + m), M = __ldg(a.I + (r0 + s) * n + g.N + m);
        acc[s][0] = cfma(mv, M, cfma(mu, J, acc[s][0]));
        acc[s][1] = cfma(Au, M, cfma(mv, J, acc[s][1]));
      }
    }
  }
#pragma unroll
  for (int s = 0; s < kS; ++s)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double2 t = blas1::warp_sum2(acc[s][c]);
      if (lane == 0) red[wp][s][c] = t;
    }
  __syncthreads();
  if (threadIdx.x >= nr) return;
  double2 su = c2(0.0, 0.0), sv = c2(0.0, 0.0);
  for (int q = 0; q < kFarSlices; ++q) {
    su = cadd(su, red[q][threadIdx.x][0]);
    sv = cadd(sv, red[q][threadIdx.x][1]);
  }
  const double2 coeff = c2(g.k1.y, -g.k1.x);
  double2* out = a.out + ((r0 + threadIdx.x) * static_cast<size_t>(a.n_total_angles) + a.angle0 + blockIdx.x) * 3;
#pragma unroll
  for (int c = 0; c < 3; ++c) out[c] = cmul(coeff, cadd(cscale(su, u[c]), cscale(sv, v[c])));
}

// One chunk of angles; kRwgs by the body's size alone, so that a solution's field
// is the same in every call. A block per angle where that gives every SM one, or
// on small bodies, for few solutions (one B200, us, far_batch_kernel / far_few_kernel):
// 361 angles, one solution: 240 unknowns 52 / 19, 960 55 / 20, 3,840 96 / 57,
// 61,440 1,049 / 868; four 3,840 118 / 71, 61,440 1,109 / 1,037; eight 240
// unknowns 58 / 26, 960 61 / 32; 37 angles, one solution: 960 unknowns 15.5 /
// 14.6, 3,840 17 / 28, 61,440 165 / 388. Tiles of 64 RWGs instead of 256 where those would
// leave blocks of a cluster without any: 32 solutions at 37 angles, 240 unknowns
// 25 -> 17 us, at 361 angles 143 -> 91.
template <bool kSkew, int kRwgs>
void launch_far(const FarBatchArg& a, cudaStream_t s) {
  const bool small = a.g.N <= 512;
  if (a.R <= (small ? 2 : 1) * kFarFewSols && (small || a.n_angles >= 148)) {
    const dim3 grid(a.n_angles, (a.R + kFarFewSols - 1) / kFarFewSols);
    if (a.R == 1)
      far_few_kernel<kSkew, kRwgs, 1><<<grid, 32 * kFarSlices, 0, s>>>(a);
    else if (a.R == 2)
      far_few_kernel<kSkew, kRwgs, 2><<<grid, 32 * kFarSlices, 0, s>>>(a);
    else
      far_few_kernel<kSkew, kRwgs, kFarFewSols><<<grid, 32 * kFarSlices, 0, s>>>(a);
    return;
  }
  const dim3 grid((a.n_angles + kFarAngles - 1) / kFarAngles, (a.R + kFarSols - 1) / kFarSols, kFarSlices);
  far_batch_kernel<kSkew, kRwgs><<<grid, kFarThreads, 0, s>>>(a);
}

struct FarMonoArg {
  Geo g;
  double dir[kFarChunk][3];
  int r0;            // first solution of this chunk
  const double2* I;  // [R][2N]
  double2* out;      // [R][3]
};

// block per solution of the chunk, observed in its own direction
template <bool kSkew>
__global__ void __launch_bounds__(256) far_mono_kernel(const __grid_constant__ FarMonoArg a) {
  __shared__ double2 sh[8];
  const Geo& g = a.g;
  const int q = blockIdx.x;
  const double r[3] = {a.dir[q][0], a.dir[q][1], a.dir[q][2]};
  double u[3], v[3];
  transverse(r, u, v);
  const double2* I = a.I + (a.r0 + q) * 2 * static_cast<size_t>(g.N);
  double2 su = c2(0.0, 0.0), sv = c2(0.0, 0.0);
  for (int m = threadIdx.x; m < g.N; m += blockDim.x) {
    double2 Au, Av;
    far_moment<kSkew>(g, m, r, u, v, Au, Av);
    const double2 IJ = I[m], IM = I[g.N + m];
    su = csub(csub(su, cmul(Av, IM)), cmul(Au, IJ));
    sv = csub(cadd(sv, cmul(Au, IM)), cmul(Av, IJ));
  }
  const double2 coeff = c2(g.k1.y, -g.k1.x);
  su = blas1::block_sum(su, sh);
  sv = blas1::block_sum(sv, sh);
  if (threadIdx.x == 0)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      a.out[(a.r0 + q) * 3 + c] = cmul(coeff, cadd(cscale(su, u[c]), cscale(sv, v[c])));
}

// Code/RCS.h:120-123: observation direction of (theta, phi) in degrees
void direction(double theta_deg, double phi_deg, double r[3]) {
  const double th = (theta_deg / 180.0) * kPi, ph = (phi_deg / 180.0) * kPi;
  r[0] = std::sin(th) * std::cos(ph);
  r[1] = std::sin(th) * std::sin(ph);
  r[2] = std::cos(th);
}

}  // namespace

void rhs_pmchwt_batch(Plan& P, int R, const double* kinc, const double* einc, const double* hinc, double2* V_dev,
                      cudaStream_t s) {
  if (R <= 0) return;
  MLFMA_CUDA(cudaSetDevice(P.device));
  RhsBatchArg a{};
  a.g = geo(P);
  for (int c0 = 0; c0 < R; c0 += kRhsChunk) {
    a.R = std::min(kRhsChunk, R - c0);
    for (int q = 0; q < a.R; ++q)
      for (int c = 0; c < 3; ++c) {
        a.inc[q][c] = kinc[3 * (c0 + q) + c];
        a.inc[q][3 + c] = einc[3 * (c0 + q) + c];
        a.inc[q][6 + c] = hinc[3 * (c0 + q) + c];
      }
    a.V = V_dev + static_cast<size_t>(c0) * 2 * P.N;
    const dim3 grid((P.N + 127) / 128, (a.R + kRhsTile - 1) / kRhsTile);
    rhs_batch_kernel<<<grid, 128, 0, s>>>(a);
    MLFMA_CUDA(cudaGetLastError());
  }
}

void rcs_pmchwt_batch(Plan& P, int R, const double2* I_dev, int n_angles, const double* theta_deg,
                      const double* phi_deg, double2* field_dev, cudaStream_t s) {
  if (R <= 0 || n_angles <= 0) return;
  MLFMA_CUDA(cudaSetDevice(P.device));
  FarBatchArg a{};
  a.g = geo(P);
  a.R = R;
  a.I = I_dev;
  a.out = field_dev;
  a.n_total_angles = n_angles;
  for (int c0 = 0; c0 < n_angles; c0 += kFarChunk) {
    a.n_angles = std::min(kFarChunk, n_angles - c0);
    a.angle0 = c0;
    for (int q = 0; q < a.n_angles; ++q) direction(theta_deg[c0 + q], phi_deg[c0 + q], a.dir[q]);
    const bool few = P.N <= (kFarSlices - 1) * kFarRwgs;
    if (a.g.skew)
      few ? launch_far<true, kFarFew>(a, s) : launch_far<true, kFarRwgs>(a, s);
    else
      few ? launch_far<false, kFarFew>(a, s) : launch_far<false, kFarRwgs>(a, s);
    MLFMA_CUDA(cudaGetLastError());
  }
}

void rcs_pmchwt_mono(Plan& P, int R, const double2* I_dev, const double* theta_deg, const double* phi_deg,
                     double2* field_dev, cudaStream_t s) {
  if (R <= 0) return;
  MLFMA_CUDA(cudaSetDevice(P.device));
  FarMonoArg a{};
  a.g = geo(P);
  a.I = I_dev;
  a.out = field_dev;
  for (int c0 = 0; c0 < R; c0 += kFarChunk) {
    const int nr = std::min(kFarChunk, R - c0);
    a.r0 = c0;
    for (int q = 0; q < nr; ++q) direction(theta_deg[c0 + q], phi_deg[c0 + q], a.dir[q]);
    if (a.g.skew)
      far_mono_kernel<true><<<nr, 256, 0, s>>>(a);
    else
      far_mono_kernel<false><<<nr, 256, 0, s>>>(a);
    MLFMA_CUDA(cudaGetLastError());
  }
}

void rcs_db(int n_angles, const double* theta_deg, const double* phi_deg, const double* field, double* out) {
  for (int i = 0; i < n_angles; ++i) {
    // theta-hat / phi-hat of EMSource::initPW (Code/EMSource.cpp:34-59):
    // degrees to radians with |a| < 1e-6 snapped to 0, components snapped too;
    // dB as the dual-static study forms them (Code/RCS.h:391-410).
    auto snap = [](double v) { return std::abs(v) < 1e-6 ? 0.0 : v; };
    const double th = snap(theta_deg[i] * kPi / 180.0), ph = snap(phi_deg[i] * kPi / 180.0);
    const double vt[3] = {snap(-std::cos(th) * std::cos(ph)), snap(-std::cos(th) * std::sin(ph)), snap(std::sin(th))};
    const double vp[3] = {snap(-std::sin(ph)), snap(std::cos(ph)), 0.0};
    const cplx E[3] = {cplx(field[6 * i], field[6 * i + 1]), cplx(field[6 * i + 2], field[6 * i + 3]),
                       cplx(field[6 * i + 4], field[6 * i + 5])};
    const cplx Ev = vt[0] * E[0] + vt[1] * E[1] + vt[2] * E[2];
    const cplx Eh = vp[0] * E[0] + vp[1] * E[1] + vp[2] * E[2];
    out[3 * i] = 10.0 * std::log10((std::norm(Ev) + std::norm(Eh)) / (4.0 * kPi));
    out[3 * i + 1] = 10.0 * std::log10(std::norm(Ev) / (4.0 * kPi));
    out[3 * i + 2] = 10.0 * std::log10(std::norm(Eh) / (4.0 * kPi));
  }
}

}  // namespace mlfma
