// The two leaf contractions of the batched complex64 operator in FP32 on the
// CUDA cores: aggregation (Code/ProcessMLFMM.h:33-56) and far-field testing
// (Code/MLFMM.cpp:285-351) of up to 16 right-hand-side slots at once.
//
// Both read each pattern value once for all slots and are bound by FP32
// issue: 30,720 RWGs, 800 directions of both media and 16 slots are 9.4 G
// fused multiply-adds each, 0.25 ms at the FP32 rate. The tensor-core forms of
// agg_tc.cu do the same contractions as three TF32 products per step, but
// splitting, transposing and storing the operands costs more than the
// multiply-adds it saves (tensor pipe 7-10 % active). One B200, 16 slots at
// 61,440 unknowns: aggregation 0.62 against 0.95 ms, testing 1.15 against 1.87;
// 8 slots at 15,360: 0.10 against 0.26 and 0.20 against 0.44 ms.
#include <stdexcept>

#include "agg_tc.hpp"
#include "bulk.cuh"
#include "cplx.cuh"
#include "plan.hpp"

namespace mlfma {
namespace {

constexpr int kAbThreads = 256;
constexpr int kAbStage = 48;  // RWGs of a box staged at a time (a multiple of 4)

// Aggregation: CTA per (leaf box, 256 pattern entries of one medium), a thread
// one entry of every (part, slot): 2 kS complex sums. The box's currents are
// staged in complex64, [RWG][part][slot], and read as broadcasts.
template <int kS>
__global__ void __launch_bounds__(kAbThreads, 2) agg_slots_kernel(const __grid_constant__ AggTcArg a, int tiles0) {
  __shared__ float4 xs4[kAbStage][kS];  // two slots per value
  float2* xs = reinterpret_cast<float2*>(xs4);
  const int b = blockIdx.x;
  const int m = static_cast<int>(blockIdx.y) >= tiles0;
  const int K3 = 3 * a.K[m];
  const int e = (blockIdx.y - m * tiles0) * kAbThreads + threadIdx.x;
  const int r0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - r0;
  const float2* V = reinterpret_cast<const float2*>(a.Vs[m]) + static_cast<size_t>(r0) * K3 + min(e, K3 - 1);
  float2 acc[2 * kS];
#pragma unroll
  for (int i = 0; i < 2 * kS; ++i) acc[i] = make_float2(0.f, 0.f);
  float2 next[4];  // the next four RWGs' values, in flight
  auto fetch = [&](int r) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      next[u] = r + u < nb ? __ldg(V + static_cast<size_t>(r + u) * K3) : make_float2(0.f, 0.f);
  };
  fetch(0);
  for (int s0 = 0; s0 < nb; s0 += kAbStage) {
    const int n = min(kAbStage, nb - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < n * 2 * kS; i += kAbThreads) {
      const int r = i / (2 * kS), col = i - r * (2 * kS), part = col / kS, j = col - part * kS;
      float2 x = make_float2(0.f, 0.f);
      if (j < a.R) x = Cx<float2>::from(__ldg(a.X + j * a.ldx + part * a.N + __ldg(a.leaf_rwg + r0 + s0 + r)));
      xs[i] = x;
    }
    __syncthreads();
    for (int r = 0; r < n; r += 4) {
      float2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = next[u];
      fetch(s0 + r + 4);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r + u < n) {
#pragma unroll
          for (int i = 0; i < kS; ++i) {
            const float4 x = xs4[r + u][i];
            acc[2 * i] = cfma(v[u], make_float2(x.x, x.y), acc[2 * i]);
            acc[2 * i + 1] = cfma(v[u], make_float2(x.z, x.w), acc[2 * i + 1]);
          }
        }
      }
    }
  }
  if (e >= K3) return;
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int j = 0; j < kS; ++j)
      if (j < a.R) a.S[m][j][(static_cast<size_t>(b) * 2 + part) * K3 + e] = acc[part * kS + j];
}

// Far-field testing. With c and e of a medium (c1, 1 or c2, etai),
//   w_J = sum over directions of Vf . c (e B_J - khat x B_M),
//   w_M = sum over directions of Vf . c (khat x B_J + B_M / e),
// because ((-khat) x Vf) . B = Vf . (khat x B): with the bracketed vectors
// formed once per (box, direction, slot), each receive-pattern value meets two
// products per slot instead of four.
// CTA per (leaf box, kRows RWGs); per 32 directions it stages the rows'
// patterns (cp.async, two stages) and the vectors of every slot, the next
// ones' B in registers. A warp multiplies an eighth of the 96 entries: lanes 2
// rows x 4 columns of (slot, J or M), kTiles row tiles. The sums of a chunk
// start from zero and are added to the running ones (at most ~100 FP32
// additions in a row), the warps' sums meet in shared memory at the end.
constexpr int kLbThreads = 256;
constexpr int kLbWarps = kLbThreads / 32;
constexpr int kLbDirs = 32;
constexpr int kLbEntries = 3 * kLbDirs;

template <int kS>
struct LeafSlots {
  static constexpr int kCols = 2 * kS;                // (J, M) x slots
  static constexpr int kColGroups = kCols / 4;        // lanes across columns
  static constexpr int kRowGroups = 32 / kColGroups;  // lanes across rows, 2 rows each
  static constexpr int kTileRows = 2 * kRowGroups;
  static constexpr int kTiles = kS == 16 ? 3 : kS == 8 ? 2 : 1;
  static constexpr int kRows = kTiles * kTileRows;    // 24, 32, 32
  static constexpr int kDPitch = kCols + 2;           // float2 per entry: 16-byte rows, spread over the banks
  static constexpr int kVPitch = kLbEntries + 2;      // float2 per row
  struct Smem {
    float2 V[2][kRows * kVPitch];
    float2 D[2][kLbEntries * kDPitch];
  };
  static_assert(sizeof(float2) * kLbWarps * kRows * kCols <= 2 * sizeof(Smem), "");
};

template <int kS>
__global__ void __launch_bounds__(kLbThreads, 2) leaf_slots_kernel(const __grid_constant__ LeafTcArg a) {
  using T = LeafSlots<kS>;
  constexpr int kCols = T::kCols, kRows = T::kRows, kTiles = T::kTiles;
  constexpr int kPerThread = (kLbDirs * kS + kLbThreads - 1) / kLbThreads;  // (direction, slot) pairs
  extern __shared__ __align__(16) unsigned char leaf_smem[];
  typename T::Smem& sm = *reinterpret_cast<typename T::Smem*>(leaf_smem);
  const int b = blockIdx.x;
  const int rb0 = a.leaf_ptr[b], nb = a.leaf_ptr[b + 1] - rb0;
  const int t0 = blockIdx.y * kRows;
  if (t0 >= nb) return;
  const int nt = min(kRows, nb - t0);
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int kk = lane;  // this thread's direction of a chunk; slots wp + kLbWarps i
  const int nc0 = (a.K[0] + kLbDirs - 1) / kLbDirs, nchunk = nc0 + (a.K[1] + kLbDirs - 1) / kLbDirs;
  float2 f[kPerThread][6];
  float kh[3];
  auto fetch = [&](int ch) {
    const int m = ch >= nc0, K = a.K[m], k = (ch - m * nc0) * kLbDirs + kk;
    const bool in = k < K;
#pragma unroll
    for (int c = 0; c < 3; ++c) kh[c] = in ? static_cast<float>(__ldg(a.khat[m] + c * K + k)) : 0.f;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
      const int j = wp + kLbWarps * i;
      const float2* B = j < a.R ? a.Bm[m][j] + static_cast<size_t>(b) * 6 * K + k : nullptr;
#pragma unroll
      for (int c = 0; c < 6; ++c)
        f[i][c] = in && j < a.R ? __ldg(B + static_cast<size_t>(c) * K) : make_float2(0.f, 0.f);
    }
  };
  auto stage = [&](int ch) {  // patterns of chunk ch: 16-byte pairs of directions
    if (ch < nchunk) {
      const int m = ch >= nc0, K = a.K[m], k0 = (ch - m * nc0) * kLbDirs;
      const float2* V = a.Vf[m] + static_cast<size_t>(rb0 + t0) * 3 * K + k0;
      float2* dst = sm.V[ch & 1];
      constexpr int kPairs = kLbDirs / 2;
      for (int i = tid; i < kRows * 3 * kPairs; i += kLbThreads) {
        const int row = i / (3 * kPairs), q = i - row * (3 * kPairs), c = q / kPairs, pr = q - c * kPairs;
        const bool take = row < nt && k0 + 2 * pr < K;  // K is even
        cp_async16_or_zero(dst + row * T::kVPitch + c * kLbDirs + 2 * pr,
                           take ? V + (static_cast<size_t>(row) * 3 + c) * K + 2 * pr : a.Vf[m], take);
      }
    }
    cp_async_commit();
  };
  float2 acc[kTiles][2][4];
#pragma unroll
  for (int t = 0; t < kTiles; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[t][i][j] = make_float2(0.f, 0.f);
  const int rg = lane / T::kColGroups, cg = lane - rg * T::kColGroups;
  stage(0);
  fetch(0);
  for (int ch = 0; ch < nchunk; ++ch) {
    {  // the chunk's vectors, J columns then M columns of each slot
      const int m = ch >= nc0;
      const float2 c = m ? a.c2 : a.c1, e = m ? a.etai : make_float2(1.f, 0.f);
      const float2 ce = cmul(c, e), cie = cdiv(c, e);
#pragma unroll
      for (int i = 0; i < kPerThread; ++i) {
        const int j = wp + kLbWarps * i;
        if (j >= kS) continue;
        const float2 *J = f[i], *M = f[i] + 3;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
          const float2 xJ = csub(cscale(J[q2], kh[q1]), cscale(J[q1], kh[q2]));  // khat x B_J
          const float2 xM = csub(cscale(M[q2], kh[q1]), cscale(M[q1], kh[q2]));
          float2* d = sm.D[ch & 1] + (q * kLbDirs + kk) * T::kDPitch;
          d[j] = csub(cmul(ce, J[q]), cmul(c, xM));
          d[kS + j] = cfma(cie, M[q], cmul(c, xJ));
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // the chunk is staged, and every warp is done with the one before it
    stage(ch + 1);
    if (ch + 1 < nchunk) fetch(ch + 1);
    const float2 *V = sm.V[ch & 1], *Dc = sm.D[ch & 1];
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      if (t * T::kTileRows >= nt) break;
      float2 s[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = make_float2(0.f, 0.f);
      const float2* v0 = V + (t * T::kTileRows + 2 * rg) * T::kVPitch;
#pragma unroll 4  // all 12 at once spill
      for (int q = 0; q < kLbEntries / kLbWarps; ++q) {
        const int en = wp * (kLbEntries / kLbWarps) + q;
        const float4 da = *reinterpret_cast<const float4*>(Dc + en * T::kDPitch + 4 * cg);
        const float4 db = *reinterpret_cast<const float4*>(Dc + en * T::kDPitch + 4 * cg + 2);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 v = v0[i * T::kVPitch + en];
          s[i][0] = cfma(v, make_float2(da.x, da.y), s[i][0]);
          s[i][1] = cfma(v, make_float2(da.z, da.w), s[i][1]);
          s[i][2] = cfma(v, make_float2(db.x, db.y), s[i][2]);
          s[i][3] = cfma(v, make_float2(db.z, db.w), s[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[t][i][j] = cadd(acc[t][i][j], s[i][j]);
    }
  }
  __syncthreads();
  float2* red = reinterpret_cast<float2*>(leaf_smem);  // [warp][row][column]
#pragma unroll
  for (int t = 0; t < kTiles; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        red[(wp * kRows + t * T::kTileRows + 2 * rg + i) * kCols + 4 * cg + j] = acc[t][i][j];
  __syncthreads();
  for (int o = tid; o < kRows * kCols; o += kLbThreads) {
    const int row = o / kCols, col = o - row * kCols, part = col / kS, j = col - part * kS;
    if (row >= nt || j >= a.R) continue;
    float2 v = red[o];
#pragma unroll
    for (int q = 1; q < kLbWarps; ++q) v = cadd(v, red[q * kRows * kCols + o]);
    double2* w = a.W + j * a.ldw + part * a.N + a.leaf_rwg[rb0 + t0 + row];
    *w = cadd(*w, Cx<float2>::to64(v));
  }
}

template <int kS>
size_t leaf_slots_smem() {
  using T = LeafSlots<kS>;
  return std::max(sizeof(typename T::Smem), sizeof(float2) * kLbWarps * T::kRows * T::kCols);
}

template <int kS>
void launch_leaf_as(const Plan& P, const LeafTcArg& a, cudaStream_t s) {
  const int smem = static_cast<int>(leaf_slots_smem<kS>());
  MLFMA_CUDA(cudaFuncSetAttribute(leaf_slots_kernel<kS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int tiles = (P.max_leaf_rwgs + LeafSlots<kS>::kRows - 1) / LeafSlots<kS>::kRows;
  leaf_slots_kernel<kS><<<dim3(P.lv[P.maxL].B, tiles), kLbThreads, smem, s>>>(a);
}

}  // namespace

// The slots are padded to 4, 8 or 16: the smallest that holds them.
void launch_agg_slots(const Plan& P, const AggTcArg& a, cudaStream_t s) {
  if (a.R < 1 || a.R > kBatchSlots) throw std::invalid_argument("batched aggregation: 1 <= R <= 16");
  const int tiles0 = (3 * a.K[0] + kAbThreads - 1) / kAbThreads, tiles1 = (3 * a.K[1] + kAbThreads - 1) / kAbThreads;
  const dim3 grid(P.lv[P.maxL].B, tiles0 + tiles1);
  if (a.R <= 4)
    agg_slots_kernel<4><<<grid, kAbThreads, 0, s>>>(a, tiles0);
  else if (a.R <= 8)
    agg_slots_kernel<8><<<grid, kAbThreads, 0, s>>>(a, tiles0);
  else
    agg_slots_kernel<16><<<grid, kAbThreads, 0, s>>>(a, tiles0);
  MLFMA_CUDA(cudaGetLastError());
}

void launch_leaf_slots(const Plan& P, const LeafTcArg& a, cudaStream_t s) {
  if (a.R < 1 || a.R > kBatchSlots) throw std::invalid_argument("batched far-field testing: 1 <= R <= 16");
  if (a.R <= 4)
    launch_leaf_as<4>(P, a, s);
  else if (a.R <= 8)
    launch_leaf_as<8>(P, a, s);
  else
    launch_leaf_as<16>(P, a, s);
  MLFMA_CUDA(cudaGetLastError());
}

}  // namespace mlfma
