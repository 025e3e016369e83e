// Warp and block sums of complex128 values.
#pragma once
#include "cplx.cuh"

namespace mlfma {
namespace blas1 {

__device__ __forceinline__ double2 warp_sum2(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// Sum over the block, valid in thread 0 (sh: one value per warp).
__device__ __forceinline__ double2 block_sum(double2 v, double2* sh) {
  v = warp_sum2(v);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) v = warp_sum2(lane < (blockDim.x >> 5) ? sh[lane] : c2(0.0, 0.0));
  return v;
}

}  // namespace blas1
}  // namespace mlfma
