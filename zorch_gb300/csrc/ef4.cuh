// EF4 loads, stores and block-wide sums shared by the sumcheck units.
#pragma once
#include "field.cuh"

namespace zc {

__device__ __forceinline__ ef4 ld4(const uint32_t* p) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  return ef4{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void st4(uint32_t* p, const ef4& a) {
  *reinterpret_cast<uint4*>(p) = make_uint4(a.c[0], a.c[1], a.c[2], a.c[3]);
}
template <class F>
__device__ __forceinline__ ef4 ef_base(const ef4& a, uint32_t b) {  // EF4 * base
  return ef_scale<F>(a, b);
}

// Block-wide EF4 sum (blockDim a multiple of 32, <= 1024); the result is
// valid in thread 0.
template <class F>
__device__ ef4 block_sum(ef4 v) {
  __shared__ uint32_t red[4][32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < 4; e++) v.c[e] = madd<F>(v.c[e], __shfl_xor_sync(0xffffffffu, v.c[e], o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // red reused across calls
  if (lane == 0)
#pragma unroll
    for (int e = 0; e < 4; e++) red[e][warp] = v.c[e];
  __syncthreads();
  ef4 r{{0, 0, 0, 0}};
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int e = 0; e < 4; e++) r.c[e] = lane < nw ? red[e][lane] : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < 4; e++) r.c[e] = madd<F>(r.c[e], __shfl_xor_sync(0xffffffffu, r.c[e], o));
  }
  return r;
}

}  // namespace zc
