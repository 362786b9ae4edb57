// solve_common.cuh - reductions and node-vector access of the solve kernels
// (private to libfastgpu).
#pragma once

#include <cstdint>

#include "internal.h"

namespace fastgpu {

constexpr int kSpmvThreads = 256;
constexpr int kVecThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-level fixed-order sum; returns the total in thread 0
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sbuf) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sbuf[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = (lane < NT / 32) ? sbuf[lane] : 0.0;
    t = warp_sum(t);
  }
  return t;
}

// padded node vectors
template <typename T> struct V4;
template <> struct V4<float> {
  static __device__ __forceinline__ void load(const float *p, float &a, float &b, float &c) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    a = v.x; b = v.y; c = v.z;
  }
  static __device__ __forceinline__ void store(float *p, float a, float b, float c) {
    *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, 0.f);
  }
};
template <> struct V4<double> {
  static __device__ __forceinline__ void load(const double *p, double &a, double &b, double &c) {
    const double2 v0 = *reinterpret_cast<const double2 *>(p);
    a = v0.x; b = v0.y; c = p[2];
  }
  static __device__ __forceinline__ void store(double *p, double a, double b, double c) {
    *reinterpret_cast<double2 *>(p) = make_double2(a, b);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(c, 0.0);
  }
};

// single-block fixed-order sum of n partials
template <int NT = 256>
__device__ __forceinline__ double sum_partials(const double *p, int n, double *sbuf) {
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += p[i];
  return block_sum<NT>(v, sbuf);
}

// z = Dinv r with Dinv stored as 3 padded rows per node
template <typename T>
__device__ __forceinline__ void apply_dinv(const T *D, T r0, T r1, T r2, T &z0, T &z1, T &z2) {
  z0 = D[0] * r0 + D[1] * r1 + D[2] * r2;
  z1 = D[4] * r0 + D[5] * r1 + D[6] * r2;
  z2 = D[8] * r0 + D[9] * r1 + D[10] * r2;
}

// true in exactly one thread of the last block to reach this point
__device__ __forceinline__ bool last_block(uint32_t *counter) {
  __shared__ bool is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t t = atomicAdd(counter, 1u);
    is_last = (t == gridDim.x - 1);
    if (is_last) *counter = 0;
  }
  __syncthreads();
  return is_last && threadIdx.x == 0;
}

}  // namespace fastgpu
