// mass_rows.cu - consistent mass of one hex bucket, row by row (sm_100a).
//
// M_ab = rho sum_g c_g N_a N_b I3 (cElmParam::MassMat, elc/elmparam.cpp:672-739)
// is one number per node pair, yet adding element after element into the 3x3
// blocks of the matrix, colour by colour, reads and writes every block once
// per element that shares it, after a zero fill: 2.5 GB for 32,760 hex20
// elements, 974 us plus 100 for the fill.  Here
//  1. mass_pairs forms the numbers of 16 elements per block as the product of
//     their weighted determinants with the N_a N_b: 105 MB, which stay in L2;
//  2. mass_rows gives a warp each node: it sums the rows (e, a) of the
//     elements at the node into shared memory, in the fixed order of the
//     node's list, and stores the node's blocks once, whole, in order.
// Measured at 32,760 hex20 elements (7.8 million blocks, 563 MB): pairs 96 us
// (32 elements a block: 107), rows 186 us, 4 TB/s with the lists and slots
// they read; together 282 us.
#include <algorithm>
#include <cstdint>

#include "elem_common.cuh"
#include "internal.h"

namespace fastgpu {
namespace {

constexpr int kPairThreads = 256, kPairElems = 16;

template <int NN>
__global__ void __launch_bounds__(kPairThreads)
mass_pairs(int64_t ne, int ng, const int32_t *__restrict__ conn, const double *__restrict__ X,
           const double *__restrict__ rho, const double *__restrict__ N, const double *__restrict__ dN,
           const double *__restrict__ w, double *__restrict__ out, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) double sm[];
  double *sX = sm;                         // [NN][3][kPairElems]
  double *sd = sX + NN * 3 * kPairElems;   // [ng][kPairElems] rho w det J
  const int tid = threadIdx.x;
  for (int64_t e0 = (int64_t)blockIdx.x * kPairElems; e0 < ne; e0 += (int64_t)gridDim.x * kPairElems) {
    const int cnt = (int)(ne - e0 < kPairElems ? ne - e0 : kPairElems);
    __syncthreads();
    for (int t = tid; t < NN * kPairElems; t += kPairThreads) {
      const int el = t % kPairElems, a = t / kPairElems;
      if (el < cnt) {
        const double *x = X + 3 * (int64_t)conn[(e0 + el) * NN + a];
        for (int c = 0; c < 3; c++) sX[(3 * a + c) * kPairElems + el] = x[c];
      }
    }
    __syncthreads();
    for (int t = tid; t < ng * kPairElems; t += kPairThreads) {
      const int el = t % kPairElems, g = t / kPairElems;
      if (el >= cnt) {
        sd[t] = 0.0;
        continue;
      }
      double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      const double *d = dN + g * NN * 3;
#pragma unroll 4
      for (int a = 0; a < NN; a++) {
        const double x0 = sX[(3 * a) * kPairElems + el], x1 = sX[(3 * a + 1) * kPairElems + el],
                     x2 = sX[(3 * a + 2) * kPairElems + el];
#pragma unroll
        for (int p = 0; p < 3; p++) {
          J[3 * p] += d[3 * a + p] * x0;
          J[3 * p + 1] += d[3 * a + p] * x1;
          J[3 * p + 2] += d[3 * a + p] * x2;
        }
      }
      const double det = J[0] * (J[4] * J[8] - J[5] * J[7]) - J[1] * (J[3] * J[8] - J[5] * J[6]) +
                         J[2] * (J[3] * J[7] - J[4] * J[6]);
      if (!(det > 0.0)) atomicOr(status, 1);
      sd[t] = rho[e0 + el] * (w[g] * det);
    }
    __syncthreads();
    for (int q = tid; q < NN * NN; q += kPairThreads) {
      const int a = q / NN, b = q - NN * a;
      double acc[kPairElems];
#pragma unroll
      for (int k = 0; k < kPairElems; k++) acc[k] = 0.0;
#pragma unroll 3
      for (int g = 0; g < ng; g++) {
        const double P = N[g * NN + a] * N[g * NN + b];
        const double2 *s = reinterpret_cast<const double2 *>(sd + g * kPairElems);
#pragma unroll
        for (int k = 0; k < kPairElems / 2; k++) {
          const double2 v = s[k];
          acc[2 * k] += P * v.x;
          acc[2 * k + 1] += P * v.y;
        }
      }
#pragma unroll
      for (int k = 0; k < kPairElems; k++)
        if (k < cnt) out[(e0 + k) * (NN * NN) + q] = acc[k];
    }
  }
}

constexpr int kRowThreads = 256, kRowCols = 128;  // columns of a row held at a time

template <int NN>
__global__ void __launch_bounds__(kRowThreads)
mass_rows(int64_t nnode, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
          const uint8_t *__restrict__ fix, const int64_t *__restrict__ gptr, const int64_t *__restrict__ ginc,
          const int32_t *__restrict__ slot, const double *__restrict__ pairs, double *__restrict__ M) {
  constexpr int PER = 32 / NN;        // list entries (e, a) a warp reads at once, a lane per b
  constexpr int U = NN == 8 ? 2 : 4;  // such reads in flight
  __shared__ double sacc[kRowThreads / 32][kRowCols];
  __shared__ uint8_t sfix[kRowThreads / 32][kRowCols];
  const int lane = threadIdx.x & 31, sub = lane / NN, b = lane - sub * NN;
  double *acc = sacc[threadIdx.x >> 5];
  uint8_t *fx = sfix[threadIdx.x >> 5];
  for (int64_t n = (blockIdx.x * (int64_t)kRowThreads + threadIdx.x) >> 5; n < nnode;
       n += ((int64_t)gridDim.x * kRowThreads) >> 5) {
    const int32_t r1 = rowptr[n + 1];
    const int64_t i0 = gptr[n], i1 = gptr[n + 1];
    const uint8_t fn = fix[n];
    for (int32_t c0 = rowptr[n]; c0 < r1; c0 += kRowCols) {
      const int nb = r1 - c0 < kRowCols ? r1 - c0 : kRowCols;
      for (int j = lane; j < nb; j += 32) {
        acc[j] = 0.0;
        fx[j] = fn | fix[col[c0 + j]];
      }
      __syncwarp();
      for (int64_t i = i0; i < i1; i += PER * U) {
        int32_t at[U];
        double m[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int64_t k = i + u * PER + sub;
          at[u] = -1;
          if (sub < PER && k < i1) {
            const int64_t ea = ginc[k] / 3;  // element NN + a
            at[u] = slot[ea * NN + b] - c0;
            m[u] = pairs[ea * NN + b];
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int k = 0; k < PER; k++) {  // one element at a time: its columns differ
            if (sub == k && at[u] >= 0 && at[u] < nb) acc[at[u]] += m[u];
            __syncwarp();
          }
      }
      double *out = M + 9 * (int64_t)c0;
      for (int t = lane; t < 9 * nb; t += 32) {
        const int j = t / 9, k = t - 9 * j;
        out[t] = (k & 3) == 0 && !((fx[j] >> (k >> 2)) & 1) ? acc[j] : 0.0;
      }
      __syncwarp();
    }
  }
}

template <int NN>
cudaError_t go(Ctx &c, const Bucket &B, double *M) {
  auto kern = mass_pairs<NN>;
  const size_t bytes = sizeof(double) * kPairElems * (NN * 3 + B.ng);
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  const int64_t need = (B.ne + kPairElems - 1) / kPairElems;
  kern<<<(unsigned)need, kPairThreads, bytes, c.stream>>>(
      B.ne, B.ng, B.d_conn, c.d_X, B.d_rho, B.d_N, B.d_dN, B.d_w, c.d_mpairs, c.d_status);
  mass_rows<NN><<<(unsigned)((c.nnode * 32 + kRowThreads - 1) / kRowThreads), kRowThreads, 0, c.stream>>>(
      c.nnode, c.d_rowptr, c.d_col, c.d_fix, c.d_gptr, c.d_ginc, B.d_slot, c.d_mpairs, M);
  c.launches += 2;
  return cudaGetLastError();
}

}  // namespace

// One hex bucket with densities and no ties (the node lists and the slots cover
// every element).  cudaErrorNotSupported: the coloured scatter has to do it,
// also where the pair numbers (8 NN^2 bytes per element) find no memory.
cudaError_t launch_mass_rows(Ctx &c, double *M) {
  if (c.buckets.size() != 1 || !c.force_gather || c.has_ties() || !c.buckets[0].has_rho) return cudaErrorNotSupported;
  const Bucket &B = c.buckets[0];
  if (B.type != FAST_ELEM_HEX8 && B.type != FAST_ELEM_HEX20) return cudaErrorNotSupported;
  if (!c.d_mpairs && cudaMalloc((void **)&c.d_mpairs, sizeof(double) * (size_t)B.ne * B.nn * B.nn) != cudaSuccess) {
    cudaGetLastError();
    c.d_mpairs = nullptr;
    return cudaErrorNotSupported;
  }
  return B.nn == 8 ? go<8>(c, B, M) : go<20>(c, B, M);
}

// The pair numbers are kept for the next assembly up to 1 GB (335,544 hex20
// elements); a larger array is given back once the stream is done with it, so
// that the solve's layouts find room.  Making it anew costs as much as the
// assembly: 11.0 ms an assembly of 648,000 elements (2.1 GB), 5.3 if it is kept,
// 19.6 by the coloured scatter; at 131,072 (420 MB) 2.1, 1.1 and 4.0.
void mass_rows_done(Ctx &c) {
  constexpr size_t kKeep = (size_t)1 << 30;
  if (!c.d_mpairs) return;
  const Bucket &B = c.buckets[0];
  if (sizeof(double) * (size_t)B.ne * B.nn * B.nn <= kKeep) return;
  cudaFree(c.d_mpairs);
  c.d_mpairs = nullptr;
}

}  // namespace fastgpu
