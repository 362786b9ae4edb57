// elem_mma.cu - FP64 hex20 element stiffness on the FP64 matrix instruction,
// and its colour-scheduled scatter (sm_100a).
//
// The element of elem_kernels.cu (cElmParam::StiffMat,
// elc/elmparam.cpp:539-597, factored as M_ij(a, b) = sum_g D_ia(g) D_jb(g)
// with D = sqrt(c_g) dN/dx, and the isotropic block per node pair;
// cSolid::QMatrix, elc/anmodel.cpp:1286-1298), scattered the same way (no
// atomics, first-touch stores), for the bucket's own scatter of a colour.
//
// What bounded that kernel: a thread per node pair reads six numbers of D from
// shared memory for nine multiply-adds, the Jacobian phases leave most of 224
// threads idle, and three elements per SM do not cover the waits between
// phases.  Here three warps take an element:
//   * warp p forms row p of the Jacobians, a lane per Gauss point (the
//     derivative table is stored Gauss point innermost: whole lines), then each
//     warp inverts them all and forms D for its third of the nodes;
//   * M is 3x3 tiles of 8x8 node pairs (20 nodes padded to 24), six with
//     a <= b, two per warp: mma.m8n8k4.f64 over the Gauss points.  A lane ends
//     up with all nine M_ij of its two pairs (a, b), (a, b+1) of each tile, so
//     the isotropic blocks need no exchange;
//   * the blocks go through shared memory (in D's place) and are added to the
//     values that cp.async fetches during the product, consecutive lanes taking
//     consecutive entries of a block.
// The next element's slots, flags and nodes are on their way meanwhile.  54 KB
// and 96 threads per element: four elements per SM.
// Measured at 32,760 hex20 elements, 27 points: 1,287 us with a thread per pair,
// 1,157 with the entry indices worked out per entry, 1,000 like this
// (with the old values fetched before the Jacobians, the launches in turn).  Half of
// it is the scatter: with the matrix instructions left out a colour takes 105 of
// 125 us, with the scatter left out 62 (loads into registers in fifteens
// instead of cp.async, five elements per SM: 122).
#include <algorithm>
#include <cstdint>

#include "elem_common.cuh"
#include "internal.h"

namespace fastgpu {
namespace {

constexpr int kN = 20, kT = 96, kLD = 77;  // (77: neither the fragments' nor D's stores pile up on a bank)

template <int NG>
struct MmaSmem {
  static constexpr int KS = (NG + 3) / 4;          // steps of the product
  static constexpr int kD = KS * 4 * kLD;          // D[g][24 i + a], then the blocks [210][9]
  static constexpr int kJ = (9 * NG + 1) / 2 * 2, kX = 3 * kN, kK = 9 * kN * kN;
  static constexpr int kV = 9 * kN * (kN + 1) / 2, kDV = kD > kV ? kD : kV;
  static constexpr size_t bytes = sizeof(double) * (kDV + kJ + kX + kK) + sizeof(int32_t) * (2 * kN * kN + 436) + 32;
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// M of the node tiles (A0, B0) and (A1, B1), 8 nodes each
template <int KS, int A0, int B0, int A1, int B1>
__device__ __forceinline__ void tiles(const double *sD, int lane, double (&M)[2][9][2]) {
  const double *d = sD + (lane & 3) * kLD + (lane >> 2);
#pragma unroll 1
  for (int s = 0; s < KS; s++, d += 4 * kLD) {
    double a0[3], b0[3], a1[3], b1[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      a0[i] = d[24 * i + 8 * A0];
      b0[i] = B0 == A0 ? a0[i] : d[24 * i + 8 * B0];
      a1[i] = A1 == A0 ? a0[i] : d[24 * i + 8 * A1];
      b1[i] = B1 == A1 ? a1[i] : (B1 == B0 ? b0[i] : d[24 * i + 8 * B1]);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        mma_f64(M[0][3 * i + j], a0[i], b0[j]);
        mma_f64(M[1][3 * i + j], a1[i], b1[j]);
      }
  }
}

// what a block (a, b) = q of the element needs: 9 times its place among the
// blocks with a <= b, whether it is the transpose, a and b
__device__ __forceinline__ int32_t block_word(int q) {
  const int a = q / kN, b = q - kN * a, lo = min(a, b), hi = max(a, b);
  return 9 * (lo * kN - lo * (lo - 1) / 2 + (hi - lo)) | (a > b ? 1 << 11 : 0) | a << 12 | b << 17;
}

template <int NG>
__global__ void __launch_bounds__(kT, 4) elem_mma20(ElemArgs A, const double *__restrict__ dNt) {
  using S = MmaSmem<NG>;
  extern __shared__ __align__(16) double sm[];
  double *sD = sm;              // and sV
  double *sKo = sD + S::kDV;
  double *sJ = sKo + S::kK;     // [9][NG]
  double *sX = sJ + S::kJ;
  int32_t *sRow = reinterpret_cast<int32_t *>(sX + S::kX);  // the element's slots [400], flags [16], nodes [20]
  int32_t *sSlot = sRow + 436;  // slots, complemented where the element writes first
  int32_t *sQ = sSlot + kN * kN;
  uint8_t *sfix = reinterpret_cast<uint8_t *>(sQ + kN * kN);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // scatter: 27 lanes of a warp take three blocks at a time, entry k of each
  chain_release();
  const int kb = lane / 9, k9 = lane - 9 * kb, kt9 = 3 * (k9 % 3) + k9 / 3, q0 = 3 * w + kb;
  for (int q = tid; q < kN * kN; q += kT) sQ[q] = block_word(q);
  auto ahead = [&](int64_t it) {  // an element's slots, flags and nodes
    if (it < A.ne) {
      const int64_t e = A.offset + it;
      for (int i = tid; i < 109; i += kT) {
        const void *g = i < 100 ? (const void *)(A.slot + e * (kN * kN) + 4 * i)
                                : (i < 104 ? (const void *)(A.first + e * 16 + 4 * (i - 100))
                                           : (const void *)(A.conn + e * kN + 4 * (i - 104)));
        if (A.first || i < 100 || i >= 104)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                           (unsigned)__cvta_generic_to_shared(sRow + 4 * i)),
                       "l"(g)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  ahead(blockIdx.x);
  for (int64_t it = blockIdx.x; it < A.ne; it += gridDim.x) {
    const int64_t e = A.offset + it;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    bool fixed_node = false;
    if (tid < 3 * kN) {
      sX[tid] = A.X[3 * (int64_t)sRow[416 + tid / 3] + tid % 3];
    } else if (tid - 3 * kN < kN) {
      const uint8_t f = A.fix[sRow[416 + tid - 3 * kN]];
      sfix[tid - 3 * kN] = f;
      fixed_node = f != 0;
    }
    for (int q = tid; q < kN * kN; q += kT) {
      const bool fst = A.first && ((uint32_t)sRow[400 + (q >> 5)] >> (q & 31) & 1u);
      sSlot[q] = fst ? ~sRow[q] : sRow[q];
    }
    const bool any_fixed = __syncthreads_or(fixed_node);
    // Jacobians J[p][q] = sum_a dN_a/dxi_p X_a,q (cShapeSolid::DrvShpXYZ, shp/shpsolid.cpp:58-126)
    for (int g = lane; g < NG; g += 32) {
      double j0 = 0.0, j1 = 0.0, j2 = 0.0;
#pragma unroll 10
      for (int a = 0; a < kN; a++) {
        const double d = dNt[(3 * a + w) * NG + g];
        j0 = fma(d, sX[3 * a], j0);
        j1 = fma(d, sX[3 * a + 1], j1);
        j2 = fma(d, sX[3 * a + 2], j2);
      }
      sJ[(3 * w) * NG + g] = j0;
      sJ[(3 * w + 1) * NG + g] = j1;
      sJ[(3 * w + 2) * NG + g] = j2;
    }
    __syncthreads();
    for (int g = lane; g < 4 * S::KS; g += 32) {
      double *D = sD + g * kLD;
      if (g >= NG) {  // the steps' padding
        for (int a = w; a < 72; a += 3) D[a] = 0.0;
        continue;
      }
      // inverse by cofactors (cShape::ShpMatInv, shp/shape.cpp:360-393) and D in
      // the expressions of elem_kernels.cu: the same bits whichever kernel runs
      const double j00 = sJ[g], j01 = sJ[NG + g], j02 = sJ[2 * NG + g], j10 = sJ[3 * NG + g], j11 = sJ[4 * NG + g],
                   j12 = sJ[5 * NG + g], j20 = sJ[6 * NG + g], j21 = sJ[7 * NG + g], j22 = sJ[8 * NG + g];
      const double det = j00 * (j11 * j22 - j12 * j21) - j01 * (j10 * j22 - j12 * j20) + j02 * (j10 * j21 - j11 * j20);
      if (!(det > 0.0)) atomicOr(A.status, 1);
      const double id = 1.0 / ((det != 0.0) ? det : 1.0);
      double J[9];
      J[0] = (j11 * j22 - j12 * j21) * id;
      J[1] = -(j01 * j22 - j02 * j21) * id;
      J[2] = (j01 * j12 - j02 * j11) * id;
      J[3] = -(j10 * j22 - j12 * j20) * id;
      J[4] = (j00 * j22 - j02 * j20) * id;
      J[5] = -(j00 * j12 - j02 * j10) * id;
      J[6] = (j10 * j21 - j11 * j20) * id;
      J[7] = -(j00 * j21 - j01 * j20) * id;
      J[8] = (j00 * j11 - j01 * j10) * id;
      const double sq = sqrt(A.w[g] * det);
#pragma unroll 7
      for (int a = w; a < kN; a += 3) {
        const double d0 = dNt[(3 * a) * NG + g], d1 = dNt[(3 * a + 1) * NG + g], d2 = dNt[(3 * a + 2) * NG + g];
        D[a] = sq * (J[0] * d0 + J[1] * d1 + J[2] * d2);
        D[24 + a] = sq * (J[3] * d0 + J[4] * d1 + J[5] * d2);
        D[48 + a] = sq * (J[6] * d0 + J[7] * d1 + J[8] * d2);
      }
    }
    if (it == blockIdx.x) chain_wait();
    if (lane < 27) {
#pragma unroll 5
      for (int q = q0; q < kN * kN; q += 9) {
        const int32_t sl = sSlot[q];
        if (sl >= 0)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                           (unsigned)__cvta_generic_to_shared(sKo + 9 * q + k9)),
                       "l"(A.K + (int64_t)sl * 9 + k9)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ahead(it + gridDim.x);
    const double E = A.E[e], nu = A.nu[e];
    __syncthreads();
    double M[2][9][2];
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int k = 0; k < 9; k++) M[t][k][0] = M[t][k][1] = 0.0;
    if (w == 0) tiles<S::KS, 0, 0, 0, 1>(sD, lane, M);
    else if (w == 1) tiles<S::KS, 0, 2, 1, 1>(sD, lane, M);
    else tiles<S::KS, 1, 2, 2, 2>(sD, lane, M);
    __syncthreads();
    // the isotropic blocks: i == j: C00 M_ii + G (tr M - M_ii); i != j: C01 M_ij + G M_ji
    double *sV = sD;
    const double dd = (1.0 + nu) * (1.0 - 2.0 * nu);
    const double C00 = E * (1.0 - nu) / dd, C01 = E * nu / dd, G = 0.5 * E / (1.0 + nu);
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const int ta = w == 0 ? 0 : (w == 1 ? t : 1 + t), tb = w == 0 ? t : (w == 1 ? 2 - t : 2);
      const int a = 8 * ta + (lane >> 2);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int b = 8 * tb + 2 * (lane & 3) + h;
        if (a > b || b >= kN) continue;
        double *v = sV + 9 * (a * kN - a * (a - 1) / 2 + (b - a));
        const double tr = M[t][0][h] + M[t][4][h] + M[t][8][h];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int j = 0; j < 3; j++)
            v[3 * i + j] = i == j ? C00 * M[t][4 * i][h] + G * (tr - M[t][4 * i][h])
                                  : C01 * M[t][3 * i + j][h] + G * M[t][3 * j + i][h];
      }
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (lane < 27 && !any_fixed) {
#pragma unroll 5
      for (int q = q0; q < kN * kN; q += 9) {
        const int32_t sl = sSlot[q], t = sQ[q];
        const double add = sV[(t & 2047) + (t & 2048 ? kt9 : k9)];
        if (sl >= 0) A.K[(int64_t)sl * 9 + k9] = sKo[9 * q + k9] + add;
        else A.K[(int64_t)~sl * 9 + k9] = add;
      }
    } else if (lane < 27) {
      const int i = k9 / 3, j = k9 - 3 * i;
      for (int q = q0; q < kN * kN; q += 9) {
        const int32_t sl = sSlot[q], t = sQ[q];
        const int a = (t >> 12) & 31, b = t >> 17;
        const bool fst = sl < 0, fixed = ((sfix[a] >> i) & 1) || ((sfix[b] >> j) & 1);
        double out;
        if (entry_value(fst, fixed, a == b && i == j, fst ? 0.0 : sKo[9 * q + k9],
                        sV[(t & 2047) + (t & 2048 ? kt9 : k9)], out))
          A.K[(int64_t)(fst ? ~sl : sl) * 9 + k9] = out;
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int NG>
cudaError_t run(Ctx &c, const Bucket &B, ElemArgs a, int64_t count) {
  auto kern = elem_mma20<NG>;
  const size_t bytes = MmaSmem<NG>::bytes;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kT, bytes);
  if (e != cudaSuccess) return e;
  per_sm = elem_per_sm(c, per_sm, a.ctas_per_sm);
  a.ne = count;
  c.launches++;
  return launch_chained(a.chain, kern, dim3((unsigned)std::min<int64_t>((int64_t)per_sm * c.sm_count, count)), dim3(kT),
                        bytes, c.stream, a, B.d_dNt);
}

}  // namespace

cudaError_t launch_mma_elements(Ctx &c, const Bucket &B, ElemArgs a, int64_t count) {
  if (count <= 0) return cudaSuccess;
  if (!B.d_dNt || !B.d_slot || !a.K) return cudaErrorInvalidValue;
  switch (B.ng) {
    case 8: return run<8>(c, B, a, count);
    case 27: return run<27>(c, B, a, count);
    case 64: return run<64>(c, B, a, count);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fastgpu
