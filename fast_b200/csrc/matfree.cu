// matfree.cu - K.u for large small-strain hex models without the assembled
// matrix (sm_100a): the operator of the PCG iteration and of its residuals.
//
// An iteration on the assembled matrix streams it: 40 (FP32) or 76 (FP64)
// bytes per 3x3 block, 57 blocks per node of a hex20 mesh, 1.26 / 2.4 GB at
// 131,072 elements, 214 / 402 us at 6 TB/s.  Applied element by element
// (matfree_math.cuh) the same product reads 9 numbers per Gauss point and the
// directions of the element's nodes: 0.19 / 0.37 GB, and about 4,700
// multiply-adds per element.  Measured there: element kernel 68 / 117 us, node
// kernel 27 / 51 us (an iteration 239 -> 102 us in FP32, with its FP64 residuals,
// 447 -> 173 us in FP64).
// What bounds the element kernel now is the latency of its dependent steps at
// 12 (9) warps per SM: with the geometry resident in L2 it still takes 62 us.
//
// One iteration is two kernels:
//  1. elements: convergence test and beta from the last update's partial sums,
//     the direction z + beta p built for every gathered node, element forces
//     K_e p_e to memory, partial p.K p (the sum over elements of p_e . K_e p_e);
//  2. nodes: alpha, w = the sum of the node's element forces in a fixed order
//     (no atomics: the same bits every run), p, u, r, z and the partial sums.
// Every block forms the scalars it needs from the partials, alike (a last block
// doing it at the end of the kernel before was slower: 98 against 93 us an
// iteration at 131,072 hex20 elements).
//
// hex20: three warps take 32 elements, a lane per element and a warp per Gauss
// plane: it collapses the nodal values onto its plane, works through the
// plane's nine points and carries them back alone; the three parts are summed
// in shared memory.  hex8: a lane takes its element whole.  Elements are
// batched by 32 in the mesh's own order (neighbours share nodes in L1 and L2);
// every per-element array has the elements of a batch innermost, so each load
// is one full line per warp.
#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include "elem_common.cuh"
#include "matfree_math.cuh"
#include "solve_common.cuh"

namespace fastgpu {

namespace {

constexpr int kT20 = 96;   // hex20: a warp per Gauss plane
constexpr int kT8 = 128;   // hex8: 4 batches
constexpr int kMfBatchChunk = 32;  // iterations of independent problems between two looks at their states

template <typename T>
struct MfArgs {
  int nb;                          // batches of 32 elements
  const int32_t *conn;             // [nb][nn][32] nodes (padding elements: node 0, zero geometry)
  const T *geo;                    // hex20 [nb][9 lines][27][32], hex8 (FP32) [nb][72][32]
  const double *X;                 // hex8 (FP64): nodal coordinates, 3 per node
  const T *lam, *mu;               // [nb][32]
  const T *p, *z;                  // directions
  T *F;                            // [nb][nn][32][4] element forces
  PcgState *st;
  const int32_t *skip;
  double *part;                    // p.K p per block (or null)
  const double *part_rr, *part_zr; // DIR: sums of the last update
  int nred;
};

// sums of n <= 8 NT partials in a fixed order, all loads in flight; every thread gets them
template <int NT, int NV>
__device__ __forceinline__ void sum_parts(const double *const (&p)[NV], int n, double (&out)[NV]) {
  __shared__ double sw[NV][NT / 32], sv[NV];
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) v[k] = 0.0;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int k = 0; k < NV; k++) {
      const int at = threadIdx.x + i * NT;
      v[k] += at < n ? p[k][at] : 0.0;
    }
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const double t = warp_sum(v[k]);
    if ((threadIdx.x & 31) == 0) sw[k][threadIdx.x >> 5] = t;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++) t += sw[threadIdx.x][w];
    sv[threadIdx.x] = t;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; k++) out[k] = sv[k];
}

// DIR: the scalars of pcg_direction_fused, formed alike in every block; returns done
template <int NT>
__device__ __forceinline__ int next_direction(const PcgState *st, const double *part_rr, const double *part_zr, int n,
                                              double &rr, double &zr, double &err, double &beta) {
  const double lenf = st->lenf, tol = st->tol, dot0 = st->dot0;
  const int iter = st->iter + 1, maxit = st->maxit;
  const double *const p[2] = {part_rr, part_zr};
  double v[2];
  sum_parts<NT>(p, n, v);
  rr = v[0];
  zr = v[1];
  err = sqrt(rr) / lenf;
  beta = zr / dot0;
  return err < tol ? 1 : (!isfinite(err) ? 3 : (iter >= maxit ? 2 : 0));
}

__device__ __forceinline__ void commit_direction(PcgState *st, int done, double rr, double zr, double err,
                                                 double beta) {
  if (last_block(&st->arrive_dir)) {
    st->iter += 1;
    st->rr = rr;
    st->err = err;
    if (done) {
      st->done = done;
    } else {
      st->beta = beta;
      st->dot0 = zr;
    }
  }
}

// Gauss plane k of 32 elements, by one warp: the nodal values in sU
// [3][20][32] -> the plane's part of the element forces in sR [3][24][32] (20
// of 24 used).  FP32 keeps the plane's polynomials and their adjoints in
// registers and finds the plane's geometry [81][32] in sR's place (each lane
// reads and writes its own column only); in FP64 neither fits: the line
// coefficients and results pass through sR (the warp's own), the geometry is
// loaded a point ahead of its use.  No other warp is involved.
template <typename T>
__device__ __forceinline__ void hex20_plane(int k, const T *sU, T *sR, const T *gp, T lam, T mu, int lane) {
  constexpr bool REG = sizeof(T) == 4;
  const T z = mf::gauss20<T>(k), zz = mf::gauss20_sq<T>(k);
  T An[9];
  if (!REG) {
#pragma unroll
    for (int q = 0; q < 9; q++) An[q] = __ldcs(gp + 32 * q);  // (read once: evict first)
  }
  mf::Plane<T> P[REG ? 3 : 1], N[REG ? 3 : 1];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    T f[20];
#pragma unroll
    for (int a = 0; a < 20; a++) f[a] = sU[(20 * c + a) * 32 + lane];
    const mf::Plane<T> Q = mf::plane_poly(f, z, zz);
    if (REG) {
      P[REG ? c : 0] = Q;
      N[REG ? c : 0] = mf::Plane<T>{};
    } else {
#pragma unroll
      for (int j = 0; j < 3; j++) {
        T L[8];
        mf::plane_line(Q, mf::gauss20<T>(j), mf::gauss20_sq<T>(j), L);
#pragma unroll
        for (int q = 0; q < 8; q++) sR[(24 * c + 8 * j + q) * 32 + lane] = L[q];
      }
    }
  }
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    if (REG && j == 0) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
    }
    const T y = mf::gauss20<T>(j), yy = mf::gauss20_sq<T>(j);
    T *sj = sR + 8 * j * 32 + lane;
    T H[3][9];
    {
      T L[3][8];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if (REG) {
          mf::plane_line(P[REG ? c : 0], y, yy, L[c]);
        } else {
#pragma unroll
          for (int q = 0; q < 8; q++) L[c][q] = sj[(24 * c + q) * 32];
        }
      }
      mf::line_gradients(L, H);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      T A[9], S[9];
      if (REG) {
#pragma unroll
        for (int q = 0; q < 9; q++) A[q] = sR[(9 * (3 * j + i) + q) * 32 + lane];
      } else {
#pragma unroll
        for (int q = 0; q < 9; q++) A[q] = An[q];
        const T *gn = gp + (3 * j + i < 8 ? 32 * 9 * (3 * j + i + 1) : 0);
#pragma unroll
        for (int q = 0; q < 9; q++) An[q] = __ldcs(gn + 32 * q);
      }
      mf::point_stress(H[i], A, lam, mu, S);
#pragma unroll
      for (int q = 0; q < 9; q++) H[i][q] = S[q];
    }
    T R[3][8];
    mf::line_gradients_t(H, R);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (REG) {
        mf::plane_line_t(R[c], y, yy, N[REG ? c : 0]);
      } else {
#pragma unroll
        for (int q = 0; q < 8; q++) sj[(24 * c + q) * 32] = R[c][q];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    T f[20];
    if (!REG) {
      N[0] = mf::Plane<T>{};
#pragma unroll
      for (int j = 0; j < 3; j++) {
        T L[8];
#pragma unroll
        for (int q = 0; q < 8; q++) L[q] = sR[(24 * c + 8 * j + q) * 32 + lane];
        mf::plane_line_t(L, mf::gauss20<T>(j), mf::gauss20_sq<T>(j), N[0]);
      }
    }
    mf::plane_poly_t(N[REG ? c : 0], z, zz, f);
#pragma unroll
    for (int a = 0; a < 20; a++) sR[(24 * c + a) * 32 + lane] = f[a];
  }
}

// element forces of the hex20 batches; DIR: x = z + beta p, otherwise x = p.
// The block's three warps meet twice per batch: after the gather and for the
// sum of their parts.
template <typename T, bool DIR>
__global__ void __launch_bounds__(kT20, sizeof(T) == 4 ? 4 : 3) mf_hex20(MfArgs<T> A) {
  extern __shared__ __align__(16) unsigned char msm[];
  __shared__ double sred[32];
  T *sU = reinterpret_cast<T *>(msm);  // [3][20][32]
  T *sR = sU + 3 * 20 * 32;            // [3 planes][PLANE]: [3][24][32], in FP32 also the geometry [81][32]
  constexpr int PLANE = (sizeof(T) == 4 ? 81 : 72) * 32;
  int32_t *sC = reinterpret_cast<int32_t *>(sR + 3 * PLANE);  // [20][32] the next batch's nodes
  if (A.skip && *A.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double pacc = 0.0;
  // the next batch on its way while this one is worked on: its nodes to shared
  // memory, its geometry (31 or 62 KB) to L2
  auto ahead = [&](int b) {
    if (b < A.nb) {
      for (int i = tid; i < 20 * 8; i += kT20)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sC + 4 * i)),
                     "l"(A.conn + (size_t)b * (20 * 32) + 4 * i)
                     : "memory");
      const char *g = reinterpret_cast<const char *>(A.geo + (size_t)b * (9 * 27 * 32));
      for (int i = tid; i < 9 * 27 * 32 * (int)sizeof(T) / 128; i += kT20)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(g + 128 * i));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  ahead(blockIdx.x);
  double rr = 0, zr = 0, err = 0, bt = 0;
  int done = 0;
  if (DIR) done = next_direction<kT20>(A.st, A.part_rr, A.part_zr, A.nred, rr, zr, err, bt);
  const T beta = (T)bt;
  for (int b = blockIdx.x; b < A.nb && !done; b += gridDim.x) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const T *gp = A.geo + ((size_t)b * 9 + 3 * w) * (27 * 32);
    T *sRw = sR + w * PLANE;
    if (sizeof(T) == 4) {  // the plane's geometry, while the block gathers
#pragma unroll 7
      for (int i = lane; i < 81 * 32 / 4; i += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sRw + 4 * i)),
                     "l"(gp + 4 * i)
                     : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int h = 0; h < 7; h++) {
      const int a = w + 3 * h;
      if (a >= 20) continue;
      const int64_t n = sC[32 * a + lane];
      T x[3];
      V4<T>::load(A.p + 4 * n, x[0], x[1], x[2]);
      if (DIR) {
        T y[3];
        V4<T>::load(A.z + 4 * n, y[0], y[1], y[2]);
#pragma unroll
        for (int q = 0; q < 3; q++) x[q] = y[q] + beta * x[q];
      }
#pragma unroll
      for (int q = 0; q < 3; q++) sU[(20 * q + a) * 32 + lane] = x[q];
    }
    __syncthreads();
    const T lam = A.lam[(size_t)b * 32 + lane], mu = A.mu[(size_t)b * 32 + lane];
    hex20_plane(w, sU, sRw, gp + lane, lam, mu, lane);
    __syncthreads();
    ahead(b + gridDim.x);
#pragma unroll
    for (int h = 0; h < 7; h++) {
      const int a = w + 3 * h;
      if (a >= 20) continue;
      T f[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const T *r = sR + (24 * i + a) * 32 + lane;
        f[i] = (r[0] + r[PLANE]) + r[2 * PLANE];
        pacc += (double)f[i] * sU[(20 * i + a) * 32 + lane];
      }
      V4<T>::store(A.F + 4 * (((size_t)b * 20 + a) * 32 + lane), f[0], f[1], f[2]);
    }
    // (the next gather writes sU, the next geometry copy sR after a barrier)
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (A.part && !done) {
    const double s = block_sum<kT20>(pacc, sred);
    if (tid == 0) A.part[blockIdx.x] = s;
  }
  if (DIR) commit_direction(A.st, done, rr, zr, err, bt);
}

// ... of the hex8 batches in FP32: a lane takes its element whole.  The geometry
// of a warp's batch (9 KB) is copied to shared memory while the warp gathers.
// (Stored, not rebuilt as in FP64: differences of FP32 coordinates would lose
// digits.)
template <bool DIR>
__global__ void __launch_bounds__(kT8) mf_hex8_32(MfArgs<float> A) {
  using T = float;
  extern __shared__ __align__(16) unsigned char msm[];
  __shared__ double sred[32];
  if (A.skip && *A.skip) return;
  const int tid = threadIdx.x, lane = tid & 31;
  T *sG = reinterpret_cast<T *>(msm) + (tid >> 5) * 72 * 32;
  double pacc = 0.0;
  const int b0 = blockIdx.x * (kT8 / 32) + (tid >> 5), db = gridDim.x * (kT8 / 32);
  auto copy_geometry = [&](int b) {
    const char *g = reinterpret_cast<const char *>(A.geo + (size_t)b * (72 * 32));
    const unsigned d = (unsigned)__cvta_generic_to_shared(sG);
#pragma unroll 9
    for (int i = lane; i < 72 * 32 * (int)sizeof(T) / 16; i += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i), "l"(g + 16 * i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (b0 < A.nb) copy_geometry(b0);
  double rr = 0, zr = 0, err = 0, bt = 0;
  int done = 0;
  if (DIR) done = next_direction<kT8>(A.st, A.part_rr, A.part_zr, A.nred, rr, zr, err, bt);
  const T beta = (T)bt;
  for (int b = b0; b < A.nb && !done; b += db) {
    T x[3][8], D[3][3][4], R[3][3][4];
    int32_t n[8];
#pragma unroll
    for (int a = 0; a < 8; a++) n[a] = A.conn[((size_t)b * 8 + a) * 32 + lane];
    const T lam = A.lam[(size_t)b * 32 + lane], mu = A.mu[(size_t)b * 32 + lane];
#pragma unroll
    for (int a = 0; a < 8; a++) V4<T>::load(A.p + 4 * (int64_t)n[a], x[0][a], x[1][a], x[2][a]);
    if (DIR) {
#pragma unroll
      for (int a = 0; a < 8; a++) {
        T y[3];
        V4<T>::load(A.z + 4 * (int64_t)n[a], y[0], y[1], y[2]);
#pragma unroll
        for (int c = 0; c < 3; c++) x[c][a] = y[c] + beta * x[c][a];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      mf::hex8_grads(x[c], D[c]);
#pragma unroll
      for (int i = 0; i < 12; i++) R[c][i / 4][i % 4] = T(0);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int gx = g & 1, gy = (g >> 1) & 1, gz = g >> 2;
      const int id[3] = {gy + 2 * gz, gx + 2 * gz, gx + 2 * gy};
      T H[9], P[9], Ag[9];
#pragma unroll
      for (int q = 0; q < 9; q++) Ag[q] = sG[(9 * g + q) * 32 + lane];
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int d = 0; d < 3; d++) H[3 * c + d] = D[c][d][id[d]];
      mf::point_stress(H, Ag, lam, mu, P);
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int d = 0; d < 3; d++) R[c][d][id[d]] += P[3 * c + d];
    }
    __syncwarp();
    if (b + db < A.nb) copy_geometry(b + db);
    T f[3][8];
#pragma unroll
    for (int c = 0; c < 3; c++) mf::hex8_grads_t(R[c], f[c]);
#pragma unroll
    for (int a = 0; a < 8; a++) {
      V4<T>::store(A.F + 4 * (((size_t)b * 8 + a) * 32 + lane), f[0][a], f[1][a], f[2][a]);
      pacc += (double)f[0][a] * x[0][a] + (double)f[1][a] * x[1][a] + (double)f[2][a] * x[2][a];
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (A.part && !done) {
    const double s = block_sum<kT8>(pacc, sred);
    if (tid == 0) A.part[blockIdx.x] = s;
  }
  if (DIR) commit_direction(A.st, done, rr, zr, err, bt);
}

// FP64 forces of a lane's hex8 element at x = z + beta p (DIR) or p, into
// F[node][32][4]; returns x . K_e x.  The geometry is rebuilt from the nodes'
// coordinates (in L1 and L2: neighbours share them): 72 stored numbers a
// visit would be 576 of an element's 900 bytes, and the 450 extra operations
// are cheap beside them.  The coordinates' derivatives wait in the lane's
// column of sJ[36][kT8].  Bound by the FP64 pipe (half busy) and its latency at
// 8 warps per SM: 248 registers hold D and R; at 168, three blocks, the spills
// cost more than the warps give (261 against 183 us for 1.5 million elements,
// which with loads at their point of use took 245).  An iteration at 127,500
// nodes went from 48.9 us with stored geometry to 44.0.
template <bool DIR>
__device__ __forceinline__ double hex8_forces(const int32_t (&n)[8], const double *__restrict__ X, const double *p,
                                              const double *z, double beta, double lam, double mu, double *sJ,
                                              double *F) {
  double D[3][3][4], R[3][3][4];
  {
    double x[3][8], y[3][8], v[3][8];  // every load in flight before the first use
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
      for (int c = 0; c < 3; c++) v[c][a] = X[3 * (int64_t)n[a] + c];
#pragma unroll
    for (int a = 0; a < 8; a++) V4<double>::load(p + 4 * (int64_t)n[a], x[0][a], x[1][a], x[2][a]);
    if (DIR) {
#pragma unroll
      for (int a = 0; a < 8; a++) V4<double>::load(z + 4 * (int64_t)n[a], y[0][a], y[1][a], y[2][a]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      mf::hex8_grads(v[c], D[c]);
#pragma unroll
      for (int i = 0; i < 12; i++) sJ[(12 * c + i) * kT8] = D[c][i / 4][i % 4];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (DIR) {
#pragma unroll
        for (int a = 0; a < 8; a++) x[c][a] = y[c][a] + beta * x[c][a];
      }
      mf::hex8_grads(x[c], D[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int i = 0; i < 12; i++) R[c][i / 4][i % 4] = 0.0;
#pragma unroll
  for (int g = 0; g < 8; g++) {
    const int gx = g & 1, gy = (g >> 1) & 1, gz = g >> 2;
    const int id[3] = {gy + 2 * gz, gx + 2 * gz, gx + 2 * gy};
    double H[9], P[9], A[9];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int d = 0; d < 3; d++) P[3 * c + d] = sJ[(12 * c + 4 * d + id[d]) * kT8];
    const double q = 1.0 / mf::cofactors(P, A);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int d = 0; d < 3; d++) H[3 * c + d] = D[c][d][id[d]];
    mf::point_stress(H, A, q * lam, q * mu, P);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int d = 0; d < 3; d++) R[c][d][id[d]] += P[3 * c + d];
  }
  double e = 0.0;  // x . G^T R = (G x) . R
  double f[3][8];
#pragma unroll
  for (int c = 0; c < 3; c++) {
#pragma unroll
    for (int i = 0; i < 12; i++) e += D[c][i / 4][i % 4] * R[c][i / 4][i % 4];
    mf::hex8_grads_t(R[c], f[c]);
  }
#pragma unroll
  for (int a = 0; a < 8; a++) V4<double>::store(F + 4 * 32 * a, f[0][a], f[1][a], f[2][a]);
  return e;
}

// what a lane needs of its next element, loaded while it works on this one
struct Hex8Ahead {
  int32_t n[8];
  double lam, mu;
  __device__ __forceinline__ void load(const MfArgs<double> &A, int b, int lane) {
#pragma unroll
    for (int a = 0; a < 8; a++) n[a] = A.conn[((size_t)b * 8 + a) * 32 + lane];
    lam = A.lam[(size_t)b * 32 + lane];
    mu = A.mu[(size_t)b * 32 + lane];
  }
};

template <bool DIR>
__global__ void __launch_bounds__(kT8, 2) mf_hex8_64(MfArgs<double> A) {
  __shared__ double sJ[36 * kT8];
  __shared__ double sred[32];
  if (A.skip && *A.skip) return;
  const int tid = threadIdx.x, lane = tid & 31;
  double pacc = 0.0, rr = 0, zr = 0, err = 0, beta = 0;
  int done = 0;
  if (DIR) done = next_direction<kT8>(A.st, A.part_rr, A.part_zr, A.nred, rr, zr, err, beta);
  Hex8Ahead h;
  int b = blockIdx.x * (kT8 / 32) + (tid >> 5);
  if (b < A.nb) h.load(A, b, lane);
  while (b < A.nb && !done) {
    const Hex8Ahead g = h;
    const int at = b;
    b += gridDim.x * (kT8 / 32);
    if (b < A.nb) h.load(A, b, lane);
    pacc += hex8_forces<DIR>(g.n, A.X, A.p, A.z, beta, g.lam, g.mu, sJ + tid, A.F + 4 * ((size_t)at * (8 * 32) + lane));
  }
  if (A.part && !done) {
    const double s = block_sum<kT8>(pacc, sred);
    if (tid == 0) A.part[blockIdx.x] = s;
  }
  if (DIR) commit_direction(A.st, done, rr, zr, err, beta);
}

// sum of the node's element forces, supports masked
template <typename T>
__device__ __forceinline__ void node_force(int64_t n, const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc,
                                           const T *__restrict__ F, const uint8_t *__restrict__ fix, T &w0, T &w1,
                                           T &w2) {
  w0 = w1 = w2 = T(0);
  const int32_t i1 = ptr[n + 1];
  for (int32_t i = ptr[n]; i < i1; i++) {  // entries in fours (the last ones padded by a zero entry): four loads in flight
    const int4 e = reinterpret_cast<const int4 *>(inc)[i];
    T a[4], b[4], c[4];
    V4<T>::load(F + 4 * (int64_t)e.x, a[0], b[0], c[0]);
    V4<T>::load(F + 4 * (int64_t)e.y, a[1], b[1], c[1]);
    V4<T>::load(F + 4 * (int64_t)e.z, a[2], b[2], c[2]);
    V4<T>::load(F + 4 * (int64_t)e.w, a[3], b[3], c[3]);
    w0 += (a[0] + a[1]) + (a[2] + a[3]);
    w1 += (b[0] + b[1]) + (b[2] + b[3]);
    w2 += (c[0] + c[1]) + (c[2] + c[3]);
  }
  const uint8_t m = fix[n];
  if (m & 1) w0 = T(0);
  if (m & 2) w1 = T(0);
  if (m & 4) w2 = T(0);
}

// one node: p = z + beta p (DIR), u += alpha p, r -= alpha w, z = Dinv r; adds
// to r.r and z.r.  dj: the inverse diagonal, 4 per node (Jacobi), or null and
// dinv, 12 per node.
template <typename T, bool DIR>
__device__ __forceinline__ void node_update(int64_t n, const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc,
                                            const T *__restrict__ F, const uint8_t *__restrict__ fix,
                                            T *__restrict__ u, T *__restrict__ r, T *__restrict__ z,
                                            T *__restrict__ p, const T *__restrict__ dj, const T *__restrict__ dinv,
                                            T alpha, T beta, double &rr, double &zr) {
  T u0, u1, u2, p0, p1, p2, r0, r1, r2, w0, w1, w2, z0, z1, z2;
  V4<T>::load(p + 4 * n, p0, p1, p2);
  if (DIR) V4<T>::load(z + 4 * n, z0, z1, z2);
  V4<T>::load(u + 4 * n, u0, u1, u2);
  V4<T>::load(r + 4 * n, r0, r1, r2);
  node_force(n, ptr, inc, F, fix, w0, w1, w2);
  if (DIR) {
    p0 = z0 + beta * p0; p1 = z1 + beta * p1; p2 = z2 + beta * p2;
    V4<T>::store(p + 4 * n, p0, p1, p2);
  }
  u0 = u0 + alpha * p0; u1 = u1 + alpha * p1; u2 = u2 + alpha * p2;
  r0 = r0 + (-alpha) * w0; r1 = r1 + (-alpha) * w1; r2 = r2 + (-alpha) * w2;
  if (dj) {
    T d0, d1, d2;
    V4<T>::load(dj + 4 * n, d0, d1, d2);
    z0 = d0 * r0; z1 = d1 * r1; z2 = d2 * r2;
  } else {
    apply_dinv(dinv + 12 * n, r0, r1, r2, z0, z1, z2);
  }
  V4<T>::store(u + 4 * n, u0, u1, u2);
  V4<T>::store(r + 4 * n, r0, r1, r2);
  V4<T>::store(z + 4 * n, z0, z1, z2);
  rr += (double)r0 * r0 + (double)r1 * r1 + (double)r2 * r2;
  zr += (double)z0 * r0 + (double)z1 * r1 + (double)z2 * r2;
}

// alpha = dot0 / p.Kp (every block), p = z + beta p (DIR), u += alpha p;
// r -= alpha w; z = Dinv r; partials r.r, z.r; the last block stores p.Kp and
// alpha, or the breakdown state (as pcg_update_fused).
template <typename T, bool DIR>
__global__ void __launch_bounds__(kVecThreads)
mf_update(int64_t nnode, const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc, const T *__restrict__ F,
          const uint8_t *__restrict__ fix, T *__restrict__ u, T *__restrict__ r, T *__restrict__ z, T *__restrict__ p,
          const T *__restrict__ dj, const T *__restrict__ dinv, PcgState *__restrict__ st,
          const double *__restrict__ part_pw, int npw, double *__restrict__ part_rr, double *__restrict__ part_zr) {
  if (st->done) return;
  __shared__ double sbuf[32];
  const double dot0 = st->dot0;
  const T beta = (T)st->beta;
  const double *const pp[1] = {part_pw};
  double pw[1];
  sum_parts<kVecThreads>(pp, npw, pw);
  const double al = dot0 / pw[0];
  const bool bad = !(al > 0.0) || !isfinite(pw[0]) || !isfinite(al);
  if (!bad) {
    double rr = 0.0, zr = 0.0;
    const T alpha = (T)al;
    for (int64_t n = blockIdx.x * (int64_t)kVecThreads + threadIdx.x; n < nnode; n += (int64_t)gridDim.x * kVecThreads)
      node_update<T, DIR>(n, ptr, inc, F, fix, u, r, z, p, dj, dinv, alpha, beta, rr, zr);
    const double t1 = block_sum<kVecThreads>(rr, sbuf);
    if (threadIdx.x == 0) part_rr[blockIdx.x] = t1;
    const double t2 = block_sum<kVecThreads>(zr, sbuf);
    if (threadIdx.x == 0) part_zr[blockIdx.x] = t2;
  }
  if (last_block(&st->arrive_update)) {
    st->pw = pw[0];
    if (bad) st->done = 3;
    else st->alpha = al;
  }
}

// r = f - (the nodes' element forces), r.r per block; nothing while *skip
__global__ void __launch_bounds__(kVecThreads)
mf_residual(int64_t nnode, const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc,
            const double *__restrict__ F, const uint8_t *__restrict__ fix, const double *__restrict__ f,
            double *__restrict__ r, double *__restrict__ part, const int32_t *__restrict__ skip) {
  if (skip && *skip) return;
  __shared__ double sbuf[32];
  double rr = 0.0;
  for (int64_t n = blockIdx.x * (int64_t)kVecThreads + threadIdx.x; n < nnode; n += (int64_t)gridDim.x * kVecThreads) {
    double w0, w1, w2, f0, f1, f2;
    V4<double>::load(f + 4 * n, f0, f1, f2);
    node_force(n, ptr, inc, F, fix, w0, w1, w2);
    f0 -= w0; f1 -= w1; f2 -= w2;
    V4<double>::store(r + 4 * n, f0, f1, f2);
    rr += f0 * f0 + f1 * f1 + f2 * f2;
  }
  const double t = block_sum<kVecThreads>(rr, sbuf);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// ---- independent problems, all of them an iteration at a time

// Four kernels an iteration: elements (batches of every running problem, shared
// out over resident warps), alpha, nodes (blocks of 256 of one problem), beta.
// The chip is filled whatever the mix of sizes, and nothing streams a matrix
// (3.4 GB an iteration for 256 cantilevers with 1.8 million nodes).  There:
// elements 183 us on average over the solve, nodes 143 (at 5.4 TB/s), alpha and
// beta 4.8 and 3.9; all problems 780 -> 225 ms.  (The last tile of a problem
// forming alpha or beta behind a fence and a counter: 317 instead of 268 ms for
// assembly and solve.)
struct MfBatch {
  const int32_t *bprob;  // [nb] problem of a batch
  const int4 *ntile;     // {first node, end, problem, }
  const int32_t *eptr;   // [nprob + 1] batches of a problem
  const int32_t *nptr;   // ... node tiles
  MfProblem *S;
  double *part_pw;            // per batch
  double *part_rr, *part_zr;  // per node tile
};

// element forces at z + beta p, p.K p per batch
__global__ void __launch_bounds__(kT8, 2) mf_batch_elements(MfArgs<double> A, MfBatch B) {
  __shared__ double sJ[36 * kT8];
  const int tid = threadIdx.x, lane = tid & 31;
  struct Next {
    Hex8Ahead e;
    double beta;
    int done;
    __device__ __forceinline__ void load(const MfArgs<double> &A, const MfBatch &B, int b, int k, int lane) {
      e.load(A, b, lane);
      beta = B.S[k].beta;
      done = B.S[k].done;
    }
  } h;
  const int step = gridDim.x * (kT8 / 32);
  int b = blockIdx.x * (kT8 / 32) + (tid >> 5), k2 = 0;
  if (b < A.nb) h.e.load(A, b, lane);
  chain_wait();
  chain_release();
  if (b < A.nb) h.load(A, B, b, B.bprob[b], lane);
  if (b + step < A.nb) k2 = B.bprob[b + step];
  while (b < A.nb) {
    const Next g = h;
    const int at = b;
    b += step;
    if (b < A.nb) h.load(A, B, b, k2, lane);
    if (b + step < A.nb) k2 = B.bprob[b + step];
    if (g.done) continue;
    const double e = warp_sum(hex8_forces<true>(g.e.n, A.X, A.p, A.z, g.beta, g.e.lam, g.e.mu, sJ + tid,
                                                A.F + 4 * ((size_t)at * (8 * 32) + lane)));
    if (lane == 0) B.part_pw[at] = e;
  }
}

// a block per problem
__global__ void __launch_bounds__(128) mf_batch_alpha(MfBatch B) {
  __shared__ double sbuf[32];
  MfProblem *S = B.S + blockIdx.x;
  chain_wait();
  chain_release();
  if (S->done) return;
  double v = 0.0;
  for (int i = B.eptr[blockIdx.x] + threadIdx.x; i < B.eptr[blockIdx.x + 1]; i += 128) v += B.part_pw[i];
  const double pw = block_sum<128>(v, sbuf);
  if (threadIdx.x == 0) {
    const double al = S->dot0 / pw;
    S->alpha = al;
    if (!(al > 0.0) || !isfinite(pw) || !isfinite(al)) S->done = 3;
  }
}

// p = z + beta p, u, r, z; r.r and z.r
__global__ void __launch_bounds__(kVecThreads)
mf_batch_update(const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc, const double *__restrict__ F,
                const uint8_t *__restrict__ fix, double *__restrict__ u, double *__restrict__ r,
                double *__restrict__ z, double *__restrict__ p, const double *__restrict__ dj,
                const double *__restrict__ dinv, MfBatch B) {
  __shared__ double sbuf[32];
  const int4 t = B.ntile[blockIdx.x];
  const MfProblem *S = B.S + t.z;
  chain_wait();
  chain_release();
  if (S->done) return;
  const double alpha = S->alpha, beta = S->beta;
  const int64_t n = t.x + (int)threadIdx.x;
  double rr = 0.0, zr = 0.0;
  if (n < t.y) node_update<double, true>(n, ptr, inc, F, fix, u, r, z, p, dj, dinv, alpha, beta, rr, zr);
  rr = block_sum<kVecThreads>(rr, sbuf);
  zr = block_sum<kVecThreads>(zr, sbuf);
  if (threadIdx.x == 0) {
    B.part_rr[blockIdx.x] = rr;
    B.part_zr[blockIdx.x] = zr;
  }
}

// the stopping test and beta, a block per problem
__global__ void __launch_bounds__(128) mf_batch_beta(MfBatch B, double tol, int maxit) {
  __shared__ double sbuf[32];
  MfProblem *S = B.S + blockIdx.x;
  chain_wait();
  chain_release();
  if (S->done) return;
  double a = 0.0, b = 0.0;
  for (int i = B.nptr[blockIdx.x] + threadIdx.x; i < B.nptr[blockIdx.x + 1]; i += 128) {
    a += B.part_rr[i];
    b += B.part_zr[i];
  }
  const double rr = block_sum<128>(a, sbuf), zr = block_sum<128>(b, sbuf);
  if (threadIdx.x == 0) {
    const double err = sqrt(rr) / S->lenf;
    S->err = err;
    S->iter += 1;
    S->beta = zr / S->dot0;
    S->dot0 = zr;
    if (err < tol) S->done = 1;
    else if (!isfinite(err)) S->done = 3;
    else if (S->iter >= maxit) S->done = 2;
  }
}

// a block per problem: |f| with the reference's normaliser, r = f unless warm
// (then r = f - K u is there), z = Dinv r, p = 0 (the first direction is z + 0 p)
__global__ void __launch_bounds__(1024)
mf_batch_init(const int32_t *__restrict__ order, const int64_t *__restrict__ noff,
              const double *__restrict__ f, const double *__restrict__ dinv, double *__restrict__ u,
              double *__restrict__ r, double *__restrict__ z, double *__restrict__ p, double tol, int warm,
              MfProblem *__restrict__ S) {
  __shared__ double sbuf[32];
  __shared__ double slen;
  const int k = order[blockIdx.x];
  const int64_t n0 = noff[k], n1 = noff[k + 1];
  double ff = 0.0;
  for (int64_t n = n0 + threadIdx.x; n < n1; n += 1024) {
    double f0, f1, f2;
    V4<double>::load(f + 4 * n, f0, f1, f2);
    ff += f0 * f0 + f1 * f1 + f2 * f2;
  }
  ff = block_sum<1024>(ff, sbuf);
  if (threadIdx.x == 0) slen = sqrt(ff);
  __syncthreads();
  const double lenf = slen;
  const bool trivial = lenf < tol;  // PCGSolver returns u = 0 at once
  double zr = 0.0;
  for (int64_t n = n0 + threadIdx.x; n < n1; n += 1024) {
    double r0, r1, r2, z0, z1, z2;
    if (trivial || !warm) V4<double>::store(u + 4 * n, 0.0, 0.0, 0.0);
    if (trivial) continue;
    V4<double>::load((warm ? r : f) + 4 * n, r0, r1, r2);
    if (!warm) V4<double>::store(r + 4 * n, r0, r1, r2);
    apply_dinv(dinv + 12 * n, r0, r1, r2, z0, z1, z2);
    V4<double>::store(z + 4 * n, z0, z1, z2);
    V4<double>::store(p + 4 * n, 0.0, 0.0, 0.0);
    zr += z0 * r0 + z1 * r1 + z2 * r2;
  }
  zr = block_sum<1024>(zr, sbuf);
  if (threadIdx.x == 0) S[blockIdx.x] = MfProblem{lenf > 1e11 ? 1.0 : lenf, zr, 0.0, 0.0, 0.0, 0, trivial ? 1 : 0};
}

// ---- set-up

// Slots: 32 per batch, at[slot] the colour-sorted position of its element, or
// ~position for padding (an element of the batch once more, without stiffness).

// colour-sorted incidence -> batches
__global__ void mf_batch_conn(int64_t n32, int nn, const int32_t *__restrict__ at, const int32_t *__restrict__ conn,
                              int32_t *__restrict__ out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n32 * nn) return;
  const int64_t ba = t >> 5, b = ba / nn, a = ba - b * nn;
  const int32_t i = at[32 * b + (t & 31)];
  out[t] = conn[(int64_t)(i < 0 ? ~i : i) * nn + a];
}

// the node lists of the gathered internal force (offsets 3 (position nn + a)
// into the colour-sorted element forces) -> entries of the batched forces, in
// fours, padded with the zero entry
__global__ void mf_lists(int64_t nnode, int nn, int32_t zero, const int64_t *__restrict__ gptr,
                         const int64_t *__restrict__ ginc, const int32_t *__restrict__ slot,
                         const int32_t *__restrict__ ptr, int32_t *__restrict__ inc) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnode) return;
  int64_t i = gptr[n];
  const int64_t i1 = gptr[n + 1];
  for (int64_t o = 4 * (int64_t)ptr[n]; o < 4 * (int64_t)ptr[n + 1]; o++, i++) {
    int32_t at = zero;
    if (i < i1) {
      const int64_t off = ginc[i] / 3, pos = off / nn, a = off - pos * nn;
      const int32_t e = slot[pos];
      at = (int32_t)(((int64_t)(e >> 5) * nn + a) * 32 + (e & 31));
    }
    inc[o] = at;
  }
}

// lambda, mu per slot, times `scale` (a power of two)
__global__ void mf_material(int64_t n32, double scale, const int32_t *__restrict__ at, const double *__restrict__ E,
                            const double *__restrict__ nu, double *__restrict__ lam, double *__restrict__ mu,
                            float *__restrict__ lam32, float *__restrict__ mu32) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= n32) return;
  double l = 0.0, m = 0.0;
  const int32_t i = at[e];
  if (i >= 0) {
    const double Ey = E[i], n = nu[i];
    l = scale * (Ey * n / ((1.0 + n) * (1.0 - 2.0 * n)));
    m = scale * (0.5 * Ey / (1.0 + n));
  }
  lam[e] = l;
  mu[e] = m;
  if (lam32) {
    lam32[e] = (float)l;
    mu32[e] = (float)m;
  }
}

// A = sqrt(w / det J) det J J^-1 from J (det > 0: the assembly has checked it)
__device__ __forceinline__ void point_geometry(const double *J, double w, double *A) {
  const double s = sqrt(w / mf::cofactors(J, A));
#pragma unroll
  for (int q = 0; q < 9; q++) A[q] *= s;
}

constexpr int kG20 = 288;  // a warp per Gauss line
__global__ void __launch_bounds__(kG20) mf_geometry20(int nb, const int32_t *__restrict__ conn,
                                                      const double *__restrict__ X, double *__restrict__ g64,
                                                      float *__restrict__ g32) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = w / 3, j = w - 3 * k;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    double L[3][8], H[3][9];
    for (int c = 0; c < 3; c++) {
      double f[20];
#pragma unroll
      for (int a = 0; a < 20; a++) f[a] = X[3 * (int64_t)conn[((size_t)b * 20 + a) * 32 + lane] + c];
      const mf::Plane<double> P = mf::plane_poly(f, mf::gauss20<double>(k), mf::gauss20_sq<double>(k));
      mf::plane_line(P, mf::gauss20<double>(j), mf::gauss20_sq<double>(j), L[c]);
#pragma unroll
      for (int q = 0; q < 8; q++) L[c][q] *= 1.0 / mf::kScale20;
    }
    mf::line_gradients(L, H);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double wt = (i == 1 ? 8.0 : 5.0) * (j == 1 ? 8.0 : 5.0) * (k == 1 ? 8.0 : 5.0) / 729.0;
      double A[9];
      point_geometry(H[i], wt, A);
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const size_t at = (((size_t)b * 9 + w) * 27 + 9 * i + q) * 32 + lane;
        g64[at] = A[q];
        if (g32) g32[at] = (float)A[q];
      }
    }
  }
}

__global__ void __launch_bounds__(kT8) mf_geometry8(int nb, const int32_t *__restrict__ conn,
                                                    const double *__restrict__ X, float *__restrict__ g32) {
  const int lane = threadIdx.x & 31;
  for (int b = blockIdx.x * (kT8 / 32) + (threadIdx.x >> 5); b < nb; b += gridDim.x * (kT8 / 32)) {
    double D[3][3][4];
    for (int c = 0; c < 3; c++) {
      double f[8];
#pragma unroll
      for (int a = 0; a < 8; a++) f[a] = X[3 * (int64_t)conn[((size_t)b * 8 + a) * 32 + lane] + c];
      mf::hex8_grads(f, D[c]);
    }
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int gx = g & 1, gy = (g >> 1) & 1, gz = g >> 2;
      double J[9], A[9];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        J[3 * c] = D[c][0][gy + 2 * gz];
        J[3 * c + 1] = D[c][1][gx + 2 * gz];
        J[3 * c + 2] = D[c][2][gx + 2 * gy];
      }
      point_geometry(J, 1.0, A);
#pragma unroll
      for (int q = 0; q < 9; q++) {
        g32[((size_t)b * 72 + 9 * g + q) * 32 + lane] = (float)A[q];
      }
    }
  }
}

// the diagonal of the 12-per-node inverse, 4 per node
template <typename T>
__global__ void mf_diag(int64_t nnode, const T *__restrict__ dinv, T *__restrict__ dj) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnode) return;
  V4<T>::store(dj + 4 * n, dinv[12 * n], dinv[12 * n + 5], dinv[12 * n + 10]);
}

constexpr size_t kSmem8 = (kT8 / 32) * 72 * 32 * sizeof(float);  // mf_hex8_32
template <typename T> constexpr size_t kSmem20 = (3 * 20 + 3 * (sizeof(T) == 4 ? 81 : 72)) * 32 * sizeof(T) + 20 * 32 * sizeof(int32_t);

template <typename T>
T *either(float *a, double *b) {
  return reinterpret_cast<T *>(sizeof(T) == 4 ? (void *)a : (void *)b);
}

// blocks of the element kernels (= p.K p partials): all resident ones, no more than the batches need
template <typename T>
int mf_grid(const Ctx &c) {
  const MatFree &M = c.mf;
  const int per_sm = sizeof(T) == 4 ? M.per_sm32 : M.per_sm64;
  const int need = M.nn == 20 ? M.nb : (M.nb + kT8 / 32 - 1) / (kT8 / 32);
  return std::max(1, std::min(std::min(per_sm * c.sm_count, need), 8 * 128));
}

template <typename T, bool DIR>
void mf_elements(Ctx &c, const T *p, const T *z, const int32_t *skip, double *part, const double *part_rr,
                 const double *part_zr, int nred) {
  const MatFree &M = c.mf;
  const MfArgs<T> a{M.nb, M.conn, either<T>(M.g32, M.g64), c.d_X, either<T>(M.lam32, M.lam64), either<T>(M.mu32, M.mu64), p, z,
                    either<T>(M.F32, M.F64), c.d_state, skip, part, part_rr, part_zr, nred};
  const int G = mf_grid<T>(c);
  if (M.nn == 20) mf_hex20<T, DIR><<<G, kT20, kSmem20<T>, c.stream>>>(a);
  else if constexpr (sizeof(T) == 4) mf_hex8_32<DIR><<<G, kT8, kSmem8, c.stream>>>(a);
  else mf_hex8_64<DIR><<<G, kT8, 0, c.stream>>>(a);
  c.launches++;
}

}  // namespace

void MatFree::release() {
  for (void *p : {(void *)conn, (void *)at, (void *)ptr, (void *)inc, (void *)g32, (void *)g64, (void *)lam32,
                  (void *)mu32, (void *)lam64, (void *)mu64, (void *)F32, (void *)F64, (void *)dj32, (void *)dj64,
                  (void *)bprob, (void *)ntile, (void *)eptr, (void *)nptr, (void *)bpart, (void *)S})
    if (p) cudaFree(p);
  *this = MatFree{};
}

// One bucket of small-strain hex8 (2x2x2 points) or hex20 (3x3x3) elements,
// no ties, the stiffness as the last assembly left it, and a system large
// enough that an iteration of two kernels beats the persistent kernel, which
// is while that one's matrix leaves shared memory and L2.  Measured, us per
// iteration on the assembled matrix / matrix-free:
//   hex20  19,623 nodes FP32 11.9 / 16.7  FP64 16.3 / 18.8
//          35,116            17.2 / 17.3       43.9 / 21.0
//          54,398            32.4 / 19.9       85.7 / 26.1
//   hex8   29,791            10.9 / 14.8       15.0 / 18.6
//          64,000            17.1 / 17.5       40.9 / 25.9
//         127,500            47.0 / 22.9       70.6 / 44.0
static bool mf_possible(const Ctx &c) {
  if (!c.K_pure || c.mf_off || c.has_ties() || c.buckets.size() != 1 || !c.force_gather) return false;
  const Bucket &B = c.buckets[0];
  if (B.tl || !((B.type == FAST_ELEM_HEX8 && B.ng == 8) || (B.type == FAST_ELEM_HEX20 && B.ng == 27))) return false;
  return (B.ne + 31 * std::max(1, (int)c.nprob)) * B.nn < (int64_t)1 << 30;
}
bool mf_active(const Ctx &c) {
  if (!mf_possible(c)) return false;
  const int64_t least = c.mf_min_nodes >= 0        ? c.mf_min_nodes
                        : c.buckets[0].nn == 20    ? (c.mf_fp32 ? 36000 : 22000)
                                                   : (c.mf_fp32 ? 66000 : 42000);
  return c.nnode >= least;
}
// Independent hex8 problems: all of them an iteration at a time, or a cluster of
// two blocks for each on the assembled matrix (pcg_batch)?  Fitted to solves of
// 1 to 1,000 cantilevers of 45 to 18,081 nodes each: an iteration of pcg_batch
// takes 6.5 us and 0.036 us per node of its problem, 148 clusters run at once
// and the largest problem may be what is waited for; a lockstep iteration takes
// 17 us (four kernels) and 0.15 ns per node of all problems.  Measured, ms
// (pcg_batch / lockstep): 8 problems of 112..637 nodes 5.7 / 3.5, 16 of 112..396
// 3.1 / 3.0, 64 of 112..225 1.9 / 2.5, 128 of 112..637 6.3 / 4.7, 256 of
// 225..1,377 26 / 14, 8 of 1,900..18,081 501 / 23, 256 of 637..18,081 780 / 225.
bool mf_batch_active(const Ctx &c) {
  if (c.nprob <= 0 || !mf_possible(c) || c.buckets[0].nn != 8) return false;
  if (c.mf_min_nodes >= 0) return c.nnode >= c.mf_min_nodes;
  double sum = 0.0, most = 0.0;
  for (int k = 0; k < c.nprob; k++) {
    const double t = 6.5 + 0.036 * (double)(c.h_noff[k + 1] - c.h_noff[k]);
    sum += t;
    most = std::max(most, t);
  }
  return 17.0 + 0.15e-3 * (double)c.nnode < std::max(most, sum / c.sm_count);
}

// The batches: elements in the mesh's own order, 32 at a time; of a context with
// independent problems (fast_gpu_set_problems) problem by problem, the largest
// first, each from a batch of its own.  at[slot]: as in mf_batch_conn;
// slot[colour-sorted position].
static void mf_slots(Ctx &c, std::vector<int32_t> &at, std::vector<int32_t> &slot) {
  MatFree &M = c.mf;
  const Bucket &B = c.buckets[0];
  slot.resize(B.ne);
  auto put = [&](int32_t pos) {
    slot[pos] = (int32_t)at.size();
    at.push_back(pos);
  };
  auto pad = [&] {
    const int32_t last = at.empty() ? 0 : at.back();
    while (at.size() % 32) at.push_back(~last);
  };
  M.h_eptr.clear();
  if (c.nprob <= 0) {
    for (int64_t e = 0; e < B.ne; e++) put(B.inv[e]);
    pad();
    return;
  }
  std::vector<int32_t> rank(c.nprob);
  for (int k = 0; k < c.nprob; k++) rank[c.h_order[k]] = k;
  std::vector<std::vector<int32_t>> of(c.nprob);
  for (int64_t e = 0; e < B.ne; e++) {
    const int64_t n = B.h_conn[(int64_t)B.inv[e] * B.nn];
    const auto up = std::upper_bound(c.h_noff.begin(), c.h_noff.end(), n);
    of[rank[up - c.h_noff.begin() - 1]].push_back(B.inv[e]);
  }
  for (int k = 0; k < c.nprob; k++) {
    M.h_eptr.push_back((int32_t)(at.size() / 32));
    for (int32_t pos : of[k]) put(pos);
    pad();
  }
  M.h_eptr.push_back((int32_t)(at.size() / 32));
}

// the batched copies of mesh, geometry and material, whichever are stale
static cudaError_t prepare(Ctx &c, bool fp32, int precond) {
  MatFree &M = c.mf;
  const Bucket &B = c.buckets[0];
  const int64_t ne = B.ne, nn = B.nn;
  const size_t ng9 = (size_t)9 * B.ng;
  cudaError_t e = cudaSuccess;
  auto alloc = [&](auto **p, size_t n) {
    if (e == cudaSuccess && !*p) e = cudaMalloc((void **)p, sizeof(**p) * n);
  };
  if (!M.built) {
    std::vector<int32_t> at, slot;
    mf_slots(c, at, slot);
    const int64_t n32 = (int64_t)at.size();
    M.nn = (int)nn;
    M.nb = (int)(n32 / 32);
    std::vector<int64_t> gptr(c.nnode + 1);
    std::vector<int32_t> ptr(c.nnode + 1, 0);
    if ((e = cudaMemcpyAsync(gptr.data(), c.d_gptr, sizeof(int64_t) * gptr.size(), cudaMemcpyDeviceToHost, c.stream)) !=
            cudaSuccess ||
        (e = cudaStreamSynchronize(c.stream)) != cudaSuccess)
      return e;
    for (int64_t n = 0; n < c.nnode; n++) ptr[n + 1] = ptr[n] + (int32_t)((gptr[n + 1] - gptr[n] + 3) / 4);
    int32_t *d_slot = nullptr;
    alloc(&M.conn, n32 * nn);
    alloc(&M.at, n32);
    alloc(&M.ptr, c.nnode + 1);
    alloc(&M.inc, 4 * (size_t)ptr[c.nnode]);
    alloc(&M.lam64, n32);
    alloc(&M.mu64, n32);
    if (nn == 20) alloc(&M.g64, n32 * ng9);
    alloc(&M.F64, n32 * nn * 4 + 4);  // one zero entry behind the last
    if (e == cudaSuccess) e = cudaMemsetAsync(M.F64 + 4 * n32 * nn, 0, sizeof(double) * 4, c.stream);
    alloc(&M.dj64, 4 * c.nnode);
    alloc(&d_slot, ne);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(M.at, at.data(), sizeof(int32_t) * n32, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(d_slot, slot.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(M.ptr, ptr.data(), sizeof(int32_t) * ptr.size(), cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess) {
      const int64_t t1 = n32 * nn;
      mf_batch_conn<<<(unsigned)((t1 + 255) / 256), 256, 0, c.stream>>>(n32, (int)nn, M.at, B.d_conn, M.conn);
      mf_lists<<<(unsigned)((c.nnode + 255) / 256), 256, 0, c.stream>>>(c.nnode, (int)nn, (int32_t)t1, c.d_gptr,
                                                                        c.d_ginc, d_slot, M.ptr, M.inc);
      c.launches += 2;
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
    if (d_slot) cudaFree(d_slot);
    if (e != cudaSuccess) return e;
    int a = 0, b = 0;
    auto sized = [&](auto kern, int threads, size_t smem, int *n) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kern, threads, smem);
    };
    if (nn == 20) {
      sized(mf_hex20<double, false>, kT20, kSmem20<double>, &a);
      sized(mf_hex20<float, false>, kT20, kSmem20<float>, &b);
      sized(mf_hex20<double, true>, kT20, kSmem20<double>, &a);
      sized(mf_hex20<float, true>, kT20, kSmem20<float>, &b);
    } else {
      sized(mf_hex8_64<false>, kT8, 0, &a);
      sized(mf_hex8_32<false>, kT8, kSmem8, &b);
      sized(mf_hex8_64<true>, kT8, 0, &a);
      sized(mf_hex8_32<true>, kT8, kSmem8, &b);
    }
    if (e != cudaSuccess) return e;
    M.per_sm64 = std::max(1, a);
    M.per_sm32 = std::max(1, b);
    M.built = true;
  }
  const int64_t n32 = 32 * (int64_t)M.nb;
  if (fp32) {
    if (!M.g32) M.geo_ok = M.mat_ok = false;
    alloc(&M.g32, n32 * ng9);
    alloc(&M.lam32, n32);
    alloc(&M.mu32, n32);
    alloc(&M.dj32, 4 * c.nnode);
    const bool fresh = !M.F32;
    alloc(&M.F32, n32 * nn * 4 + 4);
    if (e == cudaSuccess && fresh) e = cudaMemsetAsync(M.F32 + 4 * n32 * nn, 0, sizeof(float) * 4, c.stream);
    if (e != cudaSuccess) return e;
  }
  if (!M.geo_ok && (nn == 20 || M.g32)) {
    const int G = std::min(2 * M.nb, 8 * c.sm_count);
    if (nn == 20) mf_geometry20<<<G, kG20, 0, c.stream>>>(M.nb, M.conn, c.d_X, M.g64, M.g32);
    else mf_geometry8<<<G, kT8, 0, c.stream>>>(M.nb, M.conn, c.d_X, M.g32);
    c.launches++;
    M.geo_ok = true;
  }
  if (!M.mat_ok) {
    const double scale = nn == 20 ? 1.0 / (mf::kScale20 * mf::kScale20) : 1.0;
    mf_material<<<(unsigned)((n32 + 255) / 256), 256, 0, c.stream>>>(n32, scale, M.at, B.d_E, B.d_nu, M.lam64, M.mu64,
                                                                     M.lam32, M.mu32);
    c.launches++;
    M.mat_ok = true;
  }
  M.jacobi = precond == FAST_PRECOND_JACOBI;
  if (M.jacobi) {
    const unsigned g = (unsigned)((c.nnode + 255) / 256);
    mf_diag<double><<<g, 256, 0, c.stream>>>(c.nnode, c.d_dinv, M.dj64);
    c.launches++;
    if (fp32) {
      mf_diag<float><<<g, 256, 0, c.stream>>>(c.nnode, c.s_dinv, M.dj32);
      c.launches++;
    }
  }
  return cudaGetLastError();
}

cudaError_t mf_prepare(Ctx &c, bool fp32, int precond) {
  try {
    return prepare(c, fp32, precond);
  } catch (const std::bad_alloc &) {
    return cudaErrorMemoryAllocation;
  }
}

void mf_give_up(Ctx &c) {
  (void)cudaGetLastError();
  cudaStreamSynchronize(c.stream);
  c.drop_mf_graphs();
  c.mf.release();
}

template <typename T>
void mf_iterations(Ctx &c, int k, T *u, T *r, T *z, T *p, double *part_pw, double *part_rr, double *part_zr) {
  const MatFree &M = c.mf;
  PcgState *st = c.d_state;
  const T *F = either<T>(M.F32, M.F64);
  const T *dj = M.jacobi ? either<T>(M.dj32, M.dj64) : nullptr;
  const T *dinv = either<T>(c.s_dinv, c.d_dinv);
  const int R = kRedBlocks;
  for (int i = 0; i < k; i++) {
    c.begin_span(sizeof(T) == 4 ? 1 : 0);
    if (i > 0) mf_elements<T, true>(c, p, z, &st->done, part_pw, part_rr, part_zr, R);
    else mf_elements<T, false>(c, p, z, &st->done, part_pw, part_rr, part_zr, R);
    c.end_span();
    const int G = mf_grid<T>(c);
    if (i > 0)
      mf_update<T, true><<<R, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, F, c.d_fix, u, r, z, p, dj, dinv, st,
                                                          part_pw, G, part_rr, part_zr);
    else
      mf_update<T, false><<<R, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, F, c.d_fix, u, r, z, p, dj, dinv, st,
                                                           part_pw, G, part_rr, part_zr);
    c.launches++;
  }
}
template void mf_iterations<float>(Ctx &, int, float *, float *, float *, float *, double *, double *, double *);
template void mf_iterations<double>(Ctx &, int, double *, double *, double *, double *, double *, double *, double *);

cudaError_t mf_residual_of(Ctx &c, const double *f, const double *u, double *r, double *part, int nparts,
                           const int32_t *skip) {
  const MatFree &M = c.mf;
  mf_elements<double, false>(c, u, nullptr, skip, nullptr, nullptr, nullptr, 0);
  mf_residual<<<nparts, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, M.F64, c.d_fix, f, r, part, skip);
  c.launches++;
  return cudaGetLastError();
}

// Per-problem PCG of every problem, as launch_pcg_batch.  The problems lie
// largest first, so the launches shrink from the end as the small ones, which
// need fewer iterations, are done.
static cudaError_t solve_batch(Ctx &c, double tol, int maxit, bool warm, int32_t *it, double *err, int32_t *done) {
  MatFree &M = c.mf;
  cudaError_t e;
  const int np = c.nprob;
  if (!M.S) {
    std::vector<int32_t> bp(M.nb);
    std::vector<int4> nt;
    M.h_ntile.assign(1, 0);
    for (int k = 0; k < np; k++) {
      const int64_t n0 = c.h_noff[c.h_order[k]], n1 = c.h_noff[c.h_order[k] + 1];
      for (int b = M.h_eptr[k]; b < M.h_eptr[k + 1]; b++) bp[b] = k;
      for (int64_t n = n0; n < n1; n += kVecThreads)
        nt.push_back(make_int4((int)n, (int)std::min(n + kVecThreads, n1), k, 0));
      M.h_ntile.push_back((int32_t)nt.size());
    }
    e = cudaSuccess;
    auto up = [&](auto **p, const auto &v) {
      if (e == cudaSuccess && !*p) e = cudaMalloc((void **)p, sizeof(v[0]) * std::max<size_t>(1, v.size()));
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(*p, v.data(), sizeof(v[0]) * v.size(), cudaMemcpyHostToDevice, c.stream);
    };
    up(&M.bprob, bp);
    up(&M.ntile, nt);
    up(&M.eptr, M.h_eptr);
    up(&M.nptr, M.h_ntile);
    // (on the solve's own stream, which the legacy stream does not order, and done before bp and nt go)
    const cudaError_t es = cudaStreamSynchronize(c.stream);
    if (e == cudaSuccess) e = es;
    if (e == cudaSuccess && !M.bpart) e = cudaMalloc((void **)&M.bpart, sizeof(double) * (M.nb + 2 * nt.size() + 1));
    if (e == cudaSuccess) e = cudaMalloc((void **)&M.S, sizeof(MfProblem) * np);
    if (e != cudaSuccess) return e;
  }
  if (warm && (e = mf_residual_of(c, c.d_f, c.d_u, c.d_r, c.d_partials, kRedBlocks, nullptr)) != cudaSuccess) return e;
  mf_batch_init<<<np, 1024, 0, c.stream>>>(c.d_order, c.d_noff, c.d_f, c.d_dinv, c.d_u, c.d_r, c.d_z, c.d_p, tol,
                                           warm ? 1 : 0, M.S);
  c.launches++;
  MfArgs<double> a{M.nb, M.conn, M.g64, c.d_X, M.lam64, M.mu64, c.d_p, c.d_z, M.F64, nullptr, nullptr, nullptr, nullptr,
                   nullptr, 0};
  const MfBatch b{M.bprob, M.ntile, M.eptr, M.nptr, M.S, M.bpart, M.bpart + M.nb, M.bpart + M.nb + M.h_ntile[np]};
  std::vector<MfProblem> S(np);
  int live = np;  // problems [0, live) of the order may still run
  for (int chunk = 0;; chunk = std::min(chunk ? 2 * chunk : 8, kMfBatchChunk)) {
    a.nb = M.h_eptr[live];
    const int G = std::max(1, std::min(M.per_sm64 * c.sm_count, (a.nb + kT8 / 32 - 1) / (kT8 / 32)));
    for (int i = 0; i < chunk; i++) {
      // (each is scheduled while the one before it drains: 257 -> 251 ms for the
      // 256 cantilevers; the same in the captured chunks of a single solve was
      // slower, 18.4 -> 20.0 ms for hex8 61x47x33)
      launch_chained(i > 0, mf_batch_elements, G, kT8, 0, c.stream, a, b);
      launch_chained(true, mf_batch_alpha, live, 128, 0, c.stream, b);
      launch_chained(true, mf_batch_update, M.h_ntile[live], kVecThreads, 0, c.stream, M.ptr, M.inc, M.F64, c.d_fix, c.d_u,
                     c.d_r, c.d_z, c.d_p, M.jacobi ? M.dj64 : nullptr, c.d_dinv, b);
      launch_chained(true, mf_batch_beta, live, 128, 0, c.stream, b, tol, maxit);
      c.launches += 4;
    }
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(S.data(), M.S, sizeof(MfProblem) * np, cudaMemcpyDeviceToHost, c.stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(c.stream)) != cudaSuccess)
      return e;
    while (live > 0 && S[live - 1].done) live--;
    if (live == 0) break;
  }
  for (int k = 0; k < np; k++) {
    it[c.h_order[k]] = S[k].iter;
    err[c.h_order[k]] = S[k].err;
    done[c.h_order[k]] = S[k].done;
  }
  return cudaSuccess;
}

cudaError_t mf_solve_batch(Ctx &c, double tol, int maxit, bool warm, int32_t *it, double *err, int32_t *done) {
  try {
    return solve_batch(c, tol, maxit, warm, it, err, done);
  } catch (const std::bad_alloc &) {
    return cudaErrorMemoryAllocation;
  }
}

}  // namespace fastgpu
