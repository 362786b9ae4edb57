// matfree.cu - K.u for large small-strain hex models without the assembled
// matrix (sm_100a): the operator of the PCG iteration and of its residuals.
//
// An iteration on the assembled matrix streams it: 40 (FP32) or 76 (FP64)
// bytes per 3x3 block, 57 blocks per node of a hex20 mesh, 1.26 / 2.4 GB at
// 131,072 elements, 214 / 402 us at 6 TB/s.  Applied element by element
// (matfree_math.cuh) the same product reads 9 numbers per Gauss point and the
// directions of the element's nodes: 0.19 / 0.37 GB, and about 4,700
// multiply-adds per element.  Measured there: element kernel 66 / 110 us, node
// kernel 27 / 52 us (an iteration 239 -> 98 us in FP32, 447 -> 168 us in FP64).
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
#include <vector>

#include "matfree_math.cuh"
#include "solve_common.cuh"

namespace fastgpu {

namespace {

constexpr int kT20 = 96;   // hex20: a warp per Gauss plane
constexpr int kT8 = 128;   // hex8: 4 batches

template <typename T>
struct MfArgs {
  int nb;                          // batches of 32 elements
  const int32_t *conn;             // [nb][nn][32] nodes (padding elements: node 0, zero geometry)
  const T *geo;                    // hex20 [nb][9 lines][27][32], hex8 [nb][72][32]
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

// ... of the hex8 batches: a lane takes its element whole.  The geometry of a
// warp's batch (9 or 18 KB) is copied to shared memory while the warp gathers.
template <typename T, bool DIR>
__global__ void __launch_bounds__(kT8) mf_hex8(MfArgs<T> A) {
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

// alpha = dot0 / p.Kp (every block), p = z + beta p (DIR), u += alpha p;
// r -= alpha w; z = Dinv r; partials r.r, z.r; the last block stores p.Kp and
// alpha, or the breakdown state (as pcg_update_fused).  dj: the inverse
// diagonal, 4 per node (Jacobi), or null and dinv, 12 per node.
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
    for (int64_t n = blockIdx.x * (int64_t)kVecThreads + threadIdx.x; n < nnode;
         n += (int64_t)gridDim.x * kVecThreads) {
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

// ---- set-up

// colour-sorted incidence -> batches of 32 in the mesh's own element order
__global__ void mf_batch_conn(int64_t ne, int64_t n32, int nn, const int32_t *__restrict__ inv,
                              const int32_t *__restrict__ conn, int32_t *__restrict__ out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n32 * nn) return;
  const int lane = (int)(t & 31);
  const int64_t ba = t >> 5, b = ba / nn, a = ba - b * nn, e = 32 * b + lane;
  out[t] = e < ne ? conn[(int64_t)inv[e] * nn + a] : 0;
}

// the node lists of the gathered internal force (offsets 3 (position nn + a)
// into the colour-sorted element forces) -> entries of the batched forces, in
// fours, padded with the zero entry
__global__ void mf_lists(int64_t nnode, int nn, int32_t zero, const int64_t *__restrict__ gptr,
                         const int64_t *__restrict__ ginc, const int32_t *__restrict__ perm,
                         const int32_t *__restrict__ ptr, int32_t *__restrict__ inc) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnode) return;
  int64_t i = gptr[n];
  const int64_t i1 = gptr[n + 1];
  for (int64_t o = 4 * (int64_t)ptr[n]; o < 4 * (int64_t)ptr[n + 1]; o++, i++) {
    int32_t at = zero;
    if (i < i1) {
      const int64_t off = ginc[i] / 3, pos = off / nn, a = off - pos * nn;
      const int32_t e = perm[pos];
      at = (int32_t)(((int64_t)(e >> 5) * nn + a) * 32 + (e & 31));
    }
    inc[o] = at;
  }
}

// lambda, mu per element in the mesh's own order, times `scale` (a power of two)
__global__ void mf_material(int64_t ne, int64_t n32, double scale, const int32_t *__restrict__ inv,
                            const double *__restrict__ E, const double *__restrict__ nu, double *__restrict__ lam,
                            double *__restrict__ mu, float *__restrict__ lam32, float *__restrict__ mu32) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= n32) return;
  double l = 0.0, m = 0.0;
  if (e < ne) {
    const double Ey = E[inv[e]], n = nu[inv[e]];
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

// A = sqrt(w det J) J^-1 from J (J[3 c + d] = dx_c/dxi_d)
__device__ __forceinline__ void point_geometry(const double *J, double w, double *A) {
  const double c0 = J[4] * J[8] - J[5] * J[7], c1 = J[5] * J[6] - J[3] * J[8], c2 = J[3] * J[7] - J[4] * J[6];
  const double det = J[0] * c0 + J[1] * c1 + J[2] * c2;
  const double s = sqrt(w / det);  // (det > 0: the assembly has checked it)
  A[0] = s * c0;
  A[1] = s * (J[2] * J[7] - J[1] * J[8]);
  A[2] = s * (J[1] * J[5] - J[2] * J[4]);
  A[3] = s * c1;
  A[4] = s * (J[0] * J[8] - J[2] * J[6]);
  A[5] = s * (J[2] * J[3] - J[0] * J[5]);
  A[6] = s * c2;
  A[7] = s * (J[1] * J[6] - J[0] * J[7]);
  A[8] = s * (J[0] * J[4] - J[1] * J[3]);
}

constexpr int kG20 = 288;  // a warp per Gauss line
__global__ void __launch_bounds__(kG20) mf_geometry20(int64_t ne, int nb, const int32_t *__restrict__ conn,
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
    const bool real = 32 * (int64_t)b + lane < ne;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double wt = (i == 1 ? 8.0 : 5.0) * (j == 1 ? 8.0 : 5.0) * (k == 1 ? 8.0 : 5.0) / 729.0;
      double A[9];
      point_geometry(H[i], wt, A);
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const size_t at = (((size_t)b * 9 + w) * 27 + 9 * i + q) * 32 + lane;
        const double v = real ? A[q] : 0.0;
        g64[at] = v;
        if (g32) g32[at] = (float)v;
      }
    }
  }
}

__global__ void __launch_bounds__(kT8) mf_geometry8(int64_t ne, int nb, const int32_t *__restrict__ conn,
                                                    const double *__restrict__ X, double *__restrict__ g64,
                                                    float *__restrict__ g32) {
  const int lane = threadIdx.x & 31;
  for (int b = blockIdx.x * (kT8 / 32) + (threadIdx.x >> 5); b < nb; b += gridDim.x * (kT8 / 32)) {
    double D[3][3][4];
    for (int c = 0; c < 3; c++) {
      double f[8];
#pragma unroll
      for (int a = 0; a < 8; a++) f[a] = X[3 * (int64_t)conn[((size_t)b * 8 + a) * 32 + lane] + c];
      mf::hex8_grads(f, D[c]);
    }
    const bool real = 32 * (int64_t)b + lane < ne;
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
        const size_t at = ((size_t)b * 72 + 9 * g + q) * 32 + lane;
        const double v = real ? A[q] : 0.0;
        g64[at] = v;
        if (g32) g32[at] = (float)v;
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

template <typename T> constexpr size_t kSmem8 = (kT8 / 32) * 72 * 32 * sizeof(T);
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
  const MfArgs<T> a{M.nb, M.conn, either<T>(M.g32, M.g64), either<T>(M.lam32, M.lam64), either<T>(M.mu32, M.mu64), p, z,
                    either<T>(M.F32, M.F64), c.d_state, skip, part, part_rr, part_zr, nred};
  const int G = mf_grid<T>(c);
  if (M.nn == 20) mf_hex20<T, DIR><<<G, kT20, kSmem20<T>, c.stream>>>(a);
  else mf_hex8<T, DIR><<<G, kT8, kSmem8<T>, c.stream>>>(a);
  c.launches++;
}

}  // namespace

void MatFree::release() {
  for (void *p : {(void *)conn, (void *)inv, (void *)ptr, (void *)inc, (void *)g32, (void *)g64, (void *)lam32,
                  (void *)mu32, (void *)lam64, (void *)mu64, (void *)F32, (void *)F64, (void *)dj32, (void *)dj64})
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
//   hex8   29,791            11.0 / 15.4       15.1 / 19.7
//          64,000            17.3 / 18.4       40.6 / 26.7
//         127,500            47.4 / 22.1       71.2 / 48.9
bool mf_active(const Ctx &c) {
  if (!c.K_pure || c.mf_off || c.has_ties() || c.buckets.size() != 1 || !c.force_gather) return false;
  const Bucket &B = c.buckets[0];
  if (B.tl || !((B.type == FAST_ELEM_HEX8 && B.ng == 8) || (B.type == FAST_ELEM_HEX20 && B.ng == 27))) return false;
  const int64_t least = c.mf_min_nodes >= 0 ? c.mf_min_nodes
                        : B.nn == 20        ? (c.mf_fp32 ? 36000 : 22000)
                                            : (c.mf_fp32 ? 66000 : 42000);
  return c.nnode >= least && B.ne * B.nn < (int64_t)1 << 30;
}

// the batched copies of mesh, geometry and material, whichever are stale
cudaError_t mf_prepare(Ctx &c, bool fp32, int precond) {
  MatFree &M = c.mf;
  const Bucket &B = c.buckets[0];
  const int64_t ne = B.ne, nn = B.nn, n32 = (ne + 31) / 32 * 32;
  const size_t ng9 = (size_t)9 * B.ng;
  cudaError_t e = cudaSuccess;
  auto alloc = [&](auto **p, size_t n) {
    if (e == cudaSuccess && !*p) e = cudaMalloc((void **)p, sizeof(**p) * n);
  };
  if (!M.built) {
    M.nn = (int)nn;
    M.nb = (int)(n32 / 32);
    std::vector<int64_t> gptr(c.nnode + 1);
    std::vector<int32_t> ptr(c.nnode + 1, 0);
    if ((e = cudaMemcpyAsync(gptr.data(), c.d_gptr, sizeof(int64_t) * gptr.size(), cudaMemcpyDeviceToHost, c.stream)) !=
            cudaSuccess ||
        (e = cudaStreamSynchronize(c.stream)) != cudaSuccess)
      return e;
    for (int64_t n = 0; n < c.nnode; n++) ptr[n + 1] = ptr[n] + (int32_t)((gptr[n + 1] - gptr[n] + 3) / 4);
    int32_t *perm = nullptr;
    alloc(&M.conn, n32 * nn);
    alloc(&M.inv, ne);
    alloc(&M.ptr, c.nnode + 1);
    alloc(&M.inc, 4 * (size_t)ptr[c.nnode]);
    alloc(&M.lam64, n32);
    alloc(&M.mu64, n32);
    alloc(&M.g64, n32 * ng9);
    alloc(&M.F64, n32 * nn * 4 + 4);  // one zero entry behind the last
    if (e == cudaSuccess) e = cudaMemsetAsync(M.F64 + 4 * n32 * nn, 0, sizeof(double) * 4, c.stream);
    alloc(&M.dj64, 4 * c.nnode);
    alloc(&perm, ne);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(M.inv, B.inv.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(perm, B.perm.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(M.ptr, ptr.data(), sizeof(int32_t) * ptr.size(), cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess) {
      const int64_t t1 = n32 * nn;
      mf_batch_conn<<<(unsigned)((t1 + 255) / 256), 256, 0, c.stream>>>(ne, n32, (int)nn, M.inv, B.d_conn, M.conn);
      mf_lists<<<(unsigned)((c.nnode + 255) / 256), 256, 0, c.stream>>>(c.nnode, (int)nn, (int32_t)t1, c.d_gptr,
                                                                        c.d_ginc, perm, M.ptr, M.inc);
      c.launches += 2;
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
    if (perm) cudaFree(perm);
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
      sized(mf_hex8<double, false>, kT8, kSmem8<double>, &a);
      sized(mf_hex8<float, false>, kT8, kSmem8<float>, &b);
      sized(mf_hex8<double, true>, kT8, kSmem8<double>, &a);
      sized(mf_hex8<float, true>, kT8, kSmem8<float>, &b);
    }
    if (e != cudaSuccess) return e;
    M.per_sm64 = std::max(1, a);
    M.per_sm32 = std::max(1, b);
    M.built = true;
  }
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
  if (!M.geo_ok) {
    const int G = std::min(2 * M.nb, 8 * c.sm_count);
    if (nn == 20) mf_geometry20<<<G, kG20, 0, c.stream>>>(ne, M.nb, M.conn, c.d_X, M.g64, M.g32);
    else mf_geometry8<<<G, kT8, 0, c.stream>>>(ne, M.nb, M.conn, c.d_X, M.g64, M.g32);
    c.launches++;
    M.geo_ok = true;
  }
  if (!M.mat_ok) {
    const double scale = nn == 20 ? 1.0 / (mf::kScale20 * mf::kScale20) : 1.0;
    mf_material<<<(unsigned)((n32 + 255) / 256), 256, 0, c.stream>>>(ne, n32, scale, M.inv, B.d_E, B.d_nu, M.lam64,
                                                                     M.mu64, M.lam32, M.mu32);
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

}  // namespace fastgpu
