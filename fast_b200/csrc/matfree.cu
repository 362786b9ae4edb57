// matfree.cu - K.u for large small-strain hex models without the assembled
// matrix (sm_100a): the operator of the PCG iteration and of its residuals.
//
// An iteration on the assembled matrix streams it: 40 (FP32) or 76 (FP64)
// bytes per 3x3 block, 57 blocks per node of a hex20 mesh, 1.26 / 2.4 GB at
// 131,072 elements, 214 / 402 us at 6 TB/s.  Applied element by element
// (matfree_math.cuh) the same product reads 9 numbers per Gauss point and the
// directions of the element's nodes: 0.19 / 0.37 GB, and about 3,100
// multiply-adds per element, which the FP32 (and FP64) pipes do in less time
// than HBM takes for the geometry.
//
// One iteration is two kernels:
//  1. elements: convergence test and beta from the last update's partial sums
//     (every block forms the same sums), the direction z + beta p built for
//     every gathered node, element forces K_e p_e to memory, partial p.K p
//     (the sum over elements of p_e . K_e p_e);
//  2. nodes: w = the sum of the node's element forces in a fixed order (no
//     atomics: the same bits every run), p, u, r, z and the partial sums.
//
// hex20: a block of 9 warps takes 32 elements, a lane per element.  Each warp
// collapses one component onto one Gauss plane, then takes one Gauss line of
// three points, then carries one component of one plane back; the parts meet
// in shared memory (35 KB in FP32, three blocks per SM).  hex8: a thread takes
// an element, all in registers.  Elements are batched by 32 in the mesh's own
// order (neighbours share nodes in L1 and L2); every per-element array has the
// 32 elements of a batch innermost, so each load is one full line per warp.
#include <algorithm>
#include <cmath>

#include "matfree_math.cuh"
#include "solve_common.cuh"

namespace fastgpu {

namespace {

constexpr int kT20 = 288;  // hex20: 9 warps
constexpr int kT8 = 128;   // hex8: 4 batches

template <typename T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

template <typename T>
struct MfArgs {
  int nb;                          // batches of 32 elements
  const int32_t *conn;             // [nb][nn][32] nodes (padding elements: node 0, zero geometry)
  const T *geo;                    // hex20 [nb][9 lines][3][9][32], hex8 [nb][8][9][32]
  const typename Pair<T>::type *lm;  // [nb][32] lambda, mu
  const T *p, *z;                  // directions
  T *F;                            // [nb][nn][32][4] element forces
  PcgState *st;
  const int32_t *skip;
  double *part;                    // p.K p per block (or null)
  const double *part_rr, *part_zr; // DIR: sums of the last update
  int nred;
};

// DIR: the scalars of pcg_direction_fused, formed alike in every block; returns done
template <int NT>
__device__ __forceinline__ int next_direction(const PcgState *st, const double *part_rr, const double *part_zr, int n,
                                              double &rr, double &zr, double &err, double &beta) {
  __shared__ double sbuf[32];
  __shared__ double sh[3];
  __shared__ int done_sh;
  const double a = sum_partials<NT>(part_rr, n, sbuf);
  const double b = sum_partials<NT>(part_zr, n, sbuf);
  if (threadIdx.x == 0) {
    const double e = sqrt(a) / st->lenf;
    int done = 0;
    if (e < st->tol) done = 1;
    else if (!isfinite(e)) done = 3;
    else if (st->iter + 1 >= st->maxit) done = 2;
    done_sh = done;
    sh[0] = e;
    sh[1] = b / st->dot0;
  }
  __syncthreads();
  rr = a;
  zr = b;
  err = sh[0];
  beta = sh[1];
  return done_sh;
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

// element forces of the hex20 batches; DIR: x = z + beta p, otherwise x = p
template <typename T, bool DIR>
__global__ void __launch_bounds__(kT20, sizeof(T) == 4 ? 3 : 2) mf_hex20(MfArgs<T> A) {
  extern __shared__ __align__(16) unsigned char msm[];
  __shared__ double sred[32];
  T *sU = reinterpret_cast<T *>(msm);  // [3][20][32]
  T *sL = sU + 3 * 20 * 32;            // [9 lines][3][8][32]; later [3 planes][3][20][32]
  if (A.skip && *A.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, c = w / 3, k = w - 3 * c;
  double rr = 0, zr = 0, err = 0, bt = 0;
  int done = 0;
  if (DIR) done = next_direction<kT20>(A.st, A.part_rr, A.part_zr, A.nred, rr, zr, err, bt);
  const T beta = (T)bt;
  double pacc = 0.0;
  for (int b = blockIdx.x; b < A.nb && !done; b += gridDim.x) {
    const T *__restrict__ gp = A.geo + ((size_t)b * 9 + w) * (27 * 32) + lane;
    T geo[27];
    if (sizeof(T) == 4) {  // in flight while the block gathers (evict-first: read once per product)
#pragma unroll
      for (int q = 0; q < 27; q++) geo[q] = __ldcs(gp + 32 * q);
    }
    for (int a = w; a < 20; a += 9) {
      const int64_t n = A.conn[((size_t)b * 20 + a) * 32 + lane];
      T x0, x1, x2;
      V4<T>::load(A.p + 4 * n, x0, x1, x2);
      if (DIR) {
        T z0, z1, z2;
        V4<T>::load(A.z + 4 * n, z0, z1, z2);
        x0 = z0 + beta * x0; x1 = z1 + beta * x1; x2 = z2 + beta * x2;
      }
      sU[a * 32 + lane] = x0;
      sU[(20 + a) * 32 + lane] = x1;
      sU[(40 + a) * 32 + lane] = x2;
    }
    __syncthreads();
    {  // component c onto plane k
      T f[20], L[3][8];
#pragma unroll
      for (int a = 0; a < 20; a++) f[a] = sU[(20 * c + a) * 32 + lane];
      mf::plane_lines(f, k, L);
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int q = 0; q < 8; q++) sL[(((3 * k + j) * 3 + c) * 8 + q) * 32 + lane] = L[j][q];
    }
    __syncthreads();
    {  // line w
      T L[3][8];
#pragma unroll
      for (int i = 0; i < 24; i++) L[i / 8][i % 8] = sL[(24 * w + i) * 32 + lane];
      const auto lm = A.lm[(size_t)b * 32 + lane];
      if (sizeof(T) == 4)
        mf::line_points(L, [&](int i, int q) { return geo[9 * i + q]; }, (T)lm.x, (T)lm.y);
      else
        mf::line_points(L, [&](int i, int q) { return __ldcs(gp + 32 * (9 * i + q)); }, (T)lm.x, (T)lm.y);
#pragma unroll
      for (int i = 0; i < 24; i++) sL[(24 * w + i) * 32 + lane] = L[i / 8][i % 8];
    }
    __syncthreads();
    {  // component c of plane k back to the nodes
      T L[3][8], f[20];
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int q = 0; q < 8; q++) L[j][q] = sL[(((3 * k + j) * 3 + c) * 8 + q) * 32 + lane];
      mf::plane_lines_t(L, k, f);
      __syncthreads();
#pragma unroll
      for (int a = 0; a < 20; a++) sL[((3 * k + c) * 20 + a) * 32 + lane] = f[a];
    }
    __syncthreads();
    for (int a = w; a < 20; a += 9) {
      T f[3];
#pragma unroll
      for (int i = 0; i < 3; i++)
        f[i] = sL[(i * 20 + a) * 32 + lane] + sL[((3 + i) * 20 + a) * 32 + lane] + sL[((6 + i) * 20 + a) * 32 + lane];
      V4<T>::store(A.F + 4 * (((size_t)b * 20 + a) * 32 + lane), f[0], f[1], f[2]);
      pacc += (double)f[0] * sU[a * 32 + lane] + (double)f[1] * sU[(20 + a) * 32 + lane] +
              (double)f[2] * sU[(40 + a) * 32 + lane];
    }
    // (the next batch's gather writes the sU entries this thread read, its
    // plane stage writes sL only after a barrier)
  }
  if (A.part && !done) {
    const double t = block_sum<kT20>(pacc, sred);
    if (tid == 0) A.part[blockIdx.x] = t;
  }
  if (DIR) commit_direction(A.st, done, rr, zr, err, bt);
}

// ... of the hex8 batches: a thread per element
template <typename T, bool DIR>
__global__ void __launch_bounds__(kT8) mf_hex8(MfArgs<T> A) {
  __shared__ double sred[32];
  if (A.skip && *A.skip) return;
  const int tid = threadIdx.x, lane = tid & 31;
  double rr = 0, zr = 0, err = 0, bt = 0;
  int done = 0;
  if (DIR) done = next_direction<kT8>(A.st, A.part_rr, A.part_zr, A.nred, rr, zr, err, bt);
  const T beta = (T)bt;
  double pacc = 0.0;
  for (int b = blockIdx.x * (kT8 / 32) + (tid >> 5); b < A.nb && !done; b += gridDim.x * (kT8 / 32)) {
    T x[3][8], D[3][3][4], R[3][3][4];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const int64_t n = A.conn[((size_t)b * 8 + a) * 32 + lane];
      V4<T>::load(A.p + 4 * n, x[0][a], x[1][a], x[2][a]);
      if (DIR) {
        T z0, z1, z2;
        V4<T>::load(A.z + 4 * n, z0, z1, z2);
        x[0][a] = z0 + beta * x[0][a]; x[1][a] = z1 + beta * x[1][a]; x[2][a] = z2 + beta * x[2][a];
      }
    }
    const auto lm = A.lm[(size_t)b * 32 + lane];
    const T *__restrict__ gp = A.geo + (size_t)b * (72 * 32) + lane;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      mf::hex8_grads(x[c], D[c]);
#pragma unroll
      for (int i = 0; i < 12; i++) R[c][i / 4][i % 4] = T(0);
    }
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int gx = g & 1, gy = (g >> 1) & 1, gz = g >> 2;
      const int id[3] = {gy + 2 * gz, gx + 2 * gz, gx + 2 * gy};
      T H[9], P[9], Ag[9];
#pragma unroll
      for (int q = 0; q < 9; q++) Ag[q] = __ldcs(gp + 32 * (9 * g + q));
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int d = 0; d < 3; d++) H[3 * c + d] = D[c][d][id[d]];
      mf::point_stress(H, Ag, (T)lm.x, (T)lm.y, P);
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int d = 0; d < 3; d++) R[c][d][id[d]] += P[3 * c + d];
    }
    T f[3][8];
#pragma unroll
    for (int c = 0; c < 3; c++) mf::hex8_grads_t(R[c], f[c]);
#pragma unroll
    for (int a = 0; a < 8; a++) {
      V4<T>::store(A.F + 4 * (((size_t)b * 8 + a) * 32 + lane), f[0][a], f[1][a], f[2][a]);
      pacc += (double)f[0][a] * x[0][a] + (double)f[1][a] * x[1][a] + (double)f[2][a] * x[2][a];
    }
  }
  if (A.part && !done) {
    const double t = block_sum<kT8>(pacc, sred);
    if (tid == 0) A.part[blockIdx.x] = t;
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
  for (int32_t i = ptr[n]; i < i1; i++) {
    T a, b, c;
    V4<T>::load(F + 4 * (int64_t)inc[i], a, b, c);
    w0 += a; w1 += b; w2 += c;
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
  __shared__ double alpha_sh;
  __shared__ int bad_sh;
  const double pw = sum_partials(part_pw, npw, sbuf);
  if (threadIdx.x == 0) {
    const double al = st->dot0 / pw;
    bad_sh = (!(al > 0.0) || !isfinite(pw) || !isfinite(al)) ? 1 : 0;
    alpha_sh = al;
  }
  __syncthreads();
  const int bad = bad_sh;
  const double al = alpha_sh;
  if (!bad) {
    double rr = 0.0, zr = 0.0;
    const T alpha = (T)al, beta = (T)st->beta;
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
    st->pw = pw;
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
// into the colour-sorted element forces) -> entries of the batched forces
__global__ void mf_lists(int64_t nnode, int64_t nent, int nn, const int64_t *__restrict__ gptr,
                         const int64_t *__restrict__ ginc, const int32_t *__restrict__ perm,
                         int32_t *__restrict__ ptr, int32_t *__restrict__ inc) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t <= nnode) ptr[t] = (int32_t)gptr[t];
  if (t >= nent) return;
  const int64_t off = ginc[t] / 3, pos = off / nn, a = off - pos * nn;
  const int32_t e = perm[pos];
  inc[t] = (int32_t)(((int64_t)(e >> 5) * nn + a) * 32 + (e & 31));
}

// lambda, mu per element in the mesh's own order
__global__ void mf_material(int64_t ne, int64_t n32, const int32_t *__restrict__ inv, const double *__restrict__ E,
                            const double *__restrict__ nu, double2 *__restrict__ lm, float2 *__restrict__ lm32) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= n32) return;
  double2 v = make_double2(0.0, 0.0);
  if (e < ne) {
    const double Ey = E[inv[e]], n = nu[inv[e]];
    v = make_double2(Ey * n / ((1.0 + n) * (1.0 - 2.0 * n)), 0.5 * Ey / (1.0 + n));
  }
  lm[e] = v;
  if (lm32) lm32[e] = make_float2((float)v.x, (float)v.y);
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

__global__ void __launch_bounds__(kT20) mf_geometry20(int64_t ne, int nb, const int32_t *__restrict__ conn,
                                                      const double *__restrict__ X, double *__restrict__ g64,
                                                      float *__restrict__ g32) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = w / 3, j = w - 3 * k;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    double J[3][9], A[9];
    for (int c = 0; c < 3; c++) {
      double f[20], L[3][8];
#pragma unroll
      for (int a = 0; a < 20; a++) f[a] = X[3 * (int64_t)conn[((size_t)b * 20 + a) * 32 + lane] + c];
      mf::plane_lines(f, k, L);
      double l[8];
#pragma unroll
      for (int q = 0; q < 8; q++) l[q] = j == 0 ? L[0][q] : (j == 1 ? L[1][q] : L[2][q]);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const double x = (i - 1) * mf::kA20, xx = x * x;
        J[i][3 * c] = l[0] + x * l[1];
        J[i][3 * c + 1] = l[2] + x * l[3] + xx * l[4];
        J[i][3 * c + 2] = l[5] + x * l[6] + xx * l[7];
      }
    }
    const bool real = 32 * (int64_t)b + lane < ne;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double wt = (i == 1 ? 8.0 : 5.0) * (j == 1 ? 8.0 : 5.0) * (k == 1 ? 8.0 : 5.0) / 729.0;
      point_geometry(J[i], wt, A);
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

template <typename T> constexpr size_t smem20() { return (3 * 20 + 9 * 24) * 32 * sizeof(T); }

// blocks of the element kernels (= p.K p partials): all resident ones, no more than the batches need
template <typename T>
int mf_grid(const Ctx &c) {
  const MatFree &M = c.mf;
  const int per_sm = sizeof(T) == 4 ? M.per_sm32 : M.per_sm64;
  const int need = M.nn == 20 ? M.nb : (M.nb + kT8 / 32 - 1) / (kT8 / 32);
  return std::max(1, std::min(std::min(per_sm * c.sm_count, need), 2048));
}

template <typename T, bool DIR>
void mf_elements(Ctx &c, const T *p, const T *z, const int32_t *skip, double *part, const double *part_rr,
                 const double *part_zr, int nred) {
  const MatFree &M = c.mf;
  MfArgs<T> a{};
  a.nb = M.nb;
  a.conn = M.conn;
  a.geo = reinterpret_cast<const T *>(sizeof(T) == 4 ? (const void *)M.g32 : (const void *)M.g64);
  a.lm = reinterpret_cast<const typename Pair<T>::type *>(sizeof(T) == 4 ? (const void *)M.lm32 : (const void *)M.lm64);
  a.p = p;
  a.z = z;
  a.F = reinterpret_cast<T *>(M.F);
  a.st = c.d_state;
  a.skip = skip;
  a.part = part;
  a.part_rr = part_rr;
  a.part_zr = part_zr;
  a.nred = nred;
  const int G = mf_grid<T>(c);
  if (M.nn == 20) mf_hex20<T, DIR><<<G, kT20, smem20<T>(), c.stream>>>(a);
  else mf_hex8<T, DIR><<<G, kT8, 0, c.stream>>>(a);
  c.launches++;
}

}  // namespace

void MatFree::release() {
  for (void *p : {(void *)conn, (void *)inv, (void *)ptr, (void *)inc, (void *)g32, (void *)g64, (void *)lm32,
                  (void *)lm64, F, (void *)dj32, (void *)dj64})
    if (p) cudaFree(p);
  *this = MatFree{};
}

// One bucket of small-strain hex8 (2x2x2 points) or hex20 (3x3x3) elements,
// no ties, the stiffness as the last assembly left it, and a system large
// enough that an iteration of two kernels beats the persistent kernel
// (c.mf_min_nodes: measured where it is set).
bool mf_active(const Ctx &c) {
  if (!c.K_pure || c.mf_off || c.has_ties() || c.buckets.size() != 1 || !c.force_gather) return false;
  const Bucket &B = c.buckets[0];
  if (B.tl || !((B.type == FAST_ELEM_HEX8 && B.ng == 8) || (B.type == FAST_ELEM_HEX20 && B.ng == 27))) return false;
  const int64_t least = c.mf_min_nodes >= 0 ? c.mf_min_nodes : (B.nn == 20 ? kMfNodesHex20 : kMfNodesHex8);
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
    int32_t *perm = nullptr;
    alloc(&M.conn, n32 * nn);
    alloc(&M.inv, ne);
    alloc(&M.ptr, c.nnode + 1);
    alloc(&M.inc, ne * nn);
    alloc(&M.lm64, n32);
    alloc(&M.g64, n32 * ng9);
    alloc((double **)&M.F, n32 * nn * 4);
    alloc(&M.dj64, 4 * c.nnode);
    alloc(&perm, ne);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(M.inv, B.inv.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(perm, B.perm.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice, c.stream);
    if (e == cudaSuccess) {
      const int64_t t1 = n32 * nn, t2 = std::max<int64_t>(ne * nn, c.nnode + 1);
      mf_batch_conn<<<(unsigned)((t1 + 255) / 256), 256, 0, c.stream>>>(ne, n32, (int)nn, M.inv, B.d_conn, M.conn);
      mf_lists<<<(unsigned)((t2 + 255) / 256), 256, 0, c.stream>>>(c.nnode, ne * nn, (int)nn, c.d_gptr, c.d_ginc, perm,
                                                                   M.ptr, M.inc);
      c.launches += 2;
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
    if (perm) cudaFree(perm);
    if (e != cudaSuccess) return e;
    int a = 0, b = 0;
    if (nn == 20) {
      for (auto k : {mf_hex20<double, true>, mf_hex20<double, false>})
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem20<double>());
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, mf_hex20<double, true>, kT20, smem20<double>());
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, mf_hex20<float, true>, kT20, smem20<float>());
    } else {
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, mf_hex8<double, true>, kT8, 0);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, mf_hex8<float, true>, kT8, 0);
    }
    if (e != cudaSuccess) return e;
    M.per_sm64 = std::max(1, a);
    M.per_sm32 = std::max(1, b);
    M.built = true;
  }
  if (fp32) {
    if (!M.g32) M.geo_ok = M.mat_ok = false;
    alloc(&M.g32, n32 * ng9);
    alloc(&M.lm32, n32);
    alloc(&M.dj32, 4 * c.nnode);
    if (e != cudaSuccess) return e;
  }
  if (!M.geo_ok) {
    if (nn == 20) mf_geometry20<<<std::min(M.nb, 8 * c.sm_count), kT20, 0, c.stream>>>(ne, M.nb, M.conn, c.d_X, M.g64, M.g32);
    else mf_geometry8<<<std::min((M.nb + 3) / 4, 8 * c.sm_count), kT8, 0, c.stream>>>(ne, M.nb, M.conn, c.d_X, M.g64, M.g32);
    c.launches++;
    M.geo_ok = true;
  }
  if (!M.mat_ok) {
    mf_material<<<(unsigned)((n32 + 255) / 256), 256, 0, c.stream>>>(ne, n32, M.inv, B.d_E, B.d_nu, M.lm64, M.lm32);
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
void mf_iteration(Ctx &c, bool dir, T *u, T *r, T *z, T *p, double *part_pw, double *part_rr, double *part_zr) {
  const MatFree &M = c.mf;
  PcgState *st = c.d_state;
  c.begin_span(sizeof(T) == 4 ? 1 : 0);
  if (dir) mf_elements<T, true>(c, p, z, &st->done, part_pw, part_rr, part_zr, kRedBlocks);
  else mf_elements<T, false>(c, p, z, &st->done, part_pw, part_rr, part_zr, kRedBlocks);
  c.end_span();
  const T *F = reinterpret_cast<const T *>(M.F);
  const T *dj = M.jacobi ? reinterpret_cast<const T *>(sizeof(T) == 4 ? (const void *)M.dj32 : (const void *)M.dj64)
                         : nullptr;
  const T *dinv = reinterpret_cast<const T *>(sizeof(T) == 4 ? (const void *)c.s_dinv : (const void *)c.d_dinv);
  const int G = mf_grid<T>(c);
  if (dir)
    mf_update<T, true><<<kRedBlocks, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, F, c.d_fix, u, r, z, p, dj, dinv,
                                                                 st, part_pw, G, part_rr, part_zr);
  else
    mf_update<T, false><<<kRedBlocks, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, F, c.d_fix, u, r, z, p, dj,
                                                                  dinv, st, part_pw, G, part_rr, part_zr);
  c.launches++;
}
template void mf_iteration<float>(Ctx &, bool, float *, float *, float *, float *, double *, double *, double *);
template void mf_iteration<double>(Ctx &, bool, double *, double *, double *, double *, double *, double *, double *);

cudaError_t mf_residual_of(Ctx &c, const double *f, const double *u, double *r, double *part, int nparts,
                           const int32_t *skip) {
  const MatFree &M = c.mf;
  mf_elements<double, false>(c, u, nullptr, skip, nullptr, nullptr, nullptr, 0);
  mf_residual<<<nparts, kVecThreads, 0, c.stream>>>(c.nnode, M.ptr, M.inc, reinterpret_cast<const double *>(M.F),
                                                    c.d_fix, f, r, part, skip);
  c.launches++;
  return cudaGetLastError();
}

}  // namespace fastgpu
