// matfree_math.cuh - the element operator of the matrix-free solve, in pieces.
//
// K_e u_e for a small-strain isotropic hex element is evaluated as
// interpolate -> gradient at the Gauss points -> stress -> transpose, never
// forming K_e.  The reference gradients of a serendipity hex20 field at the
// 3x3x3 points come from its polynomial, one direction at a time: the nodal
// values collapse to a plane z = z_k (an 8-node serendipity polynomial of the
// field and one of its z derivative), a plane to a line y = y_j (8
// coefficients), a line to its three points.  That takes about 1/9 of the
// multiply-adds of the dense 27 x 20 x 3 derivative table; hex8 likewise.
// Every step has its transpose beside it.
//
// Geometry enters through A_g = sqrt(w_g det J_g) J_g^-1 (9 numbers per point):
//   G = H A (H_cd = du_c/dxi_d), S = lambda tr(G) I + mu (G + G^T), P = S A^T,
// and P goes back through the transposes.  Node numbering: FAST's local order
// (hex8 shp/shpsolid.cpp:173-184, hex20 :301-325).
#pragma once

#ifdef __CUDACC__
#define FG_HD __host__ __device__ __forceinline__
#else
#define FG_HD inline
#endif

namespace fastgpu {
namespace mf {

// hex20: vertical edge i (corner (-,-), (+,-), (+,+), (-,+)): nodes at z = 1, -1, 0;
// mid i ((0,-), (+,0), (0,+), (-,0)): nodes at z = 1, -1; it lies between corners i and i + 1
FG_HD int corner_top(int i) { return 2 * i; }
FG_HD int corner_bot(int i) { return 12 + 2 * i; }
FG_HD int corner_mid(int i) { return 8 + i; }
FG_HD int mid_top(int i) { return 1 + 2 * i; }
FG_HD int mid_bot(int i) { return 13 + 2 * i; }

constexpr double kA20 = 0.77459666924148337704;  // sqrt(0.6): the 3-point Gauss abscissa
constexpr double kA8 = 0.57735026918962576451;   // sqrt(1/3)

// coefficients of the 8-node serendipity polynomial from the values at the
// corners c and mids m; k: x, y, xx, yy, xy, xxy, xyy, 1
template <typename T>
FG_HD void face_poly(const T *c, const T *m, T *k) {
  const T h = T(0.5);
  const T q1 = h * (c[0] + c[1]) - m[0], q2 = h * (c[1] + c[2]) - m[1], q3 = h * (c[2] + c[3]) - m[2],
          q4 = h * (c[3] + c[0]) - m[3];
  const T s1 = h * (c[1] - c[0]), s3 = h * (c[2] - c[3]), t4 = h * (c[3] - c[0]), t2 = h * (c[2] - c[1]);
  k[2] = h * (q1 + q3);
  k[5] = h * (q3 - q1);
  k[3] = h * (q2 + q4);
  k[6] = h * (q2 - q4);
  k[4] = h * (s3 - s1);
  k[0] = h * (s1 + s3) - k[6];
  k[1] = h * (t4 + t2) - k[5];
  k[7] = h * (m[0] + m[2]) - k[3];
}

// transpose: k (overwritten) -> c, m; with_one: k[7] takes part
template <typename T>
FG_HD void face_poly_t(T *k, bool with_one, T *c, T *m) {
  const T h = T(0.5);
  T one = T(0);
  if (with_one) {
    one = h * k[7];
    k[3] -= k[7];
  }
  k[6] -= k[0];
  k[5] -= k[1];
  const T s1 = h * (k[0] - k[4]), s3 = h * (k[0] + k[4]), t = h * k[1];
  const T q1 = h * (k[2] - k[5]), q3 = h * (k[2] + k[5]), q4 = h * (k[3] - k[6]), q2 = h * (k[3] + k[6]);
  c[0] = h * (q1 + q4 - s1 - t);
  c[1] = h * (q1 + q2 + s1 - t);
  c[2] = h * (q3 + q2 + s3 + t);
  c[3] = h * (q3 + q4 - s3 + t);
  m[0] = one - q1;
  m[1] = -q2;
  m[2] = one - q3;
  m[3] = -q4;
}

// one component of a hex20 field on the plane z = (k - 1) sqrt(0.6): the 8
// line coefficients of each of its lines y = (j - 1) sqrt(0.6),
//   d/dx = L0 + L1 x, d/dy = L2 + L3 x + L4 x^2, d/dz = L5 + L6 x + L7 x^2
template <typename T>
FG_HD void plane_lines(const T *f, int k, T (*L)[8]) {
  const T a = T(kA20), h = T(0.5), z = k == 0 ? -a : (k == 1 ? T(0) : a), zz = k == 1 ? T(0) : T(0.6);
  T d[4], c[4], m[4], cz[4], mz[4];
  for (int i = 0; i < 4; i++) {
    const T fp = f[corner_top(i)], fm = f[corner_bot(i)], f0 = f[corner_mid(i)];
    const T o = h * (fp - fm);
    d[i] = h * (fp + fm) - f0;
    c[i] = f0 + z * o + zz * d[i];
    cz[i] = o + T(2) * z * d[i];
  }
  for (int i = 0; i < 4; i++) {
    const T fp = f[mid_top(i)], fm = f[mid_bot(i)];
    const T o = h * (fp - fm), e = h * (fp + fm), g = h * (d[i] + d[(i + 1) & 3]);
    m[i] = e + z * o - (T(1) - zz) * g;
    mz[i] = o + T(2) * z * g;
  }
  T p[8], q[8];
  face_poly(c, m, p);
  face_poly(cz, mz, q);
  for (int j = 0; j < 3; j++) {
    const T y = j == 0 ? -a : (j == 1 ? T(0) : a), yy = j == 1 ? T(0) : T(0.6);
    L[j][0] = p[0] + y * p[4] + yy * p[6];
    L[j][1] = T(2) * (p[2] + y * p[5]);
    L[j][2] = p[1] + T(2) * y * p[3];
    L[j][3] = p[4] + T(2) * y * p[6];
    L[j][4] = p[5];
    L[j][5] = q[7] + y * q[1] + yy * q[3];
    L[j][6] = q[0] + y * q[4] + yy * q[6];
    L[j][7] = q[2] + y * q[5];
  }
}

// transpose: the plane's line coefficients -> its part of the nodal values
template <typename T>
FG_HD void plane_lines_t(const T (*L)[8], int k, T *f) {
  const T a = T(kA20), h = T(0.5), z = k == 0 ? -a : (k == 1 ? T(0) : a), zz = k == 1 ? T(0) : T(0.6);
  const T b = T(0.6);
  T p[8], q[8], c[4], m[4], cz[4], mz[4];
  {
    const T s0 = L[0][0] + L[2][0], d0 = a * (L[2][0] - L[0][0]);
    const T s1 = L[0][1] + L[2][1], d1 = a * (L[2][1] - L[0][1]);
    const T s2 = L[0][2] + L[2][2], d2 = a * (L[2][2] - L[0][2]);
    const T s3 = L[0][3] + L[2][3], d3 = a * (L[2][3] - L[0][3]);
    p[0] = s0 + L[1][0];
    p[4] = d0 + s3 + L[1][3];
    p[6] = b * s0 + T(2) * d3;
    p[2] = T(2) * (s1 + L[1][1]);
    p[5] = T(2) * d1 + (L[0][4] + L[1][4] + L[2][4]);
    p[1] = s2 + L[1][2];
    p[3] = T(2) * d2;
    p[7] = T(0);
  }
  {
    const T s0 = L[0][5] + L[2][5], s1 = L[0][6] + L[2][6], s2 = L[0][7] + L[2][7];
    q[7] = s0 + L[1][5];
    q[1] = a * (L[2][5] - L[0][5]);
    q[3] = b * s0;
    q[0] = s1 + L[1][6];
    q[4] = a * (L[2][6] - L[0][6]);
    q[6] = b * s1;
    q[2] = s2 + L[1][7];
    q[5] = a * (L[2][7] - L[0][7]);
  }
  face_poly_t(p, false, c, m);
  face_poly_t(q, true, cz, mz);
  T g[4];
  for (int i = 0; i < 4; i++) {
    const T o = z * m[i] + mz[i];
    g[i] = T(2) * z * mz[i] - (T(1) - zz) * m[i];
    f[mid_top(i)] = h * (m[i] + o);
    f[mid_bot(i)] = h * (m[i] - o);
  }
  for (int i = 0; i < 4; i++) {
    const T o = z * c[i] + cz[i];
    const T d = zz * c[i] + T(2) * z * cz[i] + h * (g[i] + g[(i + 3) & 3]);
    f[corner_top(i)] = h * (d + o);
    f[corner_bot(i)] = h * (d - o);
    f[corner_mid(i)] = c[i] - d;
  }
}

// one Gauss point: H (3 x 3 reference gradient, H[3 c + d]) -> P
template <typename T>
FG_HD void point_stress(const T *H, const T *A, T lam, T mu, T *P) {
  T G[9];
  for (int c = 0; c < 3; c++)
    for (int j = 0; j < 3; j++) G[3 * c + j] = H[3 * c] * A[j] + H[3 * c + 1] * A[3 + j] + H[3 * c + 2] * A[6 + j];
  const T tr = lam * (G[0] + G[4] + G[8]);
  const T m2 = mu + mu;
  const T s0 = tr + m2 * G[0], s1 = tr + m2 * G[4], s2 = tr + m2 * G[8];
  const T s01 = mu * (G[1] + G[3]), s02 = mu * (G[2] + G[6]), s12 = mu * (G[5] + G[7]);
  for (int d = 0; d < 3; d++) {
    const T a0 = A[3 * d], a1 = A[3 * d + 1], a2 = A[3 * d + 2];
    P[d] = s0 * a0 + s01 * a1 + s02 * a2;
    P[3 + d] = s01 * a0 + s1 * a1 + s12 * a2;
    P[6 + d] = s02 * a0 + s12 * a1 + s2 * a2;
  }
}

// a line's three points: L[c][8] (overwritten with the transposed result),
// geometry A(i, q) of point i
template <typename T, typename Geo>
FG_HD void line_points(T (*L)[8], const Geo &A, T lam, T mu) {
  const T a = T(kA20);
  T R[3][8];
  for (int c = 0; c < 3; c++)
    for (int q = 0; q < 8; q++) R[c][q] = T(0);
  for (int i = 0; i < 3; i++) {
    const T x = i == 0 ? -a : (i == 1 ? T(0) : a), xx = i == 1 ? T(0) : T(0.6);
    T H[9], P[9], Ag[9];
    for (int q = 0; q < 9; q++) Ag[q] = A(i, q);
    for (int c = 0; c < 3; c++) {
      H[3 * c] = L[c][0] + x * L[c][1];
      H[3 * c + 1] = L[c][2] + x * L[c][3] + xx * L[c][4];
      H[3 * c + 2] = L[c][5] + x * L[c][6] + xx * L[c][7];
    }
    point_stress(H, Ag, lam, mu, P);
    for (int c = 0; c < 3; c++) {
      R[c][0] += P[3 * c];
      R[c][1] += x * P[3 * c];
      R[c][2] += P[3 * c + 1];
      R[c][3] += x * P[3 * c + 1];
      R[c][4] += xx * P[3 * c + 1];
      R[c][5] += P[3 * c + 2];
      R[c][6] += x * P[3 * c + 2];
      R[c][7] += xx * P[3 * c + 2];
    }
  }
  for (int c = 0; c < 3; c++)
    for (int q = 0; q < 8; q++) L[c][q] = R[c][q];
}

// hex8, one component: nodal values -> the derivatives, each of which is
// constant along its own direction: D[0] = d/dx at (y, z) signs 2 bits
// (y + 2 z), D[1] = d/dy at x + 2 z, D[2] = d/dz at x + 2 y
template <typename T>
FG_HD void hex8_grads(const T *f, T (*D)[4]) {
  // corner pairs of FAST's order: nodes 0..3 at z = 1: (-,-) (+,-) (+,+) (-,+); 4..7 at z = -1
  const T w = T(0.125), s = T(0.125 * kA8), t = T(0.125 / 3.0);
  T e[4], o[4];
  for (int i = 0; i < 4; i++) { e[i] = f[i] + f[4 + i]; o[i] = f[i] - f[4 + i]; }
  const T ex = (e[1] - e[0]) + (e[2] - e[3]), exy = (e[0] - e[1]) + (e[2] - e[3]),
          ey = (e[2] - e[1]) + (e[3] - e[0]);
  const T o0 = (o[0] + o[1]) + (o[2] + o[3]), ox = (o[1] - o[0]) + (o[2] - o[3]),
          oxy = (o[0] - o[1]) + (o[2] - o[3]), oy = (o[2] - o[1]) + (o[3] - o[0]);
  auto four = [](T c, T u, T v, T uv, T *out) {  // c +- u +- v +- uv
    out[0] = (c - u) - (v - uv);
    out[1] = (c + u) - (v + uv);
    out[2] = (c - u) + (v - uv);
    out[3] = (c + u) + (v + uv);
  };
  four(w * ex, s * exy, s * ox, t * oxy, D[0]);   // u: y, v: z
  four(w * ey, s * exy, s * oy, t * oxy, D[1]);   // u: x, v: z
  four(w * o0, s * ox, s * oy, t * oxy, D[2]);    // u: x, v: y
}
template <typename T>
FG_HD void hex8_grads_t(const T (*D)[4], T *f) {
  const T w = T(0.125), s = T(0.125 * kA8), t = T(0.125 / 3.0);
  auto four = [](const T *in, T &c, T &u, T &v, T &uv) {
    const T a = in[0] + in[1], b = in[2] + in[3], d = in[1] - in[0], e = in[3] - in[2];
    c = a + b;
    u = d + e;
    v = b - a;
    uv = e - d;
  };
  T c0, u0, v0, w0, c1, u1, v1, w1, c2, u2, v2, w2;
  four(D[0], c0, u0, v0, w0);
  four(D[1], c1, u1, v1, w1);
  four(D[2], c2, u2, v2, w2);
  const T ex = w * c0, exy = s * (u0 + u1), ox = s * (v0 + u2), oxy = t * (w0 + w1 + w2), ey = w * c1,
          oy = s * (v1 + v2), o0 = w * c2;
  const T e[4] = {-ex + exy - ey, ex - exy - ey, ex + exy + ey, -ex - exy + ey};
  const T o[4] = {o0 - ox + oxy - oy, o0 + ox - oxy - oy, o0 + ox + oxy + oy, o0 - ox - oxy + oy};
  for (int i = 0; i < 4; i++) { f[i] = e[i] + o[i]; f[4 + i] = e[i] - o[i]; }
}

}  // namespace mf
}  // namespace fastgpu
