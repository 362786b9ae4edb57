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
//
// The hex20 steps carry a factor of 8 (kScale20), which removes every
// halving: H comes out 8 times too large, the transposes return another 8, and
// lambda and mu are taken divided by 64 (exact).
#pragma once

#ifdef __CUDACC__
#define FG_HD __host__ __device__ __forceinline__
#else
#define FG_HD inline
#endif

namespace fastgpu {
namespace mf {

template <typename T>
FG_HD T mad(T a, T b, T c) {
  return a * b + c;
}

// hex20: vertical edge i (corner (-,-), (+,-), (+,+), (-,+)): nodes at z = 1, -1, 0;
// mid i ((0,-), (+,0), (0,+), (-,0)): nodes at z = 1, -1; it lies between corners i and i + 1
FG_HD constexpr int corner_top(int i) { return 2 * i; }
FG_HD constexpr int corner_bot(int i) { return 12 + 2 * i; }
FG_HD constexpr int corner_mid(int i) { return 8 + i; }
FG_HD constexpr int mid_top(int i) { return 1 + 2 * i; }
FG_HD constexpr int mid_bot(int i) { return 13 + 2 * i; }

constexpr double kA20 = 0.77459666924148337704;  // sqrt(0.6): the 3-point Gauss abscissa
constexpr double kA8 = 0.57735026918962576451;   // sqrt(1/3)
constexpr double kScale20 = 8.0;

// The 8-node serendipity polynomial k of values c (corners) and m (mids), from
// C = 2 c, M = 2 m: 8 k of x: A - w, y: B2 - v, xy: B, xx: u, xxy: v, yy: s, xyy: w, 1: e - s
template <typename T>
struct Face {
  T A, B, B2, u, v, s, w;
};
template <typename T>
FG_HD Face<T> face_poly(const T *C, const T *M) {
  const T two = T(-2.0);
  const T q1 = mad(two, M[0], C[0] + C[1]), q2 = mad(two, M[1], C[1] + C[2]), q3 = mad(two, M[2], C[2] + C[3]),
          q4 = mad(two, M[3], C[3] + C[0]);
  const T p = C[1] - C[0], r = C[2] - C[3];
  return {p + r, r - p, (C[3] - C[0]) + (C[2] - C[1]), q1 + q3, q3 - q1, q2 + q4, q2 - q4};
}
// transpose: the adjoints of the seven -> C, M
template <typename T>
FG_HD void face_poly_t(const Face<T> &F, T *C, T *M) {
  const T two = T(-2.0);
  const T q1 = F.u - F.v, q3 = F.u + F.v, q2 = F.s + F.w, q4 = F.s - F.w;
  const T p = F.A - F.B, r = F.A + F.B, t = F.B2;
  const T pm = p + t, pp = p - t, rp = r + t, rm = t - r;
  C[0] = (q1 + q4) - pm;
  C[1] = (q1 + q2) + pp;
  C[2] = (q2 + q3) + rp;
  C[3] = (q3 + q4) + rm;
  M[0] = two * q1;
  M[1] = two * q2;
  M[2] = two * q3;
  M[3] = two * q4;
}

// Planes z = (k - 1) sqrt(0.6) and lines y = (j - 1) sqrt(0.6) are taken by
// their coordinates, not as template parameters: one copy of the code for all
// (three unrolled copies of the planes overran the instruction cache).
template <typename T>
FG_HD T gauss20(int k) {
  return k == 0 ? T(-kA20) : (k == 1 ? T(0.0) : T(kA20));
}
template <typename T>
FG_HD T gauss20_sq(int k) {
  return k == 1 ? T(0.0) : T(0.6);
}

// one component of a hex20 field on the plane z (zz = z^2): its polynomial
// there (p) and that of its z derivative (q; d0, dy: constant and y)
template <typename T>
struct Plane {
  Face<T> p, q;
  T d0, dy;
};
template <typename T>
FG_HD Plane<T> plane_poly(const T *f, T z, T zz) {
  const T z2 = z + z, g = T(0.5) * zz - T(0.5);
  T D[4], C[4], M[4], CZ[4], MZ[4];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 4; i++) {
    const T fp = f[corner_top(i)], fm = f[corner_bot(i)], f0 = f[corner_mid(i)];
    const T O = fp - fm, F = f0 + f0;
    D[i] = (fp + fm) - F;
    C[i] = mad(z, O, mad(zz, D[i], F));
    CZ[i] = mad(z2, D[i], O);
  }
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 4; i++) {
    const T fp = f[mid_top(i)], fm = f[mid_bot(i)];
    const T O = fp - fm, G = D[i] + D[(i + 1) & 3];
    M[i] = mad(z, O, mad(g, G, fp + fm));
    MZ[i] = mad(z, G, O);
  }
  Plane<T> P;
  P.p = face_poly(C, M);
  P.q = face_poly(CZ, MZ);
  P.d0 = mad(T(2.0), MZ[0] + MZ[2], -P.q.s);
  P.dy = P.q.B2 - P.q.v;
  return P;
}
// the 8 line coefficients on y (yy = y^2), scaled by 8:
//   d/dx = L0 + 2 x L1, d/dy = L2 + x L3 + x^2 L4, d/dz = L5 + x L6 + x^2 L7
template <typename T>
FG_HD void plane_line(const Plane<T> &P, T y, T yy, T *L) {
  const T y2 = y + y, c = yy - T(1.0);
  L[0] = mad(y, P.p.B, mad(c, P.p.w, P.p.A));
  L[1] = mad(y, P.p.v, P.p.u);
  L[2] = mad(y2, P.p.s, P.p.B2 - P.p.v);
  L[3] = mad(y2, P.p.w, P.p.B);
  L[4] = P.p.v;
  L[5] = mad(y, P.dy, mad(yy, P.q.s, P.d0));
  L[6] = mad(y, P.q.B, mad(c, P.q.w, P.q.A));
  L[7] = mad(y, P.q.v, P.q.u);
}

// transposes.  A line's results R are added to the plane's adjoint N (zeroed
// before), whose p.A ... q.w, d0 and dy are the adjoints of the plane's ...
template <typename T>
FG_HD void plane_line_t(const T *R, T y, T yy, Plane<T> &N) {
  const T y2 = y + y, c = yy - T(1.0);
  N.p.A += R[0];
  N.p.B += mad(y, R[0], R[3]);
  N.p.w += mad(c, R[0], y2 * R[3]);
  N.p.u += R[1];
  N.p.v += mad(y, R[1], R[4] - R[2]);
  N.p.B2 += R[2];
  N.p.s = mad(y2, R[2], N.p.s);
  N.d0 += R[5];
  N.dy = mad(y, R[5], N.dy);
  N.q.s = mad(yy, R[5], N.q.s);
  N.q.A += R[6];
  N.q.B = mad(y, R[6], N.q.B);
  N.q.w = mad(c, R[6], N.q.w);
  N.q.u += R[7];
  N.q.v = mad(y, R[7], N.q.v);
}
// ... and the plane's adjoint goes to its part of the nodal values
template <typename T>
FG_HD void plane_poly_t(Plane<T> &N, T z, T zz, T *f) {
  const T z2 = z + z, g = T(0.5) * zz - T(0.5);
  T C[4], M[4], CZ[4], MZ[4];
  N.q.B2 = N.dy;
  N.q.v -= N.dy;
  N.q.s -= N.d0;
  face_poly_t(N.p, C, M);
  face_poly_t(N.q, CZ, MZ);
  MZ[0] = mad(T(2.0), N.d0, MZ[0]);
  MZ[2] = mad(T(2.0), N.d0, MZ[2]);
  T G[4];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 4; i++) {
    const T O = mad(z, M[i], MZ[i]);
    G[i] = mad(z, MZ[i], g * M[i]);
    f[mid_top(i)] = M[i] + O;
    f[mid_bot(i)] = M[i] - O;
  }
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 4; i++) {
    const T O = mad(z, C[i], CZ[i]);
    const T D = mad(zz, C[i], mad(z2, CZ[i], G[i] + G[(i + 3) & 3]));
    f[corner_top(i)] = D + O;
    f[corner_bot(i)] = D - O;
    const T m = C[i] - D;
    f[corner_mid(i)] = m + m;
  }
}

// one Gauss point: H (3 x 3 reference gradient, H[3 c + d]) -> P
template <typename T>
FG_HD void point_stress(const T *H, const T *A, T lam, T mu, T *P) {
  T G[9];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int c = 0; c < 3; c++)
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int j = 0; j < 3; j++) G[3 * c + j] = mad(H[3 * c], A[j], mad(H[3 * c + 1], A[3 + j], H[3 * c + 2] * A[6 + j]));
  const T tr = lam * ((G[0] + G[4]) + G[8]);
  const T m2 = mu + mu;
  const T s0 = mad(m2, G[0], tr), s1 = mad(m2, G[4], tr), s2 = mad(m2, G[8], tr);
  const T s01 = mu * (G[1] + G[3]), s02 = mu * (G[2] + G[6]), s12 = mu * (G[5] + G[7]);
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int d = 0; d < 3; d++) {
    const T a0 = A[3 * d], a1 = A[3 * d + 1], a2 = A[3 * d + 2];
    P[d] = mad(s0, a0, mad(s01, a1, s02 * a2));
    P[3 + d] = mad(s01, a0, mad(s1, a1, s12 * a2));
    P[6 + d] = mad(s02, a0, mad(s12, a1, s2 * a2));
  }
}

// a line's gradients at its three points x = -sqrt(0.6), 0, sqrt(0.6):
// L[c][8] -> H[point][3 c + d], and the transpose.  (All three at once, P in
// H's place afterwards: the line's 24 coefficients are dead while the points
// are worked on.)
template <typename T>
FG_HD void line_gradients(const T (*L)[8], T (*H)[9]) {
  const T a = T(kA20), na = T(-kA20), a2 = T(2 * kA20), na2 = T(-2 * kA20), b = T(0.6);
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int c = 0; c < 3; c++) {
    H[0][3 * c] = mad(na2, L[c][1], L[c][0]);
    H[1][3 * c] = L[c][0];
    H[2][3 * c] = mad(a2, L[c][1], L[c][0]);
    const T y = mad(b, L[c][4], L[c][2]), z = mad(b, L[c][7], L[c][5]);
    H[0][3 * c + 1] = mad(na, L[c][3], y);
    H[1][3 * c + 1] = L[c][2];
    H[2][3 * c + 1] = mad(a, L[c][3], y);
    H[0][3 * c + 2] = mad(na, L[c][6], z);
    H[1][3 * c + 2] = L[c][5];
    H[2][3 * c + 2] = mad(a, L[c][6], z);
  }
}
template <typename T>
FG_HD void line_gradients_t(const T (*P)[9], T (*R)[8]) {
  const T a = T(kA20), a2 = T(2 * kA20), b = T(0.6);
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int c = 0; c < 3; c++) {
    R[c][0] = (P[0][3 * c] + P[2][3 * c]) + P[1][3 * c];
    R[c][1] = a2 * (P[2][3 * c] - P[0][3 * c]);
    const T y = P[0][3 * c + 1] + P[2][3 * c + 1], z = P[0][3 * c + 2] + P[2][3 * c + 2];
    R[c][2] = y + P[1][3 * c + 1];
    R[c][3] = a * (P[2][3 * c + 1] - P[0][3 * c + 1]);
    R[c][4] = b * y;
    R[c][5] = z + P[1][3 * c + 2];
    R[c][6] = a * (P[2][3 * c + 2] - P[0][3 * c + 2]);
    R[c][7] = b * z;
  }
}

// A = det J J^-1 from J (J[3 c + d] = dx_c/dxi_d); returns det J
template <typename T>
FG_HD T cofactors(const T *J, T *A) {
  A[0] = J[4] * J[8] - J[5] * J[7];
  A[1] = J[2] * J[7] - J[1] * J[8];
  A[2] = J[1] * J[5] - J[2] * J[4];
  A[3] = J[5] * J[6] - J[3] * J[8];
  A[4] = J[0] * J[8] - J[2] * J[6];
  A[5] = J[2] * J[3] - J[0] * J[5];
  A[6] = J[3] * J[7] - J[4] * J[6];
  A[7] = J[1] * J[6] - J[0] * J[7];
  A[8] = J[0] * J[4] - J[1] * J[3];
  return J[0] * A[0] + J[1] * A[3] + J[2] * A[6];
}

// hex8, one component: nodal values -> the derivatives, each of which is
// constant along its own direction: D[0] = d/dx at (y, z) signs 2 bits
// (y + 2 z), D[1] = d/dy at x + 2 z, D[2] = d/dz at x + 2 y
template <typename T>
FG_HD void four_signs(T c, T u, T v, T uv, T *out) {  // c +- u +- v +- uv
  const T a = c - v, b = c + v, d = u - uv, e = u + uv;
  out[0] = a - d;
  out[1] = a + d;
  out[2] = b - e;
  out[3] = b + e;
}
template <typename T>
FG_HD void four_signs_t(const T *in, T &c, T &u, T &v, T &uv) {
  const T a = in[0] + in[1], b = in[2] + in[3], d = in[1] - in[0], e = in[3] - in[2];
  c = a + b;
  u = d + e;
  v = b - a;
  uv = e - d;
}
template <typename T>
FG_HD void hex8_grads(const T *f, T (*D)[4]) {
  // corner pairs of FAST's order: nodes 0..3 at z = 1: (-,-) (+,-) (+,+) (-,+); 4..7 at z = -1
  const T w = T(0.125), s = T(0.125 * kA8), t = T(0.125 / 3.0);
  T e[4], o[4];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 4; i++) {
    e[i] = f[i] + f[4 + i];
    o[i] = f[i] - f[4 + i];
  }
  const T ep = e[1] - e[0], er = e[2] - e[3], op = o[1] - o[0], orr = o[2] - o[3];
  const T ex = ep + er, exy = er - ep, ey = (e[2] - e[1]) + (e[3] - e[0]);
  const T o0 = (o[0] + o[1]) + (o[2] + o[3]), ox = op + orr, oxy = orr - op, oy = (o[2] - o[1]) + (o[3] - o[0]);
  const T se = s * exy, sx = s * ox, sy = s * oy, tt = t * oxy;
  four_signs(w * ex, se, sx, tt, D[0]);   // u: y, v: z
  four_signs(w * ey, se, sy, tt, D[1]);   // u: x, v: z
  four_signs(w * o0, sx, sy, tt, D[2]);   // u: x, v: y
}
template <typename T>
FG_HD void hex8_grads_t(const T (*D)[4], T *f) {
  const T w = T(0.125), s = T(0.125 * kA8), t = T(0.125 / 3.0);
  T c0, u0, v0, w0, c1, u1, v1, w1, c2, u2, v2, w2;
  four_signs_t(D[0], c0, u0, v0, w0);
  four_signs_t(D[1], c1, u1, v1, w1);
  four_signs_t(D[2], c2, u2, v2, w2);
  const T ex = w * c0, exy = s * (u0 + u1), ox = s * (v0 + u2), oxy = t * ((w0 + w1) + w2), ey = w * c1,
          oy = s * (v1 + v2), o0 = w * c2;
  const T exa = ex + exy, exb = ex - exy, oxa = ox + oxy, oxb = ox - oxy;
  const T e0 = T(-1.0) * (exb + ey), e1 = exb - ey, e2 = exa + ey, e3 = ey - exa;
  const T oa = o0 - oy, ob = o0 + oy;
  const T q0 = oa - oxb, q1 = oa + oxb, q2 = ob + oxa, q3 = ob - oxa;
  f[0] = e0 + q0; f[1] = e1 + q1; f[2] = e2 + q2; f[3] = e3 + q3;
  f[4] = e0 - q0; f[5] = e1 - q1; f[6] = e2 - q2; f[7] = e3 - q3;
}

}  // namespace mf
}  // namespace fastgpu
