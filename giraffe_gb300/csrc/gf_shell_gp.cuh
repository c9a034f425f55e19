// The Shell_1 Gauss point on the device in the global frame: its 15x15 tangent
// operator Psi^T D Psi + G and its force terms (Shell_1::Mount, reference
// src/Shell_1.cpp:899-1332), the follower pressure at a point
// (src/Shell_1.cpp:1392-1467) and the inertia at a point
// (src/Shell_1.cpp:2406-2498).
//
// FP64 is this part's scarce unit (64 cycles a warp instruction on a
// sub-partition).  The operator takes about 1,900 operations a point instead of
// the 5,000 of 3x3 matrix products in the element frame, and no rotation of the
// 27x27 result:
//  - increments stay in the global frame; the element frame enters through R_i =
//    T3^T Q_i and T3^T z_i;
//  - the operator is the Hessian of the strain energy at the point, so only its
//    blocks (r, c), r <= c, are formed, the diagonal ones as upper triangles;
//  - of the thickness-integrated operator D only 2x2 blocks and the diagonals of
//    the third components are not zero: D[n_a][n_b] = A0_ab, D[n_a][k_b] = -A1_ab
//    E, D[k_a][n_b] = E A1_ab, D[k_a][k_b] = -E A2_ab E with A_k = sum w zeta^k C
//    and E = [[0, -1], [1, 0]]; E goes into the curvatures' directions;
//  - products of skew tensors are outer products (as in gf_beam_gp.cuh).
#pragma once
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

typedef V3<double> s3;

GF_HD s3 s_cross(const s3& a, const s3& b) {
  return {{a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]}};
}
// s (x + h a x x): Xi x with h = 1/2, Xi^T x with h = -1/2 (s = g)
GF_HD s3 s_xi(const s3& a, const s3& x, double s, double h) {
  const s3 c = s_cross(a, x);
  return {{s * (x[0] + h * c[0]), s * (x[1] + h * c[1]), s * (x[2] + h * c[2])}};
}

// Kinematics of Gauss point g at the nodal increments d (27, global, entry x at
// d[x * ds]): rotation a, its derivatives b[2], z[2] and the columns of Q in the
// global frame, the strains eta[2] (less the reference's) and curvatures kap[2].
struct ShellKin {
  s3 a, b[2], z[2], Q[3], eta[2], kap[2];
  double gq, hg;
};
GF_HD void shell_kin(const ShellConst& c, const ShellHist& h, const double* d, int ds, int g, ShellKin& k) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double u1 = 0.0, u2 = 0.0, a = 0.0, b1 = 0.0, b2 = 0.0;
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const double x = d[(3 * n + i) * ds];
      u1 = fma(x, c.Nu1[g][n], u1);
      u2 = fma(x, c.Nu2[g][n], u2);
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double x = d[(18 + 3 * m + i) * ds];
      a = fma(x, c.Na[g][m], a);
      b1 = fma(x, c.Na1[g][m], b1);
      b2 = fma(x, c.Na2[g][m], b2);
    }
    k.z[0][i] = u1;
    k.z[1][i] = u2;
    k.a[i] = a;
    k.b[0][i] = b1;
    k.b[1][i] = b2;
  }
  k.gq = 4.0 / (4.0 + dot(k.a, k.a));
  k.hg = 0.5 * k.gq;
  M3<double> T;
#pragma unroll
  for (int q = 0; q < 9; ++q) T[q] = c.T3[q];
  // y = Q_delta^T z in the element frame, as z plus its small rotation: the
  // strains eta = Q_i^T y - e cancel to the last bits of y, so y takes as few
  // roundings as it can
  const s3 al = mv(T, k.a);
  s3 y[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const s3 hz = q ? s3{{h.z2[g][0], h.z2[g][1], h.z2[g][2]}} : s3{{h.z1[g][0], h.z1[g][1], h.z1[g][2]}};
    const s3 ul = mv(T, k.z[q]), zl = {{ul[0] + hz[0], ul[1] + hz[1], ul[2] + hz[2]}};
    const s3 c1 = s_cross(al, zl), c2 = s_cross(al, c1), w = tmv(T, hz);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      y[q][i] = fma(k.gq, fma(0.5, c2[i], -c1[i]), zl[i]);
      k.z[q][i] += w[i];
    }
  }
  const s3 beta1 = s_xi(k.a, k.b[0], k.gq, -0.5), beta2 = s_xi(k.a, k.b[1], k.gq, -0.5);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const s3 qi = {{h.Q[g][j], h.Q[g][3 + j], h.Q[g][6 + j]}};
    const s3 r = tmv(T, qi);  // column j of T3^T Q_i
    k.eta[0][j] = dot(qi, y[0]) - (j == 0 ? 1.0 : 0.0);
    k.eta[1][j] = dot(qi, y[1]) - (j == 1 ? 1.0 : 0.0);
    k.kap[0][j] = dot(r, beta1) + h.k1[g][j];
    k.kap[1][j] = dot(r, beta2) + h.k2[g][j];
    const s3 c1 = s_cross(k.a, r), c2 = s_cross(k.a, c1);
#pragma unroll
    for (int i = 0; i < 3; ++i) k.Q[j][i] = fma(k.gq, fma(0.5, c2[i], c1[i]), r[i]);
  }
}

// Thickness integration (three points) of the compressible neo-Hookean law: the
// stress resultants n[2], m[2] and, with TAN, the moments A[k] = sum w zeta^k C of
// the 2x2 in-plane operators: C11 (00, 01, 11), C22 (00, 01, 11), C12 (row-major).
template <bool TAN> struct ShellLaw;
template <> struct ShellLaw<false> {
  s3 n[2], m[2];
};
template <> struct ShellLaw<true> {
  s3 n[2], m[2];
  double A[3][10];
};
template <bool TAN> GF_HD void shell_law(const ShellConst& c, const ShellKin& k, ShellLaw<TAN>& s) {
  const double mu = c.mu, la = c.lambda;
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 3; ++i) s.n[q][i] = s.m[q][i] = 0.0;
  if constexpr (TAN) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int x = 0; x < 10; ++x) s.A[q][x] = 0.0;
  }
  const double jac = 0.5 * c.thick;
#pragma unroll 1
  for (int q = 0; q < 3; ++q) {
    const double zeta = q == 1 ? 0.0 : (q ? 1.0 : -1.0) * 0.77459666924148337703585307995648 * jac;
    const double w = (q == 1 ? 0.88888888888888888888888888888889 : 0.55555555555555555555555555555556) * jac;
    const double g11 = fma(zeta, k.kap[0][1], k.eta[0][0]), g12 = fma(-zeta, k.kap[0][0], k.eta[0][1]);
    const double g21 = fma(zeta, k.kap[1][1], k.eta[1][0]), g22 = fma(-zeta, k.kap[1][0], k.eta[1][1]);
    const double f1 = 1.0 + g11, f2 = 1.0 + g22, jb = f1 * f2 - g12 * g21;
    const double j2 = jb * jb, den = la * j2 + 2.0 * mu, r = 1.0 / (jb * den);
    const double v = (la * (jb * j2 - 1.0) + 2.0 * mu * (jb - 1.0)) * r, mv_ = mu * v;
    const double sh = mu * (g12 + g21), wz = w * zeta;
    const double t10 = mv_ * f2 + mu * (g11 - g22), t11 = sh - mv_ * g21;
    const double t20 = sh - mv_ * g12, t21 = mv_ * f1 + mu * (g22 - g11);
    s.n[0][0] += w * t10;
    s.n[0][1] += w * t11;
    s.n[1][0] += w * t20;
    s.n[1][1] += w * t21;
    s.m[0][0] -= wz * t11;
    s.m[0][1] += wz * t10;
    s.m[1][0] -= wz * t21;
    s.m[1][1] += wz * t20;
    if constexpr (TAN) {
      const double dv = (la + 2.0 * mu) * (3.0 * la * j2 + 2.0 * mu) * r * r, md = mu * dv, wz2 = wz * zeta;
      const double m2 = md * f2, m1 = md * f1;
      const double C[10] = {m2 * f2 + mu,      -m2 * g21, md * g21 * g21 + mu,        md * g12 * g12 + mu, -m1 * g12,
                            m1 * f1 + mu,      -m2 * g12, mv_ - mu + m2 * f1,         mu - mv_ + md * g12 * g21,
                            -m1 * g21};
#pragma unroll
      for (int x = 0; x < 10; ++x) {
        s.A[0][x] = fma(w, C[x], s.A[0][x]);
        s.A[1][x] = fma(wz, C[x], s.A[1][x]);
        s.A[2][x] = fma(wz2, C[x], s.A[2][x]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    s.n[q][2] = mu * c.thick * k.eta[q][2];
    s.m[q][2] = c.stiff_drill * k.kap[q][2];
  }
}

// Stored values of one Gauss point.  Operator blocks over the rows (x1
// derivative of u, x1 of alpha, x2 of u, x2 of alpha, alpha): diagonal ones as
// (00, 11, 22, 01, 02, 12), the others row-major.
constexpr int SP_D0 = 0, SP_D1 = 6, SP_D2 = 12, SP_D3 = 18, SP_D4 = 24, SP_M01 = 30, SP_M02 = 39, SP_M03 = 48,
              SP_M12 = 57, SP_M13 = 66, SP_M23 = 75, SP_M04 = 84, SP_M14 = 93, SP_M24 = 102, SP_M34 = 111,
              SP_COUNT = 120;
// The geometric part, added to M04, M14, M24, M34 and D4 afterwards (formed by
// other lanes), and the generalized forces of the five rows.
constexpr int SG_M04 = 0, SG_M14 = 9, SG_M24 = 18, SG_M34 = 27, SG_D4 = 36, SG_COUNT = 42;
constexpr int SQ_COUNT = 15;

// Entry (i, j) of a diagonal block.
GF_HD int sp_sym(int i, int j) { return i == j ? i : i + j + 2; }

// 3x2 directions of the in-plane strains of each kind and their third ones.
struct Dir2 {
  s3 v[2];
};
// X A with the 2x2 A = [a b; c d]
GF_HD Dir2 dir_mul(const Dir2& X, double a, double b, double c, double d) {
  Dir2 r;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    r.v[0][i] = X.v[0][i] * a + X.v[1][i] * c;
    r.v[1][i] = X.v[0][i] * b + X.v[1][i] * d;
  }
  return r;
}
GF_HD void dir_add(Dir2& r, const Dir2& X, double a, double b, double c, double d) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    r.v[0][i] = fma(X.v[1][i], c, fma(X.v[0][i], a, r.v[0][i]));
    r.v[1][i] = fma(X.v[1][i], d, fma(X.v[0][i], b, r.v[1][i]));
  }
}
GF_HD double dir_dot(const Dir2& X, const Dir2& Y, int i, int j) {
  return fma(X.v[1][i], Y.v[1][j], X.v[0][i] * Y.v[0][j]);
}
// X Y^T (+ w p q^T) to a full block
GF_HD void dir_full(const Dir2& X, const Dir2& Y, double* o, int os) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) o[(3 * i + j) * os] = dir_dot(X, Y, i, j);
}
GF_HD void dir_full(const Dir2& X, const Dir2& Y, const s3& p, const s3& q, double* o, int os) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) o[(3 * i + j) * os] = fma(p[i], q[j], dir_dot(X, Y, i, j));
}
GF_HD void dir_sym(const Dir2& X, const Dir2& Y, double w, const s3& q, double* o, int os) {
  const s3 p = {{w * q[0], w * q[1], w * q[2]}};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) o[sp_sym(i, j) * os] = fma(p[i], q[j], dir_dot(X, Y, i, j));
}

// Directions of the curvatures: W = Xi^T Q, Y = [W_2, -W_1] (W E).
GF_HD void shell_curv_dirs(const ShellKin& k, Dir2& Y, s3& W3) {
  const s3 W1 = s_xi(k.a, k.Q[0], k.gq, -0.5), W2 = s_xi(k.a, k.Q[1], k.gq, -0.5);
  W3 = s_xi(k.a, k.Q[2], k.gq, -0.5);
  Y.v[0] = W2;
  Y.v[1] = {{-W1[0], -W1[1], -W1[2]}};
}

// Part 0 of a point: the blocks of the derivative rows, and their forces.
GF_HD void shell_part0(const ShellConst& c, const ShellHist& h, const double* d, int ds, int g, double* o, double* fq,
                       int os) {
  ShellKin k;
  ShellLaw<true> s;
  shell_kin(c, h, d, ds, g, k);
  shell_law<true>(c, k, s);
  const double t3 = c.mu * c.thick;
  Dir2 S, Y;
  s3 W3;
  S.v[0] = k.Q[0];
  S.v[1] = k.Q[1];
  shell_curv_dirs(k, Y, W3);
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      fq[(6 * q + i) * os] = fma(k.Q[2][i], s.n[q][2], fma(k.Q[1][i], s.n[q][1], k.Q[0][i] * s.n[q][0]));
      // Xi^T Q m with W = [-Y_2, Y_1, W3]
      fq[(6 * q + 3 + i) * os] = fma(W3[i], s.m[q][2], fma(Y.v[0][i], s.m[q][1], -Y.v[1][i] * s.m[q][0]));
    }
  const double *A0 = s.A[0], *A1 = s.A[1], *A2 = s.A[2];
  dir_sym(dir_mul(S, A0[0], A0[1], A0[1], A0[2]), S, t3, k.Q[2], o + SP_D0 * os, os);
  dir_sym(dir_mul(S, A0[3], A0[4], A0[4], A0[5]), S, t3, k.Q[2], o + SP_D2 * os, os);
  dir_full(dir_mul(S, A0[6], A0[7], A0[8], A0[9]), S, o + SP_M02 * os, os);
  dir_full(dir_mul(S, A1[0], A1[1], A1[1], A1[2]), Y, o + SP_M01 * os, os);
  dir_full(dir_mul(S, A1[6], A1[7], A1[8], A1[9]), Y, o + SP_M03 * os, os);
  // (kappa_1, eta_2): Y A1_12 S^T
  dir_full(dir_mul(Y, A1[6], A1[7], A1[8], A1[9]), S, o + SP_M12 * os, os);
  dir_full(dir_mul(S, A1[3], A1[4], A1[4], A1[5]), Y, o + SP_M23 * os, os);
  dir_sym(dir_mul(Y, A2[0], A2[1], A2[1], A2[2]), Y, c.stiff_drill, W3, o + SP_D1 * os, os);
  dir_sym(dir_mul(Y, A2[3], A2[4], A2[4], A2[5]), Y, c.stiff_drill, W3, o + SP_D3 * os, os);
  dir_full(dir_mul(Y, A2[6], A2[7], A2[8], A2[9]), Y, o + SP_M13 * os, os);
}

// Part 1: the material part of the rotation's column (M04, M14, M24, M34, D4).
GF_HD void shell_part1(const ShellConst& c, const ShellHist& h, const double* d, int ds, int g, double* o, int os) {
  ShellKin k;
  ShellLaw<true> s;
  shell_kin(c, h, d, ds, g, k);
  shell_law<true>(c, k, s);
  const double t3 = c.mu * c.thick;
  Dir2 S, Y;
  s3 W[3], W3;
  S.v[0] = k.Q[0];
  S.v[1] = k.Q[1];
  shell_curv_dirs(k, Y, W3);
  W[0] = {{-Y.v[1][0], -Y.v[1][1], -Y.v[1][2]}};
  W[1] = Y.v[0];
  W[2] = W3;
  // rotation's directions of eta_a (B: Xi^T (q_i x z_a)) and kappa_a (U: Xi_a'^T
  // q_i = -g/2 ((a.b_a) W_i + b_a x q_i)), the kappas' through E
  Dir2 B[2], U[2];
  s3 B3[2], U3[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double ab = dot(k.a, k.b[q]);
    s3 C[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const s3 x = s_xi(k.a, s_cross(k.Q[i], k.z[q]), k.gq, -0.5);
      if (i < 2) B[q].v[i] = x;
      else B3[q] = x;
      const s3 y = s_cross(k.b[q], k.Q[i]);
#pragma unroll
      for (int j = 0; j < 3; ++j) C[i][j] = -k.hg * fma(ab, W[i][j], y[j]);
    }
    U[q].v[0] = C[1];
    U[q].v[1] = {{-C[0][0], -C[0][1], -C[0][2]}};
    U3[q] = C[2];
  }
  const double *A0 = s.A[0], *A1 = s.A[1], *A2 = s.A[2];
  double d4[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  // column a of D through the rotation's directions: H_r = sum_q (direction of
  // q) D_qr for r = eta_1, kappa_1, eta_2, kappa_2; D_21 is D_12 transposed
  auto add4 = [&](const Dir2& H, const Dir2& X, double w, const s3& q) {
    const s3 p = {{w * q[0], w * q[1], w * q[2]}};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) d4[sp_sym(i, j)] += fma(p[i], q[j], dir_dot(H, X, i, j));
  };
  auto column = [&](const Dir2& H, const Dir2& X, const s3& x3, double w, const s3& q3, double* out) {
    // block (row, alpha) = X H^T + w x3 q3^T
    dir_full(X, H, x3, s3{{w * q3[0], w * q3[1], w * q3[2]}}, out, os);
  };
  Dir2 H = dir_mul(B[0], A0[0], A0[1], A0[1], A0[2]);
  dir_add(H, U[0], A1[0], A1[1], A1[1], A1[2]);
  dir_add(H, B[1], A0[6], A0[8], A0[7], A0[9]);
  dir_add(H, U[1], A1[6], A1[8], A1[7], A1[9]);
  column(H, S, k.Q[2], t3, B3[0], o + SP_M04 * os);
  add4(H, B[0], t3, B3[0]);
  H = dir_mul(B[0], A1[0], A1[1], A1[1], A1[2]);
  dir_add(H, U[0], A2[0], A2[1], A2[1], A2[2]);
  dir_add(H, B[1], A1[6], A1[8], A1[7], A1[9]);
  dir_add(H, U[1], A2[6], A2[8], A2[7], A2[9]);
  column(H, Y, W3, c.stiff_drill, U3[0], o + SP_M14 * os);
  add4(H, U[0], c.stiff_drill, U3[0]);
  H = dir_mul(B[0], A0[6], A0[7], A0[8], A0[9]);
  dir_add(H, U[0], A1[6], A1[7], A1[8], A1[9]);
  dir_add(H, B[1], A0[3], A0[4], A0[4], A0[5]);
  dir_add(H, U[1], A1[3], A1[4], A1[4], A1[5]);
  column(H, S, k.Q[2], t3, B3[1], o + SP_M24 * os);
  add4(H, B[1], t3, B3[1]);
  H = dir_mul(B[0], A1[6], A1[7], A1[8], A1[9]);
  dir_add(H, U[0], A2[6], A2[7], A2[8], A2[9]);
  dir_add(H, B[1], A1[3], A1[4], A1[4], A1[5]);
  dir_add(H, U[1], A2[3], A2[4], A2[4], A2[5]);
  column(H, Y, W3, c.stiff_drill, U3[1], o + SP_M34 * os);
  add4(H, U[1], c.stiff_drill, U3[1]);
#pragma unroll
  for (int x = 0; x < 6; ++x) o[(SP_D4 + x) * os] = d4[x];
}

// Part 2: the geometric part of the rotation's column (symmetric parts of the
// rotation block: see gf_beam_gp.cuh, here the sum over both derivatives) and its
// force.
GF_HD void shell_part2(const ShellConst& c, const ShellHist& h, const double* d, int ds, int g, double* o, double* fq,
                       int os) {
  ShellKin k;
  ShellLaw<false> s;
  shell_kin(c, h, d, ds, g, k);
  shell_law<false>(c, k, s);
  const double hg = k.hg, g2 = hg * hg;
  const s3 ha = {{hg * k.a[0], hg * k.a[1], hg * k.a[2]}};
  const s3 X[3] = {{{k.gq, ha[2], -ha[1]}}, {{-ha[2], k.gq, ha[0]}}, {{ha[1], -ha[0], k.gq}}};  // columns of Xi
  double d4[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  s3 f4 = {{0.0, 0.0, 0.0}};
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
    const s3 b = q ? k.b[1] : k.b[0], z = q ? k.z[1] : k.z[0], nr = q ? s.n[1] : s.n[0], mr = q ? s.m[1] : s.m[0];
    s3 n, m;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      n[i] = fma(k.Q[2][i], nr[2], fma(k.Q[1][i], nr[1], k.Q[0][i] * nr[0]));
      m[i] = fma(k.Q[2][i], mr[2], fma(k.Q[1][i], mr[1], k.Q[0][i] * mr[0]));
    }
    double* og = o + (q ? SG_M24 : SG_M04) * os;
    double* om = o + (q ? SG_M34 : SG_M14) * os;
    const double ab = dot(k.a, b), zn = dot(z, n), bmd = dot(b, m);
    const s3 mu = s_xi(k.a, m, k.gq, -0.5), bm = s_cross(b, m), beta = s_xi(k.a, b, k.gq, -0.5);
    const s3 nu = s_xi(k.a, n, k.gq, -0.5), zeta = s_xi(k.a, z, k.gq, -0.5), kx = s_xi(k.a, s_cross(z, n), k.gq, -0.5);
    const s3 w = {{-hg * mu[0], -hg * mu[1], -hg * mu[2]}}, hm = {{hg * m[0], hg * m[1], hg * m[2]}};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const s3 nx = s_cross(n, X[j]);
#pragma unroll
      for (int i = 0; i < 3; ++i) og[(3 * i + j) * os] = -nx[i];
    }
    // V(a, m)^T = a w^T - g/2 skew(m)
    const double sk[9] = {0.0, -hm[2], hm[1], hm[2], 0.0, -hm[0], -hm[1], hm[0], 0.0};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) om[(3 * i + j) * os] = fma(k.a[i], w[j], -sk[3 * i + j]);
    s3 p;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      p[i] = fma(zn * g2, k.a[i], fma(hg, kx[i], g2 * fma(2.0 * ab, mu[i], bm[i])));
      f4[i] -= fma(hg, fma(ab, mu[i], bm[i]), kx[i]);
    }
    const double diag = fma(k.gq, zn, k.gq * hg * bmd);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        if (i == j) {
          d4[i] += fma(nu[i], zeta[i], fma(p[i], k.a[i], fma(w[i], b[i], hm[i] * beta[i]))) - diag;
        } else {
          double v = fma(nu[i], zeta[j], nu[j] * zeta[i]);
          v = fma(p[i], k.a[j], fma(p[j], k.a[i], v));
          v = fma(w[i], b[j], fma(w[j], b[i], v));
          v = fma(hm[i], beta[j], fma(hm[j], beta[i], v));
          d4[sp_sym(i, j)] = fma(0.5, v, d4[sp_sym(i, j)]);
        }
      }
  }
#pragma unroll
  for (int x = 0; x < 6; ++x) o[(SG_D4 + x) * os] = d4[x];
#pragma unroll
  for (int i = 0; i < 3; ++i) fq[(12 + i) * os] = f4[i];
}

// Follower pressure p at point kq (six-point rule) and the displacements pu (18,
// global, entry x at pu[x * ds]) of the nodes from the reference position: the
// surface tangents t1, t2, the unit normal, 1 / |t1 x t2|, w p, and the load.
constexpr int PP_T1 = 0, PP_T2 = 3, PP_N = 6, PP_RN = 9, PP_WP = 10, PP_F = 11, PP_COUNT = 14;
GF_HD void shell_press_point(const ShellConst& c, const double* pu, int ds, double p, bool area_update, int kq,
                             double* o, int os) {
  s3 t1, t2;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const double x = pu[(3 * n + j) * ds];
      s1 = fma(c.N41[kq][n], x, s1);
      s2 = fma(c.N42[kq][n], x, s2);
    }
    t1[j] = c.T3[j] + s1;
    t2[j] = c.T3[3 + j] + s2;
  }
  const s3 cr = s_cross(t1, t2);
  const double nc = sqrt(dot(cr, cr)), rn = 1.0 / nc, wp = c.w4[kq] * p, fac = (area_update ? nc : 1.0) * wp;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double np = rn * cr[j];
    o[(PP_T1 + j) * os] = t1[j];
    o[(PP_T2 + j) * os] = t2[j];
    o[(PP_N + j) * os] = np;
    o[(PP_F + j) * os] = fac * np;
  }
  o[PP_RN * os] = rn;
  o[PP_WP * os] = wp;
}

// Column j of the pressure's tangent blocks (a, nb), a = 0..5, into o[(6 a + nb)
// 9 + 3 i + col]: entries of that column without the area's update, else (the
// blocks are skew) the entries in which component j appears.
GF_HD void shell_press_cols(const ShellConst& c, const double* pt, int ps, int kstep, bool area_update, int nb, int j,
                            double* o) {
  if (area_update) {
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
    for (int kq = 0; kq < 6; ++kq) {
      const double* q = pt + kq * kstep;
      const double x = q[PP_WP * ps] * (q[(PP_T1 + j) * ps] * c.N42[kq][nb] - q[(PP_T2 + j) * ps] * c.N41[kq][nb]);
#pragma unroll
      for (int a = 0; a < 6; ++a) v[a] = fma(c.N4[kq][a], x, v[a]);
    }
    const int j1 = j == 2 ? 0 : j + 1, j2 = j == 0 ? 2 : j - 1;  // (j + 1) % 3, (j + 2) % 3
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      double* e = o + (6 * a + nb) * 9;
      e[4 * j] = 0.0;
      e[3 * j2 + j1] = v[a];
      e[3 * j1 + j2] = -v[a];
    }
    return;
  }
  double v[6][3];
#pragma unroll
  for (int a = 0; a < 6; ++a) v[a][0] = v[a][1] = v[a][2] = 0.0;
#pragma unroll 1
  for (int kq = 0; kq < 6; ++kq) {
    const double* q = pt + kq * kstep;
    s3 x;
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i] = q[(PP_T1 + i) * ps] * c.N42[kq][nb] - q[(PP_T2 + i) * ps] * c.N41[kq][nb];
    // column j of skew(x), less its part along the normal
    const s3 col = j == 0 ? s3{{0.0, x[2], -x[1]}} : (j == 1 ? s3{{-x[2], 0.0, x[0]}} : s3{{x[1], -x[0], 0.0}});
    const s3 n = {{q[PP_N * ps], q[(PP_N + 1) * ps], q[(PP_N + 2) * ps]}};
    const double nd = dot(n, col), w = q[PP_RN * ps] * q[PP_WP * ps];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double y = w * fma(-nd, n[i], col[i]);
#pragma unroll
      for (int a = 0; a < 6; ++a) v[a][i] = fma(c.N4[kq][a], y, v[a][i]);
    }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a)
#pragma unroll
    for (int i = 0; i < 3; ++i) o[(6 * a + nb) * 9 + 3 * i + j] = v[a][i];
}

// Inertia at Gauss point g (MountMass and the mass part of MountDyn, reference
// src/Shell_1.cpp:2406-2498, 2536-2541), global frame.  The director fibre has
// mass coef1 per unit area and, about the midsurface, rotary inertia J = coef2
// (I - e e^T) with e = Q(alpha_i) e3r; its inertial moment coef2 e x e'' equals
// J w' + w x J w:
//   dT_u = coef1 (a1 du - a2 v_i - a3 acc_i)
//   dT_a = Xi(da) h,  h = J w2 + w1 x J w1,
//   w1 = a4 da + a5 w_i + a6 dw_i,  w2 = a1 da - a2 w_i - a3 dw_i
// (Newmark in the tangent space transported by Q_delta, as for Beam_1), and the
// exact tangents d dT_u / d du = a1 coef1 I,
//   d dT_a / d da = Xi (a1 J + a4 (skew(w1) J - skew(J w1)))
//                   - g^2/2 (h + da x h / 2) da^T - g/2 skew(h).
// vel, acc: nodal velocities and accelerations, six per node: entry k of the
// element's node n at vel[at(n) + k].  Out: dT_u, dT_a, the rotation's tangent.
constexpr int SI_FU = 0, SI_FA = 3, SI_D = 6, SI_COUNT = 15;
template <typename At>
GF_HD void shell_inertia_point(const ShellConst& c, const ShellHistAux& x, const double* d, int ds, const double* vel,
                               const double* acc, At at, const double* an, int g, double* o, int os) {
  const double a1 = an[0], a2 = an[1], a3 = an[2], a4 = an[3], a5 = an[4], a6 = an[5];
  s3 fu = {{0, 0, 0}}, da = {{0, 0, 0}}, wi = {{0, 0, 0}}, dwi = {{0, 0, 0}};
  {
    s3 du = {{0, 0, 0}}, vi = {{0, 0, 0}}, ai = {{0, 0, 0}};
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const double N = c.Nu[g][n];
      const double *v = vel + at(n), *q = acc + at(n);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        du[i] = fma(d[(3 * n + i) * ds], N, du[i]);
        vi[i] = fma(v[i], N, vi[i]);
        ai[i] = fma(q[i], N, ai[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) fu[i] = c.coef1 * (a1 * du[i] - a2 * vi[i] - a3 * ai[i]);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double N = c.Na[g][m];
    const double *v = vel + at(3 + m) + 3, *q = acc + at(3 + m) + 3;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      da[i] = fma(d[(18 + 3 * m + i) * ds], N, da[i]);
      wi[i] = fma(v[i], N, wi[i]);
      dwi[i] = fma(q[i], N, dwi[i]);
    }
  }
  M3<double> T;
#pragma unroll
  for (int q = 0; q < 9; ++q) T[q] = c.T3[q];
  const M3<double> Qi = rodrigues(s3{{x.alpha[g][0], x.alpha[g][1], x.alpha[g][2]}});
  const s3 e = tmv(T, s3{{Qi[2], Qi[5], Qi[8]}});
  s3 w1, w2;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    w1[i] = a4 * da[i] + a5 * wi[i] + a6 * dwi[i];
    w2[i] = a1 * da[i] - a2 * wi[i] - a3 * dwi[i];
  }
  const double e1 = dot(e, w1), e2 = dot(e, w2);
  s3 Jw1, Jw2;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Jw1[i] = c.coef2 * (w1[i] - e[i] * e1);
    Jw2[i] = c.coef2 * (w2[i] - e[i] * e2);
  }
  const s3 cr = s_cross(w1, Jw1), h = {{Jw2[0] + cr[0], Jw2[1] + cr[1], Jw2[2] + cr[2]}};
  const double gg = 4.0 / (4.0 + dot(da, da));
  const s3 mom = s_xi(da, h, gg, 0.5);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[(SI_FU + i) * os] = fu[i];
    o[(SI_FA + i) * os] = mom[i];
  }
  // columns of a1 J + a4 (skew(w1) J - skew(J w1)): skew(w1) J = coef2 (skew(w1) -
  // (w1 x e) e^T)
  const s3 we = s_cross(w1, e), axh = s_cross(da, h);
  s3 r;
#pragma unroll
  for (int i = 0; i < 3; ++i) r[i] = c.coef2 * w1[i] - Jw1[i];
  const double hh = 0.5 * gg;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const s3 sk = j == 0 ? s3{{0.0, r[2], -r[1]}} : (j == 1 ? s3{{-r[2], 0.0, r[0]}} : s3{{r[1], -r[0], 0.0}});
    const s3 sh = j == 0 ? s3{{0.0, h[2], -h[1]}} : (j == 1 ? s3{{-h[2], 0.0, h[0]}} : s3{{h[1], -h[0], 0.0}});
    const double ej = c.coef2 * e[j];
    s3 col;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      col[i] = a1 * ((i == j ? c.coef2 : 0.0) - e[i] * ej) + a4 * (sk[i] - we[i] * ej);
    const s3 y = s_xi(da, col, gg, 0.5);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      o[(SI_D + 3 * i + j) * os] = y[i] - hh * (gg * (h[i] + 0.5 * axh[i]) * da[j] + sh[i]);
  }
}

// Columns of K_e from the stored values.  M, Q: point g at [g * gs], entries ms
// apart.  Rotation column j of midside node m: acc[0..5] the rows of the nodes'
// translations, acc[6..8] those of the rotations of the midside nodes >= m; f the
// force entry.
GF_HD void shell_col_rot(const ShellConst& c, const double* M, const double* Q, int gs, int ms, int m, int j,
                         double (&acc)[9][3], double& f) {
  f = 0.0;
#pragma unroll
  for (int n = 0; n < 9; ++n) acc[n][0] = acc[n][1] = acc[n][2] = 0.0;
#pragma unroll 1
  for (int g = 0; g < 3; ++g) {
    const double* o = M + g * gs;
    const double* q = Q + g * gs;
    const double c1 = c.alpha1 * c.Na1[g][m], c2 = c.alpha1 * c.Na2[g][m], c0 = c.alpha1 * c.Na[g][m];
    f = fma(c1, q[(3 + j) * ms], fma(c2, q[(9 + j) * ms], fma(c0, q[(12 + j) * ms], f)));
    double R[5][3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int x = 3 * i + j, t = 3 * j + i, y = sp_sym(i, j);
      R[0][i] = fma(c0, o[(SP_M04 + x) * ms], fma(c2, o[(SP_M03 + x) * ms], c1 * o[(SP_M01 + x) * ms]));
      R[1][i] = fma(c0, o[(SP_M14 + x) * ms], fma(c2, o[(SP_M13 + x) * ms], c1 * o[(SP_D1 + y) * ms]));
      R[2][i] = fma(c0, o[(SP_M24 + x) * ms], fma(c2, o[(SP_M23 + x) * ms], c1 * o[(SP_M12 + t) * ms]));
      R[3][i] = fma(c0, o[(SP_M34 + x) * ms], fma(c2, o[(SP_D3 + y) * ms], c1 * o[(SP_M13 + t) * ms]));
      R[4][i] = fma(c0, o[(SP_D4 + y) * ms], fma(c2, o[(SP_M34 + t) * ms], c1 * o[(SP_M14 + t) * ms]));
    }
#pragma unroll
    for (int n = 0; n < 6; ++n)
#pragma unroll
      for (int i = 0; i < 3; ++i) acc[n][i] = fma(c.Nu2[g][n], R[2][i], fma(c.Nu1[g][n], R[0][i], acc[n][i]));
#pragma unroll
    for (int n = 0; n < 3; ++n)
      if (n >= m)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          acc[6 + n][i] = fma(c.Na[g][n], R[4][i], fma(c.Na2[g][n], R[3][i], fma(c.Na1[g][n], R[1][i], acc[6 + n][i])));
  }
}
// Translation column j of node m: acc[n], n >= m, the rows of the translations.
GF_HD void shell_col_tr(const ShellConst& c, const double* M, const double* Q, int gs, int ms, int m, int j,
                        double (&acc)[9][3], double& f) {
  f = 0.0;
#pragma unroll
  for (int n = 0; n < 6; ++n) acc[n][0] = acc[n][1] = acc[n][2] = 0.0;
#pragma unroll 1
  for (int g = 0; g < 3; ++g) {
    const double* o = M + g * gs;
    const double* q = Q + g * gs;
    const double c1 = c.alpha1 * c.Nu1[g][m], c2 = c.alpha1 * c.Nu2[g][m];
    f = fma(c1, q[j * ms], fma(c2, q[(6 + j) * ms], f));
    double R[2][3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int y = sp_sym(i, j);
      R[0][i] = fma(c2, o[(SP_M02 + 3 * i + j) * ms], c1 * o[(SP_D0 + y) * ms]);
      R[1][i] = fma(c2, o[(SP_D2 + y) * ms], c1 * o[(SP_M02 + 3 * j + i) * ms]);
    }
#pragma unroll
    for (int n = 0; n < 6; ++n)
      if (n >= m)
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[n][i] = fma(c.Nu2[g][n], R[1][i], fma(c.Nu1[g][n], R[0][i], acc[n][i]));
  }
}

}  // namespace gf
