// The Beam_1 Gauss point on the device: its 9x9 tangent operator B^T D B + G
// and its force terms, in the global frame (Beam_1::Mount, reference
// src/Beam_1.cpp:695-835).
//
// FP64 is this part's scarce unit (64 cycles a warp instruction on a
// sub-partition), so the operator is formed from about 600 operations a point
// instead of the 1,470 of matrix products in the element frame:
//  - every increment stays in the global frame; the element frame enters only
//    through R_i = T3^T Q_i and T3^T dz_i, so no block is rotated afterwards;
//  - the operator is the Hessian of the strain energy at the point, so its
//    blocks (0,0), (1,1), (2,2) are formed as upper triangles and (2,0), (2,1)
//    are the transposes of (0,2), (1,2); (0,1) is zero;
//  - products of skew tensors are outer products: skew(a) skew(b) = b a^T -
//    (a.b) I, Xi^T Xi = g I - (g/2)^2 a a^T, Xi^T skew(m) Xi = g^2 skew(...),
//    whose antisymmetric parts cancel in the sum;
//  - Q_delta^T Xi = Xi^T for Rodrigues parameters, so the moment's stiffness
//    needs Q only through R = Q^T Xi.
// Operations are rounded explicitly: the point gives the same bits whatever
// code surrounds it, so kernels that spread an element over different numbers
// of lanes agree bit for bit.
#pragma once
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

GF_HD double rmul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
GF_HD double radd(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
GF_HD double rsub(double a, double b) { return radd(a, -b); }
GF_HD double rfma(double a, double b, double c) { return fma(a, b, c); }

typedef V3<double> d3;

GF_HD double rdot(const d3& a, const d3& b) { return rfma(a[2], b[2], rfma(a[1], b[1], rmul(a[0], b[0]))); }
GF_HD d3 rcross(const d3& a, const d3& b) {
  return {{rfma(a[1], b[2], -rmul(a[2], b[1])), rfma(a[2], b[0], -rmul(a[0], b[2])),
           rfma(a[0], b[1], -rmul(a[1], b[0]))}};
}
// s (x + h a x x): Xi x with h = 1/2, Xi^T x with h = -1/2 (s = g)
GF_HD d3 rxi(const d3& a, const d3& x, double s, double h) {
  const d3 c = rcross(a, x);
  return {{rmul(s, rfma(h, c[0], x[0])), rmul(s, rfma(h, c[1], x[1])), rmul(s, rfma(h, c[2], x[2]))}};
}
// columns of a 3x3 matrix held as three vectors: M^T x
GF_HD d3 rtmv(const d3 (&M)[3], const d3& x) { return {{rdot(M[0], x), rdot(M[1], x), rdot(M[2], x)}}; }
// M x
GF_HD d3 rmv(const d3 (&M)[3], const d3& x) {
  d3 y;
#pragma unroll
  for (int i = 0; i < 3; ++i) y[i] = rfma(M[2][i], x[2], rfma(M[1][i], x[1], rmul(M[0][i], x[0])));
  return y;
}

// Stored values of one Gauss point: operator blocks (upper triangles 00, 01,
// 02, 11, 12, 22; full blocks row-major), then the force terms n (with N'), s1
// (with N'), s2 (with N).
constexpr int GP_M00 = 0, GP_M02 = 6, GP_M11 = 15, GP_M12 = 21, GP_M22 = 30, GP_N = 36, GP_S1 = 39, GP_S2 = 42,
              GP_COUNT = 45;

// Interpolated increments at point g, global frame (reference
// src/Beam_1.cpp:700-746): rotation a, its derivative b, displacement
// derivative u1.
GF_HD void beam_gp_interp(const BeamConst& c, const double* d, int g, d3& a, d3& b, d3& u1) {
  const double N0 = c.N[g][0], N1 = c.N[g][1], N2 = c.N[g][2];
  const double D0 = c.dN[g][0], D1 = c.dN[g][1], D2 = c.dN[g][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a[i] = rfma(d[15 + i], N2, rfma(d[9 + i], N1, rmul(d[3 + i], N0)));
    b[i] = rfma(d[15 + i], D2, rfma(d[9 + i], D1, rmul(d[3 + i], D0)));
    u1[i] = rfma(d[12 + i], D2, rfma(d[6 + i], D1, rmul(d[i], D0)));
  }
}

// The point's operator and forces at the nodal increments d (18, global),
// written to o[x * os].  Parts: 1 the blocks 00, 02 and the share Y^T W of 22, 2 the
// blocks 11, 12 and the share S^T D S, 4 the geometric share of 22 and the forces;
// 22 is (Y^T W + S^T D S) + the geometric share.  A part alone writes its share at
// GP_PART + 6 (0, 1, 2) and forms what it needs of the kinematics itself.
constexpr int GP_PART = GP_COUNT;
template <int PARTS = 7>
GF_HD void beam_gp(const BeamConst& c, const BeamHist& h, const double* d, int g, double* o, int os) {
  d3 a, b, z;
  beam_gp_interp(c, d, g, a, b, z);
  d3 T[3];  // rows of T3
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) T[i][j] = c.T3[i * 3 + j];
  const double gq = 4.0 / radd(4.0, rdot(a, a));
  const double hg = rmul(0.5, gq);
  // y = Q_delta^T z' in the element frame, as z' plus its small rotation: the
  // strains eta = Q_i^T y - e3r cancel to the last bits of y, so y takes as few
  // roundings as it can
  d3 y;
  {
    const d3 al = rtmv(T, a), ul = rtmv(T, z), hz = {{h.dz[g][0], h.dz[g][1], h.dz[g][2]}};
    const d3 zl = {{radd(ul[0], hz[0]), radd(ul[1], hz[1]), radd(ul[2], hz[2])}};
    const d3 c1 = rcross(al, zl), c2 = rcross(al, c1), w = rmv(T, hz);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      y[i] = rfma(gq, rfma(0.5, c2[i], -c1[i]), zl[i]);
      z[i] = radd(z[i], w[i]);  // z' in the global frame
    }
  }
  const d3 beta = rxi(a, b, gq, -0.5);  // Xi^T b
  d3 Q[3];                              // columns of Q
  d3 kap, eta;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const d3 qi = {{h.Q[g][j], h.Q[g][3 + j], h.Q[g][6 + j]}};
    const d3 r = rmv(T, qi);  // column j of T3^T Q_i
    kap[j] = radd(rdot(r, beta), h.kap[g][j]);
    eta[j] = rdot(qi, y);
    const d3 c1 = rcross(a, r), c2 = rcross(a, c1);
#pragma unroll
    for (int i = 0; i < 3; ++i) Q[j][i] = rfma(gq, rfma(0.5, c2[i], c1[i]), r[i]);
  }
  // stress resultants (retro-rotated) and their spatial forms
  d3 nr, mr;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    nr[i] = rmul(c.Dd[i], rsub(eta[i], c.e3r[i]));
    mr[i] = rmul(c.Dd[3 + i], kap[i]);
  }
  mr[0] = rfma(c.D34, kap[1], mr[0]);
  mr[1] = rfma(c.D34, kap[0], mr[1]);
  const d3 n = rmv(Q, nr), m = rmv(Q, mr);
  // columns of Xi = g (I + A / 2)
  d3 X[3];
  {
    const d3 ha = {{rmul(hg, a[0]), rmul(hg, a[1]), rmul(hg, a[2])}};
    X[0] = {{gq, ha[2], -ha[1]}};
    X[1] = {{-ha[2], gq, ha[0]}};
    X[2] = {{ha[1], -ha[0], gq}};
  }
  // M00 = Q Dt Q^T; Y = skew(z) Xi, W = M00 Y; M02 = W - skew(n) Xi; the part
  // Y^T W of M22
  double m22[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if constexpr (PARTS & 1) {
    d3 DQ[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) DQ[j][i] = rmul(c.Dd[j], Q[j][i]);
    double s[6];
#pragma unroll
    for (int i = 0, x = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j, ++x) {
        s[x] = rfma(Q[2][i], DQ[2][j], rfma(Q[1][i], DQ[1][j], rmul(Q[0][i], DQ[0][j])));
        o[(GP_M00 + x) * os] = s[x];
      }
    d3 Y[3], W[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Y[j] = rcross(z, X[j]);
      W[j][0] = rfma(s[2], Y[j][2], rfma(s[1], Y[j][1], rmul(s[0], Y[j][0])));
      W[j][1] = rfma(s[4], Y[j][2], rfma(s[3], Y[j][1], rmul(s[1], Y[j][0])));
      W[j][2] = rfma(s[5], Y[j][2], rfma(s[4], Y[j][1], rmul(s[2], Y[j][0])));
      const d3 nx = rcross(n, X[j]);
#pragma unroll
      for (int i = 0; i < 3; ++i) o[(GP_M02 + 3 * i + j) * os] = rsub(W[j][i], nx[i]);
    }
#pragma unroll
    for (int i = 0, x = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j, ++x) {
        m22[x] = rdot(Y[i], W[j]);
        if constexpr (PARTS != 7) o[(GP_PART + x) * os] = m22[x];
      }
  }
  const double ab = rdot(a, b);
  const d3 mu = rxi(a, m, gq, -0.5);  // Xi^T m
  const d3 bm = rcross(b, m);
  const d3 w = {{rmul(-hg, mu[0]), rmul(-hg, mu[1]), rmul(-hg, mu[2])}};
  // R = Q^T Xi and S = Q^T dXi by rows; M11 = R^T Dr R, M12 = R^T Dr S + V^T,
  // the part S^T Dr S of M22
  if constexpr (PARTS & 2) {
    d3 R[3], S[3], DR[3], DS[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      R[i] = rtmv(X, Q[i]);
      const d3 tb = rcross(Q[i], b);
#pragma unroll
      for (int j = 0; j < 3; ++j) S[i][j] = rmul(-hg, rfma(ab, R[i][j], -tb[j]));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      DR[0][j] = rfma(c.D34, R[1][j], rmul(c.Dd[3], R[0][j]));
      DR[1][j] = rfma(c.D34, R[0][j], rmul(c.Dd[4], R[1][j]));
      DR[2][j] = rmul(c.Dd[5], R[2][j]);
      DS[0][j] = rfma(c.D34, S[1][j], rmul(c.Dd[3], S[0][j]));
      DS[1][j] = rfma(c.D34, S[0][j], rmul(c.Dd[4], S[1][j]));
      DS[2][j] = rmul(c.Dd[5], S[2][j]);
    }
    // V(a, m)^T = a w^T - g/2 skew(m)
    const d3 sm = {{rmul(hg, m[0]), rmul(hg, m[1]), rmul(hg, m[2])}};
    const double skew_m[9] = {0.0, -sm[2], sm[1], sm[2], 0.0, -sm[0], -sm[1], sm[0], 0.0};
#pragma unroll
    for (int i = 0, x = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double v = rfma(R[2][i], DS[2][j], rfma(R[1][i], DS[1][j], rmul(R[0][i], DS[0][j])));
        v = rfma(a[i], w[j], v);
        if (i != j) v = rsub(v, skew_m[3 * i + j]);
        o[(GP_M12 + 3 * i + j) * os] = v;
        if (j >= i) {
          o[(GP_M11 + x) * os] = rfma(R[2][i], DR[2][j], rfma(R[1][i], DR[1][j], rmul(R[0][i], DR[0][j])));
          const double y = rfma(S[2][i], DS[2][j], rfma(S[1][i], DS[1][j], rmul(S[0][i], DS[0][j])));
          if constexpr (PARTS == 7) m22[x] = radd(m22[x], y);
          else o[(GP_PART + 6 + x) * os] = y;
          ++x;
        }
      }
  }
  if constexpr (!(PARTS & 4)) return;
  // the geometric part of M22, its symmetric part:
  //   Xi^T skew(z) skew(n) Xi        = nu zeta^T - (z.n) (g I - (g/2)^2 a a^T)
  //   -V(a, z x n)                   = g/2 kappa a^T + antisymmetric
  //   dV(a, b, m)                    = c a^T + w b^T + antisymmetric
  //   -dXi^T skew(m) Xi              = g/2 (m beta^T - (b.m) Xi) + antisymmetric
  // with nu = Xi^T n, zeta = Xi^T z, kappa = Xi^T (z x n), c = g^2/2 (a.b) mu +
  // g^2/4 b x m
  const d3 nu = rxi(a, n, gq, -0.5), zeta = rxi(a, z, gq, -0.5), kx = rxi(a, rcross(z, n), gq, -0.5);
  {
    const double zn = rdot(z, n), bmd = rdot(b, m), g2 = rmul(hg, hg);  // g^2 / 4
    d3 p;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double ci = rmul(g2, rfma(rmul(2.0, ab), mu[i], bm[i]));
      p[i] = rfma(rmul(zn, g2), a[i], rfma(hg, kx[i], ci));
    }
    const double diag = rfma(gq, zn, rmul(rmul(gq, hg), bmd));
#pragma unroll
    for (int i = 0, x = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j, ++x) {
        // twice the symmetric part off the diagonal, halved at the end
        double v;
        if (i == j) {
          v = rfma(nu[i], zeta[i], rfma(p[i], a[i], rfma(w[i], b[i], rmul(rmul(hg, m[i]), beta[i]))));
          v = rsub(v, diag);
        } else {
          v = rfma(nu[i], zeta[j], rmul(nu[j], zeta[i]));
          v = rfma(p[i], a[j], rfma(p[j], a[i], v));
          v = rfma(w[i], b[j], rfma(w[j], b[i], v));
          v = rmul(0.5, rfma(rmul(hg, m[i]), beta[j], rfma(rmul(hg, m[j]), beta[i], v)));
        }
        if constexpr (PARTS == 7) o[(GP_M22 + x) * os] = radd(m22[x], v);
        else o[(GP_PART + 12 + x) * os] = v;
      }
  }
  // force terms (reference src/Beam_1.cpp:828): n, Xi^T m and Xi^T skew(z)^T n
  // + dXi^T m
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[(GP_N + i) * os] = n[i];
    o[(GP_S1 + i) * os] = mu[i];
    o[(GP_S2 + i) * os] = rsub(rmul(-hg, rfma(ab, mu[i], bm[i])), kx[i]);
  }
}

// Products of the Gauss weight and the shape functions of one point, from
// which K_e is expanded: w N' and w N per node, w N'_I N'_J and w N_I N_J for
// the node pairs I <= J (00, 01, 02, 11, 12, 22), w N'_I N_J for all.
constexpr int GC_WD = 0, GC_WN = 3, GC_DD = 6, GC_NN = 12, GC_DN = 18, GC_COUNT = 27;
GF_HD void beam_gp_coef(const BeamConst& c, int g, double* o, int os) {
  double wd[3], wn[3];
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    wd[I] = rmul(c.jac, c.dN[g][I]);
    wn[I] = rmul(c.jac, c.N[g][I]);
    o[(GC_WD + I) * os] = wd[I];
    o[(GC_WN + I) * os] = wn[I];
  }
#pragma unroll
  for (int I = 0, x = 0; I < 3; ++I)
#pragma unroll
    for (int J = 0; J < 3; ++J) {
      o[(GC_DN + 3 * I + J) * os] = rmul(wd[I], c.N[g][J]);
      if (J >= I) {
        o[(GC_DD + x) * os] = rmul(wd[I], c.dN[g][J]);
        o[(GC_NN + x) * os] = rmul(wn[I], c.N[g][J]);
        ++x;
      }
    }
}

// Coefficients of the translations written as du = u_2 - u_0 and v = u_1 - (u_0 +
// u_2) / 2, whose shape derivatives are N'_2 + N'_1 / 2 and N'_1: w D D, w D V, w
// V V, then w D N_J and w V N_J.
constexpr int GS_DD = 0, GS_DV = 1, GS_VV = 2, GS_DN = 3, GS_VN = 6, GS_COUNT = 9;
GF_HD void beam_gp_coef_sym(const BeamConst& c, int g, double* o, int os) {
  const double V = c.dN[g][1], D = rfma(0.5, V, c.dN[g][2]);
  const double wD = rmul(c.jac, D), wV = rmul(c.jac, V);
  o[GS_DD * os] = rmul(wD, D);
  o[GS_DV * os] = rmul(wD, V);
  o[GS_VV * os] = rmul(wV, V);
#pragma unroll
  for (int J = 0; J < 3; ++J) {
    o[(GS_DN + J) * os] = rmul(wD, c.N[g][J]);
    o[(GS_VN + J) * os] = rmul(wV, c.N[g][J]);
  }
}

// Index of entry (i, j), i <= j, of a 3x3 upper triangle, and of either order.
GF_HD int tri3(int i, int j) { return i <= j ? 3 * i - (i * (i - 1)) / 2 + j - i : 3 * j - (j * (j - 1)) / 2 + i - j; }

// Entries of K_e from the two points' stored values and coefficients (M and C
// hold point g at [g * gs], entries ms apart).  Translation-translation entry
// of nodes I <= J.
GF_HD double beam_k_uu(const double* M, const double* C, int gs, int ms, int pair, int x) {
  return rfma(C[gs + (GC_DD + pair) * ms], M[gs + (GP_M00 + x) * ms], rmul(C[(GC_DD + pair) * ms], M[(GP_M00 + x) * ms]));
}
// Translation i of node I against rotation j of node J.
GF_HD double beam_k_ua(const double* M, const double* C, int gs, int ms, int IJ, int x) {
  return rfma(C[gs + (GC_DN + IJ) * ms], M[gs + (GP_M02 + x) * ms], rmul(C[(GC_DN + IJ) * ms], M[(GP_M02 + x) * ms]));
}
// Rotation i of node I against rotation j of node J, I <= J.
GF_HD double beam_k_aa(const double* M, const double* C, int gs, int ms, int pair, int I, int J, int i, int j) {
  const int t = tri3(i, j), x = 3 * i + j, y = 3 * j + i;
  double v = rmul(C[(GC_DD + pair) * ms], M[(GP_M11 + t) * ms]);
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const double *m = M + g * gs, *c = C + g * gs;
    if (g) v = rfma(c[(GC_DD + pair) * ms], m[(GP_M11 + t) * ms], v);
    v = rfma(c[(GC_DN + 3 * I + J) * ms], m[(GP_M12 + x) * ms], v);
    v = rfma(c[(GC_DN + 3 * J + I) * ms], m[(GP_M12 + y) * ms], v);
    v = rfma(c[(GC_NN + pair) * ms], m[(GP_M22 + t) * ms], v);
  }
  return v;
}
// Entry of f_e: translation (rot 0) or rotation (1) component i of node I.
GF_HD double beam_f(const double* M, const double* C, int gs, int ms, int I, int rot, int i) {
  if (!rot)
    return rfma(C[gs + (GC_WD + I) * ms], M[gs + (GP_N + i) * ms], rmul(C[(GC_WD + I) * ms], M[(GP_N + i) * ms]));
  double v = rmul(C[(GC_WD + I) * ms], M[(GP_S1 + i) * ms]);
  v = rfma(C[(GC_WN + I) * ms], M[(GP_S2 + i) * ms], v);
  v = rfma(C[gs + (GC_WD + I) * ms], M[gs + (GP_S1 + i) * ms], v);
  return rfma(C[gs + (GC_WN + I) * ms], M[gs + (GP_S2 + i) * ms], v);
}

// The 162 distinct-form entries in three uniform loops: k of [0, 36) is a
// translation pair, of [0, 81) translation against rotation, of [0, 45) a
// rotation pair; (r, s) its place in K_e, r and s the element's DOFs.
GF_HD void beam_uu_place(int k, int& pair, int& x, int& I, int& J, int& i, int& j) {
  pair = k / 6;
  x = k % 6;
  I = pair < 3 ? 0 : (pair < 5 ? 1 : 2);
  J = pair < 3 ? pair : (pair < 5 ? pair - 2 : 2);
  i = x < 3 ? 0 : (x < 5 ? 1 : 2);
  j = x < 3 ? x : (x < 5 ? x - 2 : 2);
}
GF_HD void beam_aa_place(int k, int& pair, int& I, int& J, int& i, int& j) {
  if (k < 27) {  // node pairs 01, 02, 12: nine entries each
    const int q = k / 9, x = k % 9;
    pair = q == 0 ? 1 : (q == 1 ? 2 : 4);
    I = q == 2 ? 1 : 0;
    J = q == 0 ? 1 : 2;
    i = x / 3;
    j = x % 3;
  } else {  // the same node: six entries
    const int q = (k - 27) / 6, x = (k - 27) % 6;
    pair = q == 0 ? 0 : (q == 1 ? 3 : 5);
    I = J = q;
    i = x < 3 ? 0 : (x < 5 ? 1 : 2);
    j = x < 3 ? x : (x < 5 ? x - 2 : 2);
  }
}

}  // namespace gf
