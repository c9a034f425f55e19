// Beam_1 element on the device, in the element frame: interpolation, the
// inertial terms and the Gauss-point commit (reference src/Beam_1.cpp:700-753,
// 1564-1638 (MountMass) and 1494-1506 (SaveLagrange)), FP64.  The tangent and
// the internal force are in gf_beam_gp.cuh.
#pragma once
#include "gf_beam_gp.cuh"
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

// Interpolated nodal increments at one Gauss point, local frame.
struct BeamInterp {
  V3<double> alpha, dalpha, u, du;
};

// reference src/Beam_1.cpp:700-746
GF_HD BeamInterp beam_interp(const BeamConst& c, const double* d, int g) {
  const double* N = c.N[g];
  const double* dN = c.dN[g];
  V3<double> a, da, u, du;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    a[i] = d[3 + i] * N[0] + d[9 + i] * N[1] + d[15 + i] * N[2];
    da[i] = d[3 + i] * dN[0] + d[9 + i] * dN[1] + d[15 + i] * dN[2];
    u[i] = d[i] * N[0] + d[6 + i] * N[1] + d[12 + i] * N[2];
    du[i] = d[i] * dN[0] + d[6 + i] * dN[1] + d[12 + i] * dN[2];
  }
  M3<double> T;
#pragma unroll
  for (int i = 0; i < 9; ++i) T[i] = c.T3[i];
  BeamInterp r;
  r.alpha = mv(T, a);
  r.dalpha = mv(T, da);
  r.u = mv(T, u);
  r.du = mv(T, du);
  return r;
}

// Q_delta and Xi of the incremental rotation (reference src/Beam_1.cpp:748-753)
GF_HD void beam_rot(const V3<double>& alpha, double& g, M3<double>& Qd, M3<double>& Xi) {
  double n2 = dot(alpha, alpha);
  g = 4.0 / (4.0 + n2);
  M3<double> A = skew(alpha), A2 = mul(A, A);
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    Qd[i] = g * (A[i] + 0.5 * A2[i]);
    Xi[i] = g * 0.5 * A[i];
  }
  Qd[0] += 1.0; Qd[4] += 1.0; Qd[8] += 1.0;
  Xi[0] += g; Xi[4] += g; Xi[8] += g;
}

// Inertial contribution of one Gauss point (Beam_1::MountMass, reference
// src/Beam_1.cpp:1564-1638, Hooke sections: no offset of the mass centre).
// With Newmark coefficients a[0..5] = a1..a6:
//   dT_u = Mr (a1 du - a2 v_i - a3 acc_i)
//   dT_a = Xi(da) h,  h = J_i w2 + w1 x J_i w1,  J_i = Q(alpha_i) Jr Q(alpha_i)^T,
//   w1 = a4 da + a5 w_i + a6 dw_i,  w2 = a1 da - a2 w_i - a3 dw_i
// (Newmark in the tangent space transported by Q_delta, and Xi^T Q_delta = Xi
// for Rodrigues parameters), and the exact tangent
//   d dT_u/d du = a1 Mr I,
//   d dT_a/d da = Xi (a1 J_i + a4 (skew(w1) J_i - skew(J_i w1)))
//                 - g^2/2 (h + da x h / 2) da^T - g/2 skew(h).
// All in the global frame, the element frame entering through T3^T Q(alpha_i), and
// J_i symmetric: about 330 operations against 560 in the element frame with its
// rotations.  d: the nodal increments.  Returns dT_u and dT_a (fu[i * ds], fa[i *
// ds]; the element force is their sum with wJ N_I) and the rotational tangent in
// Daa[q * ds]; the translational tangent is a1 Mr I.
GF_HD void beam_gp_inertia(const BeamConst& c, const BeamHistAux& x, const double* d, const double* vel,
                           const double* acc, const double* a, int g, double* fu_out, double* fa_out, double* Daa,
                           int ds) {
  const double N0 = c.N[g][0], N1 = c.N[g][1], N2 = c.N[g][2];
  const double a1 = a[0], a2 = a[1], a3 = a[2], a4 = a[3], a5 = a[4], a6 = a[5];
  d3 al, w1, w2;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    auto at = [&](const double* v, int k) { return fma(v[12 + k], N2, fma(v[6 + k], N1, v[k] * N0)); };
    fu_out[i * ds] = c.Mr * fma(-a3, at(acc, i), fma(-a2, at(vel, i), a1 * at(d, i)));
    const double wi = at(vel, 3 + i), dwi = at(acc, 3 + i);
    al[i] = at(d, 3 + i);
    w1[i] = fma(a6, dwi, fma(a5, wi, a4 * al[i]));
    w2[i] = fma(-a3, dwi, fma(-a2, wi, a1 * al[i]));
  }
  // J = R Jr R^T with R = T3^T Q(alpha_i): Jr has the two bending inertias and their
  // product, and the polar one
  d3 J[3];  // columns
  {
    M3<double> T;
#pragma unroll
    for (int i = 0; i < 9; ++i) T[i] = c.T3[i];
    const M3<double> Q = rodrigues(V3<double>{{x.alpha[g][0], x.alpha[g][1], x.alpha[g][2]}});
    d3 R[3], S[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) R[j] = tmv(T, d3{{Q[j], Q[3 + j], Q[6 + j]}});
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      S[0][i] = fma(c.Jr[3], R[1][i], c.Jr[0] * R[0][i]);
      S[1][i] = fma(c.Jr[4], R[1][i], c.Jr[1] * R[0][i]);
      S[2][i] = c.Jr[8] * R[2][i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        const double v = fma(S[2][i], R[2][j], fma(S[1][i], R[1][j], S[0][i] * R[0][j]));
        J[j][i] = v;
        J[i][j] = v;
      }
  }
  const d3 Jw1 = rmv(J, w1), Jw2 = rmv(J, w2), cr = rcross(w1, Jw1);
  const d3 h = {{Jw2[0] + cr[0], Jw2[1] + cr[1], Jw2[2] + cr[2]}};
  const double gg = 4.0 / (4.0 + dot(al, al)), hg = 0.5 * gg;
  const d3 m = rxi(al, h, gg, 0.5), axh = rcross(al, h);
  d3 p;  // -g^2/2 (h + da x h / 2)
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    fa_out[i * ds] = m[i];
    p[i] = -hg * gg * fma(0.5, axh[i], h[i]);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const d3 t = rcross(w1, J[j]);
    // columns j of skew(J w1) and skew(h)
    const d3 sj = j == 0 ? d3{{0.0, Jw1[2], -Jw1[1]}} : j == 1 ? d3{{-Jw1[2], 0.0, Jw1[0]}} : d3{{Jw1[1], -Jw1[0], 0.0}};
    const d3 sh = j == 0 ? d3{{0.0, h[2], -h[1]}} : j == 1 ? d3{{-h[2], 0.0, h[0]}} : d3{{h[1], -h[0], 0.0}};
    d3 col;
#pragma unroll
    for (int i = 0; i < 3; ++i) col[i] = fma(a4, i == j ? t[i] : t[i] - sj[i], a1 * J[j][i]);
    const d3 y = rxi(al, col, gg, 0.5);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double v = fma(p[i], al[j], y[i]);
      Daa[(3 * i + j) * ds] = i == j ? v : fma(-hg, sh[i], v);
    }
  }
}

// Inertial tangent entry (row r, column s of the 18x18, global frame).
GF_HD double beam_M_entry(const BeamConst& c, const double* D0, const double* D1, int ds, double a1Mr, int r, int s) {
  int I = r / 6, a = r % 6, J = s / 6, b = s % 6;
  double acc = 0.0;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    double w = c.jac * c.N[g][I] * c.N[g][J];
    if (a < 3 && b < 3) {
      if (a == b) acc += w * a1Mr;
    } else if (a >= 3 && b >= 3) {
      const double* D = g ? D1 : D0;
      acc += w * D[((a - 3) * 3 + (b - 3)) * ds];
    }
  }
  return acc;
}

// SaveLagrange of one Gauss point (reference src/Beam_1.cpp:1494-1506)
GF_HD void beam_commit(const BeamConst& c, BeamHist& h, BeamHistAux& x, const double* d, int g) {
  BeamInterp ip = beam_interp(c, d, g);
  double gg;
  M3<double> Qd, Xi;
  beam_rot(ip.alpha, gg, Qd, Xi);
  M3<double> Qi;
#pragma unroll
  for (int i = 0; i < 9; ++i) Qi[i] = h.Q[g][i];
  M3<double> Q = mul(Qd, Qi);
  // kappa_r (reference src/Beam_1.cpp:785) recomputed for the history
  V3<double> t = tmv(Xi, ip.dalpha);
  V3<double> kap = tmv(Qi, t);
#pragma unroll
  for (int i = 0; i < 9; ++i) h.Q[g][i] = Q[i];
  V3<double> ai = {{x.alpha[g][0], x.alpha[g][1], x.alpha[g][2]}};
  V3<double> an = rodrigues_compose(ip.alpha, ai);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    x.u[g][i] += ip.u[i];
    h.kap[g][i] = kap[i] + h.kap[g][i];
    h.dz[g][i] = ip.du[i] + h.dz[g][i];
    x.alpha[g][i] = an[i];
  }
}

}  // namespace gf
