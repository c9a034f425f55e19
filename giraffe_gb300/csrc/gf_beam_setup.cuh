// PreCalc of a Beam_1 element and its Gauss-point state in the reference's layout,
// on the host (structures) or on the device (many elements of one call).
#pragma once
#include <cmath>

#include "../../include/giraffe_gpu.h"
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

// Rows of the element frame from the coordinate system's E1, E3 (reference
// src/CoordinateSystem.cpp:68-92).
GF_HD void cs_rows(double* Q, const double* e1e3) {
  double e1[3] = {e1e3[0], e1e3[1], e1e3[2]}, e3[3] = {e1e3[3], e1e3[4], e1e3[5]};
  double e2[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
  auto nrm = [](const double* v) { return sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); };
  double n1 = nrm(e1), n2 = nrm(e2), n3 = nrm(e3);
  for (int k = 0; k < 3; ++k) {
    Q[k] = n1 != 1.0 ? e1[k] * (1.0 / n1) : e1[k];
    Q[3 + k] = n2 != 1.0 ? e2[k] * (1.0 / n2) : e2[k];
    Q[6 + k] = n3 != 1.0 ? e3[k] * (1.0 / n3) : e3[k];
  }
}

// Beam_1::PreCalc (reference src/Beam_1.cpp:501-692): end nodes x0, x2; Hooke
// material E, nu, rho; section A, I11, I22, I12, It, I33; CS rows E1, E3;
// pre-tension T0.
GF_HD void beam_precalc(const double* x0, const double* x2, const double* mat, const double* sec, const double* cs,
                  BeamConst& c, BeamHist& h, BeamHistAux& x, double T0 = 0.0) {
  c = BeamConst{};
  h = BeamHist{};
  x = BeamHistAux{};
  double E = mat[0], nu = mat[1], rho = mat[2];
  double G = E / (2 * (1 + nu));
  double sf = 1.0;
  double A = sec[0], I1 = sec[1], I2 = sec[2], I12 = sec[3], It = sec[4], I33 = sec[5];
  c.Dd[0] = sf * G * A;
  c.Dd[1] = sf * G * A;
  c.Dd[2] = E * A;
  c.Dd[3] = E * I1;
  c.Dd[4] = E * I2;
  c.Dd[5] = G * It;
  c.D34 = E * I12;
  c.Mr = rho * A;
  c.Jr[0] = rho * I1;
  c.Jr[4] = rho * I2;
  c.Jr[8] = rho * I33;
  c.Jr[1] = c.Jr[3] = rho * I12;
  cs_rows(c.T3, cs);
  double e3[3] = {x2[0] - x0[0], x2[1] - x0[1], x2[2] - x0[2]};
  double len = sqrt(e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2]);
  double inv = 1.0 / len;
  for (int k = 0; k < 3; ++k) e3[k] = inv * e3[k];
  for (int i = 0; i < 3; ++i) c.e3r[i] = c.T3[i * 3] * e3[0] + c.T3[i * 3 + 1] * e3[1] + c.T3[i * 3 + 2] * e3[2];
  // pre-strain of a pre-tension T0: the reference length is the distance of
  // the end nodes shortened by 1 + T0 / EA, and the Gauss points start
  // stretched (reference src/Beam_1.cpp:616-621)
  const double du0 = T0 / c.Dd[2];
  c.jac = (len / (1.0 + du0)) / 2.0;
  for (int g = 0; g < 2; ++g) {
    double xi = g == 0 ? -0.577350269189626 : +0.577350269189626;
    c.N[g][0] = 0.5 * xi * (xi - 1.0);
    c.N[g][1] = 1.0 - xi * xi;
    c.N[g][2] = 0.5 * xi * (1.0 + xi);
    c.dN[g][0] = (1.0 / c.jac) * (xi - 0.5);
    c.dN[g][1] = (1.0 / c.jac) * (-2.0 * xi);
    c.dN[g][2] = (1.0 / c.jac) * (0.5 + xi);
  }
  for (int g = 0; g < 2; ++g) {
    h.Q[g][0] = h.Q[g][4] = h.Q[g][8] = 1.0;
    h.dz[g][2] = 1.0 + du0;
  }
}

// Gauss-point state in the reference's layout (Q_i column-major there, row-major
// here).
GF_HD void beam_state_in(const double* L2, BeamHist& h, BeamHistAux& x) {
  for (int g = 0; g < 2; ++g) {
    const double* L = L2 + g * GF_BEAM_LAG;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) h.Q[g][3 * i + j] = L[i + 3 * j];
    for (int i = 0; i < 3; ++i) {
      x.alpha[g][i] = L[9 + i];
      h.kap[g][i] = L[12 + i];
      x.u[g][i] = L[15 + i];
      h.dz[g][i] = L[18 + i];
    }
  }
}

}  // namespace gf
