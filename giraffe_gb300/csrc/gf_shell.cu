// Shell_1 structures on the device: element tangent and internal force with
// the follower pressure and, in Dynamic steps, the inertial terms
// (k_shell_mount, on the Gauss points of gf_shell_gp.cuh), Rayleigh damping
// (k_shell_rayleigh), the forces into P (k_shell_gather_f; k_shell_scatter with a band) and
// SaveLagrange (k_shell_commit; reference src/Shell_1.cpp:1650-1664).  The LU of
// the assembled operator is in gf_front.cu.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <vector>

#include "gf_kernels.cuh"
#include "gf_math.cuh"
#include "gf_shell_gp.cuh"
#include "gf_types.h"

namespace gf {

namespace {

__device__ __forceinline__ bool iterating_s(const StructState& s) { return s.phase == PH_ITER; }

typedef V3<double> v3;
typedef M3<double> m3;

struct SGp {
  v3 u, u1, u2, al, al1, al2;
  double g;
  m3 Xi, Xi1, Xi2, Q;
  v3 z1, z2, eta1, eta2, k1, k2;
};

// Gauss-point kinematics of the increment d (27, element DOF order, global).
__device__ void shell_gp(const ShellConst& c, const ShellHist& h, const double* d, int g, SGp& k) {
  v3 ug = {{0, 0, 0}}, u1g = {{0, 0, 0}}, u2g = {{0, 0, 0}}, ag = {{0, 0, 0}}, a1g = {{0, 0, 0}},
     a2g = {{0, 0, 0}};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      ug[j] += d[3 * n + j] * c.Nu[g][n];
      u1g[j] += d[3 * n + j] * c.Nu1[g][n];
      u2g[j] += d[3 * n + j] * c.Nu2[g][n];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      ag[j] += d[18 + 3 * m + j] * c.Na[g][m];
      a1g[j] += d[18 + 3 * m + j] * c.Na1[g][m];
      a2g[j] += d[18 + 3 * m + j] * c.Na2[g][m];
    }
  }
  m3 T;
#pragma unroll
  for (int q = 0; q < 9; ++q) T[q] = c.T3[q];
  k.u = mv(T, ug);
  k.u1 = mv(T, u1g);
  k.u2 = mv(T, u2g);
  k.al = mv(T, ag);
  k.al1 = mv(T, a1g);
  k.al2 = mv(T, a2g);
  double an2 = dot(k.al, k.al);
  k.g = 4.0 / (4.0 + an2);
  m3 A = skew(k.al), A2 = mul(A, A), Qd;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    Qd[q] = k.g * (A[q] + 0.5 * A2[q]);
    k.Xi[q] = k.g * 0.5 * A[q];
  }
  Qd[0] += 1.0; Qd[4] += 1.0; Qd[8] += 1.0;
  k.Xi[0] += k.g; k.Xi[4] += k.g; k.Xi[8] += k.g;
  m3 S1 = skew(k.al1), S2 = skew(k.al2);
  double p1 = dot(k.al, k.al1), p2 = dot(k.al, k.al2);
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    k.Xi1[q] = -0.5 * k.g * (p1 * k.Xi[q] - S1[q]);
    k.Xi2[q] = -0.5 * k.g * (p2 * k.Xi[q] - S2[q]);
  }
  m3 Qi;
#pragma unroll
  for (int q = 0; q < 9; ++q) Qi[q] = h.Q[g][q];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    k.z1[j] = k.u1[j] + h.z1[g][j];
    k.z2[j] = k.u2[j] + h.z2[g][j];
  }
  k.Q = mul(Qd, Qi);
  k.eta1 = tmv(k.Q, k.z1);
  k.eta2 = tmv(k.Q, k.z2);
  k.eta1[0] -= 1.0;
  k.eta2[1] -= 1.0;
  m3 XQ = mul(k.Xi, Qi);
  k.k1 = tmv(XQ, k.al1);
  k.k2 = tmv(XQ, k.al2);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    k.k1[j] += h.k1[g][j];
    k.k2[j] += h.k2[g][j];
  }
}

__device__ __forceinline__ void gather_d(const Batch& b, int e, double* d) {
  const int* nd = b.sh.snodes + 6 * e;
#pragma unroll
  for (int a = 0; a < 18; ++a) d[a] = b.disp[(int64_t)nd[a / 3] * 6 + a % 3];
#pragma unroll
  for (int a = 0; a < 9; ++a) d[18 + a] = b.disp[(int64_t)nd[3 + a / 3] * 6 + 3 + a % 3];
}

__device__ __forceinline__ m3 ld3(const double* p) {
  m3 r;
#pragma unroll
  for (int q = 0; q < 9; ++q) r[q] = p[q];
  return r;
}

// Table::GetValueAt (reference src/Table.cpp:73-102), first column:
// clamped outside the table, linear between the rows that bracket time.
__device__ __forceinline__ double table_value(const Batch& b, int t, double time) {
  const TableDev T = b.tables[t];
  const double* times = b.table_data + T.off;
  const double* vals = times + T.n_times;
  if (T.n_times == 0) return 0.0;
  if (time >= times[T.n_times - 1]) return vals[(int64_t)(T.n_times - 1) * T.n_cols];
  if (time <= times[0]) return vals[0];
  const int idx = table_row(T, times, time);
  double f = (time - times[idx - 1]) / (times[idx] - times[idx - 1]);
  double a = vals[(int64_t)(idx - 1) * T.n_cols], c = vals[(int64_t)idx * T.n_cols];
  return a + f * (c - a);
}

}  // namespace

// ---- tangent and internal force ----
// Ten elements per CTA of four warps.  The warps first take a part of each Gauss
// point (lane g 10 + e: derivative blocks, rotation column, its geometric part,
// pressure points and inertia), about 1,000 FP64 operations each and the chain a
// small mesh waits for; then the columns of K_e, a node block at a time (lane j 10 +
// e), the rows not above it and their transposes written together, the node
// blocks dealt out so that the warps' shares agree within 5 %.  Bound by the FP64
// pipe.  A thread per element formed the same in 32,000 operations, 1.7 ms a pass
// for 50 or 8,192 elements; with the scatter's launches 0.08 and 0.24 ms here.
constexpr int ST_E = 10, ST_THREADS = 128, ST_S = 32, ST_C = sizeof(ShellConst) / 8 + 1;
constexpr int ST_M = 0, ST_G = ST_M + SP_COUNT * ST_S, ST_P = ST_G,  // the pressure blocks take the place of G
    ST_Q = ST_P + 324 * ST_E, ST_I = ST_Q + SQ_COUNT * ST_S, ST_PT = ST_I + SI_COUNT * ST_S,
              ST_D = ST_PT + PP_COUNT * 6 * ST_E, ST_PU = ST_D + 27 * ST_E, ST_CS = ST_PU + 18 * ST_E,
              ST_SIZE = ST_CS + ST_C * ST_E;
static_assert(SG_COUNT * ST_S <= 324 * ST_E && sizeof(ShellConst) % 8 == 0, "");

// The elements of a batch's iterating structures: Mount, MountElementLoads and the
// element's ShellLoad at the step's time, and in Dynamic steps the inertia.
struct ShellBatchSrc {
  Batch b;
  __device__ int count() const { return b.sh.n_shells; }
  __device__ bool active(int e) const { return iterating_s(b.state[b.sh.sstruct[e]]); }
  __device__ const ShellConst& cst(int e) const { return b.sh.sconst[e]; }
  __device__ const ShellHist& hist(int e) const { return b.sh.shist[e]; }
  __device__ const ShellHistAux& aux(int e) const { return b.sh.saux[e]; }
  __device__ double disp(int e, int x) const {
    const int* nd = b.sh.snodes + 6 * e;
    return x < 18 ? b.disp[(int64_t)nd[x / 3] * 6 + x % 3] : b.disp[(int64_t)nd[3 + (x - 18) / 3] * 6 + 3 + x % 3];
  }
  __device__ double total(int e, int x, double d) const {
    const int64_t q = (int64_t)b.sh.snodes[6 * e + x / 3] * 6 + x % 3;
    return b.copy[q] - b.xref[q] + d;  // xref: reference positions, 6 per node
  }
  __device__ bool pressed(int e) const { return b.sh.spress[e] >= 0; }
  __device__ double pressure(int e) const {
    return table_value(b, b.sh.spress[e], b.state[b.sh.sstruct[e]].time);
  }
  __device__ bool area(int e) const { return b.sh.sarea[e] != 0; }
  __device__ bool dynamic(int e) const { return b.params[b.sh.sstruct[e]].dynamic; }
  // Rayleigh damping: on the iterations that form C_e, the stiffness (with the
  // pressure tangent, as MountLoads precedes MountDamping) goes to the damping
  // scratch, where k_shell_rayleigh turns it into C_e = alpha M_modal + beta K_e
  __device__ double* damping(int e) const {
    const StructParams& pr = b.params[b.sh.sstruct[e]];
    return pr.dynamic && pr.ray_on && (pr.ray_update || !b.state[b.sh.sstruct[e]].ray_init) ? b.sh.RD + e : nullptr;
  }
  __device__ const double* newmark(int e) const { return b.state[b.sh.sstruct[e]].a; }
  __device__ void inertia(int e, const ShellConst& c, const double* d, int ds, int g, double* o, int os) const {
    const int* nd = b.sh.snodes + 6 * e;
    shell_inertia_point(c, aux(e), d, ds, b.copy_vel, b.copy_accel, [nd](int n) { return (int64_t)nd[n] * 6; },
                        newmark(e), g, o, os);
  }
  __device__ double* K(int e) const { return b.sh.Ke + (int64_t)e * 729; }
  __device__ double* F(int e) const { return b.sh.Fe + (int64_t)e * 27; }
};

// Standalone elements (gf_shell_elements): n elements with their own constants,
// history and increments d ([n][27]); with pressure p[e] (NaN: none) at the
// displacement pu ([n][18]).
struct ShellElemSrc {
  int n, area_update;
  const ShellConst* cs;
  const ShellHist* hs;
  const double *ds, *pus, *ps;
  double *Ks, *fs;
  __device__ int count() const { return n; }
  __device__ bool active(int) const { return true; }
  __device__ const ShellConst& cst(int e) const { return cs[e]; }
  __device__ const ShellHist& hist(int e) const { return hs[e]; }
  __device__ double disp(int e, int x) const { return ds[(int64_t)e * 27 + x]; }
  __device__ double total(int e, int x, double) const { return pus[(int64_t)e * 18 + x]; }
  __device__ bool pressed(int e) const { return ps[e] == ps[e]; }
  __device__ double pressure(int e) const { return ps[e]; }
  __device__ bool area(int) const { return area_update != 0; }
  __device__ bool dynamic(int) const { return false; }
  __device__ double* damping(int) const { return nullptr; }
  __device__ const double* newmark(int) const { return nullptr; }
  __device__ void inertia(int, const ShellConst&, const double*, int, int, double*, int) const {}
  __device__ double* K(int e) const { return Ks + (int64_t)e * 729; }
  __device__ double* F(int e) const { return fs + (int64_t)e * 27; }
};

template <class Src> __global__ void __launch_bounds__(ST_THREADS) k_shell_mount(Src src) {
  extern __shared__ __align__(16) double st_sh[];
  double *M = st_sh + ST_M, *G = st_sh + ST_G, *P = st_sh + ST_P, *Q = st_sh + ST_Q, *I = st_sh + ST_I,
         *PT = st_sh + ST_PT, *D = st_sh + ST_D, *PU = st_sh + ST_PU, *CS = st_sh + ST_CS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, le = lane % ST_E, lj = lane / ST_E;
  const int e0 = blockIdx.x * ST_E, ne = min(ST_E, src.count() - e0), e = e0 + le;
  const bool live = lj < 3 && le < ne && src.active(e);
  if (!__syncthreads_or(live)) return;
  const double* cs0 = reinterpret_cast<const double*>(&src.cst(e0));
  for (int x = tid; x < ne * (ST_C - 1); x += ST_THREADS) {
    const int q = x / (ST_C - 1), y = x - q * (ST_C - 1);
    CS[q * ST_C + y] = cs0[x];
  }
  for (int x = tid; x < 27 * ST_E; x += ST_THREADS) {
    const int y = x / ST_E, q = x % ST_E;
    if (q >= ne) continue;
    const double v = src.disp(e0 + q, y);
    D[x] = v;
    if (y < 18 && src.pressed(e0 + q)) PU[x] = src.total(e0 + q, y, v);
  }
  __syncthreads();
  const ShellConst& c = *reinterpret_cast<const ShellConst*>(CS + le * ST_C);
  const bool pressed = live && src.pressed(e), dyn = live && src.dynamic(e), area = pressed && src.area(e);
  const int slot = lj * ST_E + le;
  if (live) {
    if (warp == 0) {
      shell_part0(c, src.hist(e), D + le, ST_E, lj, M + slot, Q + slot, ST_S);
    } else if (warp == 1) {
      shell_part1(c, src.hist(e), D + le, ST_E, lj, M + slot, ST_S);
    } else if (warp == 2) {
      shell_part2(c, src.hist(e), D + le, ST_E, lj, G + slot, Q + slot, ST_S);
    } else {
      if (pressed) {
        const double p = src.pressure(e);
#pragma unroll 1
        for (int kq = lj; kq < 6; kq += 3)
          shell_press_point(c, PU + le, ST_E, p, area, kq, PT + kq * ST_E + le, 6 * ST_E);
      }
      if (dyn) src.inertia(e, c, D + le, ST_E, lj, I + slot, ST_S);
    }
  }
  __syncthreads();
  if (live)
    for (int x = warp; x < SG_COUNT; x += 4)
      M[((x < SG_D4 ? SP_M04 : SP_D4 - SG_D4) + x) * ST_S + slot] += G[x * ST_S + slot];
  if (__syncthreads_or(pressed)) {
    for (int nb = warp; nb < 6; nb += 4)
      if (pressed) shell_press_cols(c, PT + le, 6 * ST_E, ST_E, area, nb, lj, P + le * 324);
    __syncthreads();
  }
  if (!live) return;
  double *K = src.K(e), *F = src.F(e), *C = src.damping(e);
  const int64_t ns = src.count();
  const double a1m = dyn ? src.newmark(e)[0] * c.coef1 : 0.0;
  auto put = [&](int x, double v, double inertia) {
    if (C) C[x * ns] = v;
    K[x] = v + inertia;
  };
  // the node blocks of this warp: midside rotation 0, 1 or 2 and translation 5, 4
  // or 3, or translations 0, 1, 2 (324 + 54, 297 + 72, 270 + 90, 144 + 126 + 108
  // operations)
#pragma unroll 1
  for (int t = 0; t < (warp == 3 ? 3 : 2); ++t) {
    const int m = warp == 3 ? t : (t ? 5 - warp : 6 + warp);
    double acc[9][3], f;
    if (m >= 6) {
      const int r = m - 6;
      shell_col_rot(c, M + le, Q + le, ST_E, ST_S, r, lj, acc, f);
      double w[3][3];  // alpha1 Na_r Na_n of the points
      if (dyn) {
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          const double x = c.alpha1 * c.Na[g][r];
          f = fma(x, I[(SI_FA + lj) * ST_S + g * ST_E + le], f);
#pragma unroll
          for (int n = 0; n < 3; ++n) w[n][g] = x * c.Na[g][n];
        }
      }
#pragma unroll
      for (int n = 0; n < 6; ++n)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          put(3 * n + i + 27 * (3 * m + lj), acc[n][i], 0.0);
          put(3 * m + lj + 27 * (3 * n + i), acc[n][i], 0.0);
        }
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        if (n < r) continue;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          double v = 0.0, u = 0.0;
          if (dyn) {
#pragma unroll
            for (int g = 0; g < 3; ++g) {
              v = fma(w[n][g], I[(SI_D + 3 * i + lj) * ST_S + g * ST_E + le], v);
              u = fma(w[n][g], I[(SI_D + 3 * lj + i) * ST_S + g * ST_E + le], u);
            }
          }
          put(18 + 3 * n + i + 27 * (3 * m + lj), acc[6 + n][i], v);
          if (n != r) put(3 * m + lj + 27 * (18 + 3 * n + i), acc[6 + n][i], u);
        }
      }
    } else {
      shell_col_tr(c, M + le, Q + le, ST_E, ST_S, m, lj, acc, f);
      const double* p = P + le * 324;
      if (pressed) {
#pragma unroll
        for (int kq = 0; kq < 6; ++kq) f = fma(c.N4[kq][m], PT[(PP_F + lj) * 6 * ST_E + kq * ST_E + le], f);
      }
      if (dyn) {
#pragma unroll
        for (int g = 0; g < 3; ++g) f = fma(c.alpha1 * c.Nu[g][m], I[(SI_FU + lj) * ST_S + g * ST_E + le], f);
      }
#pragma unroll
      for (int n = 0; n < 6; ++n) {
        if (n < m) continue;
        double w = 0.0;
        if (dyn) {
#pragma unroll
          for (int g = 0; g < 3; ++g) w = fma(c.alpha1 * c.Nu[g][m], c.Nu[g][n], w);
          w *= a1m;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          double v = acc[n][i], u = v;
          if (pressed) {
            v += p[(6 * n + m) * 9 + 3 * i + lj];
            u += p[(6 * m + n) * 9 + 3 * lj + i];
          }
          const double x = i == lj ? w : 0.0;
          put(3 * n + i + 27 * (3 * m + lj), v, x);
          if (n != m) put(3 * m + lj + 27 * (3 * n + i), u, x);
        }
      }
    }
    F[3 * m + lj] = f;
  }
}

template <class Src> static void launch_mount(const Src& src, int n, cudaStream_t st) {
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_shell_mount<Src>, ST_SIZE * 8}});
  k_shell_mount<Src><<<(n + ST_E - 1) / ST_E, ST_THREADS, ST_SIZE * 8, st>>>(src);
}

// MountDamping and the damping part of MountDyn (reference
// src/Shell_1.cpp:2501-2541).  On the iterations that form it (the step's
// first, or every one with Update 1), C_e = alpha M_modal + beta K_e.  The
// modal mass is MountMassModal (src/Shell_1.cpp:2368-2396) over the
// six-point rule: at each point the rotation vector interpolated from the
// midside nodes' accumulated rotations (copy_coordinates 3..5) gives the
// director d = Q e3r, and EvaluateMassModal (src/Shell_1.cpp:3171-) the
// 6x6 operator blockdiag(coef1 I, coef2 (|d|^2 I - d d^T) + coef3 d d^T);
// the element sums w N^T D N and turns it to the global frame.  Every
// iteration then adds a4 C_e to K_e and C_e v to f_e, v the nodes' current
// velocities.  One warp per element, lane r < 27 owning row r of C_e, K_e
// and f_e (no lane reads another's row); C_e is structure-of-arrays.
// Row r of element e's modal mass (MountMassModal over the six-point rule,
// reference src/Shell_1.cpp:2368-2396, 3171-), global frame, into row[27].
__device__ void shell_modal_row(const Batch& b, int e, int r, double* row) {
  const ShellConst& c = b.sh.sconst[e];
  const int* nd = b.sh.snodes + 6 * e;
  const int n = r / 3, i = r % 3;  // row block (node 0..5 translations, 6..8 midside rotations), row in it
#pragma unroll
  for (int x = 0; x < 27; ++x) row[x] = 0.0;
  if (n < 6) {
    // translations: coef1 times the weights on the diagonal of each 3x3
    // node block (T^T I T = I)
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
      double w = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) w += c.w4[k] * c.N4[k][n] * c.N4[k][q];
      row[3 * q + i] = c.coef1 * w;
    }
  } else {
    // rotations of midside node m: row i of T^T R[m][q] T for q = 0..2
    const int m = n - 6;
    const m3 T = ld3(c.T3);
    double R[3][9];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int x = 0; x < 9; ++x) R[q][x] = 0.0;
#pragma unroll 1
    for (int k = 0; k < 6; ++k) {
      v3 al = {{0, 0, 0}};
#pragma unroll
      for (int mm = 0; mm < 3; ++mm)
#pragma unroll
        for (int j = 0; j < 3; ++j) al[j] += b.copy[(int64_t)nd[3 + mm] * 6 + 3 + j] * c.Na4[k][mm];
      al = mv(T, al);
      const m3 Q = rodrigues(al);
      const v3 dv = {{Q[2], Q[5], Q[8]}};
      const double d2 = dot(dv, dv);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const double w = c.w4[k] * c.Na4[k][m] * c.Na4[k][q];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            R[q][a * 3 + j] += w * ((a == j ? c.coef2 * d2 : 0.0) + (c.coef3 - c.coef2) * dv[a] * dv[j]);
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      m3 Rq;
#pragma unroll
      for (int x = 0; x < 9; ++x) Rq[x] = R[q][x];
      const m3 G = tmul(T, mul(Rq, T));
#pragma unroll
      for (int j = 0; j < 3; ++j) row[18 + 3 * q + j] = G[i * 3 + j];
    }
  }
}

__global__ void __launch_bounds__(128) k_shell_rayleigh(Batch b) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int r = threadIdx.x & 31;
  if (e >= b.sh.n_shells || r >= 27) return;
  const int s = b.sh.sstruct[e];
  const StructState& st = b.state[s];
  if (!iterating_s(st)) return;
  const StructParams& p = b.params[s];
  if (!p.dynamic || !p.ray_on) return;
  const int64_t ns = b.sh.n_shells;
  double* C = b.sh.RD + e;
  const int* nd = b.sh.snodes + 6 * e;
  if (p.ray_update || !st.ray_init) {
    double row[27];
    shell_modal_row(b, e, r, row);
#pragma unroll 1
    for (int x = 0; x < 27; ++x) {
      const int64_t xi = r + 27 * x;
      C[xi * ns] = p.ray_alpha * row[x] + p.ray_beta * C[xi * ns];
    }
  }
  const double a4 = st.a[3];
  double* K = b.sh.Ke + (int64_t)e * 729;
  double acc = 0.0;
#pragma unroll 1
  for (int x = 0; x < 27; ++x) {
    const int node = x < 18 ? nd[x / 3] : nd[3 + (x - 18) / 3];
    const int k = x < 18 ? x % 3 : 3 + (x - 18) % 3;
    const double cx = C[(int64_t)(r + 27 * x) * ns];
    acc += cx * b.vel[(int64_t)node * 6 + k];
    K[r + 27 * x] += a4 * cx;
  }
  b.sh.Fe[(int64_t)e * 27 + r] += acc;
}

// The modal mass of every Shell_1 element of colour class `color` added into
// the band M (entry (i, j) at (kw + i - j) + j W, free indices of b.gl):
// one thread per element, elements of a colour share no node.
__global__ void k_modal_mass_shell(Batch b, int color, double* M, int64_t W, int kw) {
  const int k = b.sh.color_off[color] + blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.sh.color_off[color + 1]) return;
  const int e = b.sh.color_elems[k];
  const int* nd = b.sh.snodes + 6 * e;
  int g[27];
#pragma unroll 1
  for (int x = 0; x < 27; ++x) {
    const int node = x < 18 ? nd[x / 3] : nd[3 + (x - 18) / 3];
    g[x] = b.gl[(int64_t)node * 6 + (x < 18 ? x % 3 : 3 + (x - 18) % 3)];
  }
#pragma unroll 1
  for (int r = 0; r < 27; ++r) {
    if (g[r] < 0) continue;
    double row[27];
    shell_modal_row(b, e, r, row);
#pragma unroll 1
    for (int x = 0; x < 27; ++x)
      if (g[x] >= 0 && abs(g[r] - g[x]) <= kw) M[(kw + g[r] - g[x]) + (int64_t)g[x] * W] += row[x];
  }
}

void launch_shell_modal_mass(const Batch& b, double* M, int64_t W, int kw, cudaStream_t st) {
  for (int c = 0; c < b.sh.n_colors; ++c) {
    const int cnt = b.sh.color_off[c + 1] - b.sh.color_off[c];
    if (cnt > 0) k_modal_mass_shell<<<(cnt + 63) / 64, 64, 0, st>>>(b, c, M, W, kw);
  }
}

// MountGlobal: one warp per element of one colour (no two elements of a
// colour share a node, so no two writers meet).  The element's free DOFs
// (structure-local, in the structure's reverse Cuthill-McKee numbering) go
// to the wide band (where one is kept) and to P.
__global__ void k_shell_scatter(Batch b, int color) {
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int lo = b.sh.color_off[color], hi = b.sh.color_off[color + 1];
  if (lo + w >= hi) return;
  int e = b.sh.color_elems[lo + w];
  int s = b.sh.sstruct[e];
  if (!iterating_s(b.state[s])) return;
  const StructInfo& inf = b.info[s];
  const int* nd = b.sh.snodes + 6 * e;
  int myg = -1;
  if (lane < 27) {
    int node = lane < 18 ? nd[lane / 3] : nd[3 + (lane - 18) / 3];
    int k = lane < 18 ? lane % 3 : 3 + (lane - 18) % 3;
    myg = b.gl[(int64_t)node * 6 + k];
  }
  const double* K = b.sh.Ke + (int64_t)e * 729;
  const double* F = b.sh.Fe + (int64_t)e * 27;
  if (lane < 27 && myg >= 0) b.P[inf.dof_off + myg] += F[lane];
  double* band = b.sh.wband + inf.wb_off;
  const int kl = inf.wkl;
  const int64_t W = 2 * kl + 1;
  for (int base = 0; base < 729; base += 32) {
    int idx = base + lane;
    bool valid = idx < 729;
    int r = valid ? idx % 27 : 0, q = valid ? idx / 27 : 0;
    int gr = __shfl_sync(0xffffffffu, myg, r);
    int gq = __shfl_sync(0xffffffffu, myg, q);
    if (valid && gr >= 0 && gq >= 0) band[(kl + gr - gq) + (int64_t)gq * W] += K[idx];
  }
}

// The forces alone, where K_AA is not asked for: a thread per node DOF adds its
// elements' in colour order, so P has the colour scatter's bits in one launch (for 7
// of 3.3 us on the 24x24x2 plate).
__global__ void k_shell_gather_f(Batch b) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)b.n_nodes * 6) return;
  const int g = b.gl[t], i = (int)(t / 6), k = (int)(t - (int64_t)i * 6);
  const int o0 = b.sh.nref_off[i], o1 = b.sh.nref_off[i + 1];
  if (g < 0 || o0 == o1) return;
  const int s = b.node_struct[i];
  if (!iterating_s(b.state[s])) return;
  double* P = b.P + b.info[s].dof_off + g;
  double v = *P;
  for (int o = o0; o < o1; o += 4) {
    double f[4];
    bool in[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = o + q < o1 ? b.sh.nref[o + q] : 0, x = shell_dof(r & 7, k);
      in[q] = o + q < o1 && x >= 0;
      f[q] = in[q] ? b.sh.Fe[(int64_t)(r >> 3) * 27 + x] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (in[q]) v += f[q];
  }
  *P = v;
}

// SaveLagrange of Gauss point g at the converged increment d.
__device__ void shell_commit(const ShellConst& c, ShellHist& h, ShellHistAux& x, const double* d, int g) {
  SGp k;
  shell_gp(c, h, d, g, k);
  v3 ai = {{x.alpha[g][0], x.alpha[g][1], x.alpha[g][2]}};
  v3 an = rodrigues_compose(k.al, ai);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    h.k1[g][j] = k.k1[j];
    h.k2[g][j] = k.k2[j];
    h.z1[g][j] = k.z1[j];
    h.z2[g][j] = k.z2[j];
    x.u[g][j] += k.u[j];
    x.alpha[g][j] = an[j];
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) h.Q[g][q] = k.Q[q];
}

// SaveLagrange of the structures that converged this pass, a thread per Gauss
// point.
__global__ void __launch_bounds__(96) k_shell_commit(Batch b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t / 3;
  if (e >= b.sh.n_shells || !b.state[b.sh.sstruct[e]].commit) return;
  double d[27];
  gather_d(b, e, d);
  shell_commit(b.sh.sconst[e], b.sh.shist[e], b.sh.saux[e], d, t % 3);
}

__global__ void __launch_bounds__(96) k_shell_commit_elements(int n, const ShellConst* cs, ShellHist* hs,
                                                              ShellHistAux* xs, const double* ds) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t / 3;
  if (e >= n) return;
  double d[27];
  for (int a = 0; a < 27; ++a) d[a] = ds[(int64_t)e * 27 + a];
  shell_commit(cs[e], hs[e], xs[e], d, t % 3);
}

void launch_shell_mount(const Batch& b, cudaStream_t st) {
  if (b.sh.n_shells == 0) return;
  launch_mount(ShellBatchSrc{b}, b.sh.n_shells, st);
  if (b.sh.any_rayleigh) k_shell_rayleigh<<<(b.sh.n_shells + 3) / 4, 128, 0, st>>>(b);
  if (!wide_band_filled(b)) {
    k_shell_gather_f<<<(unsigned)(((int64_t)b.n_nodes * 6 + 255) / 256), 256, 0, st>>>(b);
    return;
  }
  for (int c = 0; c < b.sh.n_colors; ++c) {
    int cnt = b.sh.color_off[c + 1] - b.sh.color_off[c];
    if (cnt <= 0) continue;
    k_shell_scatter<<<(cnt + 3) / 4, 128, 0, st>>>(b, c);
  }
}

void launch_shell_elements(int n, const ShellConst* c, const ShellHist* h, const double* d, const double* pu,
                           const double* p, int area_update, double* K, double* f, cudaStream_t st) {
  if (n <= 0) return;
  launch_mount(ShellElemSrc{n, area_update, c, h, d, pu, p, K, f}, n, st);
}

// Standalone inertia (gf_shell_inertia_elements): n elements with their own
// constants, history, increments d ([n][27]), converged nodal velocities v
// and accelerations a_acc ([n][36]) and Newmark coefficients a[6].
__global__ void __launch_bounds__(64) k_shell_inertia_elements(int n, const ShellConst* cs, const ShellHistAux* xs,
                                                               const double* ds, const double* vs, const double* as,
                                                               const double* a, double* Ms, double* Fs) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const ShellConst& c = cs[e];
  double* M = Ms + (int64_t)e * 729;
  double* F = Fs + (int64_t)e * 27;
  for (int q = 0; q < 729; ++q) M[q] = 0.0;
  for (int q = 0; q < 27; ++q) F[q] = 0.0;
#pragma unroll 1
  for (int g = 0; g < 3; ++g) {
    double o[SI_COUNT];
    shell_inertia_point(c, xs[e], ds + (int64_t)e * 27, 1, vs + (int64_t)e * 36, as + (int64_t)e * 36,
                        [](int k) { return 6 * k; }, a, g, o, 1);
#pragma unroll 1
    for (int q = 0; q < 9; ++q) {
      const double w = c.alpha1 * (q < 6 ? c.Nu[g][q] : c.Na[g][q - 6]);
#pragma unroll
      for (int i = 0; i < 3; ++i) F[3 * q + i] += w * (q < 6 ? o[SI_FU + i] : o[SI_FA + i]);
#pragma unroll 1
      for (int r = q < 6 ? 0 : 6; r < (q < 6 ? 6 : 9); ++r) {
        const double x = w * (q < 6 ? c.Nu[g][r] * a[0] * c.coef1 : c.Na[g][r - 6]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            M[3 * r + i + 27 * (3 * q + j)] += x * (q < 6 ? (i == j ? 1.0 : 0.0) : o[SI_D + 3 * i + j]);
      }
    }
  }
}

void launch_shell_inertia_elements(int n, const ShellConst* c, const ShellHistAux* x, const double* d,
                                   const double* v, const double* a_acc, const double* a, double* M, double* F,
                                   cudaStream_t st) {
  if (n > 0) k_shell_inertia_elements<<<(n + 63) / 64, 64, 0, st>>>(n, c, x, d, v, a_acc, a, M, F);
}

void launch_shell_commit_elements(int n, const ShellConst* c, ShellHist* h, ShellHistAux* x, const double* d,
                                  cudaStream_t st) {
  if (n <= 0) return;
  k_shell_commit_elements<<<(n + 31) / 32, 96, 0, st>>>(n, c, h, x, d);
}

void launch_shell_commit(const Batch& b, cudaStream_t st) {
  if (b.sh.n_shells == 0) return;
  k_shell_commit<<<(b.sh.n_shells + 31) / 32, 96, 0, st>>>(b);
}

}  // namespace gf

namespace gf {
int shell_launches_per_pass(const Batch& b) {
  int n = 0;
  if (b.sh.n_shells) {
    n += 2 + (b.sh.any_rayleigh ? 1 : 0);  // tangent (+ Rayleigh damping) + commit
    if (!wide_band_filled(b)) n += 1;
    else
      for (int c = 0; c < b.sh.n_colors; ++c) n += b.sh.color_off[c + 1] > b.sh.color_off[c];
  }
  return n + shell_solve_launches(b);
}
}  // namespace gf
