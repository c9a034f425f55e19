// Device-resident Newton loop for batches of Beam_1 structures (see
// gf_kernels.cuh for the pass structure and the reference lines each kernel
// follows).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "gf_beam.cuh"
#include "gf_beam_gp.cuh"
#include "gf_chain.cuh"
#include "../../include/giraffe_model.h"
#include "gf_kernels.cuh"

namespace gf {

namespace {

__device__ __forceinline__ bool iterating(const StructState& s) { return s.phase == PH_ITER; }

__device__ __forceinline__ double table_at(const Batch& b, int t, double time, int col) {
  const TableDev T = b.tables[t];
  const double* times = b.table_data + T.off;
  const double* vals = times + T.n_times;
  if (T.n_times == 0) return 0.0;
  if (time >= times[T.n_times - 1]) return vals[(T.n_times - 1) * T.n_cols + col];
  if (time <= times[0]) return vals[col];
  const int idx = table_row(T, times, time);
  double f = (time - times[idx - 1]) / (times[idx] - times[idx - 1]);
  double a = vals[(idx - 1) * T.n_cols + col], c = vals[idx * T.n_cols + col];
  return a + f * (c - a);
}

// Magnitude bits of a double: they order like the magnitudes, with infinities
// and then NaN above every finite value.  Maxima and the divergence test work on
// them, since an FP64 comparison takes as long as an FP64 multiply-add here (16
// cycles of an SM per warp) and these kernels compare eight times per DOF.
typedef unsigned long long mag_t;
__device__ __forceinline__ mag_t mag(double v) { return (mag_t)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull; }
constexpr mag_t MAG_HUGE = 0x7E37E43C8800759Cull;  // 1e300
constexpr mag_t MAG_INF = 0x7FF0000000000000ull;
// the larger of m and v's magnitude; NaN does not count
__device__ __forceinline__ void mag_max(mag_t& m, mag_t v) {
  if (v > m && v <= MAG_INF) m = v;
}
__device__ __forceinline__ mag_t warp_max(mag_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, (mag_t)__shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---- reductions of one structure spread over several CTAs ----
__device__ __forceinline__ int red_chunks(const StructInfo& inf) {
  return inf.n_free > 0 ? (inf.n_free + GF_RED_CHUNK - 1) / GF_RED_CHUNK : 1;
}
// Max of magnitudes through their bit patterns (exact, so the result does not
// depend on the order in which warps arrive), a contribution per warp.
__device__ __forceinline__ void red_max(mag_t* p, mag_t v) {
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0 && v) atomicMax(p, v);
}
__device__ __forceinline__ void red_flag(int* p, bool f) {
  if (__any_sync(0xffffffffu, f) && (threadIdx.x & 31) == 0) atomicOr(p, 1);
}
__device__ __forceinline__ double red_value(const mag_t* p) {
  return __longlong_as_double((long long)*(volatile const mag_t*)p);
}
struct Red3 { double a, b; int f; };
// Counts this CTA in; true in every thread of the CTA that arrives last, to
// which the other CTAs' global writes are then visible (each thread fences
// its own writes before the count).
__device__ bool red_arrive(RedScratch& r, int n_chunks) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&r.ticket, 1) == n_chunks - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// UpdateDyn for one node (reference src/Dynamic.cpp:480-580): Newmark
// velocity and acceleration of the free DOFs; the rotational ones are
// transported by Q_delta.  Nodes have all rotations free or all fixed
// (checked on the host), so the rotational vectors are complete.
__device__ void update_dyn_node(const Batch& b, const double* a, int node) {
  const int64_t o = (int64_t)node * 6;
  const int* gl = b.gl + o;
  const double* d = b.disp + o;
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (gl[j] >= 0) {
      b.vel[o + j] = d[j] * a[3] + b.copy_vel[o + j] * a[4] + b.copy_accel[o + j] * a[5];
      b.accel[o + j] = d[j] * a[0] - b.copy_vel[o + j] * a[1] - b.copy_accel[o + j] * a[2];
    }
  if (gl[3] >= 0 || gl[4] >= 0 || gl[5] >= 0) {
    V3<double> al = {{d[3], d[4], d[5]}}, va, aa;
    for (int j = 0; j < 3; ++j) {
      va[j] = d[3 + j] * a[3] + b.copy_vel[o + 3 + j] * a[4] + b.copy_accel[o + 3 + j] * a[5];
      aa[j] = d[3 + j] * a[0] - b.copy_vel[o + 3 + j] * a[1] - b.copy_accel[o + 3 + j] * a[2];
    }
    M3<double> Qd = rodrigues(al);
    va = mv(Qd, va);
    aa = mv(Qd, aa);
    for (int j = 0; j < 3; ++j)
      if (gl[3 + j] >= 0) {
        b.vel[o + 3 + j] = va[j];
        b.accel[o + 3 + j] = aa[j];
      }
  }
}

// ---------------------------------------------------------------------------
// initial state: the first solution step (reference src/Static.cpp:140-170)
__global__ void k_init_state(Batch b) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.n_struct) return;
  const StructParams p = b.step_params[b.info[s].step_off];
  b.params[s] = p;
  StructState& st = b.state[s];
  StructState z = {};
  z.phase = PH_START;
  z.time = p.start_time;
  z.time_step = p.time_step0;
  z.last_converged_time = p.start_time;
  st = z;
}

// Start of a load / time step (reference src/Static.cpp:176-197): the step
// machine, a thread per structure; begin[s] tells k_step_nodes what to do (bit 0
// the step starts, bit 1 from zero velocities).
__global__ void k_step_begin(Batch b) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.n_struct) return;
  if (s == 0) *b.running = 0;
  StructState& st = b.state[s];
  const bool go = st.phase == PH_START;
  b.begin[s] = go ? 1 + 2 * (st.zero_va != 0) : 0;
  if (!go) return;
  st.zero_va = 0;
  const StructParams& p = b.params[s];
  if (st.host_step) {
    // gf_begin_step: the caller's Static::Solve / Dynamic::Solve loop
    // advanced the time itself
    st.time_step = st.current_time_step;
    st.time = st.last_converged_time + st.current_time_step;
  } else {
    st.last_converged_time = st.time;
    st.time += st.time_step;
    if (st.time > 0.99999999 * p.end_time) {
      st.time = p.end_time;
      st.time_step = p.end_time - st.last_converged_time;
    }
    st.current_time_step = st.time_step;
  }
  if (p.dynamic) {
    // reference src/Dynamic.cpp:582-590
    double dt = st.time_step;
    st.a[0] = 1.0 / (dt * dt * p.beta);
    st.a[1] = 1.0 / (dt * p.beta);
    st.a[2] = 1.0 / (2.0 * p.beta) - 1.0;
    st.a[3] = p.gamma / (dt * p.beta);
    st.a[4] = 1.0 - p.gamma / p.beta;
    st.a[5] = dt * (1.0 - p.gamma / (2.0 * p.beta));
  }
  st.it = 1;
  st.res_conv = 0;
  st.gl_conv = 0;
  st.diverged = 0;
  st.info_fail = 0;
  st.phase = PH_ITER;
}

// Zeros, the prescribed displacements of the step (NodalDisplacement::Mount,
// Euler angles or vectors) and in Dynamic steps the Newmark predictor, a thread
// per node.  disp_of[i]: the node's first entry of disps, sorted by node.
__global__ void k_step_nodes(Batch b) {
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= b.n_nodes) return;
  const int s = b.node_struct[node], begin = b.begin[s];
  if (!begin) return;
  const StructState& st = b.state[s];
  const bool dyn = b.params[s].dynamic;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const int64_t q = (int64_t)node * 6 + j;
    b.disp[q] = 0.0;
    if (begin & 2) b.vel[q] = b.accel[q] = b.copy_vel[q] = b.copy_accel[q] = 0.0;
    if (dyn) {  // back to the converged velocities (a no-op after a commit)
      b.vel[q] = b.copy_vel[q];
      b.accel[q] = b.copy_accel[q];
    }
  }
  double time = st.last_converged_time + st.current_time_step, dt = st.current_time_step;
  for (int e = b.n_disps ? b.disp_of[node] : b.n_disps; e < b.n_disps && b.disps[e].node == node; ++e) {
    const DispEntry& D = b.disps[e];
    const int* cons = b.cons + (int64_t)node * 6;
    const int* gl = b.gl + (int64_t)node * 6;
    double dl[3], dg[3];
    for (int j = 0; j < 3; ++j) dl[j] = table_at(b, D.table, time, j) - table_at(b, D.table, time - dt, j);
    for (int j = 0; j < 3; ++j) dg[j] = D.CQ[j] * dl[0] + D.CQ[3 + j] * dl[1] + D.CQ[6 + j] * dl[2];
    for (int j = 0; j < 3; ++j)
      if (cons[j] == 1 && gl[j] == -1) {
        int64_t q = (int64_t)node * 6 + j;
        b.disp[q] = dg[j];
        if (dyn) {
          b.vel[q] = dg[j] / dt;
          b.accel[q] = (b.vel[q] - b.copy_vel[q]) / dt;
        }
      }
    double phi = cons[3] == 1 ? table_at(b, D.table, time, 3) : 0.0;
    double th = cons[4] == 1 ? table_at(b, D.table, time, 4) : 0.0;
    double psi = cons[5] == 1 ? table_at(b, D.table, time, 5) : 0.0;
    M3<double> Q;
    if (D.angular == GF_ANGLES_VECTOR) {
      // Euler rotation vector (phi, th, psi): Rodrigues parameters of length
      // 2 tan(|e| / 2) along e (reference src/NodalDisplacement.cpp:330-350)
      const double en = sqrt(phi * phi + th * th + psi * psi);
      const double inv = en != 0.0 ? 1.0 / en : 0.0;
      const double rod = 2.0 * tan(en / 2.0);
      const V3<double> r = {{rod * (inv * phi), rod * (inv * th), rod * (inv * psi)}};
      const M3<double> A = skew(r), A2 = mul(A, A);
      const double g = 4.0 / (4.0 + rod * rod);
      for (int k = 0; k < 9; ++k) Q[k] = g * (A[k] + 0.5 * A2[k]);
      Q[0] += 1.0;
      Q[4] += 1.0;
      Q[8] += 1.0;
    } else {
      Q[0] = cos(th) * cos(psi);
      Q[1] = sin(phi) * sin(th) * cos(psi) - cos(phi) * sin(psi);
      Q[2] = cos(phi) * sin(th) * cos(psi) + sin(phi) * sin(psi);
      Q[3] = cos(th) * sin(psi);
      Q[4] = sin(phi) * sin(th) * sin(psi) + cos(phi) * cos(psi);
      Q[5] = cos(phi) * sin(th) * sin(psi) - sin(phi) * cos(psi);
      Q[6] = -sin(th);
      Q[7] = sin(phi) * cos(th);
      Q[8] = cos(phi) * cos(th);
    }
    M3<double> CQ, Qi;
    for (int k = 0; k < 9; ++k) { CQ[k] = D.CQ[k]; Qi[k] = b.Qn[(int64_t)node * 9 + k]; }
    Q = tmul(CQ, mul(Q, CQ));
    M3<double> Qd = mul(Q, transpose(Qi));
    double tr = Qd[0] + Qd[4] + Qd[8];
    if (tr > 3.0) tr = 3.0;
    double ax[3] = {0.5 * (Qd[7] - Qd[5]), 0.5 * (Qd[2] - Qd[6]), 0.5 * (Qd[3] - Qd[1])};
    double al = 2.0 * sqrt((3.0 - tr) / (1.0 + tr));
    double theta = 2.0 * asin(sqrt((3.0 - tr) / 4.0));
    double eu = theta != 0.0 ? theta / sin(theta) : 0.0;
    for (int j = 3; j < 6; ++j)
      if (cons[j] == 1 && gl[j] == -1) {
        int64_t q = (int64_t)node * 6 + j;
        b.disp[q] = ((4.0 + al * al) / 4.0) * ax[j - 3];
        if (dyn) {
          b.vel[q] = eu * ax[j - 3] / dt;
          b.accel[q] = (b.vel[q] - b.copy_vel[q]) / dt;
        }
      }
  }
  if (dyn) update_dyn_node(b, st.a, node);
}

// UpdateDyn after an increment (reference src/Dynamic.cpp:480-580), a thread per
// node of the Dynamic structures that have just taken one.
__global__ void k_update_dyn(Batch b) {
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= b.n_nodes) return;
  const int s = b.node_struct[node];
  const StructState& st = b.state[s];
  if (iterating(st) && st.need_solve && b.params[s].dynamic) update_dyn_node(b, st.a, node);
}

// clear band and P of iterating structures
__global__ void k_zero(Batch b) {
  int s = blockIdx.y;
  if (!iterating(b.state[s])) return;
  const StructInfo inf = b.info[s];
  // wide structures: k_wb_zero; chain structures keep no band (nodeK instead)
  const bool chain_only = inf.is_chain && !b.full_band;
  int64_t nb = (inf.wide || chain_only) ? 0 : (int64_t)inf.n_free * GF_LDB;
  if (inf.is_chain || inf.wide) {
    double* nk = b.nodeK + (int64_t)inf.node_off * 9;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_nodes * 9; i += gridDim.x * blockDim.x) nk[i] = 0.0;
  }
  double* band = b.band + inf.band_off;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nb; i += (int64_t)gridDim.x * blockDim.x)
    band[i] = 0.0;
  double* P = b.P + inf.dof_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x) P[i] = 0.0;
}

// ---------------------------------------------------------------------------
// Beam_1 Mount + MountElementLoads (k_beam_tangent) and MountGlobal
// (k_beam_scatter).
//
// k_beam_tangent: 32 elements per CTA, an element per lane, so every warp runs
// one code path and the element scratch (structure-of-arrays) is written
// coalesced.  Warps 0 and 1 form the two Gauss points' operators and forces
// (gf_beam_gp.cuh) in shared memory while warps 2 and 3 form the expansion's
// coefficients and, in Dynamic steps, the points' inertial terms; then the
// four warps share the entries of K_e and f_e.  K_e of the elastic terms is
// symmetric: each pair of entries is formed once.  FP64 throughput bounds
// large batches (about 1,900 FP64 operations an element, 4,250 with an element
// per thread and full matrix products) and the chain of a point's 620 operations
// small ones.  Keeping the band read-modify-write out of this kernel keeps
// global-load latency off its dependency chains.
// k_beam_scatter: one warp per element of one colour class; lanes walk the
// 324 tangent entries in column order, so the band updates of a column are
// contiguous.  Elements of one colour share no node, so the scatter needs no
// atomics and is deterministic.
constexpr int MOUNT_THREADS = 128;
constexpr int MP_POINT = GP_COUNT + GC_COUNT;  // doubles per Gauss point and element
// with a point's parts on three warps: their shares of block 22 before the coefficients
constexpr int MP_COEF_SPLIT = GP_PART + 18, MP_POINT_SPLIT = MP_COEF_SPLIT + GC_COUNT;
// a Gauss point's inertial terms: rotational tangent, translational and
// rotational force (global frame)
constexpr int MI_D = 0, MI_FU = 9, MI_FA = 12, MI_COUNT = 15;
constexpr int MOUNT_SMEM = 2 * MP_POINT * 32 * (int)sizeof(double);
// the batch's kernel adds the inertial terms, or in static structures of the
// symmetric chain solver their coefficients
constexpr int MOUNT_SMEM_BATCH = 2 * (MP_POINT + MI_COUNT) * 32 * (int)sizeof(double);
constexpr int MOUNT_SMEM_SPLIT = 2 * (MP_POINT_SPLIT + MI_COUNT) * 32 * (int)sizeof(double);
// Elements up to which two CTAs take 32 of them: every CTA its own SM
constexpr int MOUNT_SPLIT = 152 / 2 * 32;

// The entries of K_e and f_e of lane's element, shared by `step` warps: put(r, s, v) for one entry of every symmetric pair, force(q, v).
template <int PT, int CO, typename Put, typename Force>
__device__ __forceinline__ void beam_expand(const double* P, int warp, int step, int lane, Put put, Force force) {
  const double *M = P + lane, *C = P + CO * 32 + lane;
  constexpr int gs = PT * 32, ms = 32;
#pragma unroll 1
  for (int k = warp; k < 45; k += step) {
    int pair, I, J, i, j;
    beam_aa_place(k, pair, I, J, i, j);
    put(6 * I + 3 + i, 6 * J + 3 + j, beam_k_aa(M, C, gs, ms, pair, I, J, i, j));
  }
#pragma unroll 1
  for (int k = warp; k < 81; k += step) {
    const int IJ = k / 9, x = k % 9;
    put(6 * (IJ / 3) + x / 3, 6 * (IJ % 3) + 3 + x % 3, beam_k_ua(M, C, gs, ms, IJ, x));
  }
#pragma unroll 1
  for (int k = warp; k < 36; k += step) {
    int pair, x, I, J, i, j;
    beam_uu_place(k, pair, x, I, J, i, j);
    const double v = beam_k_uu(M, C, gs, ms, pair, x);
    put(6 * I + i, 6 * J + j, v);
    if (I != J && i != j) put(6 * I + j, 6 * J + i, v);
  }
#pragma unroll 1
  for (int k = warp; k < 18; k += step) force(k, beam_f(M, C, gs, ms, k / 6, (k % 6) / 3, k % 3));
}

// The same over (du 0-2, v 3-5, a_0 6-8, a_1 9-11, a_2 12-14), lower triangle, as
// the symmetric chain solver condenses it: put(i, j, v), i >= j.  S: the
// coefficients of du and v, point g at [g * ss].
template <int PT, int CO, typename Put, typename Force>
__device__ __forceinline__ void beam_expand_sym(const double* P, const double* S, int ss, int warp, int step, int lane, Put put,
                                                Force force) {
  const double *M = P + lane, *C = P + CO * 32 + lane;
  constexpr int gs = PT * 32, ms = 32;
#pragma unroll 1
  for (int k = warp; k < 45; k += step) {
    int pair, I, J, i, j;
    beam_aa_place(k, pair, I, J, i, j);
    const double v = beam_k_aa(M, C, gs, ms, pair, I, J, i, j);
    const int r = 6 + 3 * I + i, q = 6 + 3 * J + j;  // r <= q
    put(q, r, v);
  }
#pragma unroll 1
  for (int k = warp; k < 54; k += step) {
    const int B = k / 27, J = k % 27 / 9, x = k % 9, cf = (B ? GS_VN : GS_DN) + J;
    put(6 + 3 * J + x % 3, 3 * B + x / 3,
        rfma(S[ss + cf * ms], M[gs + (GP_M02 + x) * ms], rmul(S[cf * ms], M[(GP_M02 + x) * ms])));
  }
#pragma unroll 1
  for (int k = warp; k < 18; k += step) {
    const int B = k / 6, x = k % 6;
    const int i = x < 3 ? 0 : (x < 5 ? 1 : 2), j = x < 3 ? x : (x < 5 ? x - 2 : 2);  // i <= j
    const double v = rfma(S[ss + B * ms], M[gs + (GP_M00 + x) * ms], rmul(S[B * ms], M[(GP_M00 + x) * ms]));
    if (B == 1) {
      put(3 + i, j, v);
      if (i != j) put(3 + j, i, v);
    } else {
      put((B ? 3 : 0) + j, (B ? 3 : 0) + i, v);
    }
  }
#pragma unroll 1
  for (int k = warp; k < 18; k += step) force(k, beam_f(M, C, gs, ms, k / 6, (k % 6) / 3, k % 3));
}

// k_beam_tangent<2>: a cluster of two CTAs takes 32 elements, each one Gauss point,
// whose three parts (beam_gp) and coefficients or inertia fill the SM's four
// sub-partitions; the points' values are then exchanged and the eight warps share
// K_e.  The parts repeat the kinematics, so this is for batches that leave SMs idle.
template <int CTAS> __global__ void __launch_bounds__(MOUNT_THREADS) k_beam_tangent(Batch b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int PT = CTAS == 2 ? MP_POINT_SPLIT : MP_POINT;
  double* P = reinterpret_cast<double*>(smem_raw);  // [point][value][lane]
  double* In = P + 2 * PT * 32;                     // inertial terms, [point][value][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = CTAS == 2 ? blockIdx.x & 1 : 0;
  const int e = blockIdx.x / CTAS * 32 + lane;
  const int s = e < b.n_elem ? b.estruct[e] : -1;
  const bool live = s >= 0 && iterating(b.state[s]);
  const bool dyn = live && b.params[s].dynamic;
  if (live) {
    const BeamConst& c = b.bconst[e];
    // one CTA: warps 0, 1 the points, 2, 3 the rest; two: warps 0-2 the parts of
    // point `rank`, 3 the rest
    const int g = CTAS == 2 ? rank : warp & 1;
    const bool point = CTAS == 2 ? warp < 3 : warp < 2;
    double* M = P + g * PT * 32 + lane;
    if (!point) {
      beam_gp_coef(c, g, M + (CTAS == 2 ? MP_COEF_SPLIT : GP_COUNT) * 32, 32);
      if (!dyn) beam_gp_coef_sym(c, g, In + g * MI_COUNT * 32 + lane, 32);
    }
    if (point || dyn) {
      int nd[3] = {b.enodes[3 * e], b.enodes[3 * e + 1], b.enodes[3 * e + 2]};
      double d[18];
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int q = 0; q < 6; ++q) d[6 * j + q] = b.disp[(int64_t)nd[j] * 6 + q];
      if (point) {
        if constexpr (CTAS == 1) {
          beam_gp(c, b.bhist[e], d, g, M, 32);
        } else {
          if (warp == 0) beam_gp<1>(c, b.bhist[e], d, g, M, 32);
          else if (warp == 1) beam_gp<2>(c, b.bhist[e], d, g, M, 32);
          else beam_gp<4>(c, b.bhist[e], d, g, M, 32);
        }
      } else {
        // MountMass + MountDyn: inertial force and mass/gyroscopic tangent
        double vel[18], acc[18], a6[6];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int q = 0; q < 6; ++q) {
            vel[6 * j + q] = b.copy_vel[(int64_t)nd[j] * 6 + q];
            acc[6 * j + q] = b.copy_accel[(int64_t)nd[j] * 6 + q];
          }
#pragma unroll
        for (int q = 0; q < 6; ++q) a6[q] = b.state[s].a[q];
        double* I = In + g * MI_COUNT * 32 + lane;
        beam_gp_inertia(c, b.baux[e], d, vel, acc, a6, g, I + MI_FU * 32, I + MI_FA * 32, I, 32);
      }
    }
  }
  if constexpr (CTAS == 2) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();
    // 22 of this CTA's point, then the other's values
    double* M = P + rank * PT * 32;
    for (int x = threadIdx.x; x < 6 * 32; x += MOUNT_THREADS)
      M[GP_M22 * 32 + x] = radd(radd(M[GP_PART * 32 + x], M[(GP_PART + 6) * 32 + x]), M[(GP_PART + 12) * 32 + x]);
    cluster.sync();
    const double* other = cluster.map_shared_rank(P, rank ^ 1);
    const int o = (rank ^ 1) * PT * 32, oi = (2 * PT + (rank ^ 1) * MI_COUNT) * 32;
    for (int x = threadIdx.x; x < GP_COUNT * 32; x += MOUNT_THREADS) P[o + x] = other[o + x];
    for (int x = threadIdx.x; x < GC_COUNT * 32; x += MOUNT_THREADS)
      P[o + MP_COEF_SPLIT * 32 + x] = other[o + MP_COEF_SPLIT * 32 + x];
    for (int x = threadIdx.x; x < MI_COUNT * 32; x += MOUNT_THREADS) P[oi + x] = other[oi + x];
    cluster.sync();  // neither leaves while the other reads
  }
  if constexpr (CTAS == 1) __syncthreads();
  if (!live) return;
  const int first = warp + 4 * rank, step = 4 * CTAS;
  double* Ke = b.Ke + e;
  const int64_t ne = b.n_elem;
  constexpr int CO = CTAS == 2 ? MP_COEF_SPLIT : GP_COUNT;
  const double* Cf = P + CO * 32 + lane;
  if (!dyn) {
    if (b.info[s].sym && !b.full_band) {
      beam_expand_sym<PT, CO>(P, In + lane, MI_COUNT * 32, first, step, lane,
                      [&](int i, int j, double v) { Ke[(int64_t)(i * (i + 1) / 2 + j) * ne] = v; },
                      [&](int q, double v) { b.Fe[q * ne + e] = v; });
      return;
    }
    beam_expand<PT, CO>(P, first, step, lane,
                [&](int r, int q, double v) {
                  Ke[(r + 18 * q) * ne] = v;
                  if (r != q) Ke[(q + 18 * r) * ne] = v;
                },
                [&](int q, double v) { b.Fe[q * ne + e] = v; });
    return;
  }
  // Dynamic steps: the inertial terms on top.  Rayleigh damping: on the
  // iterations that form C_e, the stiffness part of K_e alone goes to the
  // damping scratch, where k_beam_rayleigh turns it into C_e = alpha M_modal +
  // beta K_e
  const StructParams& pr = b.params[s];
  double* Ce = pr.ray_on && (pr.ray_update || !b.state[s].ray_init) ? b.RD + e : nullptr;
  const double a1Mr = rmul(b.state[s].a[0], b.bconst[e].Mr);
  const double* I0 = In + lane;
  // K_e's entry with its inertial term, if it has one: couplings of translations
  // and rotations and of different translations do not (a zero added would take an
  // FP64 instruction's 64 cycles)
  auto with_mass = [&](int r, int q, double v) {
    const int I = r / 6, i = r % 6, J = q / 6, j = q % 6;
    const int pair = tri3(I, J);
    if ((i < 3) != (j < 3) || (i < 3 && i != j)) return v;
    if (i < 3) return radd(v, rmul(radd(Cf[(GC_NN + pair) * 32], Cf[(PT + GC_NN + pair) * 32]), a1Mr));
    const int x = (i - 3) * 3 + j - 3;
    return radd(v, rfma(Cf[(PT + GC_NN + pair) * 32], I0[(MI_COUNT + MI_D + x) * 32],
                        rmul(Cf[(GC_NN + pair) * 32], I0[(MI_D + x) * 32])));
  };
  beam_expand<PT, CO>(P, first, step, lane,
              [&](int r, int q, double v) {
                Ke[(r + 18 * q) * ne] = with_mass(r, q, v);
                if (Ce) Ce[(r + 18 * q) * ne] = v;
                if (r == q) return;
                Ke[(q + 18 * r) * ne] = with_mass(q, r, v);
                if (Ce) Ce[(q + 18 * r) * ne] = v;
              },
              [&](int q, double v) {
                const int I = q / 6, x = (q % 6) / 3 ? MI_FA + q % 3 : MI_FU + q % 3;
                v = rfma(Cf[(GC_WN + I) * 32], I0[x * 32], v);
                b.Fe[q * ne + e] = rfma(Cf[(PT + GC_WN + I) * 32], I0[(MI_COUNT + x) * 32], v);
              });
}

// MountDamping and the damping part of MountDyn (reference
// src/Beam_1.cpp:1641-1673).  On the iterations that form it (the step's
// first, or every one with Update 1), C_e = alpha M_modal + beta K_e; the
// modal mass is MountMassModal (src/Beam_1.cpp:1538-1553) with the
// EvaluateMassModal operator (src/Beam_1.cpp:1681-1774) of a section
// without a first moment of mass, blockdiag(Q Mr Q^T, Q Jr Q^T) with
// Q = Q(alpha_i) at each Gauss point, summed as wJ N^T D N (w = 1) and
// turned to the global frame block by block (T3^T B T3).  Every iteration
// then adds a4 C_e to K_e and C_e v to f_e, v the nodes' current
// velocities.  One thread per element; C_e is structure-of-arrays like K_e.
// The modal mass of a Beam_1 / Pipe_1 element: per Gauss point D[g][0] =
// Q Mr Q^T and D[g][1] = Q Jr Q^T (3x3 row-major) with Q = Q(alpha_i).
__device__ void beam_modal_D(const BeamConst& c, const BeamHistAux& x, double (*D)[2][9]) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    M3<double> Q = rodrigues(V3<double>{{x.alpha[g][0], x.alpha[g][1], x.alpha[g][2]}});
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double mt = 0.0, jt = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double qm = 0.0, qj = 0.0;
#pragma unroll
          for (int l = 0; l < 3; ++l) {
            qm += Q[i * 3 + l] * (l == k ? c.Mr : 0.0);
            qj += Q[i * 3 + l] * c.Jr[l * 3 + k];
          }
          mt += qm * Q[j * 3 + k];
          jt += qj * Q[j * 3 + k];
        }
        D[g][0][i * 3 + j] = mt;
        D[g][1][i * 3 + j] = jt;
      }
  }
}

// Block (node I, node J, translation/rotation bi, bj) of the element's modal
// mass in the global frame, 3x3 row-major: sum_g jac N_gI N_gJ D[g][bi]
// turned by T^T (.) T on the diagonal blocks bi == bj, zero off them.
__device__ void beam_modal_block(const BeamConst& c, const double (*D)[2][9], int I, int J, int bi, int bj,
                                 double* m) {
#pragma unroll
  for (int q = 0; q < 9; ++q) m[q] = 0.0;
  if (bi != bj) return;
  const double* T = c.T3;
  double loc[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    loc[q] = 0.0;
#pragma unroll
    for (int g = 0; g < 2; ++g) loc[q] += ((c.jac * c.N[g][I]) * D[g][bi][q]) * c.N[g][J];
  }
  double t2[9];  // loc T, then T^T (loc T)
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) t2[i * 3 + j] = loc[i * 3] * T[j] + loc[i * 3 + 1] * T[3 + j] + loc[i * 3 + 2] * T[6 + j];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) m[i * 3 + j] = T[i] * t2[j] + T[3 + i] * t2[3 + j] + T[6 + i] * t2[6 + j];
}

// 32 elements per CTA, an element per lane (the scratch is structure-of-arrays)
// and a row of C_e, K_e and f_e per warp, so that a row's 18 columns load side by
// side.
constexpr int RAY_THREADS = 18 * 32;
__global__ void __launch_bounds__(RAY_THREADS) k_beam_rayleigh(Batch b) {
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), q = threadIdx.x >> 5;
  if (e >= b.n_elem) return;
  const int s = b.estruct[e];
  const StructState& st = b.state[s];
  if (!iterating(st)) return;
  const StructParams& p = b.params[s];
  if (!p.dynamic || !p.ray_on) return;
  const int64_t ne = b.n_elem;
  double* C = b.RD + e;
  double c[18], k[18];
#pragma unroll
  for (int x = 0; x < 18; ++x) {
    c[x] = C[(int64_t)(q + 18 * x) * ne];
    k[x] = b.Ke[(int64_t)(q + 18 * x) * ne + e];
  }
  if (p.ray_update || !st.ray_init) {
    const BeamConst& bc = b.bconst[e];
    double D[2][2][9];  // [Gauss point][translation, rotation][3x3 row-major]
    beam_modal_D(bc, b.baux[e], D);
    const int I = q / 6, bi = q % 6 / 3, i = q % 3;
#pragma unroll
    for (int J = 0; J < 3; ++J)
#pragma unroll
      for (int bj = 0; bj < 2; ++bj) {
        double m[9];
        beam_modal_block(bc, D, I, J, bi, bj, m);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int x = 6 * J + 3 * bj + j;
          const double mv = i == 0 ? m[j] : i == 1 ? m[3 + j] : m[6 + j];
          c[x] = p.ray_alpha * mv + p.ray_beta * c[x];
          C[(int64_t)(q + 18 * x) * ne] = c[x];
        }
      }
  }
  const double a4 = st.a[3];
  double acc = 0.0;
#pragma unroll
  for (int x = 0; x < 18; ++x) {
    acc += c[x] * b.vel[(int64_t)b.enodes[3 * e + x / 6] * 6 + x % 6];
    b.Ke[(int64_t)(q + 18 * x) * ne + e] = k[x] + a4 * c[x];
  }
  b.Fe[(int64_t)q * ne + e] += acc;
}

// Pipe_1::MountPipeSpecialLoads (reference src/Pipe_1.cpp:1441-1494): the
// internal pressure p0i of a PipeLoad acting on the internal area Aint, at
// the current iterate.  At each Gauss point, with Q = Q_delta Q_i,
// kappa = Q kappa_r and e3 = Q e3r (element frame), the line load
// (f, m) = -p0i Aint (kappa x e3, Xi^T (z' x e3)) and its stiffness Kext
// (6 x 12 on (u, alpha, u', alpha'): K1ua, K1aa, K2ua, K2au) enter as
// f_e -= jac T^T N^T (f, m) and K_e -= jac p0i Aint T^T N^T Kext Upsilon T.
// Its O1 term reads the element's scalar g, which the reference's Mount
// leaves at the second Gauss point's value (src/Pipe_1.cpp:890), for both
// points.  After k_beam_tangent has written K_e and f_e and before
// k_beam_rayleigh: in a Dynamic step the reference mounts loads before damping,
// so on the iterations that form C_e the load stiffness also goes into the
// stiffness part that C_e is made from.  32 elements per CTA, an element per
// lane: warps 0 and 1 form the two Gauss points' blocks in shared memory (in the
// global frame, where K2au = -K2ua^T and kappa x e3's commutator spares the products
// of three skew matrices: 300 operations for 800), the other six the products of
// the shape functions, then the eight warps share the entries of K_e, four loads in
// flight.  Bound by these chains of FP64 operations: 500 elements 58 us with the
// element frame's matrix products and an entry at a time, 24 here.
constexpr int PP_THREADS = 256;
// blocks G1 (K1ua), G2 (K2ua), G4 (K1aa), the force and the moment; the products
// jac p0i Aint N_a N_n and N_a N'_n and jac p0i Aint N_a
constexpr int PP_G1 = 0, PP_G2 = 9, PP_G4 = 18, PP_F = 27, PP_NN = 33, PP_ND = 42, PP_N = 51, PP_COUNT = 54;
__device__ __forceinline__ void pipe_press_point(const BeamConst& c, const BeamHist& h, const double* d, int g, double* S) {
  d3 a, b, z;
  beam_gp_interp(c, d, g, a, b, z);
  const double gq = 4.0 / radd(4.0, rdot(a, a)), hg = 0.5 * gq;
  double g_last = gq;
  if (g == 0) {
    d3 y;
#pragma unroll
    for (int i = 0; i < 3; ++i) y[i] = fma(d[15 + i], c.N[1][2], fma(d[9 + i], c.N[1][1], d[3 + i] * c.N[1][0]));
    g_last = 4.0 / (4.0 + dot(y, y));
  }
  // kappa and e3 before the increment's rotation, then through it
  d3 kip = {{0.0, 0.0, 0.0}}, e3 = {{0.0, 0.0, 0.0}};
  {
    d3 T[3];  // rows of T3
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) T[i][j] = c.T3[i * 3 + j];
    const d3 w = rmv(T, d3{{h.dz[g][0], h.dz[g][1], h.dz[g][2]}}), beta = rxi(a, b, gq, -0.5);
    d3 k0 = kip, e0 = e3;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const d3 r = rmv(T, d3{{h.Q[g][j], h.Q[g][3 + j], h.Q[g][6 + j]}});
      const double kj = radd(rdot(r, beta), h.kap[g][j]);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        k0[i] = fma(r[i], kj, k0[i]);
        e0[i] = fma(r[i], c.e3r[j], e0[i]);
      }
      z[j] += w[j];
    }
    const d3 ck = rcross(a, k0), ck2 = rcross(a, ck), ce = rcross(a, e0), ce2 = rcross(a, ce);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      kip[i] = fma(gq, fma(0.5, ck2[i], ck[i]), k0[i]);
      e3[i] = fma(gq, fma(0.5, ce2[i], ce[i]), e0[i]);
    }
  }
  const d3 fl = rcross(kip, e3), c2 = rcross(e3, z);
  const d3 w = rxi(a, c2, gq, -0.5), eps = rxi(a, e3, gq, -0.5), zeta = rxi(a, z, gq, -0.5);
  const d3 ha = {{hg * a[0], hg * a[1], hg * a[2]}};
  const d3 X[3] = {{{gq, ha[2], -ha[1]}}, {{-ha[2], gq, ha[0]}}, {{ha[1], -ha[0], gq}}};  // columns of Xi
  const double hab = hg * dot(a, b), heb = hg * dot(e3, b), ze = dot(z, e3);
  const double sk[9] = {0.0, -c2[2], c2[1], c2[2], 0.0, -c2[0], -c2[1], c2[0], 0.0};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const d3 y = rcross(e3, X[j]), f = rcross(fl, X[j]);
    const double hej = hg * e3[j], aj = ze * hg * ha[j];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      S[(PP_G2 + 3 * i + j) * 32] = y[i];
      double v = fma(hej, b[i], fma(-hab, y[i], f[i]));
      if (i == j) v -= heb;
      S[(PP_G1 + 3 * i + j) * 32] = v;
      double u = i == j ? w[i] * a[j] : fma(w[i], a[j], -sk[3 * i + j]);
      u = fma(-0.5 * g_last, u, fma(eps[i], zeta[j], aj * a[i]));
      if (i == j) u = fma(-ze, gq, u);
      S[(PP_G4 + 3 * i + j) * 32] = u;
    }
    S[(PP_F + j) * 32] = fl[j];
    S[(PP_F + 3 + j) * 32] = -w[j];
  }
}
__global__ void __launch_bounds__(PP_THREADS) k_pipe_pressure(Batch b) {
  __shared__ double S[2][PP_COUNT][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * 32 + lane;
  const int e = q < b.n_pipe_press ? b.pp_elem[q] : 0;
  const int s = q < b.n_pipe_press ? b.estruct[e] : 0;
  const StructState& st = b.state[s];
  const bool on = q < b.n_pipe_press && iterating(st);
  const BeamConst& c = b.bconst[e];
  if (on) {
    const int g = warp & 1;
    if (warp < 2) {
      double d[18];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int64_t nd = b.enodes[3 * e + j];
#pragma unroll
        for (int k = 0; k < 6; ++k) d[6 * j + k] = b.disp[nd * 6 + k];
      }
      pipe_press_point(c, b.bhist[e], d, g, &S[g][0][lane]);
    } else {
      const double p0i = table_at(b, b.pp_table[q], st.last_converged_time + st.current_time_step, 0);
      const double sK = c.jac * p0i * b.pp_aint[q];
#pragma unroll 1
      for (int x = (warp >> 1) - 1; x < 9; x += 3) {  // warps 2-7: three for each point
        const double t = sK * c.N[g][x / 3];
        S[g][PP_NN + x][lane] = t * c.N[g][x % 3];
        S[g][PP_ND + x][lane] = t * c.dN[g][x % 3];
        if (x % 3 == 0) S[g][PP_N + x / 3][lane] = t;
      }
    }
  }
  __syncthreads();
  if (!on) return;
  const StructParams& pr = b.params[s];
  const bool form_c = pr.dynamic && pr.ray_on && (pr.ray_update || !st.ray_init);
  const int64_t ne = b.n_elem;
  double* Ke = b.Ke + e;
  double* Ce = form_c ? b.RD + e : nullptr;
  // f_e -= jac N (f, m) with the line load's -p0i Aint
#pragma unroll 1
  for (int k = warp; k < 18; k += 8) {
    double f = b.Fe[(int64_t)k * ne + e];
#pragma unroll
    for (int g = 0; g < 2; ++g) f = fma(S[g][PP_N + k / 6][lane], S[g][PP_F + k % 6][lane], f);
    b.Fe[(int64_t)k * ne + e] = f;
  }
  // (u_a, alpha_n): K1ua Nb + K2ua dNb; (alpha_a, u_n): K2au dNb = -K2ua^T dNb;
  // (alpha_a, alpha_n): K1aa Nb
#pragma unroll 1
  for (int k0 = warp; k0 < 243; k0 += 32) {
    int64_t at[4];
    double v[4], w[4], t[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int k = k0 + 8 * y, kind = k / 81, an = k % 81 / 9, x = k % 9, i = x / 3, j = x % 3, a = an / 3, n = an % 3;
      at[y] = ((kind == 0 ? 6 * a + i : 6 * a + 3 + i) + 18 * (kind == 1 ? 6 * n + j : 6 * n + 3 + j)) * ne;
      v[y] = k < 243 ? Ke[at[y]] : 0.0;
      w[y] = k < 243 && Ce ? Ce[at[y]] : 0.0;
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int k = k0 + 8 * y, kind = k / 81, an = k % 81 / 9, x = k % 9, xt = 3 * (x % 3) + x / 3;
      if (k >= 243) break;
      if (kind == 0) {
        t[y] = S[0][PP_NN + an][lane] * S[0][PP_G1 + x][lane];
        t[y] = fma(S[0][PP_ND + an][lane], S[0][PP_G2 + x][lane], t[y]);
        t[y] = fma(S[1][PP_NN + an][lane], S[1][PP_G1 + x][lane], t[y]);
        t[y] = fma(S[1][PP_ND + an][lane], S[1][PP_G2 + x][lane], t[y]);
      } else {
        const int cf = (kind == 1 ? PP_ND : PP_NN) + an, m = kind == 1 ? PP_G2 + xt : PP_G4 + x;
        t[y] = fma(S[1][cf][lane], S[1][m][lane], S[0][cf][lane] * S[0][m][lane]);
      }
      // (K2au's sign)
      Ke[at[y]] = kind == 1 ? v[y] + t[y] : v[y] - t[y];
      if (Ce) Ce[at[y]] = kind == 1 ? w[y] + t[y] : w[y] - t[y];
    }
  }
}

// The modal mass of every Beam_1 / Pipe_1 element of colour class `color`
// added into the band M (entry (i, j) at (kw + i - j) + j W, free indices of
// b.gl): one thread per element, elements of a colour share no node.
__global__ void k_modal_mass_beam(Batch b, int color, double* M, int64_t W, int kw) {
  const int k = b.color_off[color] + blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.color_off[color + 1]) return;
  const int e = b.color_elems[k];
  const BeamConst& c = b.bconst[e];
  double D[2][2][9];
  beam_modal_D(c, b.baux[e], D);
  int g[18];
#pragma unroll
  for (int a = 0; a < 18; ++a) g[a] = b.gl[(int64_t)b.enodes[3 * e + a / 6] * 6 + a % 6];
#pragma unroll 1
  for (int I = 0; I < 3; ++I)
#pragma unroll 1
    for (int J = 0; J < 3; ++J)
#pragma unroll 1
      for (int bi = 0; bi < 2; ++bi) {
        double m[9];
        beam_modal_block(c, D, I, J, bi, bi, m);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int gr = g[6 * I + 3 * bi + i], gq = g[6 * J + 3 * bi + j];
            if (gr >= 0 && gq >= 0 && abs(gr - gq) <= kw) M[(kw + gr - gq) + (int64_t)gq * W] += m[i * 3 + j];
          }
      }
}

__global__ void k_beam_scatter(Batch b, int color) {
  int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int lane = threadIdx.x & 31;
  int k = b.color_off[color] + w;
  if (k >= b.color_off[color + 1]) return;
  int e = b.color_elems[k];
  int s = b.estruct[e];
  if (!iterating(b.state[s])) return;
  const StructInfo inf = b.info[s];
  int myg = -1;
  if (lane < 18) myg = b.gl[(int64_t)b.enodes[3 * e + lane / 6] * 6 + lane % 6];
  if (inf.is_chain && !b.full_band) {
    // the chain solver reads K_e directly; only the residual is assembled
    if (lane < 18 && myg >= 0) b.P[inf.dof_off + myg] += b.Fe[(int64_t)lane * b.n_elem + e];
    return;
  }
  const double* Ke = b.Ke + e;
  const int64_t ne = b.n_elem;
  double* band = b.band + inf.band_off;
  // uniform trip count: every lane takes part in every shuffle
  for (int base = 0; base < 324; base += 32) {
    int idx = base + lane;
    bool valid = idx < 324;
    int r = valid ? idx % 18 : 0, q = valid ? idx / 18 : 0;
    int gr = __shfl_sync(0xffffffffu, myg, r);
    int gq = __shfl_sync(0xffffffffu, myg, q);
    if (valid && gr >= 0 && gq >= 0) band[(GF_KB + gr - gq) + (int64_t)gq * GF_LDB] += Ke[idx * ne];
  }
  if (lane < 18 && myg >= 0) b.P[inf.dof_off + myg] += b.Fe[(int64_t)lane * ne + e];
}

// MountGlobal of the internal forces when every Beam_1 element of the batch
// belongs to a chain and no band is filled (the chain solver reads K_e from
// the element scratch): one thread per node DOF gathers the forces of the one
// or two elements on its node in a single launch, in place of the two colour
// passes of k_beam_scatter.  Chain element e of a structure sits on its local
// nodes 2e, 2e+1, 2e+2.  k_zero has just cleared P, so the sum (0 + f_a) + f_b
// formed here equals the colour-ordered scatter's, whichever element's colour
// comes first (IEEE addition is commutative).
__global__ void k_chain_gather_f(Batch b) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)b.n_nodes * 6) return;
  const int g = b.gl[t];
  if (g < 0) return;
  const int i = (int)(t / 6), q = (int)(t - (int64_t)i * 6);
  const int s = b.node_struct[i];
  const StructInfo& inf = b.info[s];
  if (!inf.is_chain || !iterating(b.state[s])) return;
  const int ln = i - inf.node_off, eo = inf.elem_off;
  const int64_t ne = b.n_elem;
  double v = 0.0;
  if (ln & 1) {
    v += b.Fe[(int64_t)(6 + q) * ne + eo + (ln >> 1)];
  } else {
    const int el = ln >> 1;
    if (el >= 1) v += b.Fe[(int64_t)(12 + q) * ne + eo + el - 1];
    if (el < inf.n_elem) v += b.Fe[(int64_t)q * ne + eo + el];
  }
  b.P[inf.dof_off + g] = v;
}

// NodalLoad::Mount for every load entry of a structure, in entry order (one
// warp per structure keeps the accumulation order fixed; lanes 0-5 own the
// entry's components, lanes 0-8 the entries of its load stiffness V(alpha,
// Xi^T m)).
__global__ void __launch_bounds__(128) k_loads(Batch b) {
  const int s = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= b.n_struct || !iterating(b.state[s])) return;
  const StructInfo& inf = b.info[s];
  const StructState& st = b.state[s];
  const double time = st.last_converged_time + st.current_time_step;
  double* P = b.P + inf.dof_off;
  double* band = b.band + inf.band_off;
  const bool to_nodeK = (inf.is_chain || inf.wide) && !b.full_band;
  const bool to_wide = inf.wide && wide_band_filled(b);
  const int c6 = lane < 6 ? lane : 0, i = lane < 9 ? lane / 3 : 0, j = lane % 3;
  for (int l = inf.load_off; l < inf.load_off + inf.n_loads; ++l) {
    const LoadEntry& L = b.loads[l];
    const int node = L.node;
    const int* gl = b.gl + (int64_t)node * 6;
    const double v = L.mult[c6] * table_at(b, L.table, time, c6);
    V3<double> fl, ml;
    for (int q = 0; q < 3; ++q) {
      fl[q] = __shfl_sync(0xffffffffu, v, q);
      ml[q] = __shfl_sync(0xffffffffu, v, 3 + q);
    }
    const V3<double> al = {{b.disp[(int64_t)node * 6 + 3], b.disp[(int64_t)node * 6 + 4], b.disp[(int64_t)node * 6 + 5]}};
    const double g = 4.0 / (4.0 + dot(al, al));
    // component c6 of CQ^T (f, m): lanes 0-2 the force, 3-5 the moment
    const V3<double>& w = lane < 3 ? fl : ml;
    const int r = c6 % 3;
    double comp = L.CQ[r] * w[0] + L.CQ[3 + r] * w[1] + L.CQ[6 + r] * w[2];
    V3<double> mv3;
    for (int q = 0; q < 3; ++q) mv3[q] = __shfl_sync(0xffffffffu, comp, 3 + q);
    // Xi^T m = g (m - alpha x m / 2), and its cross product with alpha
    V3<double> am = cross(al, mv3), mm;
    for (int q = 0; q < 3; ++q) mm[q] = g * (mv3[q] - 0.5 * am[q]);
    if (lane < 6) {
      const int gi = gl[lane];
      if (gi >= 0) P[gi] += -1.0 * (lane < 3 ? comp : mm[lane - 3]);
    }
    const int gi = gl[3 + i], gj = gl[3 + j];
    if (lane < 9 && gi >= 0 && gj >= 0) {
      const double V = opV(al, mm, g)[lane];
      if (to_nodeK) b.nodeK[(int64_t)node * 9 + lane] += -1.0 * V;
      if (to_wide) b.sh.wband[inf.wb_off + (inf.wkl + gi - gj) + (int64_t)gj * (2 * inf.wkl + 1)] += -1.0 * V;
      else if (!to_nodeK) band[(GF_KB + gi - gj) + (int64_t)gj * GF_LDB] += -1.0 * V;
    }
    __syncwarp();  // the next entry may add to the same DOFs from other lanes
  }
}

// P = -P; EstablishResidualCriteria at the first iteration;
// CheckResidualConvergence (reference src/ConvergenceCriteria.cpp:187-285,
// 460-598).
__global__ void k_residual(Batch b) {
  const int s = b.chunk_struct[blockIdx.x];
  StructState& st = b.state[s];
  if (!iterating(st)) return;
  const StructInfo inf = b.info[s];
  const StructParams& p = b.params[s];
  double* P = b.P + inf.dof_off;
  const int* d6 = b.dof_node6 + inf.dof_off;
  const int i1 = min(inf.n_free, b.chunk_start[blockIdx.x] + GF_RED_CHUNK);
  mag_t va = 0, vb = 0;
  bool vf = false;
  for (int i = b.chunk_start[blockIdx.x] + threadIdx.x; i < i1; i += blockDim.x) {
    const double p0 = P[i];
    P[i] = -p0;
    const mag_t a = mag(p0);
    vf = vf || a >= MAG_HUGE;
    if (d6[i] % 6 < 3) mag_max(va, a);
    else mag_max(vb, a);
  }
  RedScratch& R = b.red[s];
  red_max(&R.a, va);
  red_max(&R.b, vb);
  red_flag(&R.f, vf);
  if (!red_arrive(R, red_chunks(inf))) return;
  Red3 r{};
  if (threadIdx.x == 0) {
    r.a = red_value(&R.a);
    r.b = red_value(&R.b);
    r.f = *(volatile int*)&R.f;
    R = RedScratch{0ull, 0ull, 0ull, 0ull, 0, 0};
  }
  if (threadIdx.x == 0) {
    if (st.it == 1) {
      double pf = st.force_crit, pm = st.moment_crit;
      double fc = r.a * p.force_tol > p.force_min * p.force_tol ? r.a * p.force_tol : p.force_min * p.force_tol;
      double mc = r.b * p.moment_tol > p.moment_min * p.moment_tol ? r.b * p.moment_tol : p.moment_min * p.moment_tol;
      st.force_crit = (st.n_conv_evaluated * pf + fc) / (st.n_conv_evaluated + 1);
      st.moment_crit = (st.n_conv_evaluated * pm + mc) / (st.n_conv_evaluated + 1);
      st.n_conv_evaluated++;
    }
    if (r.f) st.diverged = 1;
    int conv = 1;
    if (r.a > p.divergence_ref || r.b > p.divergence_ref) {
      st.diverged = 1;
      conv = 0;
    } else {
      if (inf.has_force && r.a > st.force_crit) conv = 0;
      if (inf.has_moment && r.b > st.moment_crit) conv = 0;
    }
    st.res_conv = conv;
    st.last_res = fmax(r.a, r.b);
    st.need_solve = !(st.res_conv && st.gl_conv);
  }
}

// ---------------------------------------------------------------------------
// Banded LU without pivoting, fused forward substitution, back substitution;
// FP64.  One 4-warp CTA per structure.
//
// On this GPU a dependent FP64 operation costs ~64 cycles and an FP64 divide
// ~640, so the per-column critical path is what bounds a long chain.  The
// elimination is split so that warp 0 carries only that path with one column
// of lookahead: at step j it updates column j+1, forms the next pivot's
// reciprocal (Newton-Raphson iteration r <- r (2 - p r), seeded by the FP32
// approximate reciprocal, two steps) and the next multipliers, while warps
// 1-3 apply step j's rank-1 update to columns j+2..j+17 and the right-hand
// side.  Band columns stream through a 128-column shared-memory ring filled
// 32 columns at a time, two chunks ahead.  Row j of U (with the pivot
// reciprocal in place of the pivot) goes to b.U; the forward-substituted
// right-hand side goes to P, which the back substitution overwrites with x.
constexpr int RING = 128;
constexpr int CHUNK = 32;
constexpr int SOLVE_THREADS = 128;

// Newton-Raphson reciprocal of p, seeded by the hardware FP32 approximation;
// exact division where the seed is out of FP32 range.
__device__ __forceinline__ double recip_nr(double p) {
  float pf = __double2float_rn(p);
  float af = fabsf(pf);
  if (!(af > 1e-30f && af < 1e30f)) return 1.0 / p;
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(pf));
  double r = (double)rf;
  double e = fma(-p, r, 1.0);
  r = fma(r, e, r);
  e = fma(-p, r, 1.0);
  r = fma(r, e, r);
  return r;
}

template <typename T>
__device__ __forceinline__ void load_chunk(const T* __restrict__ band, const double* __restrict__ rhs, T* ring,
                                           double* rring, int q, int n, int tid, int nthreads) {
  int c0 = q * CHUNK;
  if (c0 >= n) return;
  int nc = min(CHUNK, n - c0);
  int slot0 = c0 % RING;
  const T* src = band + (int64_t)c0 * GF_LDB;
  T* dst = ring + (int64_t)slot0 * GF_LDB;
  for (int i = tid; i < nc * GF_LDB; i += nthreads) dst[i] = src[i];
  for (int i = tid; i < nc; i += nthreads) rring[slot0 + i] = rhs[c0 + i];
}

__global__ void __launch_bounds__(SOLVE_THREADS) k_band_solve(Batch b) {
  int s = blockIdx.x;
  StructState& st = b.state[s];
  if (!iterating(st) || !st.need_solve) return;
  const StructInfo inf = b.info[s];
  if (inf.is_chain || inf.wide) return;
  const int n = inf.n_free;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  extern __shared__ unsigned char smem_raw[];
  double* ring = reinterpret_cast<double*>(smem_raw);
  double* rring = ring + RING * GF_LDB;
  __shared__ double lbuf[2][GF_KB + 1];
  __shared__ double invb[2];
  __shared__ int sfail;
  const double* band = b.band + inf.band_off;
  double* rhs = b.P + inf.dof_off;
  double* U = b.U + (int64_t)inf.dof_off * GF_UW;
  if (tid == 0) sfail = 0;
  load_chunk(band, rhs, ring, rring, 0, n, tid, SOLVE_THREADS);
  load_chunk(band, rhs, ring, rring, 1, n, tid, SOLVE_THREADS);
  load_chunk(band, rhs, ring, rring, 2, n, tid, SOLVE_THREADS);
  __syncthreads();
  // step 0 multipliers
  if (warp == 0) {
    double p = ring[GF_KB];
    double inv = recip_nr(p);
    if (lane >= 1 && lane <= GF_KB) lbuf[0][lane] = (lane < n) ? ring[GF_KB + lane] * inv : 0.0;
    if (lane == 0) {
      invb[0] = inv;
      if (!(p != 0.0) || !isfinite(p)) sfail = 1;
    }
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const int cur = j & 1;
    if (j % CHUNK == 0 && j > 0) load_chunk(band, rhs, ring, rring, j / CHUNK + 2, n, tid, SOLVE_THREADS);
    if (warp > 0) {
      // rank-1 update of columns j+2..j+17 (16 x 17 entries) and the rhs (17)
      for (int k = tid - 32; k < 16 * GF_KB + GF_KB; k += SOLVE_THREADS - 32) {
        if (k < 16 * GF_KB) {
          int r = k / 16 + 1, c = k % 16 + 2;
          int J = j + c;
          if (J < n) {
            double* col = ring + (int64_t)(J % RING) * GF_LDB;
            col[GF_KB + r - c] -= lbuf[cur][r] * col[GF_KB - c];
          }
        } else {
          int r = k - 16 * GF_KB + 1;
          if (j + r < n) rring[(j + r) % RING] -= lbuf[cur][r] * rring[j % RING];
        }
      }
    } else {
      // U row j (reciprocal pivot first), y_j
      if (lane >= 1 && lane <= GF_KB) {
        int J = j + lane;
        U[(int64_t)j * GF_UW + lane] = J < n ? ring[(int64_t)(J % RING) * GF_LDB + GF_KB - lane] : 0.0;
      } else if (lane == 0) {
        U[(int64_t)j * GF_UW] = invb[cur];
        rhs[j] = rring[j % RING];
      }
      if (j + 1 < n) {
        double* c1 = ring + (int64_t)((j + 1) % RING) * GF_LDB;
        if (lane >= 1 && lane <= GF_KB) c1[GF_KB + lane - 1] -= lbuf[cur][lane] * c1[GF_KB - 1];
        __syncwarp();
        double p = c1[GF_KB];
        double inv = recip_nr(p);
        if (lane >= 1 && lane <= GF_KB) lbuf[cur ^ 1][lane] = (j + 1 + lane < n) ? c1[GF_KB + lane] * inv : 0.0;
        if (lane == 0) {
          invb[cur ^ 1] = inv;
          if (!(p != 0.0) || !isfinite(p)) sfail = 1;
        }
      }
    }
    __syncthreads();
  }
  // back substitution, column oriented, warp 0: lane t (1..17) holds
  // y'_{j-t}; x_j = y'_j / u_jj, then y'_{j-t} -= U(j-t, j) x_j.
  if (warp == 0) {
    double yv = 0.0;  // lane 0: y'_j; lane t: y'_{j-t}
    {
      int i = n - 1 - lane;
      if (lane <= GF_KB && i >= 0) yv = rhs[i];
    }
    for (int j0 = n - 1; j0 >= 0; j0 -= CHUNK) {
      // per-chunk operands: lane t needs U(j - t, t) for j in the chunk, lane 0
      // the reciprocal pivots, lane 17 the y entering at j - 18
      double uo[CHUNK];
#pragma unroll
      for (int q = 0; q < CHUNK; ++q) {
        int j = j0 - q;
        double v = 0.0;
        if (j >= 0) {
          if (lane == 0) v = U[(int64_t)j * GF_UW];
          else if (lane <= GF_KB && j - lane >= 0) v = U[(int64_t)(j - lane) * GF_UW + lane];
          else if (lane == GF_KB + 1 && j - GF_KB - 1 >= 0) v = rhs[j - GF_KB - 1];
        }
        uo[q] = v;
      }
#pragma unroll
      for (int q = 0; q < CHUNK; ++q) {
        int j = j0 - q;
        if (j < 0) break;
        double xj = __shfl_sync(0xffffffffu, yv * uo[q], 0);
        if (lane == 0) rhs[j] = xj;
        if (lane >= 1 && lane <= GF_KB) yv = fma(-uo[q], xj, yv);
        // shift the window: lane t takes lane t+1's value; lane 17 takes y_{j-18}
        double nx = __shfl_down_sync(0xffffffffu, yv, 1);
        double ent = __shfl_sync(0xffffffffu, uo[q], GF_KB + 1);
        yv = lane < GF_KB ? nx : (lane == GF_KB ? ent : 0.0);
      }
    }
  }
  if (tid == 0) st.info_fail = sfail;
}

// UpdateDisps + CheckGLConvergence (reference src/Solution.cpp:390-423,
// src/ConvergenceCriteria.cpp:289-458)
__global__ void k_update(Batch b) {
  const int s = b.chunk_struct[blockIdx.x];
  StructState& st = b.state[s];
  if (!iterating(st) || !st.need_solve) return;
  const StructInfo inf = b.info[s];
  const StructParams& p = b.params[s];
  const double* P = b.P + inf.dof_off;
  const int* d6 = b.dof_node6 + inf.dof_off;
  const int i1 = min(inf.n_free, b.chunk_start[blockIdx.x] + GF_RED_CHUNK);
  mag_t ia = 0, ib = 0, wa = 0, wb = 0;
  bool vf = false;
  for (int i = b.chunk_start[blockIdx.x] + threadIdx.x; i < i1; i += blockDim.x) {
    int q = d6[i];
    double x = P[i];
    double nv = b.disp[q] + x;
    b.disp[q] = nv;
    const mag_t a = mag(x), v = mag(nv);
    vf = vf || a >= MAG_HUGE;
    if (q % 6 < 3) {
      mag_max(ia, a);
      mag_max(wa, v);
    } else {
      mag_max(ib, a);
      mag_max(wb, v);
    }
  }
  RedScratch& R = b.red[s];
  red_max(&R.a, ia);
  red_max(&R.b, ib);
  red_max(&R.va, wa);
  red_max(&R.vb, wb);
  red_flag(&R.f, vf);
  if (!red_arrive(R, red_chunks(inf))) return;
  Red3 ri{}, rv{};
  if (threadIdx.x == 0) {
    ri.a = red_value(&R.a);
    ri.b = red_value(&R.b);
    rv.a = red_value(&R.va);
    rv.b = red_value(&R.vb);
    ri.f = *(volatile int*)&R.f;
    R = RedScratch{0ull, 0ull, 0ull, 0ull, 0, 0};
  }
  if (threadIdx.x == 0) {
    st.res_conv = 0;
    if (ri.f) st.diverged = 1;
    st.disp_crit = rv.a * p.disp_tol > p.disp_min * p.disp_tol ? p.disp_tol * rv.a : p.disp_min * p.disp_tol;
    st.rot_crit = rv.b * p.rot_tol > p.rot_min * p.rot_tol ? p.rot_tol * rv.b : p.rot_min * p.rot_tol;
    int conv = 1;
    if (st.disp_crit > p.divergence_ref || st.rot_crit > p.divergence_ref) {
      st.diverged = 1;
      conv = 0;
    } else {
      if (inf.has_force && ri.a > st.disp_crit) conv = 0;
      if (inf.has_moment && ri.b > st.rot_crit) conv = 0;
    }
    st.gl_conv = conv;
    st.last_inc = fmax(ri.a, ri.b);
  }
}

// Newton-loop end test, divergence, commit or bisection, step growth
// (reference src/Static.cpp:236-298).
__global__ void k_control(Batch b) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.n_struct) return;
  StructState& st = b.state[s];
  st.commit = 0;
  if (st.phase != PH_ITER) {
    if (st.phase == PH_START) atomicAdd(b.running, 1);
    return;
  }
  const StructParams& p = b.params[s];
  if (p.ray_on) st.ray_init = 1;  // the step's first iteration has formed C
  int both = st.res_conv && st.gl_conv;
  if ((st.it == p.max_it && !both) || (st.need_solve && st.info_fail)) st.diverged = 1;
  if (st.time_step < p.min_time_step && st.time != p.end_time) st.aborted = 1;
  st.it++;
  st.total_it++;
  if (st.need_solve) st.n_solves++;
  bool loop = !both && !st.diverged && !st.aborted;
  if (loop) {
    atomicAdd(b.running, 1);
    return;
  }
  st.mon_now = 0;
  if (!st.diverged) {
    st.converged_number++;
    st.commit = 1;
    st.commit_dyn = p.dynamic;
    st.convergence_counter++;
    // the monitor's rule, on the solution step that converged (reference
    // src/Static.cpp:268-276, src/Dynamic.cpp:392-399)
    st.conv_in_step++;
    const StructInfo& mi = b.info[s];
    if (mi.mon_n > 0 && !st.aborted && (st.conv_in_step % mi.mon_sample == 0 || st.time == p.end_time)) {
      st.mon_now = 1;
      st.mon_rows++;
    }
    if (st.it <= p.min_it || st.convergence_counter >= p.conv_increase) {
      st.time_step = st.time_step * p.inc_factor;
      if (st.time_step > p.max_time_step) st.time_step = p.max_time_step;
      st.convergence_counter = 0;
    }
  } else {
    st.time -= st.time_step;
    st.time_step = st.time_step / 2.0;
    st.diverged = 0;
    st.convergence_counter = 0;
    st.bisections++;
  }
  if ((st.time < p.end_time || st.diverged) && !st.aborted) {
    st.phase = PH_START;
    atomicAdd(b.running, 1);
  } else if (!st.aborted && st.step + 1 < b.info[s].n_steps) {
    // the next solution step (reference src/main.cpp:52-60) starts from
    // this state: its own step control, a fresh residual-criterion average
    // (src/Static.cpp:146, src/Dynamic.cpp:261), Rayleigh matrices formed
    // anew (Dynamic::Solve's `first`), and zero nodal velocities for a
    // Static step (ZerosVelAccel) or a Dynamic one with ZeroIC.  The commit
    // kernels of this pass still save the converged state of the step that
    // ended, with the ended step's Dynamic flag (commit_dyn) deciding
    // whether its velocities are saved, as SaveConfiguration does.
    st.step++;
    st.conv_in_step = 0;
    const StructParams np = b.step_params[b.info[s].step_off + st.step];
    b.params[s] = np;
    st.time = np.start_time;
    st.last_converged_time = np.start_time;
    st.time_step = np.time_step0;
    st.convergence_counter = 0;
    st.n_conv_evaluated = 0;
    st.ray_init = 0;
    st.zero_va = np.zero_va;
    st.phase = PH_START;
    atomicAdd(b.running, 1);
  } else {
    st.phase = st.aborted ? PH_ABORTED : PH_DONE;
  }
}

// SaveConfiguration: element Gauss-point history, a thread per Gauss point ...
__device__ __forceinline__ void commit_elem(const Batch& b, int t) {
  const int e = t >> 1;
  if (e >= b.n_elem) return;
  int s = b.estruct[e];
  if (!b.state[s].commit) return;
  double d[18];
  for (int j = 0; j < 3; ++j) {
    int nd = b.enodes[3 * e + j];
    for (int q = 0; q < 6; ++q) d[6 * j + q] = b.disp[(int64_t)nd * 6 + q];
  }
  beam_commit(b.bconst[e], b.bhist[e], b.baux[e], d, t & 1);
}

// ... and nodal configuration (reference src/Node.cpp:325-370)
__device__ __forceinline__ void commit_node(const Batch& b, int i) {
  if (i >= b.n_nodes) return;
  int s = b.node_struct[i];
  if (!b.state[s].commit) return;
  double* c = b.copy + (int64_t)i * 6;
  const double* d = b.disp + (int64_t)i * 6;
  for (int k = 0; k < 3; ++k) c[k] += d[k];
  V3<double> a1 = {{c[3], c[4], c[5]}}, a2 = {{d[3], d[4], d[5]}};
  V3<double> a3 = rodrigues_compose(a2, a1);
  for (int k = 0; k < 3; ++k) c[3 + k] = a3[k];
  M3<double> Q = rodrigues(a3);
  for (int k = 0; k < 9; ++k) b.Qn[(int64_t)i * 9 + k] = Q[k];
  // the converged velocities of a Dynamic step, also of its last step when
  // the next solution step's parameters are already in place
  if (b.state[s].commit_dyn)
    for (int k = 0; k < 6; ++k) {
      b.copy_vel[(int64_t)i * 6 + k] = b.vel[(int64_t)i * 6 + k];
      b.copy_accel[(int64_t)i * 6 + k] = b.accel[(int64_t)i * 6 + k];
    }
}

// Both, the nodes in the first node_ctas CTAs: neither reads what the other writes, and
// most passes commit nothing (a launch less: 1.3 us of the roll-up's 93 us a pass).
__global__ void __launch_bounds__(128) k_commit(Batch b, int node_ctas) {
  if ((int)blockIdx.x < node_ctas) commit_node(b, blockIdx.x * blockDim.x + threadIdx.x);
  else commit_elem(b, (blockIdx.x - node_ctas) * blockDim.x + threadIdx.x);
}

// Monitor line of one monitored node (Node::WriteMonitor, reference
// src/Node.cpp:227-320) after a committed step the monitor records: time,
// copy_coordinates, the load of every numbered DOF -- the elements'
// P_loading summed at the node (global_I_A at a free DOF, global_P_B at a
// constrained one; a DOF without a number keeps its last value) with the
// moments turned from pseudo-moments by Xi(alpha)^-T, alpha the node's
// rotation increment -- and the converged velocities and accelerations.
// One thread per monitored node.
__global__ void k_monitor_record(Batch b) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= b.mon_total) return;
  const int s = b.mon_struct[q];
  const StructState& st = b.state[s];
  if (!st.commit || !st.mon_now) return;
  const int row = st.mon_rows - 1;
  const int i = b.mon_node[q];
  double* L = b.mon_load + (int64_t)q * 6;
  double sum[6] = {0, 0, 0, 0, 0, 0};
  const int64_t ne = b.n_elem;
  for (int k = b.mon_adj_off[q]; k < b.mon_adj_off[q + 1]; ++k) {
    const int2 a = b.mon_adj[k];
    const int kind = a.y >> 6, at = a.y & 63;
    if (kind == 0) {
#pragma unroll
      for (int d = 0; d < 6; ++d) sum[d] += b.Fe[(int64_t)(6 * at + d) * ne + a.x];
    } else {
      const double* F = b.sh.Fe + (int64_t)a.x * 27;
#pragma unroll
      for (int d = 0; d < 3; ++d) sum[d] += F[3 * at + d];
      if (at >= 3)
#pragma unroll
        for (int d = 0; d < 3; ++d) sum[3 + d] += F[18 + 3 * (at - 3) + d];
    }
  }
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (b.gl[(int64_t)i * 6 + d] != -2) L[d] = sum[d];
  // pseudo-moment -> moment: m = Xi(alpha)^-T m
  const V3<double> al = {{b.disp[(int64_t)i * 6 + 3], b.disp[(int64_t)i * 6 + 4], b.disp[(int64_t)i * 6 + 5]}};
  const double g = 4.0 / (4.0 + dot(al, al));
  M3<double> A = skew(al), Xt;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) Xt[r * 3 + c] = g * ((r == c ? 1.0 : 0.0) + 0.5 * A[c * 3 + r]);
  const double c00 = Xt[4] * Xt[8] - Xt[5] * Xt[7], c01 = Xt[5] * Xt[6] - Xt[3] * Xt[8],
               c02 = Xt[3] * Xt[7] - Xt[4] * Xt[6];
  const double id = 1.0 / (Xt[0] * c00 + Xt[1] * c01 + Xt[2] * c02);
  M3<double> inv;
  inv[0] = c00 * id;
  inv[1] = (Xt[2] * Xt[7] - Xt[1] * Xt[8]) * id;
  inv[2] = (Xt[1] * Xt[5] - Xt[2] * Xt[4]) * id;
  inv[3] = c01 * id;
  inv[4] = (Xt[0] * Xt[8] - Xt[2] * Xt[6]) * id;
  inv[5] = (Xt[2] * Xt[3] - Xt[0] * Xt[5]) * id;
  inv[6] = c02 * id;
  inv[7] = (Xt[1] * Xt[6] - Xt[0] * Xt[7]) * id;
  inv[8] = (Xt[0] * Xt[4] - Xt[1] * Xt[3]) * id;
  const V3<double> m = mv(inv, V3<double>{{L[3], L[4], L[5]}});
  L[3] = m[0];
  L[4] = m[1];
  L[5] = m[2];
  if (row < 0 || row >= b.mon_cap) return;
  double* o = b.mon_rec + ((int64_t)q * b.mon_cap + row) * 25;
  o[0] = st.time;
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    o[1 + d] = b.copy[(int64_t)i * 6 + d];
    o[7 + d] = L[d];
    o[13 + d] = b.copy_vel[(int64_t)i * 6 + d];
    o[19 + d] = b.copy_accel[(int64_t)i * 6 + d];
  }
}

// Element-level entry (no batch): tangent and internal force, as
// k_beam_tangent forms them.  The caller's K has an element's 324 entries
// together, so the CTA's 32 matrices are put together in shared memory (an odd
// stride apart) and written coalesced.
constexpr int BE_LD = 325;
constexpr int BE_SMEM = MOUNT_SMEM + 32 * BE_LD * (int)sizeof(double);
__global__ void __launch_bounds__(MOUNT_THREADS) k_beam_elements(int n, const BeamConst* cs, const BeamHist* hs,
                                                                 const double* ds, double* Ks, double* fs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* P = reinterpret_cast<double*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.x * 32 + lane, g = warp & 1;
  if (e < n) {
    if (warp >= 2) {
      beam_gp_coef(cs[e], g, P + (g * MP_POINT + GP_COUNT) * 32 + lane, 32);
    } else {
      double d[18];
#pragma unroll
      for (int q = 0; q < 18; ++q) d[q] = ds[(int64_t)e * 18 + q];
      beam_gp(cs[e], hs[e], d, g, P + g * MP_POINT * 32 + lane, 32);
    }
  }
  __syncthreads();
  double* tile = P + 2 * MP_POINT * 32;
  double* K = tile + lane * BE_LD;
  if (e < n)
    beam_expand<MP_POINT, GP_COUNT>(P, warp, 4, lane,
                [&](int r, int q, double v) {
                  K[r + 18 * q] = v;
                  K[q + 18 * r] = v;
                },
                [&](int q, double v) { fs[(int64_t)e * 18 + q] = v; });
  __syncthreads();
  const int64_t k0 = (int64_t)blockIdx.x * 32 * 324;
  const int m = min(32, n - (int)blockIdx.x * 32) * 324;
  for (int x = threadIdx.x; x < m; x += MOUNT_THREADS) Ks[k0 + x] = tile[x / 324 * BE_LD + x % 324];
}

// Element-level inertia (no batch): M (18x18 column-major, global) and F.
__global__ void k_beam_inertia_elements(int n, const BeamConst* cs, const BeamHistAux* xs, const double* ds,
                                        const double* vs, const double* as, const double* a, double* Ms,
                                        double* Fs) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const BeamConst& c = cs[e];
  double d[18], vel[18], acc[18], f[18], D[18];
  for (int q = 0; q < 18; ++q) {
    d[q] = ds[(int64_t)e * 18 + q];
    vel[q] = vs[(int64_t)e * 18 + q];
    acc[q] = as[(int64_t)e * 18 + q];
    f[q] = 0.0;
  }
  double an[6];
  for (int q = 0; q < 6; ++q) an[q] = a[q];
  for (int g = 0; g < 2; ++g) {
    double fu[3], fa[3];
    beam_gp_inertia(c, xs[e], d, vel, acc, an, g, fu, fa, D + 9 * g, 1);
    for (int I = 0; I < 3; ++I)
      for (int i = 0; i < 3; ++i) {
        f[6 * I + i] += c.jac * c.N[g][I] * fu[i];
        f[6 * I + 3 + i] += c.jac * c.N[g][I] * fa[i];
      }
  }
  for (int r = 0; r < 18; ++r)
    for (int q = 0; q < 18; ++q) Ms[(int64_t)e * 324 + r + 18 * q] = beam_M_entry(c, D, D + 9, 1, an[0] * c.Mr, r, q);
  for (int q = 0; q < 18; ++q) Fs[(int64_t)e * 18 + q] = f[q];
}

__global__ void k_beam_commit(int n, const BeamConst* cs, BeamHist* hs, BeamHistAux* xs, const double* ds) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t >> 1;
  if (e >= n) return;
  double d[18];
  for (int q = 0; q < 18; ++q) d[q] = ds[(int64_t)e * 18 + q];
  beam_commit(cs[e], hs[e], xs[e], d, t & 1);
}

}  // namespace

void launch_modal_mass(const Batch& b, double* M, int64_t W, int kw, cudaStream_t st) {
  for (int c = 0; c < b.n_colors; ++c) {
    const int cnt = b.color_off[c + 1] - b.color_off[c];
    if (cnt > 0) k_modal_mass_beam<<<(cnt + 63) / 64, 64, 0, st>>>(b, c, M, W, kw);
  }
  if (b.sh.n_shells) launch_shell_modal_mass(b, M, W, kw, st);
}


// ---------------------------------------------------------------------------
void launch_beam_inertia(int n, const BeamConst* c, const BeamHistAux* x, const double* d, const double* v,
                         const double* a_acc, const double* a, double* M, double* F, cudaStream_t st) {
  if (n > 0) k_beam_inertia_elements<<<(n + 63) / 64, 64, 0, st>>>(n, c, x, d, v, a_acc, a, M, F);
}

void launch_beam_commit(int n, const BeamConst* c, BeamHist* h, BeamHistAux* x, const double* d, cudaStream_t st) {
  if (n > 0) k_beam_commit<<<(n + 63) / 64, 128, 0, st>>>(n, c, h, x, d);
}

void launch_init_state(const Batch& b, cudaStream_t st) {
  if (b.n_struct == 0) return;
  k_init_state<<<(b.n_struct + 127) / 128, 128, 0, st>>>(b);
}


static void set_attrs();

static void launch_mount(const Batch& b, cudaStream_t st, LaunchProf* prof);

static void launch_loads(const Batch& b, cudaStream_t st) {
  if (b.n_loads) k_loads<<<(b.n_struct + 3) / 4, 128, 0, st>>>(b);
}

void launch_iteration_partial(const Batch& b_in, cudaStream_t st) {
  set_attrs();
  Batch b = b_in;
  b.full_band = 1;  // the assembly view: every structure's band is filled
  int ns = b.n_struct;
  launch_step_begin(b, st);
  k_zero<<<dim3(8, ns), 256, 0, st>>>(b);
  launch_wide_zero(b, st);
  launch_mount(b, st, nullptr);
  launch_shell_mount(b, st);
  launch_loads(b, st);
  k_residual<<<b.n_chunks, 256, 0, st>>>(b);
}

// The stages of one Newton iteration for a caller that runs its own step
// control (gf_begin_step, gf_assemble, gf_set_increment, gf_commit): every
// structure's band is filled (the assembly view), as the caller reads K_AA.
void launch_step_begin(const Batch& b, cudaStream_t st) {
  k_step_begin<<<(b.n_struct + 63) / 64, 64, 0, st>>>(b);
  if (b.n_nodes) k_step_nodes<<<(b.n_nodes + 127) / 128, 128, 0, st>>>(b);
}

void launch_assembly(const Batch& b_in, cudaStream_t st) {
  set_attrs();
  Batch b = b_in;
  b.full_band = 1;
  int ns = b.n_struct;
  k_zero<<<dim3(8, ns), 256, 0, st>>>(b);
  launch_wide_zero(b, st);
  launch_mount(b, st, nullptr);
  launch_shell_mount(b, st);
  launch_loads(b, st);
  k_residual<<<b.n_chunks, 256, 0, st>>>(b);
}

void launch_increment(const Batch& b, cudaStream_t st) {
  k_update<<<b.n_chunks, 256, 0, st>>>(b);
  if (b.any_dynamic) k_update_dyn<<<(b.n_nodes + 127) / 128, 128, 0, st>>>(b);
}

static void launch_commit_nodes(const Batch& b, cudaStream_t st) {
  const int nodes = (b.n_nodes + 127) / 128, elems = (b.n_elem + 63) / 64;
  if (nodes + elems) k_commit<<<nodes + elems, 128, 0, st>>>(b, nodes);
}

void launch_commit(const Batch& b, cudaStream_t st) {
  if (b.sh.n_shells) launch_shell_commit(b, st);
  launch_commit_nodes(b, st);
}

// Shared-memory limits of the large kernels (the served path's builder thread and the
// caller's thread may both get here first).
static void set_attrs() {
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_beam_tangent<2>, MOUNT_SMEM_SPLIT},
                    {(const void*)k_band_solve, (RING * GF_LDB + RING) * (int)sizeof(double)}});
}

const char* kernel_class_name(int k) {
  static const char* names[KC_COUNT] = {"step_begin", "zero", "beam_tangent", "loads", "residual", "band_solve",
                                        "update", "control", "commit_elems", "commit_nodes", "chain_solve", "scatter",
                                        "shell_mount", "wide_diag", "wide_trsm", "wide_update", "wide_subst",
                                        "wide_refine"};
  return k >= 0 && k < KC_COUNT ? names[k] : "?";
}


static void launch_mount(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  if (b.n_elem == 0) return;
  {
    ProfScope q(prof, st, KC_MOUNT);
    const int n = (b.n_elem + 31) / 32;
    if (b.n_elem <= MOUNT_SPLIT) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(2 * n);
      cfg.blockDim = dim3(MOUNT_THREADS);
      cfg.dynamicSmemBytes = MOUNT_SMEM_SPLIT;
      cfg.stream = st;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, k_beam_tangent<2>, b);
    } else {
      k_beam_tangent<1><<<n, MOUNT_THREADS, MOUNT_SMEM_BATCH, st>>>(b);
    }
    // the pressure's load stiffness is part of the K_e that Rayleigh damping
    // reads (the reference mounts loads before damping)
    if (b.n_pipe_press) k_pipe_pressure<<<(b.n_pipe_press + 31) / 32, PP_THREADS, 0, st>>>(b);
    if (b.any_rayleigh) k_beam_rayleigh<<<(b.n_elem + 31) / 32, RAY_THREADS, 0, st>>>(b);
  }
  if (!b.full_band && b.chain_sym.n_elem + b.chain_gen.n_elem == b.n_elem) {
    // chains only: the residual is all the scatter would assemble
    ProfScope q(prof, st, KC_SCATTER);
    const int64_t nt = (int64_t)b.n_nodes * 6;
    k_chain_gather_f<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(b);
    return;
  }
  for (int c = 0; c < b.n_colors; ++c) {
    int cnt = b.color_off[c + 1] - b.color_off[c];
    if (cnt <= 0) continue;
    ProfScope q(prof, st, KC_SCATTER);
    k_beam_scatter<<<(cnt + 3) / 4, 128, 0, st>>>(b, c);
  }
}

void launch_iteration(const Batch& b, cudaStream_t st, bool commit_kernels, LaunchProf* prof) {
  set_attrs();
  int ns = b.n_struct;
  { ProfScope q(prof, st, KC_STEP_BEGIN); launch_step_begin(b, st); }
  { ProfScope q(prof, st, KC_ZERO); k_zero<<<dim3(8, ns), 256, 0, st>>>(b); }
  if (b.sh.n_wide) { ProfScope q(prof, st, KC_ZERO); launch_wide_zero(b, st); }
  launch_mount(b, st, prof);
  if (b.sh.n_shells) { ProfScope q(prof, st, KC_SHELL); launch_shell_mount(b, st); }
  { ProfScope q(prof, st, KC_LOADS); launch_loads(b, st); }
  { ProfScope q(prof, st, KC_RESIDUAL); k_residual<<<b.n_chunks, 256, 0, st>>>(b); }
  if (b.n_band) { ProfScope q(prof, st, KC_SOLVE); launch_band_solve(b, st); }
  if (b.chain_gen.n_elem) { ProfScope q(prof, st, KC_CHAIN); launch_gen_chains(b, b.chain_gen, st); }
  if (b.chain_sym.n_elem) { ProfScope q(prof, st, KC_CHAIN); launch_sym_chains(b, b.chain_sym, st); }
  launch_shell_solve(b, st, prof);
  { ProfScope q(prof, st, KC_UPDATE); launch_increment(b, st); }
  { ProfScope q(prof, st, KC_CONTROL); k_control<<<(ns + 127) / 128, 128, 0, st>>>(b); }
  if (commit_kernels) {
    if (b.sh.n_shells) { ProfScope q(prof, st, KC_COMMIT_ELEMS); launch_shell_commit(b, st); }
    { ProfScope q(prof, st, KC_COMMIT_NODES); launch_commit_nodes(b, st); }
    if (b.mon_total) k_monitor_record<<<(b.mon_total + 127) / 128, 128, 0, st>>>(b);
  }
}

namespace {
template <typename T> __global__ void k_fp_probe(T* out, int iters, T a, T c) {
  T x0 = threadIdx.x, x1 = x0 + T(1), x2 = x0 + T(2), x3 = x0 + T(3), x4 = x0 + T(4), x5 = x0 + T(5),
    x6 = x0 + T(6), x7 = x0 + T(7);
  for (int i = 0; i < iters; ++i) {
    x0 = x0 * a + c; x1 = x1 * a + c; x2 = x2 * a + c; x3 = x3 * a + c;
    x4 = x4 * a + c; x5 = x5 * a + c; x6 = x6 * a + c; x7 = x7 * a + c;
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}
}  // namespace

void launch_fp_probe(bool fp64, void* out, int blocks, int threads, int iters, cudaStream_t st) {
  if (fp64)
    k_fp_probe<double><<<blocks, threads, 0, st>>>(static_cast<double*>(out), iters, 0.999, 0.001);
  else
    k_fp_probe<float><<<blocks, threads, 0, st>>>(static_cast<float*>(out), iters, 0.999f, 0.001f);
}

void launch_band_solve(const Batch& b, cudaStream_t st) {
  k_band_solve<<<b.n_struct, SOLVE_THREADS, (RING * GF_LDB + RING) * sizeof(double), st>>>(b);
}

void launch_beam_elements(int n, const BeamConst* c, const BeamHist* h, const double* d, double* K,
                          double* f, cudaStream_t st) {
  if (n <= 0) return;
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_beam_elements, BE_SMEM}});
  k_beam_elements<<<(n + 31) / 32, MOUNT_THREADS, BE_SMEM, st>>>(n, c, h, d, K, f);
}

}  // namespace gf
