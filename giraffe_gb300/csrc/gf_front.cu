// Multifrontal LU on the device (see gf_front.h): assembly of K_AA into the
// fronts, elimination height by height, back substitution.  No pivoting (a
// zero or non-finite pivot sets info_fail, as the reference's solver failure).
//
// The right-hand side is column f of every front, so the forward substitution
// is part of the elimination.  Per height, bottom up:
//   k_mf_extend   the children's Schur complements added into their parents
//                 (one launch per child ordinal: the children of a front touch
//                 common entries)
//   k_mf_small    fronts of at most MF_SMALL rows: one CTA each, in shared
//                 memory
//   larger fronts, MF_NB pivots per panel:
//     k_mf_diag   LU of the panel's diagonal block
//     k_mf_trsm   L21 = A21 U11^-1 and U12 = L11^-1 A12
//     k_mf_panel  the rest of the pivot rows and columns
//   k_mf_schur    the boundary block, once all pivots are done: C -= L21 U12
// and top down
//   k_mf_back     x of the front's own DOFs from its boundary's.
// The diagonal of U is stored as its reciprocal.
//
// What bounds it: an FP64 warp instruction holds its sub-partition's FP64 unit
// for 64 cycles whatever its active lanes (measured: one warp issues a DFMA
// every 64 cycles at any instruction-level parallelism, an SM one every 19),
// so the large fronts are bound by FP64 throughput and the chain of panels by
// the dependent results of each pivot.
#include <cuda_runtime.h>

#include <cfloat>

#include "gf_front.h"
#include "gf_kernels.cuh"
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

namespace {

// A structure whose K_AA this launch factors (in the FP64 fallback launches of
// the mixed path only those whose refinement did not finish).
__device__ __forceinline__ bool mf_active(const Batch& b, int s) {
  const StructState& st = b.state[s];
  return st.phase == PH_ITER && st.need_solve && (!b.sh.fp64_pass || st.ir_fb);
}

__device__ __forceinline__ double mf_rcp(double p) { return rcp64(p); }
__device__ __forceinline__ float mf_rcp(float p) { return __frcp_rn(p); }
__device__ __forceinline__ double mfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mfma(float a, float b, float c) { return fmaf(a, b, c); }

template <typename T> __device__ __forceinline__ T* mf_mat(const Batch& b, const Front& F) {
  return reinterpret_cast<T*>(b.sh.mf.F) + F.off;
}
template <typename T> __device__ __forceinline__ T* mf_x(const Batch& b) { return reinterpret_cast<T*>(b.sh.mf.x); }
__device__ __forceinline__ double* mf_rhs(const Batch& b, double*) { return b.P; }
__device__ __forceinline__ float* mf_rhs(const Batch& b, float*) { return b.sh.r32; }

// A zero or non-finite pivot: the FP64 LU's solver failure; the FP32 LU of the
// mixed path hands the solve to the FP64 fallback.
template <typename T> __device__ __forceinline__ void mf_fail(const Batch& b, int s) {
  if (sizeof(T) == 8) b.state[s].info_fail = 1;
  else b.state[s].ir_fb = 1;
}
template <typename T> __device__ __forceinline__ bool mf_bad(T p) { return !(p != T(0)) || !isfinite(p); }

// Index of elimination position q in front F (own DOFs, then the boundary).
__device__ __forceinline__ int mf_local(const FrontData& d, const Front& F, int q) {
  if (q < F.dof0 + F.s) return q - F.dof0;
  const int* B = d.bnd + F.bnd;
  int lo = 0, hi = F.f - F.s - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (B[mid] < q) lo = mid + 1;
    else hi = mid;
  }
  return F.s + lo;
}
// Place of the entry (row, column) given by elimination positions: the front
// of the earlier one.
__device__ __forceinline__ int64_t mf_entry(const FrontData& d, int pr, int pc) {
  const Front& F = d.fronts[d.dof_front[min(pr, pc)]];
  return F.off + mf_local(d, F, pr) + (int64_t)F.ld * mf_local(d, F, pc);
}

}  // namespace

// Destinations of the element matrices' entries, once per batch.
__global__ void k_mf_map(Batch b) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)b.sh.n_shells * 729) return;
  const int e = (int)(t / 729), x = (int)(t % 729), r = x % 27, q = x / 27;
  const int s = b.sh.sstruct[e];
  const StructInfo& inf = b.info[s];
  const int* nd = b.sh.snodes + 6 * e;
  auto dof = [&](int a) {
    const int node = a < 18 ? nd[a / 3] : nd[3 + (a - 18) / 3];
    return b.gl[(int64_t)node * 6 + (a < 18 ? a % 3 : 3 + (a - 18) % 3)];
  };
  const int gr = dof(r), gq = dof(q);
  int to = -1;
  if (gr >= 0 && gq >= 0) {
    const FrontData& d = b.sh.mf;
    to = (int)(mf_entry(d, d.pos[inf.dof_off + gr], d.pos[inf.dof_off + gq]) - d.base[s]);
  }
  b.sh.mf.map[t] = to;
}

// Clears the fronts of the structures that solve.
template <typename T> __global__ void k_mf_zero(Batch b) {
  const int s = b.sh.wide_structs[blockIdx.y];
  if (!mf_active(b, s)) return;
  const FrontData& d = b.sh.mf;
  float4* p = reinterpret_cast<float4*>(reinterpret_cast<T*>(d.F) + d.base[s]);
  const int64_t n = d.size[s] * (int64_t)sizeof(T) / 16;  // sizes are multiples of 32 entries
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// MountGlobal into the fronts: a warp per element of one colour (no two
// elements of a colour share a node, so no two writers meet).
template <typename T> __global__ void k_mf_elements(Batch b, int color) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int lo = b.sh.color_off[color], hi = b.sh.color_off[color + 1];
  if (lo + w >= hi) return;
  const int e = b.sh.color_elems[lo + w], s = b.sh.sstruct[e];
  if (!mf_active(b, s)) return;
  const double* K = b.sh.Ke + (int64_t)e * 729;
  const int* map = b.sh.mf.map + (int64_t)e * 729;
  T* F = reinterpret_cast<T*>(b.sh.mf.F) + b.sh.mf.base[s];
  for (int x = lane; x < 729; x += 32) {
    const int to = map[x];
    if (to >= 0) F[to] += (T)K[x];
  }
}

// The nodal load stiffness (3x3 rotation blocks kept per node).
template <typename T> __global__ void k_mf_nodes(Batch b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n_nodes) return;
  const int s = b.node_struct[i];
  const StructInfo& inf = b.info[s];
  if (!inf.wide || !inf.n_loads || !mf_active(b, s)) return;
  const FrontData& d = b.sh.mf;
  for (int r = 0; r < 3; ++r)
    for (int q = 0; q < 3; ++q) {
      const double v = b.nodeK[(int64_t)i * 9 + r * 3 + q];
      const int gr = b.gl[(int64_t)i * 6 + 3 + r], gq = b.gl[(int64_t)i * 6 + 3 + q];
      if (v != 0.0 && gr >= 0 && gq >= 0)
        reinterpret_cast<T*>(d.F)[mf_entry(d, d.pos[inf.dof_off + gr], d.pos[inf.dof_off + gq])] += (T)v;
    }
}

// Right-hand sides into column f of the fronts, and the solution back.
template <typename T> __global__ void k_mf_rhs(Batch b) {
  const int s = b.sh.wide_structs[blockIdx.y];
  if (!mf_active(b, s)) return;
  const StructInfo& inf = b.info[s];
  const FrontData& d = b.sh.mf;
  const T* P = mf_rhs(b, (T*)nullptr) + inf.dof_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x) {
    const int p = d.pos[inf.dof_off + i];
    const Front& F = d.fronts[d.dof_front[p]];
    mf_mat<T>(b, F)[(int64_t)F.f * F.ld + p - F.dof0] = P[i];
  }
}
template <typename T> __global__ void k_mf_out(Batch b) {
  const int s = b.sh.wide_structs[blockIdx.y];
  if (!mf_active(b, s)) return;
  const StructInfo& inf = b.info[s];
  T* P = mf_rhs(b, (T*)nullptr) + inf.dof_off;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < inf.n_free; i += gridDim.x * blockDim.x)
    P[i] = mf_x<T>(b)[b.sh.mf.pos[inf.dof_off + i]];
}

// Extend-add: sixteen columns of a child's Schur complement (and right-hand
// side) into its parent, a warp per column.
template <typename T> __global__ void __launch_bounds__(256) k_mf_extend(Batch b, int job0) {
  const FrontData& d = b.sh.mf;
  const int2 job = d.ext_jobs[job0 + blockIdx.x];
  const Front C = d.fronts[job.x];
  if (!mf_active(b, C.slot)) return;
  const Front P = d.fronts[C.parent];
  const int u = C.f - C.s, lane = threadIdx.x & 31;
  const int* rel = d.rel + C.rel;
  const T* S = mf_mat<T>(b, C);
  T* Q = mf_mat<T>(b, P);
  for (int j = job.y + (threadIdx.x >> 5); j < min(job.y + 16, u + 1); j += 8) {
    const T* sc = S + (int64_t)(C.s + j) * C.ld + C.s;
    T* qc = Q + (int64_t)(j < u ? rel[j] : P.f) * P.ld;
    for (int i = lane; i < u; i += 32) qc[rel[i]] += sc[i];
  }
}

// Partial LU of a front held in shared memory, s pivots, one CTA: the pivot
// warp (warp 3) owns column k + 1 at step k (its update, the next pivot's
// reciprocal and multipliers) while the others update the rest of the trailing
// block, packed densely over their lanes; one barrier closes the step.  Many
// CTAs share an SM, so one front's pivot chain runs beside another's updates.
constexpr int MF_SMALL_THREADS = 128;
template <typename T> __global__ void __launch_bounds__(MF_SMALL_THREADS) k_mf_small(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const Front F = d.fronts[d.list[off + blockIdx.x]];
  if (!mf_active(b, F.slot)) return;
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* A = reinterpret_cast<T*>(mf_raw);
  const int f = F.f, s = F.s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T* G = mf_mat<T>(b, F);
  for (int x = tid; x < ld * (f + 1); x += MF_SMALL_THREADS) A[x] = G[x];
  __syncthreads();
  bool bad = false;
  auto pivot = [&](int k) {  // reciprocal and multipliers of column k
    const T p = A[k + k * ld];
    bad = bad || mf_bad(p);
    const T r = mf_rcp(p);
    __syncwarp();
    for (int i = k + 1 + lane; i < f; i += 32) A[i + k * ld] *= r;
    if (lane == 0) A[k + k * ld] = r;
  };
  if (warp == 3 && s > 0) pivot(0);
  __syncthreads();
  for (int k = 0; k < s; ++k) {
    const int m = f - 1 - k;      // trailing rows
    const bool next = k + 1 < s;  // column k + 1 is a pivot column
    if (next && warp == 3) {
      const T u = A[k + (k + 1) * ld];
      for (int i = k + 1 + lane; i < f; i += 32) A[i + (k + 1) * ld] = mfma(-A[i + k * ld], u, A[i + (k + 1) * ld]);
      __syncwarp();
      pivot(k + 1);
    } else if (m > 0) {
      const int c0 = next ? k + 2 : k + 1, nt = next ? 96 : 128;
      const int tot = m * (f + 1 - c0);
      const float inv_m = 1.0f / (float)m;
      for (int e = tid; e < tot; e += nt) {
        const int jj = __float2int_rz(((float)e + 0.5f) * inv_m);  // e / m, exact for e < 2^14
        const int i = k + 1 + e - jj * m, j = c0 + jj;
        A[i + j * ld] = mfma(-A[i + k * ld], A[k + j * ld], A[i + j * ld]);
      }
    }
    __syncthreads();
  }
  for (int x = tid; x < ld * (f + 1); x += MF_SMALL_THREADS) G[x] = A[x];
  if (bad && lane == 0) mf_fail<T>(b, F.slot);
}

// LU of the diagonal block of panel p of the large fronts of a height, one CTA
// each; as k_mf_small, on the panel's block alone.
constexpr int MF_DIAG_THREADS = 160;
template <typename T> __global__ void __launch_bounds__(MF_DIAG_THREADS) k_mf_diag(Batch b, int off, int p) {
  const FrontData& d = b.sh.mf;
  const Front F = d.fronts[d.list[off + blockIdx.x]];
  if (!mf_active(b, F.slot)) return;
  const int k0 = p * MF_NB, nb = min(MF_NB, F.s - k0), ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T* G = mf_mat<T>(b, F) + k0 + (int64_t)k0 * ld;
  __shared__ T A[MF_NB][MF_NB + 1];  // A[j][i]: column j, row i
  for (int x = tid; x < nb * MF_NB; x += MF_DIAG_THREADS) {
    const int i = x % MF_NB, j = x / MF_NB;
    if (i < nb) A[j][i] = G[i + (int64_t)j * ld];
  }
  __syncthreads();
  bool bad = false;
  auto pivot = [&](int k) {
    const T q = A[k][k];
    bad = bad || mf_bad(q);
    const T r = mf_rcp(q);
    __syncwarp();
    if (lane > k && lane < nb) A[k][lane] *= r;
    if (lane == k) A[k][k] = r;
  };
  if (warp == 4) pivot(0);
  __syncthreads();
  for (int k = 0; k + 1 < nb; ++k) {
    const int m = nb - 1 - k;
    if (warp == 4) {
      const T u = A[k + 1][k];
      if (lane > k && lane < nb) A[k + 1][lane] = mfma(-A[k][lane], u, A[k + 1][lane]);
      __syncwarp();
      pivot(k + 1);
    } else {
      const int tot = m * (m - 1);
      const float inv_m = 1.0f / (float)m;
      for (int e = tid; e < tot; e += 128) {
        const int jj = __float2int_rz(((float)e + 0.5f) * inv_m);
        const int i = k + 1 + e - jj * m, j = k + 2 + jj;
        A[j][i] = mfma(-A[k][i], A[j][k], A[j][i]);
      }
    }
    __syncthreads();
  }
  for (int x = tid; x < nb * MF_NB; x += MF_DIAG_THREADS) {
    const int i = x % MF_NB, j = x / MF_NB;
    if (i < nb) G[i + (int64_t)j * ld] = A[j][i];
  }
  if (bad && lane == 0) mf_fail<T>(b, F.slot);
}

// L21 = A21 U11^-1 (blockIdx.x < nlow: 32 rows below the panel) and U12 =
// L11^-1 A12 (32 columns right of it, the right-hand side among them).  Four
// lanes per row (column), lane q holding its entries 4 j + q in registers, the
// finished entry broadcast within the four: 176 FP64 warp instructions per
// eight rows (132 with a thread per row, but four times the latency).
template <typename T> __global__ void __launch_bounds__(128) k_mf_trsm(Batch b, int off, int p, int nlow) {
  const FrontData& d = b.sh.mf;
  const Front F = d.fronts[d.list[off + blockIdx.y]];
  if (!mf_active(b, F.slot)) return;
  const int k0 = p * MF_NB, nb = min(MF_NB, F.s - k0), k1 = k0 + nb, ld = F.ld, tid = threadIdx.x;
  const bool lower = (int)blockIdx.x < nlow;
  const int first = k1 + 32 * (lower ? (int)blockIdx.x : (int)blockIdx.x - nlow);
  if (first >= (lower ? F.f : F.f + 1)) return;
  T* G = mf_mat<T>(b, F);
  __shared__ T U[MF_NB][MF_NB + 1];  // U[k][j]: the factor this side reads, identity beyond nb
  for (int x = tid; x < MF_NB * MF_NB; x += 128) {
    const int i = x % MF_NB, j = x / MF_NB;
    T v = i == j ? T(1) : T(0);
    if (i < nb && j < nb && (lower ? i <= j : i > j)) v = G[k0 + i + (int64_t)(k0 + j) * ld];
    if (lower) U[i][j] = v;  // U11(i, j), the reciprocal on the diagonal
    else U[j][i] = v;        // L11(i, j) at [j][i]
  }
  const int r = tid >> 2, q = tid & 3, g = first + r;  // row (lower) or column of the front
  const bool live = g < (lower ? F.f : F.f + 1);
  T v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 4 * j + q;
    v[j] = (live && c < nb) ? (lower ? G[g + (int64_t)(k0 + c) * ld] : G[k0 + c + (int64_t)g * ld]) : T(0);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < MF_NB; ++k) {
    // the finished entry k, from the lane that holds it
    T x = v[k >> 2];
    if (lower) x *= U[k][k];
    x = __shfl_sync(0xffffffffu, x, k & 3, 4);
    if (lower && q == (k & 3)) v[k >> 2] = x;
#pragma unroll
    for (int j = k >> 2; j < 8; ++j)
      if (4 * j + q > k) v[j] = mfma(-x, U[k][4 * j + q], v[j]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 4 * j + q;
    if (!live || c >= nb) continue;
    if (lower) G[g + (int64_t)(k0 + c) * ld] = v[j];
    else G[k0 + c + (int64_t)g * ld] = v[j];
  }
}

// The pivot rows and columns right of and below panel p: rows k1..s-1 of all
// later columns (blockIdx.x < na) and the boundary rows of the later pivot
// columns, minus L U over the panel's pivots.  16 x 32 tiles, so that the few
// tiles of the top fronts spread over the SMs (a tile holds an SM's FP64 units
// for 512 warp instructions, about 5 us).
template <typename T>
__global__ void __launch_bounds__(128) k_mf_panel(Batch b, int off, int p, int na, int nca, int ncb) {
  const FrontData& d = b.sh.mf;
  const Front F = d.fronts[d.list[off + blockIdx.y]];
  if (!mf_active(b, F.slot)) return;
  const int k0 = p * MF_NB, k1 = k0 + MF_NB, ld = F.ld, tid = threadIdx.x;
  if (k1 >= F.s) return;
  int r0, c0, r1, c1;
  if ((int)blockIdx.x < na) {
    r0 = k1 + 16 * ((int)blockIdx.x / nca);
    c0 = k1 + 32 * ((int)blockIdx.x % nca);
    r1 = F.s;
    c1 = F.f + 1;
  } else {
    const int x = (int)blockIdx.x - na;
    r0 = F.s + 16 * (x / ncb);
    c0 = k1 + 32 * (x % ncb);
    r1 = F.f;
    c1 = F.s;
  }
  if (r0 >= r1 || c0 >= c1) return;
  T* G = mf_mat<T>(b, F);
  __shared__ T Ls[MF_NB][17];  // [k][row]
  __shared__ T Us[32][MF_NB + 1];  // [column][k]
  for (int x = tid; x < MF_NB * 16; x += 128) {
    const int i = x & 15, k = x >> 4;
    Ls[k][i] = r0 + i < r1 ? G[r0 + i + (int64_t)(k0 + k) * ld] : T(0);
  }
  for (int x = tid; x < 32 * MF_NB; x += 128) {
    const int k = x & 31, c = x >> 5;
    Us[c][k] = c0 + c < c1 ? G[k0 + k + (int64_t)(c0 + c) * ld] : T(0);
  }
  const int i = tid & 15, cg = tid >> 4;  // row, columns cg + 8 q
  T acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    acc[q] = (r0 + i < r1 && c0 + cg + 8 * q < c1) ? G[r0 + i + (int64_t)(c0 + cg + 8 * q) * ld] : T(0);
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < MF_NB; ++k) {
    const T l = -Ls[k][i];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = mfma(l, Us[cg + 8 * q][k], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (r0 + i < r1 && c0 + cg + 8 * q < c1) G[r0 + i + (int64_t)(c0 + cg + 8 * q) * ld] = acc[q];
}

// The Schur complement of the large fronts of a height: C -= L21 U12 over all
// pivots, 32 x 32 tiles, 2 x 4 outputs per thread, the next 32 pivots' operands
// loading into registers while this one's products run.
template <typename T> __global__ void __launch_bounds__(128) k_mf_schur(Batch b, int job0) {
  const FrontData& d = b.sh.mf;
  const int2 job = d.schur_jobs[job0 + blockIdx.x];
  const Front F = d.fronts[job.x];
  if (!mf_active(b, F.slot)) return;
  const int r0 = F.s + 32 * (job.y & 0xFFFF), c0 = F.s + 32 * (job.y >> 16), ld = F.ld, s = F.s, tid = threadIdx.x;
  T* G = mf_mat<T>(b, F);
  __shared__ T Ls[2][32][33];  // [k][row]
  __shared__ T Us[2][32][33];  // [column][k]
  const int lx = tid & 31, ly = tid >> 5;
  const bool row_ok = r0 + lx < F.f;
  T lr[8], ur[8];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int y = ly + 4 * q;
      lr[q] = (row_ok && k0 + y < s) ? G[r0 + lx + (int64_t)(k0 + y) * ld] : T(0);
      ur[q] = (c0 + y <= F.f && k0 + lx < s) ? G[k0 + lx + (int64_t)(c0 + y) * ld] : T(0);
    }
  };
  auto stash = [&](int w) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      Ls[w][ly + 4 * q][lx] = lr[q];
      Us[w][ly + 4 * q][lx] = ur[q];
    }
  };
  const int ti = tid & 15, tj = tid >> 4;  // rows ti, ti + 16; columns tj + 8 q
  T acc[2][4];
  fetch(0);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + ti + 16 * h, c = c0 + tj + 8 * q;
      acc[h][q] = (r < F.f && c <= F.f) ? G[r + (int64_t)c * ld] : T(0);
    }
  stash(0);
  __syncthreads();
  for (int k0 = 0, w = 0; k0 < s; k0 += 32, w ^= 1) {
    if (k0 + 32 < s) fetch(k0 + 32);
    const int kn = min(32, s - k0);
    for (int k = 0; k < kn; ++k) {
      const T l0 = -Ls[w][k][ti], l1 = -Ls[w][k][ti + 16];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const T u = Us[w][tj + 8 * q][k];
        acc[0][q] = mfma(l0, u, acc[0][q]);
        acc[1][q] = mfma(l1, u, acc[1][q]);
      }
    }
    if (k0 + 32 < s) stash(w ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + ti + 16 * h, c = c0 + tj + 8 * q;
      if (r < F.f && c <= F.f) G[r + (int64_t)c * ld] = acc[h][q];
    }
}

// Back substitution of every front of a height, one CTA each: w = y - U12 x2,
// then x1 = U11^-1 w in blocks of 32 (warp 0 solves a block's triangle, then
// every thread takes its rows above it).
constexpr int MF_BACK_THREADS = 256;
template <typename T> __global__ void __launch_bounds__(MF_BACK_THREADS) k_mf_back(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const Front F = d.fronts[d.list[off + blockIdx.x]];
  if (!mf_active(b, F.slot)) return;
  const int f = F.f, s = F.s, u = f - s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const T* G = mf_mat<T>(b, F);
  T* x = mf_x<T>(b);
  const int* B = d.bnd + F.bnd;
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* w = reinterpret_cast<T*>(mf_raw);  // [f]: w of the own DOFs, then x2
  T* part = w + f + (f & 1);            // [8][32]
  for (int i = tid; i < s; i += MF_BACK_THREADS) w[i] = G[i + (int64_t)f * ld];
  for (int i = tid; i < u; i += MF_BACK_THREADS) w[s + i] = x[B[i]];
  __syncthreads();
  if (u > 0)
    for (int i0 = 0; i0 < s; i0 += 32) {
      // 32 rows, the eight warps an eighth of the columns each
      const int i = i0 + lane;
      T acc = T(0);
      if (i < s)
        for (int j = s + warp; j < f; j += 8) acc = mfma(G[i + (int64_t)j * ld], w[j], acc);
      part[warp * 32 + lane] = acc;
      __syncthreads();
      if (warp == 0 && i < s) {
        T t = part[lane];
        for (int q = 1; q < 8; ++q) t += part[q * 32 + lane];
        w[i] -= t;
      }
      __syncthreads();
    }
  for (int j0 = (s - 1) / 32 * 32; j0 >= 0; j0 -= 32) {
    const int nb = min(32, s - j0);
    if (warp == 0) {
      T v = lane < nb ? w[j0 + lane] : T(0);
      for (int k = nb - 1; k >= 0; --k) {
        const T ukk = G[j0 + k + (int64_t)(j0 + k) * ld];  // the reciprocal
        const T uk = lane < k ? G[j0 + lane + (int64_t)(j0 + k) * ld] : T(0);
        const T xk = __shfl_sync(0xffffffffu, v, k) * ukk;
        if (lane == k) v = xk;
        if (lane < k) v = mfma(-uk, xk, v);
      }
      if (lane < nb) {
        w[j0 + lane] = v;
        x[F.dof0 + j0 + lane] = v;
      }
    }
    __syncthreads();
    for (int i = tid; i < j0; i += MF_BACK_THREADS) {
      T a0 = T(0), a1 = T(0);
      for (int k = 0; k < nb; k += 2) {
        a0 = mfma(G[i + (int64_t)(j0 + k) * ld], w[j0 + k], a0);
        if (k + 1 < nb) a1 = mfma(G[i + (int64_t)(j0 + k + 1) * ld], w[j0 + k + 1], a1);
      }
      w[i] -= a0 + a1;
    }
    __syncthreads();
  }
}

// Forward substitution alone, on fronts that hold their LU: every front of a
// height, one CTA each.  w = the right-hand side of the own DOFs with what the
// children leave (their column f, read through their parent indices, one child
// after the other), then y1 = L11^-1 w1 in blocks of 32 and w2 -= L21 y1; both
// into column f.
template <typename T> __global__ void __launch_bounds__(MF_BACK_THREADS) k_mf_fwd(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const int id = d.list[off + blockIdx.x];
  const Front F = d.fronts[id];
  if (!mf_active(b, F.slot)) return;
  const int f = F.f, s = F.s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T* G = mf_mat<T>(b, F);
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* w = reinterpret_cast<T*>(mf_raw);  // [f]
  const T* P = mf_rhs(b, (T*)nullptr);
  for (int i = tid; i < f; i += MF_BACK_THREADS) w[i] = i < s ? P[d.dof_at[F.dof0 + i]] : T(0);
  for (int k = d.kid_off[id]; k < d.kid_off[id + 1]; ++k) {
    __syncthreads();
    const Front C = d.fronts[d.kids[k]];
    const T* cw = mf_mat<T>(b, C) + (int64_t)C.f * C.ld + C.s;
    const int* rel = d.rel + C.rel;
    for (int i = tid; i < C.f - C.s; i += MF_BACK_THREADS) w[rel[i]] += cw[i];
  }
  __syncthreads();
  for (int j0 = 0; j0 < s; j0 += 32) {
    const int nb = min(32, s - j0);
    if (warp == 0) {
      T v = lane < nb ? w[j0 + lane] : T(0);
      for (int k = 0; k + 1 < nb; ++k) {
        const T l = lane > k && lane < nb ? G[j0 + lane + (int64_t)(j0 + k) * ld] : T(0);
        const T yk = __shfl_sync(0xffffffffu, v, k);
        if (lane > k) v = mfma(-l, yk, v);
      }
      if (lane < nb) w[j0 + lane] = v;
    }
    __syncthreads();
    for (int i = j0 + nb + tid; i < f; i += MF_BACK_THREADS) {
      T a0 = T(0), a1 = T(0);
      for (int k = 0; k < nb; k += 2) {
        a0 = mfma(G[i + (int64_t)(j0 + k) * ld], w[j0 + k], a0);
        if (k + 1 < nb) a1 = mfma(G[i + (int64_t)(j0 + k + 1) * ld], w[j0 + k + 1], a1);
      }
      w[i] -= a0 + a1;
    }
    __syncthreads();
  }
  for (int i = tid; i < f; i += MF_BACK_THREADS) G[i + (int64_t)f * ld] = w[i];
}

// ---- standalone systems (one structure): matrix entries into the fronts ----

// A CSR row per thread: distinct rows own distinct entries, and the entries of
// a row are summed in order, so repeated entries add up the same way each run.
__global__ void k_mf_csr(Batch b, int n, const int* rp, const int* ci, const double* v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const FrontData& d = b.sh.mf;
  const int pi = d.pos[i];
  for (int k = rp[i]; k < rp[i + 1]; ++k) d.F[mf_entry(d, pi, d.pos[ci[k]])] += v[k];
}

// The stored entries of LAPACK GB columns (entry (i, j) at ab[kl + ku + i - j +
// j ldab]), one thread each.
__global__ void k_mf_band(Batch b, int n, int kl, int ku, int ldab, const double* ab) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int W = kl + ku + 1;
  if (t >= (int64_t)n * W) return;
  const int j = (int)(t / W), i = j - ku + (int)(t % W);
  if (i < 0 || i >= n) return;
  const FrontData& d = b.sh.mf;
  d.F[mf_entry(d, d.pos[i], d.pos[j])] = ab[kl + ku + i - j + (int64_t)j * ldab];
}

// ---------------------------------------------------------------------------
namespace {
constexpr int ZERO_CTAS = 8 * 152;

// Shared-memory limit, once per process (thread-safe).
template <typename T> void mf_attrs() {
  static const bool done = [] {
    cudaFuncSetAttribute(k_mf_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         MF_SMALL * (MF_SMALL + 1) * (int)sizeof(T));
    cudaFuncSetAttribute(k_mf_fwd<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_mf_back<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    return true;
  }();
  (void)done;
}

int dof_blocks(const Batch& b) { return std::max(1, std::min(152, (b.n_free + 255) / 256)); }
}  // namespace

void launch_front_map(const Batch& b, cudaStream_t st) {
  const int64_t n = (int64_t)b.sh.n_shells * 729;
  if (n) k_mf_map<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(b);
}

template <typename T> void launch_front_zero(const Batch& b, cudaStream_t st) {
  k_mf_zero<T><<<dim3(ZERO_CTAS, b.sh.n_wide), 256, 0, st>>>(b);
}

// K_AA of the wide structures from the element matrices and nodal loads.
template <typename T> void launch_front_assemble(const Batch& b, cudaStream_t st) {
  launch_front_zero<T>(b, st);
  for (int c = 0; c < b.sh.n_colors; ++c) {
    const int cnt = b.sh.color_off[c + 1] - b.sh.color_off[c];
    if (cnt > 0) k_mf_elements<T><<<(cnt + 3) / 4, 128, 0, st>>>(b, c);
  }
  if (b.n_loads) k_mf_nodes<T><<<(b.n_nodes + 127) / 128, 128, 0, st>>>(b);
}

// Factorization of the assembled fronts and solution of the right-hand side (P
// or r32, overwritten).
template <typename T> void launch_front_factor(const Batch& b, cudaStream_t st) {
  mf_attrs<T>();
  const FrontSchedule& sc = *b.sh.mf.sched;
  const dim3 dofs(dof_blocks(b), b.sh.n_wide);
  k_mf_rhs<T><<<dofs, 256, 0, st>>>(b);
  for (const FrontLevel& V : sc.level) {
    for (size_t o = 0; o < V.ext_off.size(); ++o) k_mf_extend<T><<<V.ext_cnt[o], 256, 0, st>>>(b, V.ext_off[o]);
    if (V.n_small)
      k_mf_small<T><<<V.n_small, MF_SMALL_THREADS, (size_t)((V.small_f + 1) & ~1) * (V.small_f + 1) * sizeof(T), st>>>(
          b, V.small_off);
    for (size_t p = 0; p < V.n_at.size(); ++p) {
      const int n = V.n_at[p], k0 = (int)p * MF_NB, k1 = k0 + MF_NB, f = V.f_at[p], s = V.s_at[p];
      k_mf_diag<T><<<n, MF_DIAG_THREADS, 0, st>>>(b, V.big_off, (int)p);
      // the panels of fronts whose last panel this is end before k1
      const int m = f - k0 - 1;
      if (m >= 0) {
        const int nlow = (m + 31) / 32, nup = (m + 1 + 31) / 32;
        k_mf_trsm<T><<<dim3(nlow + nup, n), 128, 0, st>>>(b, V.big_off, (int)p, nlow);
      }
      if (s > k1) {
        const int nca = (f + 1 - k1 + 31) / 32, na = (s - k1 + 15) / 16 * nca;
        const int ncb = (s - k1 + 31) / 32, nb = (f + 15) / 16 * ncb;
        k_mf_panel<T><<<dim3(na + nb, n), 128, 0, st>>>(b, V.big_off, (int)p, na, nca, ncb);
      }
    }
    if (V.schur_cnt) k_mf_schur<T><<<V.schur_cnt, 128, 0, st>>>(b, V.schur_off);
  }
}

template <typename T> void launch_front_back(const Batch& b, cudaStream_t st) {
  const FrontSchedule& sc = *b.sh.mf.sched;
  for (size_t l = sc.level.size(); l-- > 0;) {
    const FrontLevel& V = sc.level[l];
    const int f = std::max(V.small_f, V.big_f);
    k_mf_back<T><<<V.n_small + V.n_big, MF_BACK_THREADS, (size_t)(f + 2 + 8 * 32) * sizeof(T), st>>>(b, V.small_off);
  }
  k_mf_out<T><<<dim3(dof_blocks(b), b.sh.n_wide), 256, 0, st>>>(b);
}

void launch_front_solve(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  if (b.sh.n_wide == 0) return;
  { ProfScope q(prof, st, KC_WIDE_DIAG); launch_front_assemble<double>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_UPDATE); launch_front_factor<double>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_SUBST); launch_front_back<double>(b, st); }
}

// The same with the FP32 factor, on r32.
void launch_front_solve32(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  { ProfScope q(prof, st, KC_WIDE_DIAG); launch_front_assemble<float>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_UPDATE); launch_front_factor<float>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_SUBST); launch_front_back<float>(b, st); }
}
// Another right-hand side (r32) with the FP32 factor.
void launch_front_resolve32(const Batch& b, cudaStream_t st) {
  for (const FrontLevel& V : b.sh.mf.sched->level) {
    const int f = std::max(V.small_f, V.big_f);
    k_mf_fwd<float><<<V.n_small + V.n_big, MF_BACK_THREADS, (size_t)f * sizeof(float), st>>>(b, V.small_off);
  }
  launch_front_back<float>(b, st);
}
int front_resolve_launches(const Batch& b) { return b.sh.mf.sched ? 2 * (int)b.sh.mf.sched->level.size() + 1 : 0; }

void launch_front_csr(const Batch& b, int n, const int* rp, const int* ci, const double* v, cudaStream_t st) {
  launch_front_zero<double>(b, st);
  k_mf_csr<<<(n + 127) / 128, 128, 0, st>>>(b, n, rp, ci, v);
  launch_front_factor<double>(b, st);
  launch_front_back<double>(b, st);
}

void launch_front_band(const Batch& b, int n, int kl, int ku, int ldab, const double* ab, cudaStream_t st) {
  launch_front_zero<double>(b, st);
  const int64_t t = (int64_t)n * (kl + ku + 1);
  k_mf_band<<<(unsigned)((t + 255) / 256), 256, 0, st>>>(b, n, kl, ku, ldab, ab);
  launch_front_factor<double>(b, st);
  launch_front_back<double>(b, st);
}

// Launches of one assembly, factorization and solve of the batch.
int front_launches(const Batch& b) {
  if (!b.sh.n_wide || !b.sh.mf.sched) return 0;
  int n = b.sh.mf.sched->launches + (b.n_loads ? 1 : 0);
  for (int c = 0; c < b.sh.n_colors; ++c) n += b.sh.color_off[c + 1] > b.sh.color_off[c];
  return n;
}

}  // namespace gf
