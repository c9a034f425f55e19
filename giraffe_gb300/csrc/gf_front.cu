// Multifrontal LU on the device (see gf_front.h): assembly of K_AA into the
// fronts, elimination height by height, back substitution.  No pivoting (a
// zero or non-finite pivot sets info_fail, as the reference's solver failure).
//
// The right-hand side is column f of every front, so the forward substitution
// is part of the elimination.  Per height, bottom up:
//   k_mf_extend   the children's Schur complements added into the large fronts, all
//                 children of a front's column by one warp
//   k_mf_small    fronts up to the height's line (at most MF_SMALL rows): one CTA each,
//                 in shared memory, the children's complements added as it loads
//   larger fronts, MF_NB pivots per panel:
//     k_mf_diag   LU of the first panel's diagonal block
//     k_mf_trsm   L21 = A21 U11^-1 and U12 = L11^-1 A12
//     k_mf_panel  the rest of the pivot rows and columns, and the LU of the next
//                 panel's diagonal block
//   k_mf_schur    the boundary block, once all pivots are done: C -= L21 U12 (the largest
//                 fronts' in gf_front_t5.cu)
// and top down
//   k_mf_back     x of the front's own DOFs from its boundary's.
// The diagonal of U is stored as its reciprocal.
//
// What bounds it: an FP64 warp instruction holds its sub-partition's FP64 unit
// for 64 cycles whatever its active lanes (measured: one warp issues a DFMA
// every 64 cycles at any instruction-level parallelism, an SM one every 19),
// so the large fronts are bound by FP64 throughput and the chain of panels by
// the dependent results of each pivot.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cfloat>

#include "gf_front.h"
#include "gf_kernels.cuh"
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

namespace {

namespace cg = cooperative_groups;

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
__device__ __forceinline__ bool mf_bad(double p) { return bad_pivot(p); }
__device__ __forceinline__ bool mf_bad(float p) {
  const int h = __float_as_int(p) & 0x7FFFFFFF;
  return h == 0 || h >= 0x7F800000;
}

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

// Destinations of the element matrices' entries and the chains of entries that share
// one, in colour order, once per batch: a thread per pair of an element's nodes.  The
// elements with both nodes are among the first one's (nref).
__global__ void k_mf_map(Batch b) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)b.sh.n_shells * 36) return;
  const int e = (int)(t / 36), la = (int)(t % 36) / 6, lb = (int)(t % 6), s = b.sh.sstruct[e];
  const StructInfo& inf = b.info[s];
  const FrontData& d = b.sh.mf;
  const int na = b.sh.snodes[6 * (int64_t)e + la], nb = b.sh.snodes[6 * (int64_t)e + lb];
  const int o0 = b.sh.nref_off[na], o1 = b.sh.nref_off[na + 1];
  // translations or rotations of either node
  for (int ka = 0; ka < (la < 3 ? 1 : 2); ++ka)
    for (int kb = 0; kb < (lb < 3 ? 1 : 2); ++kb) {
      bool first = true, past = false;
      int ne = -1, xa = 0, xb = 0;  // the next element and its rows of the first DOFs
      for (int o = o0; o < o1 && ne < 0; ++o) {
        const int v = b.sh.nref[o];
        if (v == 8 * e + la) {
          past = true;
          continue;
        }
        const int ra = shell_dof(v & 7, 3 * ka);
        if (ra < 0) continue;
        for (int m = 0; m < 6; ++m) {
          if (b.sh.snodes[6 * (int64_t)(v >> 3) + m] != nb) continue;
          const int rb = shell_dof(m, 3 * kb);
          if (rb < 0) continue;
          if (!past) first = false;
          else {
            ne = v >> 3;
            xa = ra;
            xb = rb;
          }
          break;
        }
      }
      for (int ca = 0; ca < 3; ++ca)
        for (int cb = 0; cb < 3; ++cb) {
          const int x = shell_dof(la, 3 * ka + ca) + 27 * shell_dof(lb, 3 * kb + cb);
          const int gr = b.gl[(int64_t)na * 6 + 3 * ka + ca], gq = b.gl[(int64_t)nb * 6 + 3 * kb + cb];
          int2 to = make_int2(-1, 0);
          if (gr >= 0 && gq >= 0) {
            if (first) to.x = (int)(mf_entry(d, d.pos[inf.dof_off + gr], d.pos[inf.dof_off + gq]) - d.base[s]);
            if (ne >= 0) to.y = (ne - e) * 729 + xa + ca + 27 * (xb + cb) - x;
          }
          d.map[(int64_t)e * 729 + x] = to;
        }
    }
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

// MountGlobal into the fronts: a warp per element; the first entry of a destination
// takes the others' along its chain (at most as long as the elements on a node), so an
// entry of the fronts is written once, with the bits of one colour of elements after the
// other.  Bound by the chains' loads, twelve entries in flight a lane; a launch per
// colour that adds in place took 5.6 us for each of 7 on small meshes, 13 on the 64x64x2
// plate; this 11 and 45 in all.
template <typename T> __global__ void __launch_bounds__(128) k_mf_elements(Batch b) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= b.sh.n_shells) return;
  const int s = b.sh.sstruct[e];
  const bool active = mf_active(b, s);
  const double* K = b.sh.Ke + (int64_t)e * 729;
  const int2* map = b.sh.mf.map + (int64_t)e * 729;
  T* F = reinterpret_cast<T*>(b.sh.mf.F) + b.sh.mf.base[s];
#pragma unroll 1
  for (int x0 = lane; x0 < 729; x0 += 12 * 32) {
    int2 m[12];
    int at[12];
    T v[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      at[q] = x0 + 32 * q;
      m[q] = at[q] < 729 ? map[at[q]] : make_int2(-1, 0);
      v[q] = at[q] < 729 ? (T)K[at[q]] : T(0);
    }
    if (!active) return;
    bool more = false;
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      if (m[q].x < 0) m[q].y = 0;
      more = more || m[q].y != 0;
    }
    while (more) {
      T k[12];
      int next[12];
#pragma unroll
      for (int q = 0; q < 12; ++q) {
        at[q] += m[q].y;
        k[q] = m[q].y ? (T)K[at[q]] : T(0);
        next[q] = m[q].y ? map[at[q]].y : 0;
      }
      more = false;
#pragma unroll
      for (int q = 0; q < 12; ++q) {
        if (m[q].y) v[q] += k[q];
        m[q].y = next[q];
        more = more || next[q] != 0;
      }
    }
#pragma unroll
    for (int q = 0; q < 12; ++q)
      if (m[q].x >= 0) F[m[q].x] = v[q];
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

// Extend-add: eight columns of a large front with its children's Schur
// complements, a warp per column, two children and four rows a lane at a time (the
// small fronts gather theirs as they load).  Bound by dependent loads from L2: front,
// child, its index of the column, of the rows, the entries.
template <typename T> __global__ void __launch_bounds__(256) k_mf_extend(Batch b, int job0) {
  const FrontData& d = b.sh.mf;
  const int2 job = d.ext_jobs[job0 + blockIdx.x];
  const Front F = d.fronts[job.x];
  const bool active = mf_active(b, F.slot);
  const int lane = threadIdx.x & 31, j = job.y + (threadIdx.x >> 5), kid1 = F.kid1;
  if (j > F.f) return;
  T* g = mf_mat<T>(b, F) + (int64_t)j * F.ld;
  for (int k = F.kid0; k < kid1; k += 2) {
    const int* inv[2];
    const T* sc[2];
    bool on[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int2 kid = d.kids[min(k + q, kid1 - 1)];
      const Front& C = d.fronts[kid.x];
      inv[q] = d.inv + kid.y;
      const int cj = j < F.f ? inv[q][j] : C.f - C.s;
      on[q] = cj >= 0 && k + q < kid1;
      sc[q] = reinterpret_cast<const T*>(d.F) + C.off + C.s + (int64_t)(C.s + cj) * C.ld;
    }
    if (!on[0] && !on[1]) continue;
    for (int i0 = lane; i0 < F.f; i0 += 128) {
      int c[2][4];
      T v[4], a[2][4];
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int i = i0 + 32 * y;
#pragma unroll
        for (int q = 0; q < 2; ++q) c[q][y] = on[q] && i < F.f ? inv[q][i] : -1;
        v[y] = i < F.f ? g[i] : T(0);
      }
      if (!active) return;
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int q = 0; q < 2; ++q) a[q][y] = c[q][y] >= 0 ? sc[q][c[q][y]] : T(0);
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        if (c[0][y] >= 0) v[y] += a[0][y];
        if (c[1][y] >= 0) v[y] += a[1][y];
        if (c[0][y] >= 0 || c[1][y] >= 0) g[i0 + 32 * y] = v[y];
      }
    }
  }
}

// Partial LU of a front held in shared memory, s pivots, one CTA: the front and its
// children's Schur complements are summed as they load, then warp 3, the pivot
// warp, owns column k + 1 at step k (its update, the next pivot's reciprocal and
// multipliers) while the others update the rest of the trailing block, packed
// densely over their lanes; one barrier closes the step.  Bound by its SM's FP64
// rate, for which one CTA needs two warps a sub-partition (f = 87, s = 15, a CTA an
// SM: four warps 80 us, eight 50).
constexpr int MF_SMALL_THREADS = 256;
template <typename T> __global__ void __launch_bounds__(MF_SMALL_THREADS) k_mf_small(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.x];
  if (!mf_active(b, F.slot)) return;
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* A = reinterpret_cast<T*>(mf_raw);
  const int f = F.f, s = F.s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int WARPS = MF_SMALL_THREADS / 32;
  T* G = mf_mat<T>(b, F);
  const int size = ld * (f + 1);
  for (int x0 = tid; x0 < size; x0 += 8 * MF_SMALL_THREADS) {
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = x0 + q * MF_SMALL_THREADS < size ? G[x0 + q * MF_SMALL_THREADS] : T(0);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (x0 + q * MF_SMALL_THREADS < size) A[x0 + q * MF_SMALL_THREADS] = v[q];
  }
  for (int k = F.kid0; k < F.kid1; ++k) {
    const int2 kid = d.kids[k];
    const int* inv = d.inv + kid.y;
    const Front& C = d.fronts[kid.x];
    const int u = C.f - C.s, cld = C.ld;
    const T* S = reinterpret_cast<const T*>(d.F) + C.off + C.s + (int64_t)C.s * cld;
    int ci[MF_SMALL / 32];
#pragma unroll
    for (int q = 0; q < MF_SMALL / 32; ++q) ci[q] = lane + 32 * q < f ? inv[lane + 32 * q] : -1;
    // the child's column of each of the warp's columns, one a lane
    const int jl = warp + WARPS * lane, cjl = jl < f ? inv[jl] : jl == f ? u : -1;
    __syncthreads();  // A is complete, or holds the child before
    for (int y0 = 0; warp + WARPS * y0 <= f; y0 += 4) {
      T a[4][MF_SMALL / 32];
      int cj[4];
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        cj[y] = __shfl_sync(0xffffffffu, cjl, y0 + y);
#pragma unroll
        for (int q = 0; q < MF_SMALL / 32; ++q)
          a[y][q] = cj[y] >= 0 && ci[q] >= 0 ? S[ci[q] + (int64_t)cj[y] * cld] : T(0);
      }
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int q = 0; q < MF_SMALL / 32; ++q)
          if (cj[y] >= 0 && ci[q] >= 0) A[lane + 32 * q + (warp + WARPS * (y0 + y)) * ld] += a[y][q];
    }
  }
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
      const int c0 = next ? k + 2 : k + 1, nt = MF_SMALL_THREADS - (next ? 32 : 0);
      const int tot = m * (f + 1 - c0);
      const float inv_m = 1.0f / (float)m;
      for (int e = next && warp > 3 ? tid - 32 : tid; e < tot; e += nt) {
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

// LU of a 32 x 32 diagonal block in shared memory (A[j][i]: column j, row i; nb of it)
// by a CTA of MF_DIAG_THREADS: a chain of pivots (update of a column, reciprocal,
// multipliers), 540 cycles each if nothing holds them up.  The pivot warp (warp 3) has
// a sub-partition to itself; six warps on the other three update the remaining
// columns, lane i row i, a column at a time (FP64 instructions take their 64 cycles
// even where a predicate turns every lane off, so the loop ends at the last column;
// three warps with the columns in registers took 1,120 cycles a pivot, packed lanes
// 1,150, this 700).  True where a pivot failed.
constexpr int MF_DIAG_THREADS = 256;
template <typename T> __device__ __forceinline__ bool mf_block_lu(T (*A)[MF_NB + 1], int nb, int warp, int lane) {
  bool bad = false;
  T a = T(0), l = T(0);
  // pivot k of the updated column a: lane i keeps the multiplier of row i
  auto pivot = [&](int k) {
    const T q = __shfl_sync(0xffffffffu, a, k);
    bad = bad || mf_bad(q);
    const T r = mf_rcp(q);
    l = a * r;
    if (lane > k && lane < nb) A[k][lane] = l;
    if (lane == k) A[k][k] = r;
  };
  if (warp == 3) {
    a = A[0][lane];
    pivot(0);
  }
  __syncthreads();
  for (int k = 0; k + 1 < nb; ++k) {
    if (warp == 3) {
      a = A[k + 1][lane];
      const T u = __shfl_sync(0xffffffffu, a, k);
      if (lane > k) a = mfma(-l, u, a);
      pivot(k + 1);
    } else if (warp < 7) {
      const T x = -A[k][lane];
      for (int j = k + 2 + (warp < 3 ? warp : warp - 1); j < nb; j += 6) {
        const T v = mfma(x, A[j][k], A[j][lane]);
        if (lane > k) A[j][lane] = v;
      }
    }
    __syncthreads();
  }
  return bad;
}

// The first diagonal block of the large fronts of a height, one CTA each (k_mf_panel
// factors the next one of a front as it forms it).
template <typename T> __global__ void __launch_bounds__(MF_DIAG_THREADS) k_mf_diag(Batch b, int off) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.x];
  const bool on = mf_active(b, F.slot);
  const int nb = min(MF_NB, F.s), ld = F.ld, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* G = mf_mat<T>(b, F);
  __shared__ T A[MF_NB][MF_NB + 1];
#pragma unroll
  for (int q = 0; q < MF_NB / 8; ++q) {
    const int j = warp + 8 * q;
    if (j < nb) A[j][lane] = lane < nb ? G[lane + (int64_t)j * ld] : T(0);
  }
  if (!on) return;
  __syncthreads();
  const bool bad = mf_block_lu<T>(A, nb, warp, lane);
#pragma unroll
  for (int q = 0; q < MF_NB / 8; ++q) {
    const int j = warp + 8 * q;
    if (lane < nb && j < nb) G[lane + (int64_t)j * ld] = A[j][lane];
  }
  if (bad && lane == 0) mf_fail<T>(b, F.slot);
}

// L21 = A21 U11^-1 (blockIdx.x < nlow: the rows below the panel, 128 / L a CTA) and
// U12 = L11^-1 A12 (the columns right of it, the right-hand side among them).  L
// lanes per row (column), lane q holding its entries L j + q in registers, the
// finished entry broadcast within the L: 176 FP64 warp instructions per eight rows
// with L = 4 (132 with a thread per row, but four times the latency), 80 per two
// with L = 16, which has half the latency where the rows leave SMs idle.
template <typename T, int L> __global__ void __launch_bounds__(128) k_mf_trsm(Batch b, int off, int p, int nlow) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.y];
  const bool on = mf_active(b, F.slot);
  const int k0 = p * MF_NB, nb = min(MF_NB, F.s - k0), k1 = k0 + nb, ld = F.ld, tid = threadIdx.x;
  const bool lower = (int)blockIdx.x < nlow;
  constexpr int R = 128 / L, E = MF_NB / L;
  const int first = k1 + R * (lower ? (int)blockIdx.x : (int)blockIdx.x - nlow);
  if (first >= (lower ? F.f : F.f + 1)) return;
  T* G = mf_mat<T>(b, F);
  __shared__ T U[MF_NB][MF_NB + 1];  // U[k][j]: the factor this side reads, identity beyond nb
  T u[MF_NB / 4];
#pragma unroll
  for (int y = 0; y < MF_NB / 4; ++y) {
    const int i = tid % MF_NB, j = tid / MF_NB + 4 * y;
    u[y] = i == j ? T(1) : T(0);
    if (i < nb && j < nb && (lower ? i <= j : i > j)) u[y] = G[k0 + i + (int64_t)(k0 + j) * ld];
  }
  const int r = tid / L, q = tid % L, g = first + r;  // row (lower) or column of the front
  const bool live = g < (lower ? F.f : F.f + 1);
  T v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int c = L * j + q;
    v[j] = (live && c < nb) ? (lower ? G[g + (int64_t)(k0 + c) * ld] : G[k0 + c + (int64_t)g * ld]) : T(0);
  }
#pragma unroll
  for (int y = 0; y < MF_NB / 4; ++y) {
    const int i = tid % MF_NB, j = tid / MF_NB + 4 * y;
    if (lower) U[i][j] = u[y];  // U11(i, j), the reciprocal on the diagonal
    else U[j][i] = u[y];        // L11(i, j) at [j][i]
  }
  if (!on) return;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < MF_NB; ++k) {
    if (k % 8 == 0 && k >= nb) break;  // the factor is the identity beyond nb
    // the finished entry k, from the lane that holds it
    T x = v[k / L];
    if (lower) x *= U[k][k];
    x = __shfl_sync(0xffffffffu, x, k % L, L);
    if (lower && q == k % L) v[k / L] = x;
#pragma unroll
    for (int j = k / L; j < E; ++j)
      if (L * j + q > k) v[j] = mfma(-x, U[k][L * j + q], v[j]);
  }
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int c = L * j + q;
    if (!live || c >= nb) continue;
    if (lower) G[g + (int64_t)(k0 + c) * ld] = v[j];
    else G[k0 + c + (int64_t)g * ld] = v[j];
  }
}

// The pivot rows and columns right of and below panel p: rows k1..s-1 of all
// later columns (the first na tiles) and the boundary rows of the later pivot
// columns, minus L U over the panel's pivots.  16 x 32 tiles, so that the few
// tiles of the top fronts spread over the SMs (a tile holds an SM's FP64 units
// for 512 warp instructions, about 5 us).  The first C CTAs of a front, a cluster, take
// the 32 x 32 tile of the next diagonal block, 32 / C columns each, and the first of
// them factors it (mf_block_lu) while the others run: a launch per panel and 14 us less
// on the chain of panels.  On one CTA the tile takes 8 us of its SM's FP64 rate, all of
// them on the chain where a height has few fronts (24 us a panel with one, 17 with
// four).  FP32 fronts take one: their tile is a few us in either form (24x24x2 mixed
// plate 10.49 ms with one CTA and with four).
constexpr int MF_PANEL_THREADS = 256;
static_assert(MF_PANEL_THREADS == MF_DIAG_THREADS, "the panel's first CTA factors a block");
template <typename T, int C>
__global__ void __launch_bounds__(MF_PANEL_THREADS) k_mf_panel(Batch b, int off, int p, int na, int nca, int ncb) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.y];
  const bool on = mf_active(b, F.slot);
  const int k0 = p * MF_NB, k1 = k0 + MF_NB, ld = F.ld, tid = threadIdx.x;
  if (k1 >= F.s) return;
  T* G = mf_mat<T>(b, F);
  __shared__ T Ls[MF_NB][33];  // [k][row]
  __shared__ T Us[32][MF_NB + 1];  // [column][k]
  if (blockIdx.x < C) {
    constexpr int Q = 4 / C;
    __shared__ T Ds[MF_NB][MF_NB + 1];  // the diagonal block (the first CTA's)
    cg::cluster_group cl = cg::this_cluster();
    const int lane = tid & 31, warp = tid >> 5, r1 = F.s, c1 = F.f + 1, nb = min(MF_NB, F.s - k1);
    const int y0 = warp + 8 * Q * (int)blockIdx.x;  // this warp's columns y0 + 8 q
    T acc[Q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = warp + 8 * q;
      Ls[k][lane] = k1 + lane < r1 ? G[k1 + lane + (int64_t)(k0 + k) * ld] : T(0);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int y = y0 + 8 * q;
      Us[y][lane] = k1 + y < c1 ? G[k0 + lane + (int64_t)(k1 + y) * ld] : T(0);
      acc[q] = (k1 + lane < r1 && k1 + y < c1) ? G[k1 + lane + (int64_t)(k1 + y) * ld] : T(0);
    }
    if (!on) return;
    if (C > 1) cl.barrier_arrive();
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < MF_NB; ++k) {
      const T l = -Ls[k][lane];
#pragma unroll
      for (int q = 0; q < Q; ++q) acc[q] = mfma(l, Us[y0 + 8 * q][k], acc[q]);
    }
    if (C > 1) cl.barrier_wait();  // every CTA of the cluster runs
    T* D0 = C > 1 ? cl.map_shared_rank(&Ds[0][0], 0) : &Ds[0][0];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int y = y0 + 8 * q;
      if (y < nb) D0[y * (MF_NB + 1) + lane] = acc[q];
      else if (lane < nb && k1 + y < c1) G[k1 + lane + (int64_t)(k1 + y) * ld] = acc[q];
    }
    if (C > 1) cl.sync();
    else __syncthreads();
    if (blockIdx.x > 0) return;
    const bool bad = mf_block_lu<T>(Ds, nb, warp, lane);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int y = warp + 8 * q;
      if (lane < nb && y < nb) G[k1 + lane + (int64_t)(k1 + y) * ld] = Ds[y][lane];
    }
    if (bad && lane == 0) mf_fail<T>(b, F.slot);
    return;
  }
  const int tile = (int)blockIdx.x - C;
  int r0, c0, r1, c1;
  if (tile < na) {
    r0 = k1 + 16 * (tile / nca);
    c0 = k1 + 32 * (tile % nca);
    r1 = F.s;
    c1 = F.f + 1;
    if (r0 <= k1 + 16 && c0 == k1) return;  // the first CTAs'
  } else {
    const int x = tile - na;
    r0 = F.s + 16 * (x / ncb);
    c0 = k1 + 32 * (x % ncb);
    r1 = F.f;
    c1 = F.s;
  }
  if (r0 >= r1 || c0 >= c1) return;
  const int i = tid & 15, cg = tid >> 4;  // row, columns cg + 16 q
#pragma unroll
  for (int q = 0; q < 2; ++q) Ls[cg + 16 * q][i] = r0 + i < r1 ? G[r0 + i + (int64_t)(k0 + cg + 16 * q) * ld] : T(0);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = tid & 31, c = (tid >> 5) + 8 * q;
    Us[c][k] = c0 + c < c1 ? G[k0 + k + (int64_t)(c0 + c) * ld] : T(0);
  }
  T acc[2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
    acc[q] = (r0 + i < r1 && c0 + cg + 16 * q < c1) ? G[r0 + i + (int64_t)(c0 + cg + 16 * q) * ld] : T(0);
  if (!on) return;
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < MF_NB; ++k) {
    const T l = -Ls[k][i];
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[q] = mfma(l, Us[cg + 16 * q][k], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (r0 + i < r1 && c0 + cg + 16 * q < c1) G[r0 + i + (int64_t)(c0 + cg + 16 * q) * ld] = acc[q];
}

// The Schur complement of the large fronts of a height: C -= L21 U12 over all
// pivots, R x R tiles, 2 x 4 (R = 32) or 1 x 2 (16) outputs per thread, the next 32
// pivots' operands loading into registers while this one's products run.  Bound by
// the FP64 pipes.
template <typename T, int R> __global__ void __launch_bounds__(128) k_mf_schur(Batch b, int job0) {
  const FrontData& d = b.sh.mf;
  const int2 job = d.schur_jobs[job0 + blockIdx.x];
  const Front F = d.fronts[job.x];
  const bool on = mf_active(b, F.slot);
  constexpr int H = R / 16, Q = R / 8, N = R / 4;  // row halves, column groups, entries a thread loads
  const int r0 = F.s + R * (job.y & 0xFFFF), c0 = F.s + R * (job.y >> 16), ld = F.ld, s = F.s, tid = threadIdx.x;
  T* G = mf_mat<T>(b, F);
  __shared__ T Ls[2][32][R + 1];  // [k][row]
  __shared__ T Us[2][R][33];      // [column][k]
  const int lr_ = tid % R, lk = tid / R;      // L: row, pivots lk + (128 / R) q
  const int uk = tid & 31, uc = tid >> 5;     // U: pivot, columns uc + 4 q
  const bool row_ok = r0 + lr_ < F.f;
  const int rows = F.f - r0, cols = F.f + 1 - c0;
  const bool full = rows > R - 16 && cols > R - 8;
  T lr[N], ur[N];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int k = lk + 128 / R * q, c = uc + 4 * q;
      lr[q] = (row_ok && k0 + k < s) ? G[r0 + lr_ + (int64_t)(k0 + k) * ld] : T(0);
      ur[q] = (c0 + c <= F.f && k0 + uk < s) ? G[k0 + uk + (int64_t)(c0 + c) * ld] : T(0);
    }
  };
  auto stash = [&](int w) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      Ls[w][lk + 128 / R * q][lr_] = lr[q];
      Us[w][uc + 4 * q][uk] = ur[q];
    }
  };
  const int ti = tid & 15, tj = tid >> 4;  // rows ti + 16 h; columns tj + 8 q
  T acc[H][Q];
  fetch(0);
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int r = r0 + ti + 16 * h, c = c0 + tj + 8 * q;
      acc[h][q] = (r < F.f && c <= F.f) ? G[r + (int64_t)c * ld] : T(0);
    }
  if (!on) return;
  stash(0);
  __syncthreads();
  for (int k0 = 0, w = 0; k0 < s; k0 += 32, w ^= 1) {
    if (k0 + 32 < s) fetch(k0 + 32);
    const int kn = min(32, s - k0);
    if (full) {
      for (int k = 0; k < kn; ++k) {
        T l[H];
#pragma unroll
        for (int h = 0; h < H; ++h) l[h] = -Ls[w][k][ti + 16 * h];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const T u = Us[w][tj + 8 * q][k];
#pragma unroll
          for (int h = 0; h < H; ++h) acc[h][q] = mfma(l[h], u, acc[h][q]);
        }
      }
    } else {
      // the halves and column groups of an edge tile that hold entries
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if (16 * h < rows && 8 * q < cols)
#pragma unroll 8
            for (int k = 0; k < kn; ++k) acc[h][q] = mfma(-Ls[w][k][ti + 16 * h], Us[w][tj + 8 * q][k], acc[h][q]);
    }
    if (k0 + 32 < s) stash(w ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int r = r0 + ti + 16 * h, c = c0 + tj + 8 * q;
      if (r < F.f && c <= F.f) G[r + (int64_t)c * ld] = acc[h][q];
    }
}

// Substitution on a 32 x 32 diagonal block: D[j][i] its column j, row i (zero outside
// the nb used).  Lane i holds w_i of the block.  Eight columns at a time from
// registers, so that no load waits on the chain.
template <typename T> __device__ __forceinline__ T mf_block_back(const T (*D)[33], int nb, int lane, T v) {
  const T r = D[lane][lane];  // the reciprocal
#pragma unroll
  for (int k0 = 24; k0 >= 0; k0 -= 8) {
    if (k0 >= nb) continue;
    T c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = -D[k0 + q][lane];
#pragma unroll
    for (int q = 7; q >= 0; --q) {
      if (k0 + q >= nb) continue;
      const T xk = __shfl_sync(0xffffffffu, v * r, k0 + q);
      if (lane == k0 + q) v = xk;
      if (lane < k0 + q) v = mfma(c[q], xk, v);
    }
  }
  return v;
}
template <typename T> __device__ __forceinline__ T mf_block_fwd(const T (*D)[33], int nb, int lane, T v) {
#pragma unroll
  for (int k0 = 0; k0 < 32; k0 += 8) {
    if (k0 >= nb) continue;
    T c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = -D[k0 + q][lane];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const T yk = __shfl_sync(0xffffffffu, v, k0 + q);
      if (lane > k0 + q) v = mfma(c[q], yk, v);
    }
  }
  return v;
}

// The substitutions take a front by a cluster of C CTAs (C = 1, 2, 4 or 8, see
// subst_ctas); its rows go in groups of 32 to the ranks in turn, and every row's
// sums are in the same order whatever C is.  A block of 32 own DOFs is solved by
// warp 0 of the rank that owns it and handed to all of them in their shared memory
// (xb); then four warps take a group's rows, a quarter of the block's columns each
// from registers that were loaded while the block was solved.
//
// Bound by latency: the blocks' chain (two dependent FP64 operations and a shuffle a
// DOF) and the rounds of loads before it.  One CTA a front took 70 us a height on the 64x64x2
// plate (0.84 ms of a 6.2 ms pass), where the top fronts' U12 alone is 44 us of one
// SM's FP64 rate, and 11 us a height and sweep on the 24x24x2 plate's FP32 fronts,
// most of it four loads at a time from L2 over U12's columns.
constexpr int MF_BACK_THREADS = 256;

template <typename T> struct MfSubst {
  T D[2][32][33];   // diagonal blocks: column j, row i
  T xb[2][32];      // a solved block
  T part[8 * 32];   // quarter sums of two groups
};

__device__ __forceinline__ void mf_sync(cg::cluster_group& cl, int C) {
  if (C == 1) __syncthreads();
  else cl.sync();
}

// The rows of group h (one per lane) less a solved block's columns: quarter q of the
// columns j0 .. j0 + 31 into g, zero outside the front's s columns.
template <typename T> __device__ __forceinline__ void mf_cols(T* g, const T* G, int ld, int row, bool in, int j0, int s, int q) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = j0 + q + 4 * i;
    g[i] = (in && k < s) ? G[row + (int64_t)k * ld] : T(0);
  }
}

// One step of either substitution: the block's x in xb, the rank's groups first,
// first + dir C, ... (n of them) less its columns, two groups at a time; rows in
// [lo, hi).  g: the quarter of the first pair's columns that this warp loaded ahead.
template <typename T>
__device__ __forceinline__ void mf_apply(MfSubst<T>& m, T* w, const T* g0, const T* xb, const T* G, int ld, int first,
                                         int step, int n, int lo, int hi, int j0, int s) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3;
  T g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = g0[i];
  for (int t = 0; t < n; t += 2) {
    const int mine = t + (warp >> 2);
    if (t > 0) {
      const int row = 32 * (first + step * mine) + lane;
      mf_cols(g, G, ld, row, mine < n && row >= lo && row < hi, j0, s, q);
    }
    if (mine < n) {
      T a = T(0);
#pragma unroll
      for (int i = 0; i < 8; ++i) a = mfma(g[i], xb[q + 4 * i], a);
      m.part[warp * 32 + lane] = a;
    }
    __syncthreads();
    // group t by warp 0, which solves the next block from it, and t + 1 by warp 4
    if (q == 0 && mine < n) {
      const int row = 32 * (first + step * mine) + lane;
      const T* z = m.part + warp * 32 + lane;
      if (row >= lo && row < hi) w[row] -= (z[0] + z[32]) + (z[64] + z[96]);
    }
    if (t + 2 < n) __syncthreads();
  }
}

// Back substitution of every front of a height: w = y - U12 x2, the eight warps an
// eighth of the columns each, then x1 = U11^-1 w in blocks of 32.
template <typename T> __global__ void __launch_bounds__(MF_BACK_THREADS) k_mf_back(Batch b, int off, int C) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.x / C];
  if (!mf_active(b, F.slot)) return;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = C == 1 ? 0 : (int)cl.block_rank();
  const int f = F.f, s = F.s, u = f - s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const T* G = mf_mat<T>(b, F);
  T* x = mf_x<T>(b);
  const int* B = d.bnd + F.bnd;
  __shared__ MfSubst<T> m;
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* w = reinterpret_cast<T*>(mf_raw);  // [f]: w of the rank's own DOFs, then x2
  T* part = w + f + (f & 1);            // [8][rows of a chunk of the rank's groups]
  const int ng = (s + 31) / 32, own = (ng - rank + C - 1) / C;
  const int sp = min(own * 32, MF_PART);
  // the diagonal block of group h into E, by warps w0 to 7
  auto block = [&](T (*E)[33], int h, int w0) {
    const int j0 = 32 * h, i = lane;
    if (warp < w0) return;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int j = warp - w0 + (8 - w0) * q;
      if (j < 32) E[j][i] = (j0 + i < s && j0 + j < s) ? G[j0 + i + (int64_t)(j0 + j) * ld] : T(0);
    }
  };
  if (own > 0) block(m.D[0], rank + C * (own - 1), 0);
  for (int i = tid; i < own * 32; i += MF_BACK_THREADS) {
    const int r = 32 * (rank + C * (i / 32)) + i % 32;
    if (r < s) w[r] = G[r + (int64_t)f * ld];
  }
  if (own > 0)
    for (int i = tid; i < u; i += MF_BACK_THREADS) w[s + i] = x[B[i]];
  mf_sync(cl, C);  // every rank runs before the first block is handed over
  for (int c0 = 0; u > 0 && c0 < own * 32; c0 += MF_PART) {
    const int c1 = min(own * 32, c0 + MF_PART);
    for (int i0 = c0; i0 < c1; i0 += 32) {
      const int r = 32 * (rank + C * (i0 / 32)) + lane;
      T acc[4] = {T(0), T(0), T(0), T(0)};
      const T* g = G + min(r, s - 1);
      for (int j = s + warp; j < f; j += 128) {
        T v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = j + 8 * q < f ? g[(int64_t)(j + 8 * q) * ld] : T(0);
#pragma unroll
        for (int q = 0; q < 16; ++q)
          if (j + 8 * q < f) acc[q & 3] = mfma(v[q], w[j + 8 * q], acc[q & 3]);
      }
      part[warp * sp + i0 - c0 + lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    __syncthreads();
    for (int i = c0 + tid; i < c1; i += MF_BACK_THREADS) {
      const int r = 32 * (rank + C * (i / 32)) + i % 32;
      T t = part[i - c0];
      for (int q = 1; q < 8; ++q) t += part[q * sp + i - c0];
      if (r < s) w[r] -= t;
    }
    __syncthreads();
  }
  int cur = 0;
  for (int h = ng - 1; h >= 0; --h) {
    const int j0 = 32 * h, nb = min(32, s - j0), p = h & 1;
    // the rank's groups below h, downwards
    const int n = (h - rank + C - 1) / C, first = rank + C * (n - 1);
    T g[8];
    {
      const int mine = warp >> 2, row = 32 * (first - C * mine) + lane;
      mf_cols(g, G, ld, row, mine < n, j0, s, warp & 3);
    }
    if (h % C == rank) {
      if (warp == 0) {
        const T v = mf_block_back<T>(m.D[cur], nb, lane, lane < nb ? w[j0 + lane] : T(0));
        if (lane < nb) x[F.dof0 + j0 + lane] = v;
        if (C == 1) m.xb[p][lane] = v;
        else
          for (int c = 0; c < C; ++c) cl.map_shared_rank(&m.xb[p][0], c)[lane] = v;
      }
      cur ^= 1;
      if (n > 0) block(m.D[cur], first, 1);
    }
    mf_sync(cl, C);
    if (n > 0) mf_apply(m, w, g, m.xb[p], G, ld, first, -C, n, 0, s, j0, s);
  }
}

// Forward substitution alone, on fronts that hold their LU: every front of a height.
// w = the right-hand side of the own DOFs with what the children leave (column f of
// theirs, one child after the other), then y1 = L11^-1 w1 in blocks of 32 and w2 -=
// L21 y1; both into column f.
template <typename T> __global__ void __launch_bounds__(MF_BACK_THREADS) k_mf_fwd(Batch b, int off, int C) {
  const FrontData& d = b.sh.mf;
  const Front F = d.list[off + blockIdx.x / C];
  if (!mf_active(b, F.slot)) return;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = C == 1 ? 0 : (int)cl.block_rank();
  const int f = F.f, s = F.s, ld = F.ld, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T* G = mf_mat<T>(b, F);
  __shared__ MfSubst<T> m;
  extern __shared__ __align__(16) unsigned char mf_raw[];
  T* w = reinterpret_cast<T*>(mf_raw);  // [f], the rank's rows used
  const T* P = mf_rhs(b, (T*)nullptr);
  const int ng = (s + 31) / 32, nr = (f + 31) / 32, own = (nr - rank + C - 1) / C;
  auto block = [&](T (*E)[33], int h, int w0) {
    const int j0 = 32 * h, i = lane;
    if (warp < w0) return;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int j = warp - w0 + (8 - w0) * q;
      if (j < 32) E[j][i] = (j0 + i < s && j0 + j < s) ? G[j0 + i + (int64_t)(j0 + j) * ld] : T(0);
    }
  };
  if (rank < ng) block(m.D[0], rank, 0);
  for (int i = tid; i < own * 32; i += MF_BACK_THREADS) {
    const int r = 32 * (rank + C * (i / 32)) + i % 32;
    if (r >= f) continue;
    T v = r < s ? P[d.dof_at[F.dof0 + r]] : T(0);
    for (int k = F.kid0; k < F.kid1; k += 2) {  // two children's loads side by side
      const bool two = k + 1 < F.kid1;
      const int2 k0 = d.kids[k], k1 = d.kids[two ? k + 1 : k];
      const Front &C0 = d.fronts[k0.x], &C1 = d.fronts[k1.x];
      const int i0 = d.inv[k0.y + r], i1 = two ? d.inv[k1.y + r] : -1;
      const T* X = reinterpret_cast<const T*>(d.F);
      const T v0 = i0 >= 0 ? X[C0.off + C0.s + i0 + (int64_t)C0.f * C0.ld] : T(0);
      const T v1 = i1 >= 0 ? X[C1.off + C1.s + i1 + (int64_t)C1.f * C1.ld] : T(0);
      if (i0 >= 0) v += v0;
      if (i1 >= 0) v += v1;
    }
    w[r] = v;
  }
  mf_sync(cl, C);
  int cur = 0;
  for (int h = 0; h < ng; ++h) {
    const int j0 = 32 * h, nb = min(32, s - j0), p = h & 1;
    // the rank's groups with rows below the block, upwards: the block's own where it
    // is short
    const int g0 = nb < 32 ? h : h + 1, first = g0 + (rank - g0 % C + C) % C;
    const int n = first < nr ? (nr - first + C - 1) / C : 0;
    T g[8];
    {
      const int mine = warp >> 2, row = 32 * (first + C * mine) + lane;
      mf_cols(g, G, ld, row, mine < n && row >= j0 + nb && row < f, j0, s, warp & 3);
    }
    if (h % C == rank) {
      if (warp == 0) {
        const T v = mf_block_fwd<T>(m.D[cur], nb, lane, lane < nb ? w[j0 + lane] : T(0));
        if (lane < nb) w[j0 + lane] = v;
        if (C == 1) m.xb[p][lane] = v;
        else
          for (int c = 0; c < C; ++c) cl.map_shared_rank(&m.xb[p][0], c)[lane] = v;
      }
      cur ^= 1;
      if (h + C < ng) block(m.D[cur], h + C, 1);
    }
    mf_sync(cl, C);
    if (n > 0) mf_apply(m, w, g, m.xb[p], G, ld, first, C, n, j0 + nb, f, j0, s);
  }
  __syncthreads();
  for (int i = tid; i < own * 32; i += MF_BACK_THREADS) {
    const int r = 32 * (rank + C * (i / 32)) + i % 32;
    if (r < f) G[r + (int64_t)f * ld] = w[r];
  }
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

// r = rhs - A x and whether a row's backward error is above the limit; a non-finite
// one is.  mx: the largest |x_j| of the row's columns as its bits.
__device__ __forceinline__ void mf_row_error(int i, double rhs, double ax, double sum, unsigned long long mx, double* r, int* bad) {
  const double res = rhs - ax, d = fma(sum, __longlong_as_double((long long)mx), fabs(rhs));
  r[i] = res;
  if (!(fabs(res) <= MF_ERROR_LIMIT * d && d <= DBL_MAX)) *bad = 1;
}
__device__ __forceinline__ unsigned long long mf_mag(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// Eight lanes a row of a CSR matrix.
__global__ void __launch_bounds__(128) k_csr_residual(int n, const int* rp, const int* ci, const double* v, const double* rhs,
                                                      const double* x, double* r, int* bad) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, lane = threadIdx.x & 7;
  double ax = 0.0, sum = 0.0;
  unsigned long long mx = 0;
  const int k1 = i < n ? rp[i + 1] : 0;
  for (int k = i < n ? rp[i] + lane : 0; k < k1; k += 8) {
    const double a = v[k], xk = x[ci[k]];
    ax = fma(a, xk, ax);
    sum += fabs(a);
    mx = max(mx, mf_mag(xk));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (i < n && lane == 0) mf_row_error(i, rhs[i], ax, sum, mx, r, bad);
}

// A thread a row of LAPACK GB columns.
__global__ void __launch_bounds__(64) k_band_residual(int n, int kl, int ku, int ldab, const double* ab, const double* rhs,
                                                      const double* x, double* r, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double ax = 0.0, sum = 0.0;
  unsigned long long mx = 0;
  const int j1 = min(n - 1, i + ku);
#pragma unroll 4
  for (int j = max(0, i - kl); j <= j1; ++j) {
    const double a = ab[kl + ku + i - j + (int64_t)j * ldab], xj = x[j];
    ax = fma(a, xj, ax);
    sum += fabs(a);
    mx = max(mx, mf_mag(xj));
  }
  mf_row_error(i, rhs[i], ax, sum, mx, r, bad);
}

__global__ void k_mf_add(int n, const double* d, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += d[i];
}

// ---------------------------------------------------------------------------
namespace {
constexpr int ZERO_CTAS = 8 * 152;

template <typename T> void mf_attrs() {
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_mf_small<T>, MF_SMALL * (MF_SMALL + 1) * (int)sizeof(T)},
                    {(const void*)k_mf_fwd<T>, MF_SUBST_SMEM},
                    {(const void*)k_mf_back<T>, MF_SUBST_SMEM}});
}

// A launch in clusters of C CTAs along x.
template <typename... P, typename... A>
void launch_clusters(void (*kernel)(P...), dim3 grid, int threads, int C, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

int dof_blocks(const Batch& b) { return std::max(1, std::min(152, (b.n_free + 255) / 256)); }
}  // namespace

void launch_front_map(const Batch& b, cudaStream_t st) {
  const int64_t n = (int64_t)b.sh.n_shells * 36;
  if (n) k_mf_map<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(b);
}

template <typename T> void launch_front_zero(const Batch& b, cudaStream_t st) {
  k_mf_zero<T><<<dim3(ZERO_CTAS, b.sh.n_wide), 256, 0, st>>>(b);
}

// K_AA of the wide structures from the element matrices and nodal loads.
template <typename T> void launch_front_assemble(const Batch& b, cudaStream_t st) {
  launch_front_zero<T>(b, st);
  if (b.sh.n_shells) k_mf_elements<T><<<(b.sh.n_shells + 3) / 4, 128, 0, st>>>(b);
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
    if (V.ext_cnt) k_mf_extend<T><<<V.ext_cnt, 256, 0, st>>>(b, V.ext_off);
    if (V.n_small)
      k_mf_small<T><<<V.n_small, MF_SMALL_THREADS, (size_t)((V.small_f + 1) & ~1) * (V.small_f + 1) * sizeof(T), st>>>(
          b, V.small_off);
    for (size_t p = 0; p < V.n_at.size(); ++p) {
      if (p == 0) k_mf_diag<T><<<V.n_at[p], MF_DIAG_THREADS, 0, st>>>(b, V.big_off);
      for (int q = 0; q < front_grids(V.n_at[p]); ++q) {
        const int n = std::min(V.n_at[p] - q * MF_GRID_FRONTS, MF_GRID_FRONTS), off = V.big_off + q * MF_GRID_FRONTS;
        const int k0 = (int)p * MF_NB, k1 = k0 + MF_NB, f = V.f_at[p], s = V.s_at[p];
        // the panels of fronts whose last panel this is end before k1
        const int m = f - k0 - 1;
        if (m >= 0) {
          // sixteen lanes a row while that leaves an SM at most one CTA
          if ((2 * m + 1) * (int64_t)n <= 8 * 152) {
            const int nlow = (m + 7) / 8, nup = (m + 1 + 7) / 8;
            k_mf_trsm<T, 16><<<dim3(nlow + nup, n), 128, 0, st>>>(b, off, (int)p, nlow);
          } else {
            const int nlow = (m + 31) / 32, nup = (m + 1 + 31) / 32;
            k_mf_trsm<T, 4><<<dim3(nlow + nup, n), 128, 0, st>>>(b, off, (int)p, nlow);
          }
        }
        if (s > k1) {
          const int nca = (f + 1 - k1 + 31) / 32, na = (s - k1 + 15) / 16 * nca;
          const int ncb = (s - k1 + 31) / 32, nb = (f + 15) / 16 * ncb;
          if (sizeof(T) == 8 && 4 * n <= 152)
            launch_clusters(k_mf_panel<T, 4>, dim3((na + nb + 4 + 3) / 4 * 4, n), MF_PANEL_THREADS, 4, 0, st, b, off,
                            (int)p, na, nca, ncb);
          else
            k_mf_panel<T, 1><<<dim3(na + nb + 1, n), MF_PANEL_THREADS, 0, st>>>(b, off, (int)p, na, nca, ncb);
        }
      }
    }
    if constexpr (sizeof(T) == 8) launch_front_t5(b, V, st);
    const int jobs = sizeof(T) == 8 ? V.schur_cnt : V.schur_all;
    if (jobs) {
      if (V.tile == 16) k_mf_schur<T, 16><<<jobs, 128, 0, st>>>(b, V.schur_off);
      else k_mf_schur<T, 32><<<jobs, 128, 0, st>>>(b, V.schur_off);
    }
  }
}

namespace {
// CTAs of a front in the substitutions: as many as leave an SM one, up to eight and a
// group of 32 rows each (the 24x24x2 mixed plate's step with at most two 10.9 ms, four
// 10.3, eight 10.3; the 64x64x2 plate's with one 33.0, eight 31.4).
int subst_ctas(int n, int rows) {
  int C = 1;
  while (C < 8 && 2 * C * n <= 152 && C * 32 < rows) C *= 2;
  return C;
}
}  // namespace

template <typename T> void launch_front_back(const Batch& b, cudaStream_t st) {
  const FrontSchedule& sc = *b.sh.mf.sched;
  for (size_t l = sc.level.size(); l-- > 0;) {
    const FrontLevel& V = sc.level[l];
    const int n = V.n_small + V.n_big, C = subst_ctas(n, V.max_s), f = std::max(V.small_f, V.big_f);
    const size_t w = (size_t)f + 2 + 8 * (size_t)std::min(((V.max_s + 31) / 32 + C - 1) / C * 32, MF_PART);
    launch_clusters(k_mf_back<T>, dim3(n * C), MF_BACK_THREADS, C, w * sizeof(T), st, b, V.small_off, C);
  }
  if constexpr (sizeof(T) == 8) k_mf_out<T><<<dim3(dof_blocks(b), b.sh.n_wide), 256, 0, st>>>(b);
}

void launch_front_solve(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  if (b.sh.n_wide == 0) return;
  { ProfScope q(prof, st, KC_WIDE_DIAG); launch_front_assemble<double>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_UPDATE); launch_front_factor<double>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_SUBST); launch_front_back<double>(b, st); }
}

// The same with the FP32 factor, on r32; the solution stays in the fronts' order.
void launch_front_solve32(const Batch& b, cudaStream_t st, LaunchProf* prof) {
  { ProfScope q(prof, st, KC_WIDE_DIAG); launch_front_assemble<float>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_UPDATE); launch_front_factor<float>(b, st); }
  { ProfScope q(prof, st, KC_WIDE_SUBST); launch_front_back<float>(b, st); }
}
// Another right-hand side (P or r32) with the factor that the fronts hold.
template <typename T> void launch_front_resolve(const Batch& b, cudaStream_t st) {
  for (const FrontLevel& V : b.sh.mf.sched->level) {
    const int n = V.n_small + V.n_big, f = std::max(V.small_f, V.big_f);
    const int C = subst_ctas(n, f);
    launch_clusters(k_mf_fwd<T>, dim3(n * C), MF_BACK_THREADS, C, (size_t)f * sizeof(T), st, b, V.small_off, C);
  }
  launch_front_back<T>(b, st);
}
void launch_front_resolve32(const Batch& b, cudaStream_t st) { launch_front_resolve<float>(b, st); }
int front_resolve_launches(const Batch& b) { return b.sh.mf.sched ? 2 * (int)b.sh.mf.sched->level.size() : 0; }

void launch_front_csr(const Batch& b, int n, const int* rp, const int* ci, const double* v, cudaStream_t st) {
  launch_front_zero<double>(b, st);
  k_mf_csr<<<(n + 127) / 128, 128, 0, st>>>(b, n, rp, ci, v);
}

void launch_front_band(const Batch& b, int n, int kl, int ku, int ldab, const double* ab, cudaStream_t st) {
  launch_front_zero<double>(b, st);
  const int64_t t = (int64_t)n * (kl + ku + 1);
  k_mf_band<<<(unsigned)((t + 255) / 256), 256, 0, st>>>(b, n, kl, ku, ldab, ab);
}

void launch_front_lu(const Batch& b, double* x, cudaStream_t st) {
  launch_front_factor<double>(b, st);
  Batch out = b;
  out.P = x;
  launch_front_back<double>(out, st);
}

void launch_front_refine(const Batch& b, int n, double* r, double* x, cudaStream_t st) {
  Batch rb = b;
  rb.P = r;
  launch_front_resolve<double>(rb, st);
  k_mf_add<<<(n + 255) / 256, 256, 0, st>>>(n, r, x);
}

void launch_csr_residual(int n, const int* rp, const int* ci, const double* v, const double* rhs, const double* x,
                         double* r, int* bad, cudaStream_t st) {
  k_csr_residual<<<(n + 15) / 16, 128, 0, st>>>(n, rp, ci, v, rhs, x, r, bad);
}

void launch_band_residual(int n, int kl, int ku, int ldab, const double* ab, const double* rhs, const double* x, double* r,
                          int* bad, cudaStream_t st) {
  k_band_residual<<<(n + 63) / 64, 64, 0, st>>>(n, kl, ku, ldab, ab, rhs, x, r, bad);
}

// Launches of one assembly, factorization and solve of the batch.
int front_launches(const Batch& b) {
  if (!b.sh.n_wide || !b.sh.mf.sched) return 0;
  return b.sh.mf.sched->launches + (b.n_loads ? 1 : 0) + (b.sh.n_shells ? 1 : 0);
}

}  // namespace gf
