// Multifrontal LU of K_AA under a nested-dissection ordering: the plan (host,
// gf_order.cu), the device data and the launches (gf_front.cu).
//
// The graph of K_AA's nodes is split recursively by small vertex separators;
// every separator (and every leaf) is a supernode, eliminated after the parts
// it separates.  A supernode's front is the dense matrix over its own DOFs and
// the DOFs of later supernodes its elimination touches (its boundary).  The
// fronts form a forest; all fronts of one height are independent, so the
// factorization is one sequence of launches per height, whatever the number
// of structures.  For a mesh of m x m squares the dense fronts cost about
// 20 (m d)^3 flops (d DOFs per grid line and square) and the longest dependent
// chain is about 3.3 m d pivots, against 2 n kl^2 flops and n pivots of a
// banded LU.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace gf {

// One front, column-major: entry (i, j) at F[off + i + j ld], rows and columns
// 0..s-1 the supernode's own DOFs, s..f-1 its boundary, column f the
// right-hand side.
struct Front {
  int64_t off;
  int f, s, ld;
  int slot;    // structure
  int dof0;    // its first own DOF in the elimination order (batch-wide index)
  int bnd;     // boundary DOFs (batch-wide elimination positions, ascending): bnd[bnd .. bnd + f - s)
  int rel;     // (host) the parent's front index of every boundary DOF: rel[rel .. rel + f - s)
  int parent;  // -1: a root
  int kid0, kid1;  // its children: kids[kid0 .. kid1)
};

// Fronts up to this size may take one CTA for the elimination, the whole matrix
// in its shared memory (k_mf_small); the others run panel by panel on many.  The line of
// a height is at or below it (small_limit, gf_order.cu).
constexpr int MF_SMALL = 96;
constexpr int MF_NB = 32;  // pivots per panel of a large front
// Shared memory of the substitutions beside their static part (gf_front.cu), and the rows
// of a front whose vector fits it with the partial sums of MF_PART rows.
constexpr int MF_SUBST_SMEM = 200 * 1024, MF_PART = 512;
constexpr int MF_MAX_ROWS = MF_SUBST_SMEM / 8 - 2 - 8 * MF_PART;
// Large fronts of a height that one launch takes where they are its grid's y or z (which
// end at 65,535): more of them, as a band of 200,000 blocks has, take several.
constexpr int MF_GRID_FRONTS = 65535;
inline int front_grids(int n) { return (n + MF_GRID_FRONTS - 1) / MF_GRID_FRONTS; }

// Large fronts whose Schur complement takes this many multiply-adds run it on the
// tensor cores (gf_front_t5.cu) where the caller lets them (GF_WIDE_TENSOR, the
// default): a 128 x 64 tile takes about 10 us for 64 pivots, an SM's FP64 units 40.
// Below, the tiles are too few and the slicing's launches (15 us a height) too dear.
// A rule on the front alone, so a structure is eliminated the same way in any batch.
constexpr double MF_T5_WORK = 1.5e6;
// Largest backward error of a row of a standalone system, in units of sum_j |a_ij| max_j
// |x_j| + |b_i| (j over the row's entries): sixteen roundings.  Dominant matrices, mesh
// and beam tangents reach 1 to 8 of them in either order, a tridiagonal system with a
// diagonal entry of 1e-3 that the dissection puts first 130, one of 1e-6 350,000.
constexpr double MF_ERROR_LIMIT = 0x1p-49;
// Such a front: its slices, exponents (per 64 pivots) and pivot maxima.
struct FrontT5 {
  int64_t slices;  // L21's at oz[slices], U12's behind: [64 pivots][slice][rows][64]
  int exps, kmax;  // [operand][64 pivots][rows], [operand][s]
  int rows;        // rows of L21 and columns of U12, padded to 128
  int front;
};

// Host schedule of one height.
struct FrontLevel {
  int small_off = 0, n_small = 0, small_f = 0;  // list range, largest small front
  int big_off = 0, n_big = 0;                   // list range, by descending s
  int big_f = 0, max_s = 0;                     // largest large front, most own DOFs of any
  std::vector<int> n_at;                        // large fronts that have panel k
  std::vector<int> f_at;                        // largest f among them
  std::vector<int> s_at;                        // largest s among them
  int ext_off = 0, ext_cnt = 0;                 // extend-add jobs of the large fronts
  int t5_off = 0, t5_cnt = 0, t5_rows = 0, t5_s = 0;  // fronts on the tensor cores, their most rows and pivots
  int t5_job_off = 0, t5_job_cnt = 0;
  // Schur jobs (FP32: all of them, the tensor-core fronts' too) and the rows and columns
  // of one
  int schur_off = 0, schur_cnt = 0, schur_all = 0, tile = 32;
};
struct FrontSchedule {
  std::vector<FrontLevel> level;
  int launches = 0;  // of one factorization and solve
};

// Device arrays; the schedule is host memory owned by the batch.
struct FrontData {
  Front* fronts;
  int* bnd;
  Front* list;      // the fronts by height
  int2* ext_jobs;   // (front, column block)
  int2* schur_jobs; // (front, row tile | column tile << 16), tiles of FrontLevel::tile rows
  int2* kids;       // (child front, offset in inv)
  int* inv;         // per child: its boundary index of every row of the parent (-1: none)
  int* dof_at;      // elimination position -> free DOF (batch-wide)
  int* pos;         // free DOF (batch-wide) -> elimination position (batch-wide)
  int* dof_front;   // elimination position -> its front
  // [n_shells][729] per K_e entry: x, its destination in F relative to the structure's first
  // front (-1: none, or an earlier element's entry takes the sum); y, the distance in K_e
  // entries to the next one of the same destination (0: the last)
  int2* map;
  int64_t* base;    // per structure: offset of its fronts in F
  int64_t* size;    // per structure: doubles of its fronts
  FrontT5* t5;      // by height
  int2* t5_jobs;    // (t5 entry, row tile | column tile << 16)
  __nv_bfloat16* oz;
  int* oz_exp;
  unsigned long long* oz_kmax;
  double* F;
  double* x;        // solution in the elimination order
  const FrontSchedule* sched;
};

}  // namespace gf

namespace gfh {

// Vertices of a symmetric graph with weights (DOFs); the splits are taken
// across level sets of the scalar fields, the first n_pref of them where those
// give a separator as small as a surface mesh's.
struct NdGraph {
  int n = 0;
  int n_pref = 0;
  std::vector<int> ptr, adj, w;
  std::vector<std::vector<float>> field;
};

// The fronts of one system of n DOFs; indices relative to the system.
struct FrontPlan {
  std::vector<gf::Front> fronts;
  std::vector<int> bnd, rel, height;
  std::vector<int> pos;        // DOF -> elimination position
  std::vector<int> dof_front;  // elimination position -> front
  int64_t size = 0;            // doubles
};

// Graph of a CSR matrix's symmetrised pattern, consecutive rows with the same columns (the
// DOFs of a mesh node) as one vertex: its rows are dptr[v] .. dptr[v + 1).
void csr_graph(int n, const int* rp, const int* ci, NdGraph& g, std::vector<int>& dptr);
// Landmark fields of a graph without coordinates: differences of squared
// distances to far-apart vertices (linear functions of the position where the
// graph is a mesh).
void nd_landmark_fields(NdGraph& g);
// The plan of a graph whose vertex v holds the DOFs dofs[dptr[v] .. dptr[v + 1]).
FrontPlan plan_fronts(const NdGraph& g, const std::vector<int>& dptr, const std::vector<int>& dofs);

// Whether the kernels take a plan: 32-bit offsets, and every front's vector in shared
// memory.
bool fronts_fit(const FrontPlan& P);

// Plans of several structures joined into one schedule; device offsets are
// batch-wide.
struct FrontBuild {
  std::vector<gf::Front> fronts;
  std::vector<gf::Front> list;
  std::vector<int> bnd, rel, pos, dof_front, inv, dof_at;
  std::vector<int2> kids, ext_jobs, schur_jobs;
  std::vector<int64_t> base, size;  // per structure (0 for the others)
  int64_t total = 0;
  std::vector<gf::FrontT5> t5;
  std::vector<int2> t5_jobs;
  int64_t oz = 0, oz_exp = 0, oz_kmax = 0;  // entries of the slice buffers (every height uses them in turn)
  gf::FrontSchedule sched;
};
// plans[k] belongs to structure slots[k], whose DOFs start at dof_off[k] of
// n_dofs; base and size are sized for n_struct.  tensor: large Schur complements on
// the tensor cores.
void join_fronts(const std::vector<const FrontPlan*>& plans, const std::vector<int>& slots,
                 const std::vector<int>& dof_off, int n_struct, int n_dofs, bool tensor, FrontBuild& out);

}  // namespace gfh
