// Standalone linear solves in the reference's matrix layouts:
//
//   gf_sparse_solve   K in SparseMatrix's layout (Eigen row-major CSR,
//                     0-based), replaces sparsesystem (reference
//                     src/SparseMatrix.cpp:74-166)
//   wide_band_solve   K in BandMatrix's LAPACK GB layout with a half
//                     bandwidth above 17, the wide branch of gf_band_solve
//                     (bandsystem, src/BandMatrix.cpp:257-287)
//
// Both factor on the GPU without pivoting: by the multifrontal LU of the
// Shell_1 path (gf_front.cu) under a nested-dissection ordering of the CSR's
// graph or of the band's blocks; by the 35-row band solver and the wide-band LU
// (gf_wideband.cu) where those are estimated faster (short bands) or the fronts
// would be too large.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/giraffe_gpu.h"
#include "gf_host_internal.h"
#include "gf_front_system.h"
#include "gf_kernels.cuh"
#include "gf_types.h"
#include "gf_wide.h"

using namespace gf;

namespace gf {

// CSR rows scattered into the wide band (column-major, W = 2w + 1 rows,
// entry (i, j) at (w + i - j) + j W) under the symmetric permutation perm,
// one thread per row: distinct rows own distinct band entries, and the
// entries of a row are summed in order, so duplicates add up the same way
// on every run.  The right-hand side is permuted alongside.
__global__ void k_csr_to_wide(int n, const int* rp, const int* ci, const double* v, const int* perm, double* a,
                              int w, int64_t W, const double* b, double* P) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int pi = perm[i];
  for (int k = rp[i]; k < rp[i + 1]; ++k) {
    const int pj = perm[ci[k]];
    a[(w + pi - pj) + (int64_t)pj * W] += v[k];
  }
  P[pi] = b[i];
}

// x[i] = y[perm[i]]
__global__ void k_unpermute(int n, const int* perm, const double* y, double* x) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = y[perm[i]];
}

}  // namespace gf

namespace {

using namespace gfh;

// Half-bandwidth max |i - j| of the pattern under the ordering pos (row or
// column i at pos[i]).
int csr_bandwidth(int n, const int* rp, const int* ci, const int* pos) {
  int w = 0;
  for (int i = 0; i < n; ++i)
    for (int k = rp[i]; k < rp[i + 1]; ++k) w = std::max(w, std::abs(pos[i] - pos[ci[k]]));
  return w;
}

}  // namespace

namespace gfh {

// The multifrontal LU eliminates a band of half-bandwidth w in blocks of w,
// about 6.3 w^3 multiply-adds a block on a chain of log2(n / w) blocks; the
// banded LU takes w^2 per column on a chain of n.  Both are estimated: the 35-row
// band solver at 0.9 us a column, the wide-band LU at 85 us per 64 columns plus its
// updates at 5.4 TFLOP/s, either with 0.17 ms of allocations and copies; the fronts
// at 0.9 TFLOP/s, 0.6 us a pivot of the chain and 12 us a height.  Measured, band
// against fronts, half-bandwidth and n: 2 and 60 0.26 / 0.09 ms, 12 and 2,000 1.92 /
// 0.32, 17 and 60,000 52.5 / 5.0, 60 and 20,000 30.0 / 4.5, 120 and 600 1.20 / 0.76,
// 240 and 2,000 3.42 / 2.78, 240 and 60,000 92.9 / 71.8; the other way 480 and 2,000
// 3.56 / 5.07, 480 and 60,000 98 / 166, 900 and 20,000 34 / 130.
bool band_takes_fronts(int n, int kl, int ku) {
  const double w = std::max(std::max(kl, ku), 12);
  const double blocks = n / w;
  if (blocks < 4.0) return false;
  const double chain = w * (std::ceil(std::log2(blocks)) + 1.0);
  const double t_front = 12.6 * w * w * n / 0.9e12 + 0.6e-6 * chain + 12e-6 * chain / w;
  const double t_band =
      0.17e-3 + (kl <= GF_KB && ku <= GF_KB ? 0.9e-6 * n : n / 64.0 * 85e-6 + 2.0 * n * w * w / 5.4e12);
  return t_front < t_band;
}

static int band_on_fronts(gf_ctx* ctx, int n, int kl, int ku, const double* ab, int ldab, double* b, bool* done) {
  // blocks of at least the half-bandwidth: their graph is a path
  const int B = std::max(std::max(kl, ku), 12), nb = (n + B - 1) / B, W = kl + ku + 1;
  NdGraph g;
  g.n = nb;
  g.ptr.push_back(0);
  g.field.resize(1);
  std::vector<int> dptr(1, 0), dofs(n);
  for (int v = 0; v < nb; ++v) {
    if (v) g.adj.push_back(v - 1);
    if (v + 1 < nb) g.adj.push_back(v + 1);
    g.ptr.push_back((int)g.adj.size());
    dptr.push_back(std::min(n, (v + 1) * B));
    g.w.push_back(dptr[v + 1] - dptr[v]);
    g.field[0].push_back((float)v);
  }
  for (int i = 0; i < n; ++i) dofs[i] = i;
  const FrontPlan plan = plan_fronts(g, dptr, dofs);
  if (!fronts_fit(plan)) return GF_OK;
  std::vector<double> packed((size_t)n * W);
  for (int j = 0; j < n; ++j)
    std::memcpy(&packed[(size_t)j * W], ab + (size_t)j * ldab + kl, sizeof(double) * (size_t)W);
  FrontSystem S;
  std::vector<int> part;
  if (S.init(ctx, plan, n, b, {{packed.data(), sizeof(double) * packed.size()}}, &part) != GF_OK) return GF_OK;
  const double* A = S.at<double>(part[0]) - kl;
  return S.solve(ctx, n, [&](const Batch& q) { launch_front_band(q, n, kl, ku, W, A, ctx->stream); },
                 [&](const double* x, double* r, int* bad) { launch_band_residual(n, kl, ku, W, A, S.b.P, x, r, bad, ctx->stream); },
                 b, done);
}

static int sparse_on_fronts(gf_ctx* ctx, int n, const int* rp, const int* ci, const double* val, double* b, bool* done) {
  if (rp[n] > INT_MAX / 2) return GF_OK;  // both directions of its edges are counted in 32 bits
  NdGraph g;
  std::vector<int> dptr, dofs(n);
  csr_graph(n, rp, ci, g, dptr);
  for (int i = 0; i < n; ++i) dofs[i] = i;
  nd_landmark_fields(g);
  std::vector<float> place(g.n);
  for (int v = 0; v < g.n; ++v) place[v] = (float)v;
  g.field.push_back(std::move(place));
  const FrontPlan plan = plan_fronts(g, dptr, dofs);
  if (!fronts_fit(plan)) return GF_OK;
  const size_t nnz = rp[n];
  FrontSystem S;
  std::vector<int> part;
  if (S.init(ctx, plan, n, b, {{rp, sizeof(int) * ((size_t)n + 1)}, {ci, sizeof(int) * nnz}, {val, sizeof(double) * nnz}},
             &part) != GF_OK)
    return GF_OK;
  const int *drp = S.at<int>(part[0]), *dci = S.at<int>(part[1]);
  const double* dv = S.at<double>(part[2]);
  return S.solve(ctx, n, [&](const Batch& q) { launch_front_csr(q, n, drp, dci, dv, ctx->stream); },
                 [&](const double* x, double* r, int* bad) { launch_csr_residual(n, drp, dci, dv, S.b.P, x, r, bad, ctx->stream); },
                 b, done);
}

// A front solve that host memory does not allow leaves *done false too.
template <typename Solve> static int front_solve(bool* done, Solve solve) {
  *done = false;
  try {
    return solve();
  } catch (const std::bad_alloc&) {
    return GF_OK;
  }
}
int front_band_solve(gf_ctx* ctx, int n, int kl, int ku, const double* ab, int ldab, double* b, bool* done) {
  return front_solve(done, [&] { return band_on_fronts(ctx, n, kl, ku, ab, ldab, b, done); });
}
int front_sparse_solve(gf_ctx* ctx, int n, const int* rp, const int* ci, const double* val, double* b, bool* done) {
  return front_solve(done, [&] { return sparse_on_fronts(ctx, n, rp, ci, val, b, done); });
}

// Wide branch of gf_band_solve: the GB array goes into the wide band with
// one strided copy (each column's kl + ku + 1 stored entries keep their
// order), then the blocked LU runs.
int wide_band_solve(gf_ctx* ctx, int n, int kl, int ku, const double* ab, int ldab, double* b, int* info) {
  const int w = std::max(kl, ku);
  const int64_t W = 2 * (int64_t)w + 1;
  DevBufs mem;
  Helpers hl;
  double *dband = nullptr, *dP = nullptr, *dY = nullptr;
  if (!mem.get(&dband, (size_t)n * W) || !mem.get(&dP, (size_t)n) || !mem.get(&dY, (size_t)n)) {
    set_err(ctx, "gf_band_solve: device allocation of %lld bytes failed", (long long)(8 * ((size_t)n * W + 2 * n)));
    return GF_ERR_CUDA;
  }
  cudaStream_t s = ctx->stream;
  // GB entry (i, j) sits at row kl + ku + i - j of column j; the wide band
  // holds it at row w + i - j, so rows kl .. 2 kl + ku of a GB column land
  // on rows w - ku .. w + kl
  GF_CK(cudaMemsetAsync(dband, 0, sizeof(double) * (size_t)n * W, s));
  GF_CK(cudaMemcpy2DAsync(dband + (w - ku), sizeof(double) * W, ab + kl, sizeof(double) * ldab,
                          sizeof(double) * (kl + ku + 1), n, cudaMemcpyHostToDevice, s));
  GF_CK(cudaMemcpyAsync(dP, b, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  WideBatch wb;
  if (!wb.init(ctx, mem, hl, n, w, dband, dP, dY)) {
    set_err(ctx, "gf_band_solve: set-up of the wide-band solve failed");
    return GF_ERR_CUDA;
  }
  int fail = 0;
  GF_CK(wb.solve(ctx, &fail));
  GF_CK(cudaMemcpy(b, dP, sizeof(double) * n, cudaMemcpyDeviceToHost));
  if (info) *info = fail;
  return GF_OK;
}

}  // namespace gfh

extern "C" {

int gf_sparse_solve(gf_ctx* ctx, int n, const int* row_ptr, const int* col_idx, const double* val, double* b,
                    int* info) {
  if (!ctx || n <= 0 || !row_ptr || !col_idx || !val || !b) {
    if (ctx) gfh::set_err(ctx, "gf_sparse_solve: invalid arguments");
    return GF_ERR_ARG;
  }
  if (row_ptr[0] != 0) {
    gfh::set_err(ctx, "gf_sparse_solve: row_ptr[0] must be 0 (0-based CSR)");
    return GF_ERR_ARG;
  }
  for (int i = 0; i < n; ++i)
    if (row_ptr[i + 1] < row_ptr[i]) {
      gfh::set_err(ctx, "gf_sparse_solve: row_ptr decreases at row %d", i);
      return GF_ERR_ARG;
    }
  const int nnz = row_ptr[n];
  for (int k = 0; k < nnz; ++k)
    if (col_idx[k] < 0 || col_idx[k] >= n) {
      gfh::set_err(ctx, "gf_sparse_solve: column index %d out of range at entry %d", col_idx[k], k);
      return GF_ERR_ARG;
    }
  // a narrow band in the natural order goes to the band solvers, anything
  // wider to the multifrontal LU under a nested-dissection ordering
  bool wide = false;
  for (int i = 0; i < n && !wide; ++i)
    for (int k = row_ptr[i]; k < row_ptr[i + 1] && !wide; ++k) wide = std::abs(i - col_idx[k]) > GF_KB;
  if (wide) {
    bool done = false;
    const int rc = gfh::front_sparse_solve(ctx, n, row_ptr, col_idx, val, b, &done);
    if (rc == GF_OK && done && info) *info = 0;
    if (rc != GF_OK || done) return rc;
  }
  // a system that the multifrontal LU does not take or not solve to the accuracy that it
  // asks of it, or a narrow band: ordering natural, or reverse Cuthill-McKee on the
  // symmetrised pattern when that narrows the band
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = i;
  int w = csr_bandwidth(n, row_ptr, col_idx, perm.data());
  if (w > 2 * GF_KB) {
    std::vector<std::vector<int>> adj(n);
    for (int i = 0; i < n; ++i)
      for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
        const int j = col_idx[k];
        if (j == i) continue;
        adj[i].push_back(j);
        adj[j].push_back(i);
      }
    for (auto& v : adj) {
      std::sort(v.begin(), v.end());
      v.erase(std::unique(v.begin(), v.end()), v.end());
    }
    const std::vector<int> order = gfh::rcm_order(n, adj);  // order[k] = row placed k-th
    std::vector<int> pos(n);
    for (int k = 0; k < n; ++k) pos[order[k]] = k;
    const int w_rcm = csr_bandwidth(n, row_ptr, col_idx, pos.data());
    if (w_rcm < w) {
      w = w_rcm;
      perm = pos;
    }
  }
  w = std::max(w, 1);
  if (w <= GF_KB) {
    // narrow: LAPACK GB of the permuted matrix, through gf_band_solve
    const int ldab = 3 * w + 1;
    std::vector<double> ab((size_t)n * ldab, 0.0), x(n);
    for (int i = 0; i < n; ++i)
      for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
        const int pi = perm[i], pj = perm[col_idx[k]];
        ab[(size_t)(2 * w + pi - pj) + (size_t)pj * ldab] += val[k];
      }
    for (int i = 0; i < n; ++i) x[perm[i]] = b[i];
    int rc = gf_band_solve(ctx, n, w, w, ab.data(), ldab, x.data(), info);
    if (rc != GF_OK) return rc;
    for (int i = 0; i < n; ++i) b[i] = x[perm[i]];
    return GF_OK;
  }
  const int64_t W = 2 * (int64_t)w + 1;
  DevBufs mem;
  Helpers hl;
  double *dband = nullptr, *dP = nullptr, *dY = nullptr, *dv = nullptr, *db = nullptr;
  int *drp = nullptr, *dci = nullptr, *dperm = nullptr;
  if (!mem.get(&dband, (size_t)n * W) || !mem.get(&dP, (size_t)n) || !mem.get(&dY, (size_t)n) ||
      !mem.get(&dv, (size_t)nnz) || !mem.get(&db, (size_t)n) || !mem.get(&drp, (size_t)n + 1) ||
      !mem.get(&dci, (size_t)nnz) || !mem.get(&dperm, (size_t)n)) {
    gfh::set_err(ctx, "gf_sparse_solve: device allocation failed (half-bandwidth %d, %lld band bytes)", w,
                 (long long)(8 * (size_t)n * W));
    return GF_ERR_CUDA;
  }
  cudaStream_t s = ctx->stream;
  GF_CK(cudaMemsetAsync(dband, 0, sizeof(double) * (size_t)n * W, s));
  GF_CK(cudaMemcpyAsync(drp, row_ptr, sizeof(int) * (n + 1), cudaMemcpyHostToDevice, s));
  GF_CK(cudaMemcpyAsync(dci, col_idx, sizeof(int) * std::max(nnz, 1), cudaMemcpyHostToDevice, s));
  GF_CK(cudaMemcpyAsync(dv, val, sizeof(double) * std::max(nnz, 1), cudaMemcpyHostToDevice, s));
  GF_CK(cudaMemcpyAsync(db, b, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  GF_CK(cudaMemcpyAsync(dperm, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
  k_csr_to_wide<<<(n + 127) / 128, 128, 0, s>>>(n, drp, dci, dv, dperm, dband, w, W, db, dP);
  WideBatch wbt;
  if (!wbt.init(ctx, mem, hl, n, w, dband, dP, dY)) {
    gfh::set_err(ctx, "gf_sparse_solve: set-up of the wide-band solve failed");
    return GF_ERR_CUDA;
  }
  int fail = 0;
  GF_CK(wbt.solve(ctx, &fail));
  k_unpermute<<<(n + 127) / 128, 128, 0, s>>>(n, dperm, dP, db);
  GF_CK(cudaGetLastError());
  GF_CK(cudaMemcpyAsync(b, db, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  GF_CK(cudaStreamSynchronize(s));
  if (info) *info = fail;
  return GF_OK;
}

}  // extern "C"
