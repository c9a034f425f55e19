// What the two chain eliminations (gf_chain.cu, gf_chain_sym.cu) share on the
// device: the structure-of-arrays access and the solve of a chain's last part.
#pragma once
#include "gf_beam_gp.cuh"
#include "gf_math.cuh"
#include "gf_types.h"

namespace gf {

// Entry x of item i (n entries each): the first `soa` items structure-of-arrays,
// the others item by item behind them.
__device__ __forceinline__ double& chain_at(double* a, int soa, int n, int i, int x) {
  return a[i < soa ? (int64_t)x * soa + i : (int64_t)i * n + x];
}

__device__ __forceinline__ bool solving(const Batch& b, int s) {
  const StructState& st = b.state[s];
  return st.phase == PH_ITER && st.need_solve;
}

// The last merges of a chain (at most CHAIN_TOP - 1) as its CTA takes them: where
// the parts and the neighbours' solutions of each come from, the forces of its
// corner.
constexpr int TOP_MERGES = CHAIN_TOP - 1, TOP_FIRST = TOP_MERGES, TOP_LAST = TOP_MERGES + 1, TOP_THREADS = 256;
struct ChainTopShared {
  ChainMerge m[TOP_MERGES];
  int part1[TOP_MERGES], part2[TOP_MERGES];  // the merge that made e1 (e2), or -1: an earlier kernel
  int p[TOP_MERGES], n[TOP_MERGES];          // the merge of corner p (n), TOP_FIRST or TOP_LAST
  double f[TOP_MERGES][6];                   // forces of the corner's free DOFs, zero at its fixed ones
  double x[TOP_MERGES + 2][6];               // solution of the corners, then of the chain's ends
};
__device__ __forceinline__ void top_load(const Batch& b, const ChainParts& c, const ChainTop& ch, int tid, ChainTopShared& S) {
  const int n = ch.n_top - 1;
  for (int t = tid; t < n; t += TOP_THREADS) S.m[t] = c.merge[ch.top + t];
  __syncthreads();
  for (int y = tid; y < 6 * n; y += TOP_THREADS) {
    const ChainMerge& m = S.m[y / 6];
    const int i = y % 6;
    S.f[y / 6][i] = m.mask >> i & 1 ? b.P[m.dof + __popc(m.mask & ((1 << i) - 1))] : 0.0;
  }
  for (int y = tid; y < 4 * n; y += TOP_THREADS) {
    const int t = y >> 2, q = y & 3;
    const ChainMerge& m = S.m[t];
    const int key = q == 0 ? m.e1 : q == 1 ? m.e2 : q == 2 ? m.p : m.n;
    int at = q < 2 ? -1 : key == ch.first ? TOP_FIRST : TOP_LAST;
    for (int o = 0; o < n; ++o)
      if ((q < 2 ? S.m[o].out : S.m[o].k) == key) at = o;
    (q == 0 ? S.part1 : q == 1 ? S.part2 : q == 2 ? S.p : S.n)[t] = at;
  }
  __syncthreads();
}

// The last part of a chain with its end nodes, by one warp: 12 unknowns (u_p, a_p, u_n,
// a_n) by Gauss-Jordan, column j of the matrix in lanes j (rows 0-5) and 16 + j
// (rows 6-11), column 12 the right-hand side; fixed DOFs are identity rows and
// columns, their pivots skipped.  Bound by the chain of its pivots, 64 cycles an
// FP64 operation: six updates a pivot here against eleven with a lane per column.
template <typename Root>
__device__ void chain_root(const Batch& b, const ChainParts& c, const ChainTop& ch, int lane, Root R, double* xs) {
  const int s = ch.structure, j = lane & 15, half = lane >> 4;
  const int node0 = c.corner_node[ch.first], node1 = c.corner_node[ch.last];
  const int g = lane < 12 ? b.gl[(int64_t)(lane < 6 ? node0 : node1) * 6 + lane % 6] : -1;
  const unsigned live = __ballot_sync(0xffffffffu, g >= 0);
  double* P = b.P + b.info[s].dof_off;
  const double* nk = b.nodeK + (int64_t)(half ? node1 : node0) * 9;
  // an entry and what comes on top of it, every load before the first sum
  double col[6], add[6];
  bool on[6], more[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const int r = 6 * half + i, gi = __shfl_sync(0xffffffffu, g, r);
    on[i] = (live >> r & 1) && (j == 12 || (j < 12 && (live >> j & 1)));
    more[i] = on[i] && (j == 12 || (i >= 3 && j - 6 * half >= 3 && j - 6 * half < 6));
    col[i] = on[i] ? (j == 12 ? R.f(r) : R.k(r, j)) : 0.0;
    const double* at = j == 12 ? P + gi : nk + (i - 3) * 3 + j - 6 * half - 3;
    add[i] = more[i] ? *at : 0.0;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    if (j < 12 && R.minus(6 * half + i, j)) col[i] = -col[i];
    if (!on[i]) col[i] = 6 * half + i == j ? 1.0 : 0.0;
    if (more[i]) col[i] = radd(col[i], add[i]);
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    if (!(live >> k & 1)) continue;
    const int kh = k / 6, kr = k % 6;
    const double p = __shfl_sync(0xffffffffu, col[kr], 16 * kh + k);
    ok = ok && !bad_pivot(p);
    const double inv = rcp64(p);
    const double xk = __shfl_sync(0xffffffffu, col[kr], 16 * kh + j);
    double m[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) m[i] = __shfl_sync(0xffffffffu, col[i], 16 * half + k);
    if (j > k && j < 13) {
      const double rk = rmul(xk, inv);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        if (i == kr && half == kh) col[i] = rk;
        else col[i] = rfma(-m[i], rk, col[i]);
      }
    }
  }
  if (!ok && lane == 0) b.state[s].info_fail = 1;
  double x = 0.0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const double v = __shfl_sync(0xffffffffu, col[i], lane < 6 ? 12 : 28);
    if (lane % 6 == i) x = v;
  }
  if (lane < 12) {
    xs[lane] = g >= 0 ? x : 0.0;
    c.x[6 * (int64_t)(lane < 6 ? ch.first : ch.last) + lane % 6] = g >= 0 ? x : 0.0;
    if (g >= 0) P[g] = x;
  }
}

}  // namespace gf
