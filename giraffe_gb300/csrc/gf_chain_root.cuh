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

// The last part of a chain with its end nodes, by one warp: 12 unknowns (u_p, a_p, u_n,
// a_n), lane j column j of the matrix, lane 12 the right-hand side; fixed DOFs
// are identity rows and columns, their pivots skipped.
template <typename Root>
__device__ void chain_root(const Batch& b, const ChainParts& c, const ChainTop& ch, int lane, Root R) {
  const int s = ch.structure;
  const int node[2] = {c.corner_node[ch.first], c.corner_node[ch.last]};
  const int g = lane < 12 ? b.gl[(int64_t)node[lane / 6] * 6 + lane % 6] : -1;
  const unsigned live = __ballot_sync(0xffffffffu, g >= 0);
  double* P = b.P + b.info[s].dof_off;
  double col[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    double v = 0.0;
    if (lane < 12) {
      if ((live >> i & 1) && (live >> lane & 1)) {
        v = R.k(i, lane);
        if (i % 6 >= 3 && lane % 6 >= 3 && i / 6 == lane / 6)
          v = radd(v, b.nodeK[(int64_t)node[i / 6] * 9 + (i % 6 - 3) * 3 + lane % 6 - 3]);
      } else {
        v = i == lane ? 1.0 : 0.0;
      }
    } else if (lane == 12 && (live >> i & 1)) {
      v = radd(P[b.gl[(int64_t)node[i / 6] * 6 + i % 6]],
               R.f(i));
    }
    col[i] = v;
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    if (!(live >> k & 1)) continue;
    const double p = __shfl_sync(0xffffffffu, col[k], k);
    if (!(p != 0.0) || !isfinite(p)) ok = false;
    const double inv = rcp64(p);
    double m[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) m[i] = __shfl_sync(0xffffffffu, col[i], k);
    if (lane > k && lane < 13) {
      const double rk = rmul(col[k], inv);
      col[k] = rk;
#pragma unroll
      for (int i = 0; i < 12; ++i)
        if (i != k) col[i] = rfma(-m[i], rk, col[i]);
    }
  }
  if (!ok && lane == 0) b.state[s].info_fail = 1;
  double x = 0.0;
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    const double v = __shfl_sync(0xffffffffu, col[i], 12);
    if (lane == i) x = v;
  }
  if (lane < 12) {
    c.x[6 * (int64_t)(lane < 6 ? ch.first : ch.last) + lane % 6] = g >= 0 ? x : 0.0;
    if (g >= 0) P[g] = x;
  }
}

}  // namespace gf
