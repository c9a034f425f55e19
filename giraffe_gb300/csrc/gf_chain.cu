// General elimination of Beam_1 chains (see gf_chain.cuh): Dynamic steps and loads
// with stiffness of their own, whose K_AA is not symmetric (the symmetric one is
// in gf_chain_sym.cu).  Parts are 12x12 matrices over the DOFs (u_p, a_p, u_n,
// a_n) of their two corners.  An elimination of six unknowns is Gauss-Jordan on
// [D | b | K_p | K_n] (19 columns) and the products of the two coupling rows with
// the 13 solved columns, about 1,550 FP64 operations that form the new part
// outright.
//
// Two forms with the same operations on every entry, so the same bits: one item
// per thread, whose FP64 warp instructions carry 32 items, for the large levels,
// and one item per warp for the small ones, where an item's chain of dependent
// operations (64 cycles each on this part) is what counts.
#include <cuda_runtime.h>

#include "gf_chain.cuh"
#include "gf_chain_root.cuh"
#include "gf_kernels.cuh"
#include "gf_math.cuh"

namespace gf {

namespace {

constexpr int CT = 64;  // threads per block of the item-per-thread form
constexpr int NC = 19;  // augmented columns: 6 (matrix) + 13 (right-hand sides)

// Part: the matrix ([row * 12 + column]), then the forces on p and n.
constexpr int GP_F = 144;

// The item-per-warp form's staging area (doubles): two parts or an 18x18 K_e, a
// zero, the forces of a midside node.
constexpr int GEN_E2 = CHAIN_GEN_PART, GEN_ZERO = 324, GEN_F = 325, GEN_STAGE = 332;
static_assert(2 * CHAIN_GEN_PART <= GEN_ZERO, "two parts");

// Gauss-Jordan on a thread's augmented matrix [D | R] in two phases, both in
// registers: gj6_factor eliminates D (6x6, row-major, every index static under
// the full unroll) and records each pivot's reciprocal and multipliers;
// gj6_apply then takes one right-hand-side column through the same steps in
// the same order (r_k *= 1/p_k, then r_i -= m_ik r_k), so each column needs
// its six entries only and no shared memory.  The operations on every entry
// are those of the joined elimination.  No pivoting; gj6_factor returns false
// on a zero or non-finite pivot.
__device__ __forceinline__ bool gj6_factor(double (&D)[36], double (&inv)[6], double (&mult)[36]) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double p = D[k * 6 + k];
    ok = ok && !bad_pivot(p);
    inv[k] = rcp64(p);
    double dk[6];
#pragma unroll
    for (int c = k + 1; c < 6; ++c) {
      dk[c] = D[k * 6 + c] * inv[k];
      D[k * 6 + c] = dk[c];
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (i == k) continue;
      const double m = D[i * 6 + k];
      mult[k * 6 + i] = m;
#pragma unroll
      for (int c = k + 1; c < 6; ++c) D[i * 6 + c] = fma(-m, dk[c], D[i * 6 + c]);
    }
  }
  return ok;
}
__device__ __forceinline__ void gj6_apply(const double (&inv)[6], const double (&mult)[36], double (&r)[6]) {
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double rk = r[k] * inv[k];
    r[k] = rk;
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i != k) r[i] = fma(-mult[k * 6 + i], rk, r[i]);
  }
}

// Condensation of the midside node of part t: K_e (column-major 18x18, DOFs of
// the first corner, the midside node, the last corner) and the midside node's
// load stiffness.  Fixed DOFs of the corners have zero rows and columns.
struct GenCondense {
  const Batch& b;
  const ChainParts& c;
  int t, s, mask, nm;
  const double *K, *P;
  int64_t ne;
  __device__ __forceinline__ void init(int t_) {
    t = t_;
    const int e = c.elem[t];
    s = c.elem_struct[t];
    mask = c.elem_mask[t];
    nm = b.enodes[3 * e + 1];
    K = b.Ke + e;
    P = b.P + c.elem_dof[t];
    ne = b.n_elem;
  }
  __device__ __forceinline__ bool active() const { return solving(b, s); }
  __device__ __forceinline__ static int place(int x) { return x < 6 ? x : 6 + x; }  // corner DOF 0..11 in K_e
  __device__ __forceinline__ bool live(int x) const { return mask >> x & 1; }
  __device__ __forceinline__ double ke(int i, int j) const { return K[(int64_t)(i + 18 * j) * ne]; }
  __device__ __forceinline__ double d(int i, int j) const {
    double v = ke(6 + i, 6 + j);
    if (i >= 3 && j >= 3) v += b.nodeK[(int64_t)nm * 9 + (i - 3) * 3 + j - 3];
    return v;
  }
  __device__ __forceinline__ double r(int i, int q) const {
    return q == 0 ? P[i] : live(q - 1) ? ke(6 + i, place(q - 1)) : 0.0;
  }
  // coupling of corner DOF x to unknown k
  __device__ __forceinline__ double left(int x, int k) const { return live(x) ? ke(place(x), 6 + k) : 0.0; }
  __device__ __forceinline__ double base(int x, int q) const {
    return q == 0 || !live(x) || !live(q - 1) ? 0.0 : ke(place(x), place(q - 1));
  }
  // The item-per-warp form: K_e with its fixed corner DOFs cleared at s[0], the
  // midside node's forces at s[GEN_F], its load stiffness added.
  __device__ __forceinline__ void stage(int lane, double* s) const {
    double v[11], extra = 0.0;
#pragma unroll
    for (int q = 0; q < 11; ++q) {
      const int x = lane + 32 * q, i = x % 18, j = x / 18;
      const bool fixed = (i < 6 && !live(i)) || (i >= 12 && !live(i - 6)) || (j < 6 && !live(j)) || (j >= 12 && !live(j - 6));
      v[q] = x < 324 && !fixed ? K[(int64_t)x * ne] : 0.0;
    }
    const double* at = lane < 9 ? b.nodeK + (int64_t)nm * 9 + lane : P + lane - 9;
    if (lane < 15) extra = *at;
#pragma unroll
    for (int q = 0; q < 11; ++q)
      if (lane + 32 * q < 324) s[lane + 32 * q] = v[q];
    if (lane == 31) s[GEN_ZERO] = 0.0;
    if (lane >= 9 && lane < 15) s[GEN_F + lane - 9] = extra;
    __syncwarp();
    if (lane < 9) s[9 + lane / 3 + 18 * (9 + lane % 3)] += extra;
    __syncwarp();
  }
  // where column `lane` of [D | R] is the sum of: entries a + i sa and o + i so
  __device__ __forceinline__ void column(int lane, int& a, int& sa, int& o, int& so) const {
    a = lane < 6 ? 6 + 18 * (6 + lane) : lane == 6 ? GEN_F : lane < NC ? 6 + 18 * place(lane - 7) : GEN_ZERO;
    sa = lane < NC ? 1 : 0;
    o = GEN_ZERO;
    so = 0;
  }
  __device__ __forceinline__ static double pinned(int, int, double v) { return v; }
  __device__ __forceinline__ static double left_s(const double* s, int x, int k) { return s[place(x) + 18 * (6 + k)]; }
  __device__ __forceinline__ static double base_s(const double* s, int x, int q) {
    return s[q == 0 ? GEN_ZERO : place(x) + 18 * place(q - 1)];
  }
  __device__ __forceinline__ void keep(int x, double v) const { chain_at(c.ez, c.elem_soa, CHAIN_GEN_KEEP, t, x) = v; }
  __device__ __forceinline__ void out(int x, int q, double v) const {
    chain_at(c.part, c.part_soa, CHAIN_GEN_PART, t, q == 0 ? GP_F + x : x * 12 + q - 1) = v;
  }
  __device__ void fail() const { b.state[s].info_fail = 1; }
};

// Elimination of corner k between parts e1 (p to k) and e2 (k to n).
struct GenMerge {
  const Batch& b;
  const ChainParts& c;
  ChainMerge m;
  int t, node;
  __device__ __forceinline__ void init(int t_) {
    t = t_;
    m = c.merge[t];
    node = c.corner_node[m.k];
  }
  __device__ __forceinline__ bool active() const { return solving(b, m.structure); }
  __device__ __forceinline__ double E(int e, int x) const { return chain_at(c.part, c.part_soa, CHAIN_GEN_PART, e, x); }
  __device__ __forceinline__ bool live(int i) const { return m.mask >> i & 1; }
  __device__ __forceinline__ double d(int i, int j) const {
    if (!live(i) || !live(j)) return i == j ? 1.0 : 0.0;
    double v = E(m.e1, (6 + i) * 12 + 6 + j);
    if (i >= 3 && j >= 3) v += b.nodeK[(int64_t)node * 9 + (i - 3) * 3 + j - 3];
    return v + E(m.e2, i * 12 + j);
  }
  __device__ __forceinline__ double r(int i, int q) const {
    if (q == 0)  // the corner's own force with what both parts leave on it
      return live(i) ? b.P[m.dof + __popc(m.mask & ((1 << i) - 1))] + E(m.e1, GP_F + 6 + i) + E(m.e2, GP_F + i) : 0.0;
    return q < 7 ? E(m.e1, (6 + i) * 12 + q - 1) : E(m.e2, i * 12 + q - 1);
  }
  __device__ __forceinline__ double left(int x, int k) const {
    return x < 6 ? E(m.e1, x * 12 + 6 + k) : E(m.e2, x * 12 + k);
  }
  __device__ __forceinline__ double base(int x, int q) const {
    if (q == 0) return x < 6 ? E(m.e1, GP_F + x) : E(m.e2, GP_F + x);
    if ((x < 6) != (q < 7)) return 0.0;
    return E(x < 6 ? m.e1 : m.e2, x * 12 + q - 1);
  }
  // The item-per-warp form: e1 at s[0], e2 at s[GEN_E2], the corner's load stiffness
  // and force added to e1.
  __device__ __forceinline__ void stage(int lane, double* s) const {
    double v1[5], v2[5], extra = 0.0;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int x = lane + 32 * q;
      v1[q] = x < CHAIN_GEN_PART ? E(m.e1, x) : 0.0;
      v2[q] = x < CHAIN_GEN_PART ? E(m.e2, x) : 0.0;
    }
    const int f = lane - 9;
    const double* at = lane < 9 ? b.nodeK + (int64_t)node * 9 + lane : b.P + m.dof + __popc(m.mask & ((1 << f) - 1));
    if (lane < 9 || (lane < 15 && live(f))) extra = *at;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int x = lane + 32 * q;
      if (x < CHAIN_GEN_PART) {
        s[x] = v1[q];
        s[GEN_E2 + x] = v2[q];
      }
    }
    if (lane == 31) s[GEN_ZERO] = 0.0;
    __syncwarp();
    if (lane < 15) s[lane < 9 ? (9 + lane / 3) * 12 + 9 + lane % 3 : GP_F + 6 + f] += extra;
    __syncwarp();
  }
  __device__ __forceinline__ static void column(int lane, int& a, int& sa, int& o, int& so) {
    const int q = lane - 6;
    const bool first = lane < 6 || q == 0 || (q > 0 && q < 7), second = lane < 6 || q == 0 || (q >= 7 && lane < NC);
    a = !first ? GEN_ZERO : q == 0 ? GP_F + 6 : 72 + (lane < 6 ? 6 + lane : q - 1);
    sa = !first ? 0 : q == 0 ? 1 : 12;
    o = !second ? GEN_ZERO : GEN_E2 + (q == 0 ? GP_F : lane < 6 ? lane : q - 1);
    so = !second ? 0 : q == 0 ? 1 : 12;
  }
  // entry i of column `lane` where the corner is fixed
  __device__ __forceinline__ double pinned(int i, int lane, double v) const { return pinned(m.mask, i, lane, v); }
  __device__ __forceinline__ static double pinned(int mask, int i, int lane, double v) {
    if (lane < 6 && !((mask >> i & 1) && (mask >> lane & 1))) return i == lane ? 1.0 : 0.0;
    return lane == 6 && !(mask >> i & 1) ? 0.0 : v;
  }
  __device__ __forceinline__ static double left_s(const double* s, int x, int k) {
    return s[x < 6 ? x * 12 + 6 + k : GEN_E2 + x * 12 + k];
  }
  __device__ __forceinline__ static double base_s(const double* s, int x, int q) {
    const int o = (x < 6 ? 0 : GEN_E2) + (q == 0 ? GP_F + x : x * 12 + q - 1);
    return s[q != 0 && (x < 6) != (q < 7) ? GEN_ZERO : o];
  }
  __device__ __forceinline__ void keep(int x, double v) const { chain_at(c.mz, c.merge_soa, CHAIN_GEN_KEEP, t, x) = v; }
  __device__ __forceinline__ void out(int x, int q, double v) const {
    chain_at(c.part, c.part_soa, CHAIN_GEN_PART, m.out, q == 0 ? GP_F + x : x * 12 + q - 1) = v;
  }
  __device__ void fail() const { b.state[m.structure].info_fail = 1; }
};

// An item per thread: Z = D^-1 R a column at a time into shared memory, then the
// new part a row at a time, so that every coupling entry is loaded once.
constexpr int GEN_SMEM = 78 * CT * (int)sizeof(double);
template <typename Item> __global__ void __launch_bounds__(CT) k_gen(Batch b, ChainParts c, int lo, int hi) {
  extern __shared__ double gen_z[];
  double* z = gen_z + threadIdx.x;  // [row * 13 + column][thread]
  const int t = lo + blockIdx.x * CT + threadIdx.x;
  if (t >= hi) return;
  Item I{b, c};
  I.init(t);
  if (!I.active()) return;
  {
    double D[36];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < 6; ++j) D[i * 6 + j] = I.d(i, j);
    double inv[6], mult[36];
    if (!gj6_factor(D, inv, mult)) I.fail();
#pragma unroll 1
    for (int q = 0; q < 13; ++q) {
      double r[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) r[i] = I.r(i, q);
      gj6_apply(inv, mult, r);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        z[(i * 13 + q) * CT] = r[i];
        I.keep(i * 13 + q, r[i]);
      }
    }
  }
#pragma unroll 1
  for (int x = 0; x < 12; ++x) {
    double left[6], acc[13];
#pragma unroll
    for (int k = 0; k < 6; ++k) left[k] = I.left(x, k);
#pragma unroll
    for (int q = 0; q < 13; ++q) acc[q] = I.base(x, q);
#pragma unroll
    for (int q = 0; q < 13; ++q) {
#pragma unroll
      for (int k = 0; k < 6; ++k) acc[q] = fma(-left[k], z[(k * 13 + q) * CT], acc[q]);
      I.out(x, q, acc[q]);
    }
  }
}

// An item per warp: its operands go to shared memory in one round of loads (read
// entry by entry under the conditions of each column they took a memory round
// trip per condition), lane q < 19 holds column q of [D | R], the pivot column is
// broadcast by shuffle; then the lanes share the entries of the new part.
template <typename Item> __device__ __forceinline__ bool gen_item(const Item& I, int lane, double* st, double (*zs)[13]) {
  I.stage(lane, st);
  if (!I.active()) return true;
  double col[6];
  {
    int a, sa, o, so;
    I.column(lane, a, sa, o, so);
#pragma unroll
    for (int i = 0; i < 6; ++i) col[i] = I.pinned(i, lane, st[a + i * sa] + st[o + i * so]);
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double p = __shfl_sync(0xffffffffu, col[k], k);
    ok = ok && !bad_pivot(p);
    const double inv = rcp64(p);
    double m[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) m[i] = __shfl_sync(0xffffffffu, col[i], k);
    if (lane > k && lane < NC) {
      const double rk = col[k] * inv;
      col[k] = rk;
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (i != k) col[i] = fma(-m[i], rk, col[i]);
    }
  }
  if (lane >= 6 && lane < NC)
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      zs[i][lane - 6] = col[i];
      I.keep(i * 13 + lane - 6, col[i]);
    }
  __syncwarp();
#pragma unroll 1
  for (int o = lane; o < 156; o += 32) {
    const int x = o / 13, q = o % 13;
    double acc = I.base_s(st, x, q);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc = fma(-I.left_s(st, x, k), zs[k][q], acc);
    I.out(x, q, acc);
  }
  __syncwarp();
  return ok;
}
template <typename Item> __global__ void __launch_bounds__(128) k_gen_w(Batch b, ChainParts c, int lo, int hi) {
  __shared__ double zs[4][6][13], stage[4][GEN_STAGE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lo + blockIdx.x * 4 + warp;
  if (t >= hi) return;
  Item I{b, c};
  I.init(t);
  const bool ok = gen_item(I, lane, stage[warp], zs[warp]);
  if (!ok && lane == 0) I.fail();
}

struct GenRoot {
  const double* part;
  __device__ __forceinline__ double k(int i, int j) const { return part[i * 12 + j]; }
  __device__ __forceinline__ double f(int i) const { return part[GP_F + i]; }
  __device__ __forceinline__ static bool minus(int, int) { return false; }
};

// Back substitution x = Z_0 - Z_p x_p - Z_n x_n, row i.
template <typename Kept>
__device__ __forceinline__ double gen_back(const double* xps, const double* xns, int i, Kept kept) {
  double z[13], xp[6], xn[6];
#pragma unroll
  for (int j = 0; j < 13; ++j) z[j] = kept(i * 13 + j);
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    xp[j] = xps[j];
    xn[j] = xns[j];
  }
  double x = z[0];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    x = fma(-z[1 + j], xp[j], x);
    x = fma(-z[7 + j], xn[j], x);
  }
  return x;
}
__device__ __forceinline__ void gen_corner(const Batch& b, const ChainParts& c, int t, const ChainMerge& m, int i) {
  const double x = gen_back(c.x + 6 * (int64_t)m.p, c.x + 6 * (int64_t)m.n, i, [&](int q) { return chain_at(c.mz, c.merge_soa, CHAIN_GEN_KEEP, t, q); });
  c.x[6 * (int64_t)(m.k) + i] = x;
  if (m.mask >> i & 1) b.P[m.dof + __popc(m.mask & ((1 << i) - 1))] = x;
}
// Corners of one level: a row per lane, six lanes per item, five items per warp.
__global__ void k_gen_back(Batch b, ChainParts c, int lo, int hi) {
  const int lane = threadIdx.x & 31;
  const int t = lo + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 5 + lane / 6;
  if (lane >= 30 || t >= hi) return;
  const ChainMerge m = c.merge[t];
  if (solving(b, m.structure)) gen_corner(b, c, t, m, lane % 6);
}
__global__ void k_gen_mid(Batch b, ChainParts c) {
  const int lane = threadIdx.x & 31, i = lane % 6;
  const int t = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 5 + lane / 6;
  if (lane >= 30 || t >= c.n_elem || !solving(b, c.elem_struct[t])) return;
  const int p = c.elem_corner[t];
  b.P[c.elem_dof[t] + i] = gen_back(c.x + 6 * (int64_t)p, c.x + 6 * (int64_t)(p + 1), i, [&](int q) { return chain_at(c.ez, c.elem_soa, CHAIN_GEN_KEEP, t, q); });
}

// The last levels of a chain, its root and their back substitution in one CTA, a
// merge per warp, as k_sym_top.
struct GenTopShared {
  ChainTopShared t;
  double nk[TOP_MERGES][9];  // load stiffness of the corners
  double part[TOP_MERGES][CHAIN_GEN_PART];
  double kept[TOP_MERGES][CHAIN_GEN_KEEP];
  double zs[TOP_THREADS / 32][6][13], stage[TOP_THREADS / 32][GEN_STAGE];
};
struct GenTopMerge {
  const ChainParts& c;
  GenTopShared& S;
  int t;
  __device__ __forceinline__ static bool active() { return true; }
  __device__ __forceinline__ void stage(int lane, double* s) const {
    double v[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      const int y = lane + 32 * (q % 5), o = q < 5 ? S.t.part1[t] : S.t.part2[t], e = q < 5 ? S.t.m[t].e1 : S.t.m[t].e2;
      v[q] = y >= CHAIN_GEN_PART ? 0.0 : o >= 0 ? S.part[o][y] : chain_at(c.part, c.part_soa, CHAIN_GEN_PART, e, y);
    }
#pragma unroll
    for (int q = 0; q < 10; ++q)
      if (lane + 32 * (q % 5) < CHAIN_GEN_PART) s[(q < 5 ? 0 : GEN_E2) + lane + 32 * (q % 5)] = v[q];
    if (lane == 31) s[GEN_ZERO] = 0.0;
    __syncwarp();
    if (lane < 15)
      s[lane < 9 ? (9 + lane / 3) * 12 + 9 + lane % 3 : GP_F + 6 + lane - 9] += lane < 9 ? S.nk[t][lane] : S.t.f[t][lane - 9];
    __syncwarp();
  }
  __device__ __forceinline__ static void column(int lane, int& a, int& sa, int& o, int& so) { GenMerge::column(lane, a, sa, o, so); }
  __device__ __forceinline__ double pinned(int i, int lane, double v) const { return GenMerge::pinned(S.t.m[t].mask, i, lane, v); }
  __device__ __forceinline__ static double left_s(const double* s, int x, int k) { return GenMerge::left_s(s, x, k); }
  __device__ __forceinline__ static double base_s(const double* s, int x, int q) { return GenMerge::base_s(s, x, q); }
  __device__ __forceinline__ void keep(int x, double v) const { S.kept[t][x] = v; }
  __device__ __forceinline__ void out(int x, int q, double v) const { S.part[t][q == 0 ? GP_F + x : x * 12 + q - 1] = v; }
};
__global__ void __launch_bounds__(TOP_THREADS) k_gen_top(Batch b, ChainParts c) {
  extern __shared__ __align__(16) unsigned char gen_top_raw[];
  GenTopShared& S = *reinterpret_cast<GenTopShared*>(gen_top_raw);
  const ChainTop ch = c.chain[blockIdx.x];
  if (!solving(b, ch.structure)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = ch.n_top - 1;
  top_load(b, c, ch, tid, S.t);
  for (int y = tid; y < 9 * n; y += TOP_THREADS)
    S.nk[y / 9][y % 9] = b.nodeK[(int64_t)c.corner_node[S.t.m[y / 9].k] * 9 + y % 9];
  __syncthreads();
  int t0 = 0;
  for (int k = ch.n_top; k > 1; t0 += k / 2, k = (k + 1) / 2) {
    for (int w = warp; w < k / 2; w += TOP_THREADS / 32) {
      const GenTopMerge I{c, S, t0 + w};
      const bool ok = gen_item(I, lane, S.stage[warp], S.zs[warp]);
      if (!ok && lane == 0) b.state[ch.structure].info_fail = 1;
    }
    __syncthreads();
  }
  if (warp == 0) {
    if (n == 0) {
      for (int x = lane; x < CHAIN_GEN_PART; x += 32)
        S.part[0][x] = chain_at(c.part, c.part_soa, CHAIN_GEN_PART, ch.root, x);
      __syncwarp();
    }
    chain_root(b, c, ch, lane, GenRoot{S.part[max(n - 1, 0)]}, S.t.x[TOP_FIRST]);
  }
  __syncthreads();
  int cnt[6], nl = 0;
  for (int k = ch.n_top; k > 1; k = (k + 1) / 2) cnt[nl++] = k / 2;
  for (int l = nl - 1; l >= 0; --l) {
    t0 -= cnt[l];
    const int i = lane % 6, q = warp * 5 + lane / 6;
    if (lane < 30 && q < cnt[l]) {
      const int t = t0 + q;
      const ChainMerge& m = S.t.m[t];
      const double x = gen_back(S.t.x[S.t.p[t]], S.t.x[S.t.n[t]], i, [&](int y) { return S.kept[t][y]; });
      S.t.x[t][i] = x;
      c.x[6 * (int64_t)m.k + i] = x;
      if (m.mask >> i & 1) b.P[m.dof + __popc(m.mask & ((1 << i) - 1))] = x;
    }
    __syncthreads();
  }
}

dim3 grid_for(int n, int per) { return dim3((n + per - 1) / per); }

}  // namespace

void launch_gen_chains(const Batch& b, const ChainParts& c, cudaStream_t st) {
  if (c.n_elem == 0) return;
  if (c.elem_soa) k_gen<GenCondense><<<grid_for(c.n_elem, CT), CT, GEN_SMEM, st>>>(b, c, 0, c.n_elem);
  else k_gen_w<GenCondense><<<grid_for(c.n_elem, 4), 128, 0, st>>>(b, c, 0, c.n_elem);
  for (int l = 0; l < c.n_levels; ++l) {
    const int lo = c.merge_off[l], hi = c.merge_off[l + 1];
    if (hi <= c.merge_soa) k_gen<GenMerge><<<grid_for(hi - lo, CT), CT, GEN_SMEM, st>>>(b, c, lo, hi);
    else k_gen_w<GenMerge><<<grid_for(hi - lo, 4), 128, 0, st>>>(b, c, lo, hi);
  }
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_gen_top, (int)sizeof(GenTopShared)}});
  k_gen_top<<<c.n_chains, TOP_THREADS, sizeof(GenTopShared), st>>>(b, c);
  for (int l = c.n_levels - 1; l >= 0; --l) {
    const int lo = c.merge_off[l], hi = c.merge_off[l + 1];
    k_gen_back<<<grid_for(hi - lo, 20), 128, 0, st>>>(b, c, lo, hi);
  }
  k_gen_mid<<<grid_for(c.n_elem, 20), 128, 0, st>>>(b, c);
}

}  // namespace gf
