// Symmetric elimination of Beam_1 chains: Static steps, whose K_AA is symmetric
// and whose elements do not resist a common translation.
//
// The elements (and, as the elimination goes on, runs of elements) of such a
// chain are "parts" between two corner nodes p and n: a symmetric 9x9 stiffness
// over (du = u_n - u_p, a_p, a_n) and the forces they leave on the two nodes.
//   condensation  a midside node, written u_1 = (u_p + u_n) / 2 + v, couples to
//                 du, a_p, a_n: 6 unknowns against 9 columns
//   merge         two parts p-k-n become one: with u_k = u_p + w the unknowns
//                 (w, a_k) couple to du = u_n - u_p, a_p, a_n
//   root          the last part of a chain with its end conditions (12 unknowns,
//                 Gauss-Jordan: an end moment's stiffness is not symmetric)
//   back          corners merge by merge, then the midside nodes
// Merging pairs of parts level by level takes ceil(log2 m) levels.  Against a
// cyclic reduction on 6x6 blocks with 12 coupling columns this halves the
// coupling products (54 against 90 dot products of six per elimination by LDL^T,
// 234 by Gauss-Jordan) and needs no separate update of the surviving corners:
// about 700 FP64 operations per eliminated node against 1,100 and 1,520, in
// kernels that FP64 throughput bounds.
//
// Two forms with the same operations on every entry, so the same bits: one item
// per thread for the large levels and one per half warp for the small ones,
// where an item's chain of dependent operations (64 cycles each on this part)
// is what counts.
#include <cuda_runtime.h>

#include "gf_beam_gp.cuh"
#include "gf_chain.cuh"
#include "gf_chain_root.cuh"
#include "gf_kernels.cuh"
#include "gf_math.cuh"

namespace gf {

namespace {

constexpr int CT = 64;

__device__ __forceinline__ constexpr int lo6(int i, int j) { return i * (i + 1) / 2 + j; }

// Part: lower triangle over (du 0-2, a_p 3-5, a_n 6-8), then the forces on p and
// n (translation, rotation each).
constexpr int PT_HP = 45, PT_HN = 51;
static_assert(PT_HN + 6 == CHAIN_SYM_PART, "a part's entries");
// Kept of an elimination: W = L^-1 R ([row * 10 + column]), the entries of L E below
// the diagonal, the reciprocals of E.
constexpr int KP_M = 60, KP_R = 75;
static_assert(KP_R + 6 == CHAIN_SYM_KEEP, "an elimination's kept entries");
// The half-warp form's staging area (doubles): two parts or K_e's triangle, zeros,
// the forces of a midside node.
constexpr int SYM_E2 = CHAIN_SYM_PART, SYM_ZERO = 120, SYM_F = 128, SYM_STAGE = 134;
// Outputs: the 45 entries of the new stiffness, then the 9 forces h over (du,
// a_p, a_n).
constexpr int N_OUT = 54;

// Columns (0: right-hand side, 1-9: du, a_p, a_n) of output o.
__device__ __forceinline__ void out_pair(int o, int& p, int& q) {
  if (o >= 45) {
    p = 0;
    q = o - 44;
    return;
  }
  // row of the triangle: exact for o < 45, whose roots are at least 1/18 apart
  const int i = (int)((sqrtf(8.0f * (float)o + 1.5f) - 1.0f) * 0.5f);
  p = 1 + o - i * (i + 1) / 2;
  q = 1 + i;
}

// One elimination of six unknowns: D = L E L^T (d(i, j), j <= i), W = L^-1 R (r(i,
// q), ten columns), V = E^-1 W, and the outputs base(o) - W_p^T V_q.  L E stays
// unscaled: W_i -= (L E)_ik V_k.
template <typename Item> __device__ __forceinline__ bool eliminate(const Item& I) {
  double D[21], r[6];
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) D[lo6(i, j)] = I.d(i, j);
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double p = D[lo6(k, k)];
    ok = ok && !bad_pivot(p);
    r[k] = rcp64(p);
    I.keep(KP_R + k, r[k]);
#pragma unroll
    for (int j = k + 1; j < 6; ++j) {
      const double t = rmul(r[k], D[lo6(j, k)]);
      I.keep(KP_M + lo6(j - 1, k), D[lo6(j, k)]);
#pragma unroll
      for (int i = j; i < 6; ++i) D[lo6(i, j)] = rfma(-D[lo6(i, k)], t, D[lo6(i, j)]);
    }
  }
  double W[10][6];
#pragma unroll
  for (int q = 0; q < 10; ++q) {
    double v[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) W[q][i] = I.r(i, q);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      v[k] = rmul(r[k], W[q][k]);
#pragma unroll
      for (int i = k + 1; i < 6; ++i) W[q][i] = rfma(-D[lo6(i, k)], v[k], W[q][i]);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) I.keep(i * 10 + q, W[q][i]);
    if (q == 0) continue;
#pragma unroll
    for (int p = 0; p <= q; ++p) {
      const int o = p == 0 ? 44 + q : lo6(q - 1, p - 1);
      double acc = I.start(o, p, q);
#pragma unroll
      for (int i = 0; i < 6; ++i) acc = rfma(-W[p][i], v[i], acc);
      I.out(o, acc);
    }
  }
  return ok;
}

// What a lane of the half-warp form reads of an item's staged operands, the same for
// every item: entry i of its column is st[a[i]] plus (minus where neg's bit i is
// set) st[b[i]]; output o[x] & 63 starts from st[o[x] >> 16] and takes columns p, q
// (bits 6-9, 10-13).
template <int LANES> struct SymLane {
  static constexpr int OUTS = (N_OUT + LANES - 1) / LANES;
  int a[6], b[6], o[OUTS];
  unsigned neg;
  bool sum;  // both terms (else the first alone)
  template <typename Item> __device__ __forceinline__ void init(int lane) {
    neg = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) Item::column(i, lane & 15, a[i], b[i], neg, sum);
#pragma unroll
    for (int x = 0; x < OUTS; ++x) {
      const int y = lane + LANES * x;
      int p = 0, q = 1;
      if (y < N_OUT) out_pair(y, p, q);
      o[x] = min(y, N_OUT) | p << 6 | q << 10 | Item::base(min(y, N_OUT - 1), p, q) << 16;
    }
  }
};

// The same by a half warp (lane 0-15; LANES = 16) or by both halves of a warp, which
// then share the outputs (LANES = 32): lane q < 10 holds column q of R, lane 10 + j
// column j of D from row j on; W and V go through shared memory to the lanes that
// form the outputs.  The operands go to shared memory first (st), in one round of
// loads.
template <int LANES, typename Item>
__device__ __forceinline__ bool eliminate_h(const Item& I, const SymLane<LANES>& L, int lane, unsigned lanes, double* st,
                                            double (*ws)[10][6]) {
  const int x = lane & 15, dj = x - 10;
  const bool rhs = dj < 0, writes = lane == x;
  I.stage(lane, lanes, st);
  if (!I.active()) return true;
  double col[6], r[6], v[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    col[i] = st[L.a[i]];
    if (Item::SUMS) {
      double y = st[L.b[i]];
      if (L.neg >> i & 1) y = -y;
      y = radd(col[i], y);
      col[i] = L.sum ? y : L.neg >> i & 1 ? -col[i] : col[i];
    }
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double p = __shfl_sync(lanes, col[k], 10 + k, 16);
    ok = ok && !bad_pivot(p);
    r[k] = rcp64(p);
    double d[6], y = col[k];
#pragma unroll
    for (int i = k + 1; i < 6; ++i) {
      d[i] = __shfl_sync(lanes, col[i], 10 + k, 16);
      if (dj == i) y = d[i];
      if (lane == 15) I.keep(KP_M + lo6(i - 1, k), d[i]);
    }
    v[k] = rmul(r[k], y);
#pragma unroll
    for (int i = k + 1; i < 6; ++i)
      if (rhs || (dj > k && i >= dj)) col[i] = rfma(-d[i], v[k], col[i]);
    if (lane == 15) I.keep(KP_R + k, r[k]);
  }
  if (rhs && writes)
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      ws[0][x][i] = col[i];
      ws[1][x][i] = v[i];
      I.keep(i * 10 + x, col[i]);
    }
  __syncwarp(lanes);
#pragma unroll
  for (int y = 0; y < SymLane<LANES>::OUTS; ++y) {
    const int o = L.o[y] & 63;
    if (o >= N_OUT) break;
    const double *w = ws[0][L.o[y] >> 6 & 15], *u = ws[1][L.o[y] >> 10 & 15];
    double acc = st[L.o[y] >> 16];
#pragma unroll
    for (int i = 0; i < 6; ++i) acc = rfma(-w[i], u[i], acc);
    I.out_s(st, o, acc);
  }
  __syncwarp(lanes);
  return ok;
}

// Condensation of the midside node of part t.  The tangent kernel writes K_e of
// such an element over (du, v, a_0, a_1, a_2), lower triangle (beam_expand_sym).
struct Condense {
  const Batch& b;
  const ChainParts& c;
  int t, s;
  const double *K, *P;
  int64_t ne;
  __device__ __forceinline__ void init(int t_) {
    t = t_;
    const int e = c.elem[t];
    s = c.elem_struct[t];
    K = b.Ke + e;
    P = b.P + c.elem_dof[t];
    ne = b.n_elem;
  }
  __device__ __forceinline__ bool active() const { return solving(b, s); }
  // place of unknown i (v, a_1) and of column q (du, a_0, a_2) among the 15
  __device__ static constexpr int row(int i) { return i < 3 ? 3 + i : 6 + i; }
  __device__ static constexpr int place(int q) { return q < 4 ? q - 1 : q < 7 ? q + 2 : q + 5; }
  __device__ static int tri(int i, int j) { return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i; }
  __device__ __forceinline__ double k15(int i, int j) const { return K[(int64_t)tri(i, j) * ne]; }
  __device__ __forceinline__ double d(int i, int j) const { return k15(row(i), row(j)); }
  __device__ __forceinline__ double force(int i) const { return P[i]; }
  __device__ __forceinline__ double r(int i, int q) const { return q == 0 ? force(i) : k15(row(i), place(q)); }
  __device__ __forceinline__ double start(int o, int p, int q) const { return o >= 45 ? 0.0 : k15(place(q), place(p)); }
  __device__ __forceinline__ void keep(int x, double v) const { chain_at(c.ez, c.elem_soa, CHAIN_SYM_KEEP, t, x) = v; }
  __device__ __forceinline__ void put(int x, double v) const { chain_at(c.part, c.part_soa, CHAIN_SYM_PART, t, x) = v; }
  __device__ __forceinline__ void out(int o, double h) const { out_f(o, h, [&](int i) { return force(i); }); }
  template <typename Force> __device__ __forceinline__ void out_f(int o, double h, Force fo) const {
    if (o < 45) {
      put(o, h);
    } else if (o < 48) {  // half of the midside force to each end, and the pull of du
      const double f = rmul(0.5, fo(o - 45));
      put(PT_HP + o - 45, rsub(f, h));
      put(PT_HN + o - 45, radd(f, h));
    } else if (o < 51) {
      put(PT_HP + 3 + o - 48, h);
    } else {
      put(PT_HN + 3 + o - 51, h);
    }
  }
  // The half-warp form: K_e's triangle at st[0], the midside node's forces at
  // st[SYM_F].
  __device__ __forceinline__ void stage(int lane, unsigned lanes, double* st) const {
    double v[8], f = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = lane + 16 * q < 120 ? K[(int64_t)(lane + 16 * q) * ne] : 0.0;
    if (lane < 6) f = P[lane];
#pragma unroll
    for (int q = 0; q < 8; ++q) st[lane + 16 * q] = v[q];  // st[120 ..]: zeros
    if (lane < 6) st[SYM_F + lane] = f;
    __syncwarp(lanes);
  }
  static constexpr bool SUMS = false;
  __device__ __forceinline__ static void column(int i, int lane, int& a, int& b, unsigned& neg, bool& sum) {
    const int x = row(i), y = lane < 10 ? place(lane) : row(lane - 10);
    a = lane == 0 ? SYM_F + i : tri(x, y);
    b = SYM_ZERO;
    sum = false;
  }
  __device__ __forceinline__ static int base(int o, int p, int q) { return o >= 45 ? SYM_ZERO : tri(place(q), place(p)); }
  __device__ __forceinline__ void out_s(const double* st, int o, double h) const { out_f(o, h, [&](int i) { return st[SYM_F + i]; }); }
  __device__ void fail() const { b.state[s].info_fail = 1; }
};

// Elimination of corner k between parts e1 and e2.
struct Merge {
  const Batch& b;
  const ChainParts& c;
  ChainMerge m;
  int t;
  __device__ __forceinline__ void init(int t_) {
    t = t_;
    m = c.merge[t];
  }
  __device__ __forceinline__ bool active() const { return solving(b, m.structure); }
  __device__ __forceinline__ double E(int e, int i, int j) const {
    return chain_at(c.part, c.part_soa, CHAIN_SYM_PART, e, i >= j ? lo6(i, j) : lo6(j, i));
  }
  __device__ __forceinline__ double d(int i, int j) const {  // j <= i, unknowns (w, a_k)
    if (i < 3) return radd(E(m.e1, i, j), E(m.e2, i, j));
    if (j < 3) return rsub(E(m.e1, 3 + i, j), E(m.e2, i, j));  // a_k: a_n of e1, a_p of e2
    return radd(E(m.e1, 3 + i, 3 + j), E(m.e2, i, j));
  }
  // the corner's own force with what both parts leave on it
  __device__ __forceinline__ double force(int i) const {
    return radd(radd(b.P[m.dof + i], chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e1, PT_HN + i)), chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e2, PT_HP + i));
  }
  __device__ __forceinline__ double r(int i, int q) const {
    if (q == 0) return force(i);
    if (q < 4) return i < 3 ? -E(m.e2, i, q - 1) : E(m.e2, i, q - 1);        // du = u_n - u_p
    if (q < 7) return i < 3 ? E(m.e1, q - 1, i) : E(m.e1, 3 + i, q - 1);     // a_p (place 3 + q - 4)
    return i < 3 ? -E(m.e2, q - 1, i) : E(m.e2, q - 1, i);                   // a_n (place 6 + q - 7)
  }
  __device__ __forceinline__ double start(int o, int p, int q) const {
    if (o >= 45) return 0.0;
    const int i = q - 1, j = p - 1;  // i >= j: places of the new part
    if (i < 3) return E(m.e2, i, j);
    if (i < 6) return j < 3 ? 0.0 : E(m.e1, i, j);
    return j >= 3 && j < 6 ? 0.0 : E(m.e2, i, j);
  }
  __device__ __forceinline__ void keep(int x, double v) const { chain_at(c.mz, c.merge_soa, CHAIN_SYM_KEEP, t, x) = v; }
  __device__ __forceinline__ void put(int x, double v) const { chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.out, x) = v; }
  __device__ __forceinline__ double e1(int x) const { return chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e1, x); }
  __device__ __forceinline__ double e2(int x) const { return chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e2, x); }
  __device__ __forceinline__ void out(int o, double h) const {
    if (o < 45) {
      put(o, h);
    } else if (o < 48) {  // u_k = u_p + w: the corner's force passes to p
      const int i = o - 45;
      put(PT_HP + i, radd(e1(PT_HP + i), rsub(force(i), h)));
      put(PT_HN + i, radd(e2(PT_HN + i), h));
    } else if (o < 51) {
      put(PT_HP + o - 45, radd(e1(PT_HP + o - 45), h));
    } else {
      put(PT_HN + o - 48, radd(e2(PT_HN + o - 48), h));
    }
  }
  // The half-warp form: e1 at st[0], the corner's force added to its force on n,
  // e2 at st[SYM_E2].
  __device__ __forceinline__ void stage(int lane, unsigned lanes, double* st) const {
    double v1[4], v2[4], f = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = lane + 16 * q;
      v1[q] = x < CHAIN_SYM_PART ? chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e1, x) : 0.0;
      v2[q] = x < CHAIN_SYM_PART ? chain_at(c.part, c.part_soa, CHAIN_SYM_PART, m.e2, x) : 0.0;
    }
    if (lane < 6) f = b.P[m.dof + lane];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = lane + 16 * q;
      if (x < CHAIN_SYM_PART) {
        st[x] = v1[q];
        st[SYM_E2 + x] = v2[q];
      }
    }
    if (lane == 15) st[SYM_ZERO] = 0.0;
    __syncwarp(lanes);
    if (lane < 6) st[PT_HN + lane] = radd(f, st[PT_HN + lane]);
    __syncwarp(lanes);
  }
  // Column lane (0: force, 1-3 du, 4-6 a_p, 7-9 a_n, 10 + j: column j of D): e1's
  // entry plus or minus e2's, or one of them.
  static constexpr bool SUMS = true;
  __device__ __forceinline__ static void column(int i, int lane, int& a, int& b, unsigned& neg, bool& sum) {
    const int j = lane - 10, x1 = i < 3 ? i : 3 + i;  // the unknown among e1's places
    const bool d = j >= 0, first = d || lane == 0 || (lane >= 4 && lane < 7);
    const int y1 = d ? (j < 3 ? j : 3 + j) : lane - 1, y2 = d ? j : lane - 1;
    const int p1 = lane == 0 ? PT_HN + i : x1 >= y1 ? lo6(x1, y1) : lo6(y1, x1);
    const int p2 = SYM_E2 + (lane == 0 ? PT_HP + i : i >= y2 ? lo6(i, y2) : lo6(y2, i));
    sum = d || lane == 0;
    a = first ? p1 : p2;
    b = sum ? p2 : SYM_ZERO;
    if (d ? (i >= 3 && j < 3) : (i < 3 && lane > 0 && !first)) neg |= 1u << i;
  }
  __device__ __forceinline__ static int base(int o, int p, int q) {
    const int i = q - 1, j = p - 1;  // i >= j: places of the new part
    const bool none = o >= 45 || (i >= 3 && i < 6 ? j < 3 : i >= 6 && j >= 3 && j < 6);
    return none ? SYM_ZERO : (i >= 3 && i < 6 ? 0 : SYM_E2) + lo6(i, j);
  }
  __device__ __forceinline__ void out_s(const double* st, int o, double h) const {
    out_st(st, o, h, [&](int x, double v) { put(x, v); });
  }
  // out() from the staged parts, the force outputs along one path
  template <typename Put> __device__ __forceinline__ static void out_st(const double* st, int o, double h, Put put) {
    if (o < 45) {
      put(o, h);
      return;
    }
    const int i = o - 45;
    double t = h;
    if (i < 3) t = rsub(radd(st[PT_HN + i], st[SYM_E2 + PT_HP + i]), h);
    put(i < 6 ? PT_HP + i : PT_HN + i - 3, radd(st[i < 6 ? PT_HP + i : SYM_E2 + PT_HN + i - 3], t));
    if (i < 3) put(PT_HN + i, radd(st[SYM_E2 + PT_HN + i], h));
  }
  __device__ void fail() const { b.state[m.structure].info_fail = 1; }
};

template <typename Item> __global__ void __launch_bounds__(CT) k_sym(Batch b, ChainParts c, int lo, int hi) {
  const int t = lo + blockIdx.x * CT + threadIdx.x;
  if (t >= hi) return;
  Item I{b, c};
  I.init(t);
  if (!I.active()) return;
  if (!eliminate(I)) I.fail();
}
template <typename Item> __global__ void __launch_bounds__(128) k_sym_h(Batch b, ChainParts c, int lo, int hi) {
  __shared__ double ws[8][2][10][6], stage[8][SYM_STAGE];
  const int half = threadIdx.x >> 4, lane = threadIdx.x & 15, t = lo + blockIdx.x * 8 + half;
  const unsigned lanes = 0xFFFFu << (threadIdx.x & 16);
  if (t >= hi) return;
  Item I{b, c};
  I.init(t);
  SymLane<16> L;
  L.init<Item>(lane);
  const bool ok = eliminate_h<16>(I, L, lane, lanes, stage[half], ws[half]);
  if (!ok && lane == 0) I.fail();
}

// The last part as a 12x12 matrix: the sign of u_p in du.
struct SymRoot {
  const double* part;
  __device__ __forceinline__ double k(int i, int j) const {
    const int x = i < 6 ? i : i < 9 ? i - 6 : i - 3, y = j < 6 ? j : j < 9 ? j - 6 : j - 3;
    return part[x >= y ? lo6(x, y) : lo6(y, x)];
  }
  __device__ __forceinline__ static bool minus(int i, int j) { return (i < 3) != (j < 3); }
  __device__ __forceinline__ double f(int i) const { return part[PT_HP + i]; }
};

// Back substitution of one elimination: E x = L^-1-reduced right-hand side, i.e.
// y = W_0 - W_du du - W_p a_p - W_n a_n, then x_k = y_k / E_k and y_i -= (L E)_ki x_k
// from the last row up; a row per lane, six lanes from l0 on.  Returns row i.
template <typename Kept>
__device__ __forceinline__ double back(unsigned lanes, int l0, int i, const double (&z)[9], Kept kept) {
  double w[10], le[6];
#pragma unroll
  for (int j = 0; j < 10; ++j) w[j] = kept(i * 10 + j);
#pragma unroll
  for (int k = 1; k < 6; ++k) le[k] = i < k ? kept(KP_M + lo6(k - 1, i)) : 0.0;
  const double r = kept(KP_R + i);
  double y = w[0];
#pragma unroll
  for (int j = 0; j < 9; ++j) y = rfma(-w[1 + j], z[j], y);
#pragma unroll
  for (int k = 5; k > 0; --k) {
    const double xk = __shfl_sync(lanes, rmul(y, r), l0 + k);
    if (i < k) y = rfma(-le[k], xk, y);
  }
  return rmul(y, r);
}
__device__ __forceinline__ void around(const double* xp, const double* xn, double (&z)[9]) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    z[j] = rsub(xn[j], xp[j]);
    z[3 + j] = xp[3 + j];
    z[6 + j] = xn[3 + j];
  }
}
// Corner of merge t, row i.
__device__ __forceinline__ void back_corner(const Batch& b, const ChainParts& c, int t, const ChainMerge& m, unsigned lanes,
                                            int l0, int i) {
  double z[9];
  around(c.x + 6 * (int64_t)m.p, c.x + 6 * (int64_t)m.n, z);
  double x = back(lanes, l0, i, z, [&](int q) { return chain_at(c.mz, c.merge_soa, CHAIN_SYM_KEEP, t, q); });
  if (i < 3) x = radd(x, c.x[6 * (int64_t)(m.p) + i]);  // u_k = u_p + w
  c.x[6 * (int64_t)(m.k) + i] = x;
  b.P[m.dof + i] = x;
}
// Corners of one level, five per warp.
__global__ void k_sym_back(Batch b, ChainParts c, int lo, int hi) {
  const int lane = threadIdx.x & 31, i = lane % 6;
  const int t = lo + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 5 + lane / 6;
  bool on = lane < 30 && t < hi;
  ChainMerge m{};
  if (on) {
    m = c.merge[t];
    on = solving(b, m.structure);
  }
  const unsigned lanes = __ballot_sync(0xffffffffu, on);
  if (on) back_corner(b, c, t, m, lanes, lane - i, i);
}
// Midside nodes.
__global__ void k_sym_mid(Batch b, ChainParts c) {
  const int lane = threadIdx.x & 31, i = lane % 6;
  const int t = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 5 + lane / 6;
  const bool on = lane < 30 && t < c.n_elem && solving(b, c.elem_struct[t]);
  const unsigned lanes = __ballot_sync(0xffffffffu, on);
  if (!on) return;
  const int p = c.elem_corner[t];
  double z[9];
  around(c.x + 6 * (int64_t)p, c.x + 6 * (int64_t)(p + 1), z);
  double x = back(lanes, lane - i, i, z, [&](int q) { return chain_at(c.ez, c.elem_soa, CHAIN_SYM_KEEP, t, q); });
  if (i < 3) x = rfma(0.5, radd(c.x[6 * (int64_t)(p) + i], c.x[6 * (int64_t)(p + 1) + i]), x);
  b.P[c.elem_dof[t] + i] = x;
}

// The same an item per thread, for what the item-per-thread kernels kept
// structure-of-arrays: the loads of a warp are 32 items side by side (six lanes an
// item read five at a time: 270,000 midside nodes 89 us for 45).
template <typename Kept> __device__ __forceinline__ void back_item(const double (&z)[9], double (&x)[6], Kept kept) {
  double y[6], r[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    r[i] = kept(KP_R + i);
    y[i] = kept(i * 10);
#pragma unroll
    for (int j = 0; j < 9; ++j) y[i] = rfma(-kept(i * 10 + 1 + j), z[j], y[i]);
  }
#pragma unroll
  for (int k = 5; k > 0; --k) {
    const double xk = rmul(y[k], r[k]);
#pragma unroll
    for (int i = 0; i < k; ++i) y[i] = rfma(-kept(KP_M + lo6(k - 1, i)), xk, y[i]);
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = rmul(y[i], r[i]);
}
__global__ void __launch_bounds__(128) k_sym_back_t(Batch b, ChainParts c, int lo, int hi) {
  const int t = lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= hi) return;
  const ChainMerge m = c.merge[t];
  if (!solving(b, m.structure)) return;
  const double *xp = c.x + 6 * (int64_t)m.p, *xn = c.x + 6 * (int64_t)m.n;
  double z[9], x[6];
  around(xp, xn, z);
  back_item(z, x, [&](int q) { return c.mz[(int64_t)q * c.merge_soa + t]; });
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    if (i < 3) x[i] = radd(x[i], xp[i]);  // u_k = u_p + w
    c.x[6 * (int64_t)m.k + i] = x[i];
    b.P[m.dof + i] = x[i];
  }
}
__global__ void __launch_bounds__(128) k_sym_mid_t(Batch b, ChainParts c) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= c.n_elem || !solving(b, c.elem_struct[t])) return;
  const double *xp = c.x + 6 * (int64_t)c.elem_corner[t], *xn = xp + 6;
  double z[9], x[6];
  around(xp, xn, z);
  back_item(z, x, [&](int q) { return c.ez[(int64_t)q * c.elem_soa + t]; });
  double* P = b.P + c.elem_dof[t];
#pragma unroll
  for (int i = 0; i < 6; ++i) P[i] = i < 3 ? rfma(0.5, radd(xp[i], xn[i]), x[i]) : x[i];
}

// The last levels of a chain in one CTA, from at most CHAIN_TOP parts on: its
// merges level by level, the root, and their back substitution, the
// parts, kept entries and solutions in shared memory all along.  Bound by the chain
// of dependent FP64 operations: the roll-up's 20 parts take 38 us, 50 when the last
// 10 went through L2 between the levels and the first level had its own launches.
struct SymTopShared {
  ChainTopShared t;
  double part[TOP_MERGES][CHAIN_SYM_PART + 1];
  double kept[TOP_MERGES][CHAIN_SYM_KEEP + 1];
  double ws[TOP_THREADS / 16][2][10][6], stage[TOP_THREADS / 16][SYM_STAGE];
};
struct TopMerge {
  static constexpr bool SUMS = true;
  const ChainParts& c;
  SymTopShared& S;
  int t;
  int width;  // lanes of an item
  __device__ __forceinline__ static bool active() { return true; }
  __device__ __forceinline__ void stage(int lane, unsigned lanes, double* st) const {
    const int o1 = S.t.part1[t], o2 = S.t.part2[t], e1 = S.t.m[t].e1, e2 = S.t.m[t].e2;
    double v1[4], v2[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int y = lane + width * q;
      const bool on = y < CHAIN_SYM_PART;
      v1[q] = !on ? 0.0 : o1 >= 0 ? S.part[o1][y] : chain_at(c.part, c.part_soa, CHAIN_SYM_PART, e1, y);
      v2[q] = !on ? 0.0 : o2 >= 0 ? S.part[o2][y] : chain_at(c.part, c.part_soa, CHAIN_SYM_PART, e2, y);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int y = lane + width * q;
      if (y < CHAIN_SYM_PART) {
        st[y] = v1[q];
        st[SYM_E2 + y] = v2[q];
      }
    }
    if (lane == 15) st[SYM_ZERO] = 0.0;
    __syncwarp(lanes);
    if (lane < 6) st[PT_HN + lane] = radd(S.t.f[t][lane], st[PT_HN + lane]);
    __syncwarp(lanes);
  }
  __device__ __forceinline__ void keep(int x, double v) const { S.kept[t][x] = v; }
  __device__ __forceinline__ void out_s(const double* st, int o, double h) const {
    Merge::out_st(st, o, h, [&](int x, double v) { S.part[t][x] = v; });
  }
};
__global__ void __launch_bounds__(TOP_THREADS) k_sym_top(Batch b, ChainParts c) {
  extern __shared__ __align__(16) unsigned char sym_top_raw[];
  SymTopShared& S = *reinterpret_cast<SymTopShared*>(sym_top_raw);
  const ChainTop ch = c.chain[blockIdx.x];
  if (!solving(b, ch.structure)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = ch.n_top - 1;
  top_load(b, c, ch, tid, S.t);
  int t0 = 0;
  {
    // two items a warp while there are more than sub-partitions, then one
    SymLane<16> L;
    L.init<Merge>(lane & 15);
    const int half = tid >> 4;
    int k = ch.n_top;
    for (; k / 2 > 4; t0 += k / 2, k = (k + 1) / 2) {
      if (half < k / 2) {
        const TopMerge I{c, S, t0 + half, 16};
        const bool ok = eliminate_h<16>(I, L, lane & 15, 0xFFFFu << (tid & 16), S.stage[half], S.ws[half]);
        if (!ok && (lane & 15) == 0) b.state[ch.structure].info_fail = 1;
      }
      __syncthreads();
    }
    SymLane<32> W;
    W.init<Merge>(lane);
    for (; k > 1; t0 += k / 2, k = (k + 1) / 2) {
      if (warp < k / 2) {
        const TopMerge I{c, S, t0 + warp, 32};
        const bool ok = eliminate_h<32>(I, W, lane, 0xffffffffu, S.stage[warp], S.ws[warp]);
        if (!ok && lane == 0) b.state[ch.structure].info_fail = 1;
      }
      __syncthreads();
    }
  }
  if (warp == 0) {
    if (n == 0) {
      for (int x = lane; x < CHAIN_SYM_PART; x += 32)
        S.part[0][x] = chain_at(c.part, c.part_soa, CHAIN_SYM_PART, ch.root, x);
      __syncwarp();
    }
    chain_root(b, c, ch, lane, SymRoot{S.part[max(n - 1, 0)]}, S.t.x[TOP_FIRST]);
  }
  __syncthreads();
  // the levels again from the last: their merges end at t0
  int cnt[6], nl = 0;
  for (int k = ch.n_top; k > 1; k = (k + 1) / 2) cnt[nl++] = k / 2;
  for (int l = nl - 1; l >= 0; --l) {
    t0 -= cnt[l];
    const int i = lane % 6, q = warp * 5 + lane / 6;
    const bool on = lane < 30 && q < cnt[l];
    const unsigned on_lanes = __ballot_sync(0xffffffffu, on);
    if (on) {
      const int t = t0 + q;
      const ChainMerge& m = S.t.m[t];
      double z[9];
      around(S.t.x[S.t.p[t]], S.t.x[S.t.n[t]], z);
      double x = back(on_lanes, lane - i, i, z, [&](int y) { return S.kept[t][y]; });
      if (i < 3) x = radd(x, S.t.x[S.t.p[t]][i]);  // u_k = u_p + w
      S.t.x[t][i] = x;
      c.x[6 * (int64_t)m.k + i] = x;
      b.P[m.dof + i] = x;
    }
    __syncthreads();
  }
}

dim3 grid_for(int n, int per) { return dim3((n + per - 1) / per); }

}  // namespace

void launch_sym_chains(const Batch& b, const ChainParts& c, cudaStream_t st) {
  if (c.n_elem == 0) return;
  if (c.elem_soa) k_sym<Condense><<<grid_for(c.n_elem, CT), CT, 0, st>>>(b, c, 0, c.n_elem);
  else k_sym_h<Condense><<<grid_for(c.n_elem, 8), 128, 0, st>>>(b, c, 0, c.n_elem);
  for (int l = 0; l < c.n_levels; ++l) {
    const int lo = c.merge_off[l], hi = c.merge_off[l + 1];
    if (hi <= c.merge_soa) k_sym<Merge><<<grid_for(hi - lo, CT), CT, 0, st>>>(b, c, lo, hi);
    else k_sym_h<Merge><<<grid_for(hi - lo, 8), 128, 0, st>>>(b, c, lo, hi);
  }
  static DeviceOnce once;
  set_limits(once, {{(const void*)k_sym_top, (int)sizeof(SymTopShared)}});
  k_sym_top<<<c.n_chains, TOP_THREADS, sizeof(SymTopShared), st>>>(b, c);
  for (int l = c.n_levels - 1; l >= 0; --l) {
    const int lo = c.merge_off[l], hi = c.merge_off[l + 1];
    if (hi <= c.merge_soa) k_sym_back_t<<<grid_for(hi - lo, 128), 128, 0, st>>>(b, c, lo, hi);
    else k_sym_back<<<grid_for(hi - lo, 20), 128, 0, st>>>(b, c, lo, hi);
  }
  if (c.elem_soa) k_sym_mid_t<<<grid_for(c.n_elem, 128), 128, 0, st>>>(b, c);
  else k_sym_mid<<<grid_for(c.n_elem, 20), 128, 0, st>>>(b, c);
}

}  // namespace gf
