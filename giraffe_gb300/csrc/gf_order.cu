// Nested-dissection ordering and symbolic factorization for the multifrontal
// LU (gf_front.h): host code.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <exception>
#include <numeric>
#include <system_error>
#include <thread>

#include "gf_front.h"

namespace gfh {

namespace {

// A part of at most this weight (DOFs) is not split further: below it a split
// only adds fronts (a 2-element patch of the six-node mesh weighs 6 to 50).
constexpr int ND_LEAF = 24;

// Runs f on a thread of its own, or at once where one is not wanted or cannot be had;
// join() throws what f threw.
struct Beside {
  std::thread t;
  std::exception_ptr error;
  template <typename F> Beside(bool own, F f) {
    if (own) {
      try {
        t = std::thread([this, f] {
          try {
            f();
          } catch (...) {
            error = std::current_exception();
          }
        });
        return;
      } catch (const std::system_error&) {
      }
    }
    f();
  }
  void join() {
    if (t.joinable()) t.join();
    if (error) std::rethrow_exception(error);
  }
  ~Beside() {
    if (t.joinable()) t.join();
  }
};

struct Dissection {
  const NdGraph& g;
  std::vector<int> perm;            // elimination order
  std::vector<char> start;          // a supernode starts at this place of perm
  std::vector<int> label;           // 2 id + side of the part a vertex is in
  std::atomic<int> next_id{1};

  explicit Dissection(const NdGraph& gr) : g(gr), perm(gr.n), start(gr.n, 0), label(gr.n, 0) {
    std::iota(perm.begin(), perm.end(), 0);
  }
  // labels of other threads' parts are read but never equal the reader's own
  int lab(int v) const { return __atomic_load_n(&label[v], __ATOMIC_RELAXED); }
  void set(int v, int l) { __atomic_store_n(&label[v], l, __ATOMIC_RELAXED); }

  // Splits perm[lo, hi) into [part A | part B | separator] and recurses.
  void split(int lo, int hi, int depth) {
    const int m = hi - lo;
    if (m <= 0) return;
    long long wt = 0;
    for (int i = lo; i < hi; ++i) wt += g.w[perm[i]];
    if (m == 1 || wt <= ND_LEAF) {
      start[lo] = 1;
      return;
    }
    double best = -1.0;
    int bf = -1, bside = 0, bless = 0;
    float bt = 0.f;
    std::vector<float> val(m);
    auto classify = [&](int f, float t, int less, int id) {
      const std::vector<float>& x = g.field[f];
      for (int i = lo; i < hi; ++i) {
        const float v = x[perm[i]];
        set(perm[i], 2 * id + ((less ? v < t : v <= t) ? 0 : 1));
      }
    };
    // weights of the two boundary sets under the current labels
    auto boundary = [&](int id, long long* wb, long long* wp) {
      wb[0] = wb[1] = wp[0] = wp[1] = 0;
      for (int i = lo; i < hi; ++i) {
        const int v = perm[i], l = lab(v), side = l & 1;
        wp[side] += g.w[v];
        for (int k = g.ptr[v]; k < g.ptr[v + 1]; ++k)
          if (lab(g.adj[k]) == (l ^ 1)) {
            wb[side] += g.w[v];
            break;
          }
      }
    };
    for (int f = 0; f < (int)g.field.size(); ++f) {
      // a mesh of weight wt has separators of about 2 sqrt(wt)
      if (f >= g.n_pref && best >= 0.0 && best * best < 9.0 * (double)wt) break;
      const std::vector<float>& x = g.field[f];
      for (int i = 0; i < m; ++i) val[i] = x[perm[lo + i]];
      std::nth_element(val.begin(), val.begin() + m / 2, val.end());
      const float t = val[m / 2];
      int nl = 0, ne = 0;
      for (int i = 0; i < m; ++i) {
        nl += val[i] < t;
        ne += val[i] == t;
      }
      if (ne == m) continue;
      // the level set of t goes to the side that balances the parts
      const int less = std::abs(2 * nl - m) <= std::abs(2 * (nl + ne) - m);
      const int na = less ? nl : nl + ne;
      if (na == 0 || na == m) continue;
      const int id = next_id.fetch_add(1);
      classify(f, t, less, id);
      long long wb[2], wp[2];
      boundary(id, wb, wp);
      for (int side = 0; side < 2; ++side) {
        const double a = (double)wp[side] - wb[side], b = (double)wp[1 - side];
        const double imb = std::abs(a - b) / (double)wt;
        // a smaller separator is worth some imbalance of the parts
        const double cost = (double)wb[side] * (1.0 + 1.5 * imb * imb) + 1e-3 * imb;
        if (best < 0.0 || cost < best) {
          best = cost;
          bf = f;
          bt = t;
          bless = less;
          bside = side;
        }
      }
    }
    const int id = next_id.fetch_add(1);
    if (bf < 0) {
      // no field tells the vertices apart: halves of the present order
      for (int i = lo; i < hi; ++i) set(perm[i], 2 * id + (i - lo < m / 2 ? 0 : 1));
      bside = 0;
    } else {
      classify(bf, bt, bless, id);
    }
    std::vector<int> a, b, s;
    for (int i = lo; i < hi; ++i) {
      const int v = perm[i], l = lab(v), side = l & 1;
      bool cut = false;
      if (side == bside)
        for (int k = g.ptr[v]; k < g.ptr[v + 1] && !cut; ++k) cut = lab(g.adj[k]) == (l ^ 1);
      (cut ? s : side ? b : a).push_back(v);
    }
    if (a.empty() && b.empty()) {  // all of it is separator: one supernode
      start[lo] = 1;
      return;
    }
    std::copy(a.begin(), a.end(), perm.begin() + lo);
    std::copy(b.begin(), b.end(), perm.begin() + lo + a.size());
    std::copy(s.begin(), s.end(), perm.begin() + lo + a.size() + b.size());
    const int ma = lo + (int)a.size(), mb = ma + (int)b.size();
    if (!s.empty()) start[mb] = 1;
    auto first = [this, lo, ma, depth] { split(lo, ma, depth + 1); };
    Beside t(depth < 4 && m > 1000, first);
    split(ma, mb, depth + 1);
    t.join();
  }
};

// Distances from vertex v0 (n where unreachable); returns the last vertex reached.
int bfs(const NdGraph& g, int v0, std::vector<int>& dist, std::vector<int>& queue) {
  std::fill(dist.begin(), dist.end(), g.n);
  queue.clear();
  queue.push_back(v0);
  dist[v0] = 0;
  for (size_t q = 0; q < queue.size(); ++q) {
    const int v = queue[q];
    for (int k = g.ptr[v]; k < g.ptr[v + 1]; ++k)
      if (dist[g.adj[k]] == g.n) {
        dist[g.adj[k]] = dist[v] + 1;
        queue.push_back(g.adj[k]);
      }
  }
  return queue.back();
}

}  // namespace

void nd_landmark_fields(NdGraph& g) {
  if (g.n == 0) return;
  constexpr int L = 4;
  std::vector<int> queue, d[L], far(g.n, INT_MAX), d0(g.n);
  int v = bfs(g, bfs(g, 0, d0, queue), d0, queue);
  for (int l = 0; l < L; ++l) {
    d[l].resize(g.n);
    bfs(g, v, d[l], queue);
    // the next landmark: the vertex farthest from all so far, of those of the
    // lowest degree (a corner of the mesh)
    int best = 0;
    for (int i = 0; i < g.n; ++i) {
      far[i] = std::min(far[i], d[l][i]);
      if (far[i] >= g.n) far[i] = -1;  // another component
      const int deg = g.ptr[i + 1] - g.ptr[i], bd = g.ptr[best + 1] - g.ptr[best];
      if (far[i] > far[best] || (far[i] == far[best] && deg < bd)) best = i;
    }
    v = best;
  }
  auto add = [&](auto f) {
    std::vector<float> x(g.n);
    for (int i = 0; i < g.n; ++i) x[i] = f(i);
    g.field.push_back(std::move(x));
  };
  auto sq = [&](int l, int i) { return (float)d[l][i] * (float)d[l][i]; };
  for (int a = 0; a < L; ++a)
    for (int b = a + 1; b < L; ++b) add([&](int i) { return sq(a, i) - sq(b, i); });
  add([&](int i) { return sq(0, i) + sq(1, i) - sq(2, i) - sq(3, i); });
  add([&](int i) { return sq(0, i) + sq(2, i) - sq(1, i) - sq(3, i); });
  add([&](int i) { return sq(0, i) + sq(3, i) - sq(1, i) - sq(2, i); });
}

void csr_graph(int n, const int* rp, const int* ci, NdGraph& g, std::vector<int>& dptr) {
  std::vector<int> id(n);
  for (int i = 0; i < n; ++i) {
    const int len = rp[i + 1] - rp[i];
    const bool same = i > 0 && len == rp[i] - rp[i - 1] && len > 0 &&
                      std::memcmp(ci + rp[i], ci + rp[i - 1], sizeof(int) * (size_t)len) == 0;
    if (!same) dptr.push_back(i);
    id[i] = (int)dptr.size() - 1;
  }
  g.n = (int)dptr.size();
  dptr.push_back(n);
  for (int v = 0; v < g.n; ++v) g.w.push_back(dptr[v + 1] - dptr[v]);
  // Rows in ascending order of a symmetric pattern are the lists already: each column u met
  // while the rows go by has to be the next one of row u's own list.  (A sort of both
  // directions of every edge took 30 ns an entry, most of a call with long rows.)
  g.ptr.assign(1, 0);
  bool plain = true;
  for (int v = 0; v < g.n; ++v) {
    int last = -1;
    for (int k = rp[dptr[v]]; plain && k < rp[dptr[v] + 1]; ++k) {
      const int u = id[ci[k]];
      plain = u >= last;
      if (u != v && u != last) g.adj.push_back(u);
      last = u;
    }
    g.ptr.push_back((int)g.adj.size());
  }
  std::vector<int> at(g.ptr.begin(), g.ptr.end() - 1);
  for (int v = 0; v < g.n && plain; ++v)
    for (int k = g.ptr[v]; k < g.ptr[v + 1] && plain; ++k) {
      const int u = g.adj[k], q = at[u]++;
      plain = q < g.ptr[u + 1] && g.adj[q] == v;
    }
  if (plain) return;
  // any other: both directions of every edge, a list's transpose (which comes out sorted)
  // transposed again and the two merged without repeats
  struct Lists {
    std::vector<int> ptr, to;
  };
  auto transpose = [&](auto each) {
    Lists T;
    T.ptr.assign(g.n + 1, 0);
    each([&](int, int u) { T.ptr[u + 1]++; });
    for (int v = 0; v < g.n; ++v) T.ptr[v + 1] += T.ptr[v];
    T.to.resize(T.ptr[g.n]);
    at.assign(T.ptr.begin(), T.ptr.end() - 1);
    each([&](int v, int u) { T.to[at[u]++] = v; });
    return T;
  };
  const Lists col = transpose([&](auto f) {
    for (int v = 0; v < g.n; ++v) {
      int last = -1;
      for (int k = rp[dptr[v]]; k < rp[dptr[v] + 1]; ++k) {
        const int u = id[ci[k]];
        if (u != v && u != last) f(v, u);
        last = u;
      }
    }
  });
  const Lists row = transpose([&](auto f) {
    for (int v = 0; v < g.n; ++v)
      for (int k = col.ptr[v]; k < col.ptr[v + 1]; ++k)
        if (k == col.ptr[v] || col.to[k] != col.to[k - 1]) f(v, col.to[k]);
  });
  g.ptr.assign(1, 0);
  g.adj.clear();
  for (int v = 0; v < g.n; ++v) {
    int i = row.ptr[v], j = col.ptr[v], last = -1;
    const int i1 = row.ptr[v + 1], j1 = col.ptr[v + 1];
    while (i < i1 || j < j1) {
      const int u = j >= j1 || (i < i1 && row.to[i] <= col.to[j]) ? row.to[i++] : col.to[j++];
      if (u != last) g.adj.push_back(u);
      last = u;
    }
    g.ptr.push_back((int)g.adj.size());
  }
}

FrontPlan plan_fronts(const NdGraph& g, const std::vector<int>& dptr, const std::vector<int>& dofs) {
  FrontPlan P;
  Dissection D(g);
  D.split(0, g.n, 0);
  const std::vector<int>& perm = D.perm;
  std::vector<int> place(g.n), first, node_of(g.n);
  for (int i = 0; i < g.n; ++i) {
    place[perm[i]] = i;
    if (D.start[i]) first.push_back(i);
    node_of[i] = (int)first.size() - 1;
  }
  const int ns = (int)first.size();
  first.push_back(g.n);
  // boundary of every supernode (places of vertices, ascending); its parent
  // holds the first of them
  std::vector<std::vector<int>> bnd(ns), kids(ns);
  std::vector<int> mark(g.n, -1), parent(ns, -1);
  for (int k = 0; k < ns; ++k) {
    const int end = first[k + 1];
    std::vector<int>& B = bnd[k];
    auto take = [&](int p) {
      if (p >= end && mark[p] != k) {
        mark[p] = k;
        B.push_back(p);
      }
    };
    for (int i = first[k]; i < end; ++i)
      for (int q = g.ptr[perm[i]]; q < g.ptr[perm[i] + 1]; ++q) take(place[g.adj[q]]);
    for (int c : kids[k])
      for (int p : bnd[c]) take(p);
    std::sort(B.begin(), B.end());
    if (!B.empty()) {
      parent[k] = node_of[B[0]];
      kids[parent[k]].push_back(k);
    }
  }
  // DOFs: elimination positions by place, then the fronts
  const int nd = (int)dofs.size();
  std::vector<int> dpos(g.n + 1, 0);  // first elimination position of a place
  for (int i = 0; i < g.n; ++i) dpos[i + 1] = dpos[i] + dptr[perm[i] + 1] - dptr[perm[i]];
  P.pos.assign(nd, -1);
  P.dof_front.assign(nd, -1);
  for (int i = 0; i < g.n; ++i)
    for (int q = dptr[perm[i]], p = dpos[i]; q < dptr[perm[i] + 1]; ++q, ++p) P.pos[dofs[q]] = p;
  P.fronts.resize(ns);
  P.height.assign(ns, 0);
  for (int k = 0; k < ns; ++k) {
    gf::Front& F = P.fronts[k];
    F.s = dpos[first[k + 1]] - dpos[first[k]];
    F.dof0 = dpos[first[k]];
    F.bnd = (int)P.bnd.size();
    F.parent = parent[k];
    F.slot = 0;
    for (int p : bnd[k])
      for (int d = dpos[p]; d < dpos[p + 1]; ++d) P.bnd.push_back(d);
    F.f = F.s + (int)P.bnd.size() - F.bnd;
    F.ld = (F.f + 1) & ~1;
    F.off = P.size;
    P.size += ((int64_t)F.ld * (F.f + 1) + 31) / 32 * 32;
    for (int d = F.dof0; d < F.dof0 + F.s; ++d) P.dof_front[d] = k;
    if (F.parent >= 0) P.height[F.parent] = std::max(P.height[F.parent], P.height[k] + 1);
  }
  // front index, in the parent, of every boundary DOF
  P.rel.assign(P.bnd.size(), -1);
  for (int k = 0; k < ns; ++k) {
    gf::Front& F = P.fronts[k];
    F.rel = F.bnd;
    if (F.parent < 0) continue;
    const gf::Front& Q = P.fronts[F.parent];
    const int u = F.f - F.s, qu = Q.f - Q.s;
    for (int i = 0, j = 0; i < u; ++i) {
      const int d = P.bnd[F.bnd + i];
      if (d < Q.dof0 + Q.s) {
        P.rel[F.rel + i] = d - Q.dof0;
      } else {
        while (j < qu && P.bnd[Q.bnd + j] < d) ++j;
        P.rel[F.rel + i] = Q.s + j;
      }
    }
  }
  return P;
}

bool fronts_fit(const FrontPlan& P) {
  int f = 0;
  for (const gf::Front& F : P.fronts) f = std::max(f, F.f);
  return P.size <= INT_MAX && f <= gf::MF_MAX_ROWS;
}

// The largest front of a height that takes one CTA.  One CTA runs at its SM's FP64
// rate (16 cycles a warp instruction) and has no launches between its steps: the
// way for many fronts.  Panel by panel a front spreads over the SMs at about 30 us
// a panel (diagonal block, rows and columns, update): the way for a few, whose one
// CTA each would take longer (a front of 96 with 69 pivots 190 us, panel by panel
// 90).  Both give the same bits.  Estimates in us; W is the elimination's time on
// an SM of its own.
static int small_limit(const std::vector<gf::Front>& fronts, const std::vector<int>& at) {
  static const int lims[] = {gf::MF_SMALL, 88, 80, 72, 64, 48, 32, 0};
  int best = gf::MF_SMALL;
  double best_t = -1.0;
  for (int lim : lims) {
    double one = 0.0, ws = 0.0, wb = 0.0;
    int sb = 0, n_small = 0, n_big = 0;
    for (int k : at) {
      const double f = fronts[k].f, s = fronts[k].s, w = (s * f * f - s * s * f + s * s * s / 3.0) * (0.5 / 1930.0);
      if (fronts[k].f <= lim) {
        one = std::max(one, 1.6 * w + 0.5 * s);
        ws += w;
        ++n_small;
      } else {
        sb = std::max(sb, fronts[k].s);
        wb += w;
        ++n_big;
      }
    }
    double t = 0.0;
    if (n_small) t += 5.0 + std::max(one, 1.4 * ws / 152.0);
    if (n_big) t += 10.0 + 30.0 * ((sb + gf::MF_NB - 1) / gf::MF_NB) + 1.5 * wb / 152.0;
    if (best_t < 0.0 || t < best_t) {
      best_t = t;
      best = lim;
    }
  }
  return best;
}

void join_fronts(const std::vector<const FrontPlan*>& plans, const std::vector<int>& slots,
                 const std::vector<int>& dof_off, int n_struct, int n_dofs, bool tensor, FrontBuild& out) {
  out.pos.assign(n_dofs, -1);
  out.dof_front.assign(n_dofs, -1);
  out.base.assign(n_struct, 0);
  out.size.assign(n_struct, 0);
  std::vector<int> height;
  {
    size_t nf = 0, nb = 0;
    for (const FrontPlan* P : plans) {
      nf += P->fronts.size();
      nb += P->bnd.size();
    }
    out.fronts.reserve(nf);
    height.reserve(nf);
    out.bnd.resize(nb);
    out.rel.reserve(nb);
  }
  int b0 = 0;
  for (size_t q = 0; q < plans.size(); ++q) {
    const FrontPlan& P = *plans[q];
    const int f0 = (int)out.fronts.size(), d0 = dof_off[q];
    out.base[slots[q]] = out.total;
    out.size[slots[q]] = P.size;
    for (gf::Front F : P.fronts) {
      F.off += out.total;
      F.slot = slots[q];
      F.dof0 += d0;
      F.bnd += b0;
      F.rel += b0;
      if (F.parent >= 0) F.parent += f0;
      out.fronts.push_back(F);
    }
    for (size_t i = 0; i < P.bnd.size(); ++i) out.bnd[b0 + i] = P.bnd[i] + d0;
    b0 += (int)P.bnd.size();
    out.rel.insert(out.rel.end(), P.rel.begin(), P.rel.end());
    height.insert(height.end(), P.height.begin(), P.height.end());
    for (size_t i = 0; i < P.pos.size(); ++i) out.pos[d0 + i] = P.pos[i] + d0;
    for (size_t i = 0; i < P.dof_front.size(); ++i) out.dof_front[d0 + i] = P.dof_front[i] + f0;
    out.total += P.size;
  }
  const int nf = (int)out.fronts.size();
  int nl = 0;
  for (int h : height) nl = std::max(nl, h + 1);
  std::vector<std::vector<int>> at(nl);
  auto parent = [&](int k) { return out.fronts[k].f > out.fronts[k].s ? out.fronts[k].parent : -1; };
  size_t n_inv = 0;
  for (int k = 0; k < nf; ++k) {
    at[height[k]].push_back(k);
    out.fronts[k].kid0 = out.fronts[k].kid1 = 0;
  }
  for (int k = 0; k < nf; ++k)
    if (parent(k) >= 0) {
      ++out.fronts[parent(k)].kid1;
      n_inv += out.fronts[parent(k)].f;
    }
  int n_kids = 0;
  for (int k = 0; k < nf; ++k) {
    const int n = out.fronts[k].kid1;
    out.fronts[k].kid0 = out.fronts[k].kid1 = n_kids;
    n_kids += n;
  }
  out.kids.resize(n_kids);
  for (int k = 0; k < nf; ++k)
    if (parent(k) >= 0) out.kids[out.fronts[parent(k)].kid1++].x = k;
  out.inv.assign(n_inv, -1);
  n_inv = 0;
  for (int k = 0; k < nf; ++k)
    for (int q = out.fronts[k].kid0; q < out.fronts[k].kid1; ++q) {
      const gf::Front& C = out.fronts[out.kids[q].x];
      out.kids[q].y = (int)n_inv;
      int* inv = out.inv.data() + n_inv;
      for (int i = 0; i < C.f - C.s; ++i) inv[out.rel[C.rel + i]] = i;
      n_inv += out.fronts[k].f;
    }
  out.dof_at.assign(n_dofs, -1);
  for (int i = 0; i < n_dofs; ++i)
    if (out.pos[i] >= 0) out.dof_at[out.pos[i]] = i;
  out.sched.level.resize(nl);
  out.sched.launches = 3;  // zero, right-hand sides, gather of the solution
  for (int l = 0; l < nl; ++l) {
    gf::FrontLevel& V = out.sched.level[l];
    std::vector<int> small, big;
    const int lim = small_limit(out.fronts, at[l]);
    for (int k : at[l]) (out.fronts[k].f <= lim ? small : big).push_back(k);
    auto larger = [&](int a, int b) {
      const gf::Front &A = out.fronts[a], &B = out.fronts[b];
      return A.s != B.s ? A.s > B.s : a < b;
    };
    std::sort(big.begin(), big.end(), larger);
    std::sort(small.begin(), small.end(), larger);
    for (int k : at[l]) V.max_s = std::max(V.max_s, out.fronts[k].s);
    V.small_off = (int)out.list.size();
    V.n_small = (int)small.size();
    for (int k : small) V.small_f = std::max(V.small_f, out.fronts[k].f);
    for (int k : small) out.list.push_back(out.fronts[k]);
    V.big_off = (int)out.list.size();
    V.n_big = (int)big.size();
    for (int k : big) out.list.push_back(out.fronts[k]);
    V.ext_off = (int)out.ext_jobs.size();
    for (int k : big)
      if (out.fronts[k].kid1 > out.fronts[k].kid0)
        for (int c = 0; c <= out.fronts[k].f; c += 8) out.ext_jobs.push_back(make_int2(k, c));
    V.ext_cnt = (int)out.ext_jobs.size() - V.ext_off;
    const int panels = big.empty() ? 0 : (out.fronts[big[0]].s + gf::MF_NB - 1) / gf::MF_NB;
    for (int p = 0; p < panels; ++p) {
      int n = 0, f = 0, s = 0;
      while (n < V.n_big && out.fronts[big[n]].s > p * gf::MF_NB) {
        f = std::max(f, out.fronts[big[n]].f);
        s = std::max(s, out.fronts[big[n]].s);
        ++n;
      }
      V.n_at.push_back(n);
      V.f_at.push_back(f);
      V.s_at.push_back(s);
    }
    V.schur_off = (int)out.schur_jobs.size();
    // 32 x 32 tiles, or 16 x 16 where their waves are shorter: a tile holds an SM's FP64
    // units for its whole product, four parts of work for the large one and one for the
    // small, which takes 1.3 with its operands' loads for a quarter of the products.  16
    // everywhere: FP32 fronts of the 64x64x2 plate 122.0 -> 123.5 ms (whole waves of either);
    // 32 everywhere: four vibrating plates 18.1 -> 18.7 ms, one 6x6x2 plate 4.02 -> 4.25
    // (a part of one wave); batches of 16 to 128 plates and the FP64 64x64x2 plate
    // within 1 % either way
    auto on_t5 = [&](int k) {
      const double u = out.fronts[k].f - out.fronts[k].s;
      return tensor && out.fronts[k].s * u * u >= gf::MF_T5_WORK;
    };
    auto tiles = [&](int t) {
      int64_t n = 0;
      for (int k : big) {
        if (on_t5(k)) continue;
        const int u = out.fronts[k].f - out.fronts[k].s;
        if (u > 0) n += (int64_t)((u + t) / t) * ((u + t - 1) / t);
      }
      return n;
    };
    if (4 * ((tiles(32) + 151) / 152) * 10 > 13 * ((tiles(16) + 151) / 152)) V.tile = 16;
    auto jobs = [&](int k) {
      const int u = out.fronts[k].f - out.fronts[k].s;
      if (u > 0)
        for (int tj = 0; tj < (u + V.tile) / V.tile; ++tj)
          for (int ti = 0; ti < (u + V.tile - 1) / V.tile; ++ti) out.schur_jobs.push_back(make_int2(k, ti | (tj << 16)));
    };
    for (int k : big) {
      V.big_f = std::max(V.big_f, out.fronts[k].f);
      if (!on_t5(k)) jobs(k);
    }
    V.schur_cnt = (int)out.schur_jobs.size() - V.schur_off;
    for (int k : big)
      if (on_t5(k)) jobs(k);
    V.schur_all = (int)out.schur_jobs.size() - V.schur_off;
    V.t5_off = (int)out.t5.size();
    V.t5_job_off = (int)out.t5_jobs.size();
    int64_t oz = 0, exps = 0, kmax = 0;
    for (int k : big) {
      if (!on_t5(k)) continue;
      const gf::Front& F = out.fronts[k];
      const int u = F.f - F.s, rows = (u + 127) / 128 * 128, id = (int)out.t5.size();
      out.t5.push_back(gf::FrontT5{oz, (int)exps, (int)kmax, rows, k});
      oz += (int64_t)2 * ((F.s + 63) / 64) * 8 * rows * 64;
      exps += (int64_t)2 * ((F.s + 63) / 64) * rows;
      kmax += 2 * F.s;
      V.t5_rows = std::max(V.t5_rows, rows);
      V.t5_s = std::max(V.t5_s, F.s);
      for (int tj = 0; tj < (u + 63) / 64; ++tj)
        for (int ti = 0; ti < (u + 127) / 128; ++ti) out.t5_jobs.push_back(make_int2(id, ti | (tj << 16)));
    }
    out.oz = std::max(out.oz, oz);
    out.oz_exp = std::max(out.oz_exp, exps);
    out.oz_kmax = std::max(out.oz_kmax, kmax);
    V.t5_cnt = (int)out.t5.size() - V.t5_off;
    V.t5_job_cnt = (int)out.t5_jobs.size() - V.t5_job_off;
    out.sched.launches += (V.ext_cnt ? 1 : 0) + (V.n_small ? 1 : 0) + (V.schur_cnt ? 1 : 0) +
                          (V.t5_cnt ? 1 + 2 * gf::front_grids(V.t5_cnt) : 0) + 1;
    for (int p = 0; p < panels; ++p)
      out.sched.launches += (p == 0 ? 1 : 0) + gf::front_grids(V.n_at[p]) * ((V.f_at[p] > p * gf::MF_NB ? 1 : 0) +
                                                                           (V.s_at[p] > (p + 1) * gf::MF_NB ? 1 : 0));
  }
}

}  // namespace gfh
