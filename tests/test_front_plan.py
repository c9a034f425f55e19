"""The multifrontal LU's plan on the host (csrc/gf_order.cu, compiled here with a driver):
the limits of what the kernels take."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "giraffe_gb300", "csrc")


@pytest.fixture(scope="module")
def compiled(tmp_path_factory):
    """compile(name, source): an executable of the source with gf_order.cu."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_bf16.h")):
        pytest.skip("no CUDA headers")
    path = tmp_path_factory.mktemp("plan")

    def build(name, source):
        src, exe = path / (name + ".cpp"), path / name
        src.write_text(source)
        subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", include, "-I", CSRC, "-x", "c++",
                        os.path.join(CSRC, "gf_order.cu"), str(src), "-o", str(exe)], check=True)
        return lambda *args, **kw: subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, **kw)

    return build


def test_limits_of_the_kernels(compiled):
    # the substitutions keep a front's vector and the partial sums of 512 rows in 200 KB:
    # 21,502 rows; 2^31 - 1 entries
    run = compiled("limits", r"""
#include <cstdio>
#include <cstdlib>
#include "gf_front.h"
int main(int, char** v) {
  gfh::FrontPlan P;
  P.fronts.resize(2);
  P.fronts[1].f = std::atoi(v[1]);
  P.size = std::atoll(v[2]);
  std::printf("%d\n", (int)gfh::fronts_fit(P));
}
""")
    rows = 200 * 1024 // 8 - 2 - 8 * 512
    for f, size, fit in ((rows, 10 ** 9, 1), (rows + 1, 10 ** 9, 0), (10, 2 ** 31 - 1, 1), (10, 2 ** 31, 0)):
        assert int(run(f, size).stdout) == fit


def test_graph_of_a_csr_pattern(compiled):
    # symmetric and sorted rows take a way of their own: 2,000 patterns of either kind,
    # with repeated and unsorted columns and equal neighbouring rows, against sets
    run = compiled("graph", r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include <set>
#include "gf_front.h"
int main() {
  std::mt19937 r(1);
  int wrong = 0;
  for (int t = 0; t < 2000; ++t) {
    const int n = 1 + r() % 60, kind = r() % 4;
    std::vector<std::vector<int>> R(n);
    for (auto& x : R)
      for (int q = r() % 8; q > 0; --q) x.push_back(r() % n);
    if (kind & 1) {  // symmetric
      const auto S = R;
      for (int i = 0; i < n; ++i)
        for (int u : S[i]) R[u].push_back(i);
    }
    if (kind & 2)  // ascending, now and then without repeats
      for (auto& x : R) {
        std::sort(x.begin(), x.end());
        if (r() % 2) x.erase(std::unique(x.begin(), x.end()), x.end());
      }
    if (r() % 2)
      for (int i = 1; i < n; ++i)
        if (r() % 3 == 0) R[i] = R[i - 1];
    std::vector<int> rp(1, 0), ci, dptr, id(n);
    for (auto& x : R) {
      ci.insert(ci.end(), x.begin(), x.end());
      rp.push_back((int)ci.size());
    }
    gfh::NdGraph g;
    gfh::csr_graph(n, rp.data(), ci.data(), g, dptr);
    bool ok = (int)dptr.size() == g.n + 1 && dptr[0] == 0 && dptr[g.n] == n && (int)g.ptr.size() == g.n + 1;
    std::vector<std::set<int>> A(g.n);
    for (int v = 0; v < g.n; ++v)
      for (int i = dptr[v]; i < dptr[v + 1]; ++i) {
        id[i] = v;
        ok = ok && R[i] == R[dptr[v]] && g.w[v] == dptr[v + 1] - dptr[v];
      }
    for (int i = 0; i < n; ++i)
      for (int u : R[i])
        if (id[u] != id[i]) {
          A[id[i]].insert(id[u]);
          A[id[u]].insert(id[i]);
        }
    for (int v = 0; v < g.n && ok; ++v)
      ok = std::vector<int>(A[v].begin(), A[v].end()) == std::vector<int>(g.adj.begin() + g.ptr[v], g.adj.begin() + g.ptr[v + 1]);
    wrong += !ok;
  }
  std::printf("%d", wrong);
}
""")
    assert run().stdout == "0"


def test_plan_without_threads(compiled):
    # the dissection's threads are a help, not a need: where a thread cannot be made (its
    # stack does not fit the address space allowed) the plan is the same
    run = compiled("threads", r"""
#include <cstdio>
#include "gf_front.h"
int main() {
  const int m = 90, n = m * m;
  gfh::NdGraph g;
  g.n = n;
  g.ptr.push_back(0);
  std::vector<int> dptr(1, 0), dofs(2 * n);
  for (int v = 0; v < n; ++v) {
    if (v >= m) g.adj.push_back(v - m);
    if (v % m) g.adj.push_back(v - 1);
    if (v % m < m - 1) g.adj.push_back(v + 1);
    if (v + m < n) g.adj.push_back(v + m);
    g.ptr.push_back((int)g.adj.size());
    g.w.push_back(2);
    dptr.push_back(2 * v + 2);
    dofs[2 * v] = 2 * v;
    dofs[2 * v + 1] = 2 * v + 1;
  }
  gfh::nd_landmark_fields(g);
  const gfh::FrontPlan P = gfh::plan_fronts(g, dptr, dofs);
  unsigned long long h = 1469598103934665603ull;
  for (int p : P.pos) h = (h ^ (unsigned)p) * 1099511628211ull;
  std::printf("%zu %lld %llu", P.fronts.size(), (long long)P.size, h);
}
""")

    def no_threads():
        import resource

        resource.setrlimit(resource.RLIMIT_STACK, (4 << 30, resource.RLIM_INFINITY))
        resource.setrlimit(resource.RLIMIT_AS, (1 << 30, 1 << 30))

    free, bound = run(), run(preexec_fn=no_threads)
    assert free.returncode == 0 and bound.returncode == 0, bound.stderr
    assert free.stdout == bound.stdout
