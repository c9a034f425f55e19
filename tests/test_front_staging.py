"""A standalone system's host data on its way to the device (csrc/gf_front_system.h):
pinned staging up to a bound, pageable copies where it cannot be had or the data are
larger, nothing left of a failed allocation in CUDA's last error.  Host code, compiled
here against a CUDA runtime of memcpy and malloc."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "giraffe_gb300", "csrc")
MAIN = r"""
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "gf_front_system.h"
static size_t pin_limit, pinned_now = 0, pinned_peak = 0;
static cudaError_t last = cudaSuccess;
static double* answer;
static int n_answer;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (n > pin_limit) return last = cudaErrorMemoryAllocation;
  pinned_now = n;
  if (n > pinned_peak) pinned_peak = n;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}
namespace gfh {
bool set_err(gf_ctx*, const char*, ...) { return false; }
}
namespace gf {
void launch_front_lu(const Batch& b, double* x, cudaStream_t) { std::memcpy(x, b.P, sizeof(double) * n_answer); }
void launch_front_refine(const Batch&, int, double*, double*, cudaStream_t) {}
}
// A path of n unknowns; the "solution" is the right-hand side as it reached the device.
int main(int, char** v) {
  const int n = std::atoi(v[1]);
  pin_limit = std::strtoull(v[2], nullptr, 10);
  const size_t extra = std::strtoull(v[3], nullptr, 10);
  n_answer = n;
  gfh::NdGraph g;
  std::vector<int> dptr(1, 0), dofs(n);
  g.n = n;
  g.ptr.push_back(0);
  g.field.resize(1);
  for (int i = 0; i < n; ++i) {
    if (i) g.adj.push_back(i - 1);
    if (i + 1 < n) g.adj.push_back(i + 1);
    g.ptr.push_back((int)g.adj.size());
    g.w.push_back(1);
    g.field[0].push_back((float)i);
    dptr.push_back(i + 1);
    dofs[i] = i;
  }
  const gfh::FrontPlan plan = gfh::plan_fronts(g, dptr, dofs);
  gf_ctx ctx;
  std::vector<double> b(n), x(n, -1.0), data(extra / 8);
  for (int i = 0; i < n; ++i) b[i] = i + 0.5;
  for (size_t i = 0; i < data.size(); ++i) data[i] = 3.0 * (double)i;
  gfh::FrontSystem S;
  std::vector<int> part;
  const int rc = S.init(&ctx, plan, n, b.data(), {{data.data(), data.size() * 8}}, &part);
  bool done = false, same = true;
  int rs = -1;
  if (rc == 0) {
    same = std::memcmp(S.at<double>(part[0]), data.data(), data.size() * 8) == 0;
    rs = S.solve(&ctx, n, [](const gf::Batch&) {}, [](const double*, double*, int*) {}, x.data(), &done);
  }
  std::printf("%d %d %d %d %d %d %d\n", rc, rs, (int)done, (int)same, (int)(std::memcmp(x.data(), b.data(), n * 8) == 0),
              (int)last, (int)(pinned_peak >> 20));
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_bf16.h")):
        pytest.skip("no CUDA headers")
    path = tmp_path_factory.mktemp("staging")
    src, exe = path / "staging.cpp", path / "staging"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", include, "-I", CSRC, "-x", "c++",
                    os.path.join(CSRC, "gf_order.cu"), str(src), "-o", str(exe), "-ldl"], check=True)
    return lambda *a: subprocess.run([str(exe), *map(str, a)], check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("pin_limit,extra,staged", [(1 << 40, 1 << 20, True), (0, 1 << 20, False),
                                                    (1 << 40, 300 << 20, False)])
def test_the_data_arrive_with_and_without_pinned_staging(run, pin_limit, extra, staged):
    rc, rs, done, same, solution, last, pinned = map(int, run(2000, pin_limit, extra))
    assert (rc, rs, done, same, solution, last) == (0, 0, 1, 1, 1, 0)
    assert (pinned > 0) == staged
