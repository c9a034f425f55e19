"""rcp64 (csrc/gf_math.cuh), the reciprocal of every pivot of the fronts and chains, on
the device against 1 / p: its third-order step leaves 2^-69 before the one rounding of the
last operation, so half a unit in the last place and 2^-15 of one for exponents 64 to 1982;
outside them the division itself, and bad_pivot names zeros, infinities and NaN."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "giraffe_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include <vector>
#include "gf_math.cuh"
__global__ void k(int n, const double* p, double* r, double* q, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = gf::rcp64(p[i]);
  q[i] = 1.0 / p[i];
  bad[i] = gf::bad_pivot(p[i]);
}
int main(int, char** v) {
  FILE* f = std::fopen(v[1], "rb");
  std::fseek(f, 0, SEEK_END);
  const int n = (int)(std::ftell(f) / 8);
  std::rewind(f);
  std::vector<double> h(n);
  if ((int)std::fread(h.data(), 8, n, f) != n) return 1;
  std::fclose(f);
  double *p, *r, *q;
  int* bad;
  if (cudaMalloc(&p, n * 8) || cudaMalloc(&r, n * 8) || cudaMalloc(&q, n * 8) || cudaMalloc(&bad, n * 4)) return 2;
  cudaMemcpy(p, h.data(), n * 8, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(n, p, r, q, bad);
  std::vector<double> hr(n), hq(n);
  std::vector<int> hb(n);
  cudaMemcpy(hr.data(), r, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(hq.data(), q, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(hb.data(), bad, n * 4, cudaMemcpyDeviceToHost);
  if (cudaGetLastError() != cudaSuccess) return 3;
  f = std::fopen(v[2], "wb");
  std::fwrite(hr.data(), 8, n, f);
  std::fwrite(hq.data(), 8, n, f);
  std::fwrite(hb.data(), 4, n, f);
  std::fclose(f);
}
"""


def test_reciprocal_of_pivots(tmp_path):
    from giraffe_gb300 import build

    (tmp_path / "rcp.cu").write_text(MAIN)
    exe = str(tmp_path / "rcp")
    subprocess.run(["nvcc", *build.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
                    str(tmp_path / "rcp.cu"), "-o", exe], check=True)
    rng = np.random.default_rng(0)
    ex = np.arange(0, 2048, dtype=np.uint64)[:, None]
    frac = np.concatenate([[0, 1, 2, 2 ** 29 - 1, 2 ** 29, 2 ** 51, 2 ** 52 - 2, 2 ** 52 - 1],
                           rng.integers(0, 2 ** 52, 56)]).astype(np.uint64)[None]
    bits = ((ex << np.uint64(52)) | frac).ravel()
    bits = np.concatenate([bits, bits | np.uint64(2 ** 63)])
    p = bits.view(np.float64)
    p.tofile(tmp_path / "in")
    subprocess.run([exe, str(tmp_path / "in"), str(tmp_path / "out")], check=True)
    raw = np.fromfile(tmp_path / "out", dtype=np.uint8)
    n = len(p)
    r, q, bad = raw[:8 * n].view(np.float64), raw[8 * n:16 * n].view(np.float64), raw[16 * n:].view(np.int32)
    assert np.array_equal(bad != 0, ~np.isfinite(p) | (p == 0))
    e = (bits >> np.uint64(52)) & np.uint64(2047)
    own = (e >= 64) & (e <= 1982)
    assert np.array_equal(r[~own].view(np.uint64)[p[~own] == p[~own]], q[~own].view(np.uint64)[p[~own] == p[~own]])
    x = r[own].astype(np.longdouble)
    # (1/p - r) in units of r's last place, from the residual 1 - p r with the longer
    # significand; that of 64 bits leaves 2^-11 of a unit
    err = np.abs((1 - p[own].astype(np.longdouble) * x) / p[own]) / np.spacing(np.abs(r[own]))
    slack = 2.0 ** -15 + (2.0 ** -10 if np.finfo(np.longdouble).nmant < 100 else 0.0)
    assert float(err.max()) <= 0.5 + slack
