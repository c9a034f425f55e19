"""Kernel limits are set once per device (csrc/gf_device_once.h): for each of two devices
that one process uses, again after a failure, and for an ordinal beyond the kept ones at
every call.  Host code, compiled here against a count in place of the CUDA call."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "giraffe_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include "gf_device_once.h"
int main() {
  gf::DeviceOnce once;
  int calls[2] = {0, 0}, beyond = 0, failing = 0;
  for (int k = 0; k < 3; ++k)
    for (int d = 0; d < 2; ++d) once(d, [&] { ++calls[d]; return true; });
  for (int k = 0; k < 2; ++k) once(1000, [&] { ++beyond; return true; });
  for (int k = 0; k < 4; ++k) once(7, [&] { return ++failing == 3; });
  std::printf("%d %d %d %d\n", calls[0], calls[1], beyond, failing);
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "2", "3"]


def test_no_limit_is_set_outside_it():
    # the one place that sets a kernel's attribute is the helper that goes through it
    where = [f for f in sorted(os.listdir(CSRC)) if "cudaFuncSetAttribute(" in open(os.path.join(CSRC, f)).read()]
    assert where == ["gf_kernels.cuh"]
