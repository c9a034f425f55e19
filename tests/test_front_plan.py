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
