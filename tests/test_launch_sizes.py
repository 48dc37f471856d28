"""Grid sizes of the quartet kernels, on the CPU: lists of more items than an
int counts lanes of."""
import os
import re
import subprocess


from conftest import ROOT

CSRC = os.path.join(ROOT, "pyquante_b200", "csrc")

PROGRAM = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include "pqb_types.h"
int main()
{
    using namespace pqb;
    const long long n[] = {0, 1, 16, 17, 1000, 1LL << 28, 274600000LL, 300000000LL, 2147483647LL};
    for (long long m : n) {
        const int nsm = 148;
        printf("%lld %d %d %d\n", m, grid_blocks(m, 128 / kCoopLanes, nsm * 32), grid_blocks(m, 128, nsm * 32),
               grid_blocks(m, 1, 2147483647));
    }
}
"""


def test_grids_of_very_long_lists(tmp_path):
    src = tmp_path / "grids.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "grids"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)],
                   check=True)
    for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]:
        m, shared, threads, whole = (int(x) for x in line.split())
        assert shared == min(-(-m // 16), 148 * 32) and threads == min(-(-m // 128), 148 * 32) and whole == m


def test_the_quartet_launches_use_it():
    for name in ("eri_engine.cuh", "eri_grad.cu"):
        src = open(os.path.join(CSRC, name)).read()
        assert "grid_blocks(" in src
        assert not re.search(r"\bint grid = \(", src), "%s: a grid in 32-bit arithmetic" % name
