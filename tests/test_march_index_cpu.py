"""The packed march keeps a voxel's index in bits 18..31 of one register, above
three 6-bit counts, and loads the voxel of the step that leaves the box before
it looks at the counts.  For every world that mc_packed_world admits, every
index up to one layer before and after the world must come back from that
field, whatever the counts hold (compiled from the library's own header, run on
the CPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <stdio.h>
#include "mc_internal.h"

static int bad(int idx, unsigned counts) {
    const int packed = (int)(((unsigned)idx << 18) + counts);
    return (packed >> 18) != idx;
}

int main() {
    long long worlds = 0, wrong = 0;
    for (int wx = 1; wx <= 40; ++wx)
        for (int wy = 1; wy <= 40; ++wy)
            for (int wz = 1; wz <= 40; ++wz) {
                if (!mc_packed_world(wx, wy, wz)) continue;
                ++worlds;
                int n = 0;
                for (int idx = -wx * wz; idx < wx * wz * (wy + 1); ++idx)
                    n += bad(idx, 0u) | bad(idx, (33u << 12) | (33u << 6) | 33u);
                if (n || wx > 31 || wy > 31 || wz > 31) {
                    if (!wrong) printf("first: %d x %d x %d\n", wx, wy, wz);
                    ++wrong;
                }
            }
    printf("worlds %lld wrong %lld\n", worlds, wrong);
    printf("whole %d %d %d\n", mc_packed_world(16, 16, 16), mc_packed_world(24, 16, 20), mc_packed_world(16, 31, 16));
    return wrong != 0;
}
"""


def test_every_index_the_packed_march_loads_fits_its_field(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "index.cpp", tmp_path / "index"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "mine.cu_b200", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "whole 1 1 1" in out.stdout  # the common small worlds keep the packed march
