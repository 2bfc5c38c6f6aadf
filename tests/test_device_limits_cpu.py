"""A kernel's shared-memory limit is a setting of each device: it is made on every
device that launches the kernel, once, whichever device was first and whatever
the order of sizes (the library's own helper, compiled here with a setter that
counts)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <stdio.h>
#include <thread>
#include <vector>
#include "mc_internal.h"

int main() {
    mc_once_per_device limit;
    int sets[80] = {0};
    auto set = [&](int d) { return limit(d, [&] { ++sets[d]; return 0; }); };
    for (int round = 0; round < 3; ++round)
        for (int d : {0, 1, 7, 63}) if (set(d)) return 1;
    for (int d : {0, 1, 7, 63}) if (sets[d] != 1) return 2;
    if (sets[2]) return 3;
    set(70); set(70);                                // beyond the remembered devices: every time
    if (sets[70] != 2) return 4;
    int tries = 0;                                   // a failure is reported and tried again
    auto fails = [&] { return ++tries < 3 ? 700 : 0; };
    if (limit(5, fails) != 700 || limit(5, fails) != 700 || limit(5, fails) != 0 || limit(5, fails) != 0 || tries != 3)
        return 5;
    mc_once_per_device shared;
    std::atomic<int> done[4] = {};
    std::vector<std::thread> th;
    std::atomic<int> late{0};
    for (int t = 0; t < 8; ++t)
        th.emplace_back([&, t] {
            for (int k = 0; k < 2000; ++k) {
                const int d = (k + t) & 3;
                if (shared(d, [&] { done[d]++; return 0; }) || !done[d]) late++;
            }
        });
    for (auto& t : th) t.join();
    return late ? 6 : 0;
}
"""


def test_a_limit_is_set_once_on_every_device(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "mine.cu_b200", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_launch_remembers_a_limit_for_all_devices():
    """Every limit of a kernel goes through the helper."""
    src = open(os.path.join(ROOT, "mine.cu_b200", "csrc", "mc_backend_impl.cuh")).read()
    assert src.count("cudaFuncSetAttribute(") == 1
    body = src[src.index("static int allow_smem"):]
    assert body.index("limit(dev") < body.index("cudaFuncSetAttribute(") < body.index("\n}\n")
