"""A kernel's shared-memory limit is set once on every device that a process
opens (csrc/dk_smem_limit.h, compiled for the host)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "denrimrendererkit_gb300", "csrc")

SOURCE = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "dk_smem_limit.h"
int main() {
    dk::SmemLimit limit, other;
    std::vector<int> calls;
    auto raise = [&](dk::SmemLimit& l, int device, int result) {
        return l.raise(device, [&] { calls.push_back(device); return result; });
    };
    if (raise(limit, 0, 0) || raise(limit, 0, 0) || raise(limit, 1, 0) || raise(limit, 0, 0) || raise(limit, 1, 0)) return 1;
    if (calls != std::vector<int>{0, 1}) return 2;                       // once on each
    if (raise(limit, 2, 7) != 7 || raise(limit, 2, 0) != 0 || raise(limit, 2, 7) != 0) return 3;  // a failure is not kept
    if (raise(other, 0, 0) || calls.back() != 0 || calls.size() != 5u) return 4;  // each kernel has its own
    if (raise(limit, 200, 0) || raise(limit, 200, 0) || calls.size() != 7u) return 5;  // beyond the table: every time
    if (raise(limit, -1, 3) != 3) return 6;
    std::atomic<int> set{0};
    dk::SmemLimit shared;
    std::vector<std::thread> threads;
    for (int k = 0; k < 8; ++k)
        threads.emplace_back([&, k] { for (int i = 0; i < 1000; ++i) shared.raise(k % 4, [&] { ++set; return 0; }); });
    for (auto& t : threads) t.join();
    if (set.load() < 4 || set.load() > 8) return 7;
    std::puts("ok");
}
"""


def test_once_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "limit.cpp").write_text(SOURCE)
    exe = tmp_path / "limit"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(tmp_path / "limit.cpp"), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"
