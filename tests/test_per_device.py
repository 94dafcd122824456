"""The guard of settings that hold on one device (per_device.hpp), compiled for
the host with a counted setting in the place of the CUDA call: each device gets
its own, a failure is tried again, threads may call at once.  CPU only."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lithoinv3d_b200", "csrc")

PROGRAM = r"""
#include "per_device.hpp"
#include <cstdio>
#include <thread>
#include <vector>
using litho_b200::PerDevice;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
enum status { OK = 0, BAD = 3 };
int main() {
    PerDevice a, b;
    int calls[70] = {0};
    auto set = [&](PerDevice& p, int dev, status s = OK) { return p.once(dev, [&] { ++calls[dev]; return s; }); };
    CHECK(set(a, 1) == OK && set(a, 1) == OK && calls[1] == 1);
    CHECK(set(a, 0) == OK && calls[0] == 1);                      // another device: set there too
    CHECK(set(a, 63) == OK && set(a, 63) == OK && calls[63] == 1);
    CHECK(set(b, 1) == OK && calls[1] == 2);                      // another kernel
    CHECK(set(a, 5, BAD) == BAD && set(a, 5) == OK && set(a, 5, BAD) == OK && calls[5] == 2);
    CHECK(set(a, 64) == OK && set(a, 64) == OK && calls[64] == 2);  // beyond the mask: each time
    PerDevice shared;
    std::atomic<int> n{0};
    std::vector<std::thread> t;
    for (int i = 0; i < 8; ++i) t.emplace_back([&, i] { shared.once(i % 4, [&] { ++n; return OK; }); });
    for (auto& x : t) x.join();
    CHECK(n >= 4 && n <= 8);
    int again = 0;
    for (int i = 0; i < 4; ++i) shared.once(i, [&] { ++again; return OK; });
    CHECK(again == 0);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_no_launcher_keeps_a_guard_of_its_own():
    """A process-wide flag beside cudaFuncSetAttribute leaves every device but
    the first without the setting."""
    for name in ("mlp.cu", "capi.cu", "noalloc.cu"):
        text = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"static\s+(const\s+)?(bool|cudaError_t)\s+\w+\s*=", text), name
