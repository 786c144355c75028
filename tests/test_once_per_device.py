"""What has to be set once for each device of a process (csrc/once_per_device.h), compiled with the host compiler: a second device of the
same process gets its own, a failure is tried again, threads that come together agree.  And all kernels are set by that one place."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dragon-alpha-v1.0_b200", "csrc")

PROGRAM = r"""
#include "once_per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main()
{
    alpha::OncePerDevice once;
    int runs[alpha::kMaxDevices + 1] = {}, bad = 0;
    auto set = [&](int d, int rc) { return once(d, [&] { ++runs[d]; return rc; }); };
    for (int again = 0; again < 3; ++again)
        for (int d = 0; d < alpha::kMaxDevices; ++d) {
            if (d == 5) continue;
            bad += set(d, 0) != 0 || runs[d] != 1;
        }
    bad += set(5, 1) != 1 || set(5, 7) != 7 || set(5, 0) != 0 || set(5, 1) != 0 || runs[5] != 3;
    bad += set(alpha::kMaxDevices, 0) != 0 || runs[alpha::kMaxDevices] != 1;
    alpha::OncePerDevice shared;
    std::atomic<int> count{0}, wrong{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            for (int d = 0; d < alpha::kMaxDevices; ++d) {
                std::atomic<int> done{0};
                if (shared(d, [&] { ++count; done = 1; return 0; }) != 0) ++wrong;
            }
        });
    for (auto& t : threads) t.join();
    bad += wrong.load() != 0 || count.load() < alpha::kMaxDevices || count.load() > 8 * alpha::kMaxDevices;
    printf("%d bad\n", bad);
    return bad != 0;
}
"""


def test_every_device_is_set_once(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "once.cpp", str(tmp_path / "once")
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", "-I", CSRC, "-o", exe, str(src)], check=True, capture_output=True, timeout=120)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout


def test_one_place_sets_the_shared_memory_of_kernels():
    found = {}
    for name in os.listdir(CSRC):
        text = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"static bool \w*(done|set)\b", text), name
        if "cudaFuncSetAttribute" in text:
            found[name] = text.count("cudaFuncSetAttribute")
    assert found == {"dependent_launch.cuh": 1}, found
