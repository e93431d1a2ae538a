"""Shared-memory limits of the kernels are raised once per device, also when several threads launch first, and a refusal is reported and
asked for again.  The helper is compiled for the host against a stand-in of the three runtime calls that it makes."""
import glob
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "surogate_b200", "csrc")

PROGRAM = r"""
#include "launch_limits.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int device = 0;
static bool refuse = false;
static std::atomic<int> raised[80];
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int bytes) {
    if (refuse || a != cudaFuncAttributeMaxDynamicSharedMemorySize || bytes != 230000) return cudaErrorInvalidValue;
    ++raised[device];
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
#define EXPECT(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    int k1, k2;
    std::atomic<uint64_t> a{0}, b{0}, c{0};
    refuse = true;
    EXPECT(!sg::raise_smem_limit(&k1, 230000, a));
    refuse = false;
    for (int i = 0; i < 3; ++i)
        for (device = 0; device < 3; ++device) EXPECT(sg::raise_smem_limit(&k1, 230000, a));
    for (int d = 0; d < 3; ++d) EXPECT(raised[d] == 1);
    device = 1;
    EXPECT(sg::raise_smem_limit(&k2, 230000, b) && raised[1] == 2);          // another kernel on the same device
    device = 70;
    EXPECT(sg::raise_smem_limit(&k1, 230000, a) && sg::raise_smem_limit(&k1, 230000, a) && raised[70] == 2);
    std::vector<std::thread> ts;
    std::atomic<int> bad{0};
    for (int t = 0; t < 16; ++t)
        ts.emplace_back([&, t] {
            for (int i = 0; i < 1000; ++i) {
                device = 8 + (t + i) % 8;
                if (!sg::raise_smem_limit(&k1, 230000, c) || raised[device] == 0) ++bad;
            }
        });
    for (auto& t : ts) t.join();
    EXPECT(bad == 0);
    return 0;
}
"""


def test_limits_are_raised_once_per_device(tmp_path):
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", f"-I{home}/include", str(src), "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_kernels_ask_through_the_helper(path):
    """A flag of the whole process, or a call whose result is dropped, leaves the second device of a process without the limit."""
    text = open(path).read()
    assert not re.search(r"static\s+bool\s+attr_set", text)
    assert not re.search(r"cudaFuncSetAttribute\s*\(", text)
