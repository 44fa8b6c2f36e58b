"""Launch attributes are set once for each device: csrc/cc_per_device.h against a stand-in for the CUDA
runtime with several devices, and no other once-only flag in the CUDA sources."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crashcat_gb300", "csrc")

RUNTIME = """
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidDevice = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
inline int g_device = 0, g_bytes[80] = {}, g_sets = 0;
inline bool g_fail = false;
inline cudaError_t cudaGetDevice(int *d) { *d = g_device; return cudaSuccess; }
inline cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int v) {
    g_sets++;
    if (g_fail) return cudaErrorInvalidDevice;
    g_bytes[g_device] = v;
    return cudaSuccess;
}
"""
MAIN = """
#include <cstdio>
#include <thread>
#include <vector>
#include "cc_per_device.h"
void kernel() {}
int main() {
    cc::PerDevice shared, value;
    auto set = [&] { return shared.get([] { return cc::allow_shared(70000, kernel); }); };
    g_fail = true;
    if (set() != 0) return 1;  // not kept
    g_fail = false;
    for (int round = 0; round < 2; round++)
        for (int d : {0, 1, 5, 63}) {
            g_device = d;
            if (set() != 1 || g_bytes[d] != 70000) return 2;
        }
    if (g_sets != 1 + 4) return 3;  // once a device
    g_device = 64;  // past the table: set each time
    if (set() != 1 || set() != 1 || g_bytes[64] != 70000 || g_sets != 5 + 2) return 4;
    g_device = 3;
    std::vector<std::thread> all;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; t++)
        all.emplace_back([&] {
            for (int k = 0; k < 1000; k++) wrong += value.get([] { return 152; }) != 152;
        });
    for (auto &t : all) t.join();
    return wrong ? 5 : 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="no host compiler")
def test_values_are_kept_for_each_device(tmp_path):
    (tmp_path / "cuda_runtime_api.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "per_device"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_launch_attribute_is_set_once_for_the_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert not re.search(r"static bool \w*(attr|sized|ready)\w* *=", open(path).read()), path
