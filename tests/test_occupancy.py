"""blocks_per_sm on several devices, on the CPU: its source compiled against a fake of the four CUDA
calls it makes.  A kernel's dynamic shared-memory limit belongs to one device and starts at 48 KB
there; a kernel asked about beyond its limit has no resident block."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

FAKE = r"""
#include <cstdio>
#include <map>
#include "internal.hpp"

static int g_device = 0, g_queries = 0;
static std::map<std::pair<int, const void*>, int> g_limit;

extern "C" cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "fake"; }
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    g_limit[{g_device, f}] = v;
    return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int, size_t smem) {
    auto it = g_limit.find({g_device, f});
    const size_t most = it == g_limit.end() ? 49152 : size_t(it->second);
    *n = smem <= most ? int(227 * 1024 / (smem ? smem : 1)) : 0;
    ++g_queries;
    return cudaSuccess;
}

int main() {
    static const int a = 0, b = 0;
    for (int round = 0; round < 2; ++round)
        for (int dev = 0; dev < 3; ++dev) {
            g_device = dev;
            for (const void* k : {static_cast<const void*>(&a), static_cast<const void*>(&b)})
                for (size_t smem : {size_t(160000), size_t(60000), size_t(100000), size_t(1000)})
                    if (tgtp::blocks_per_sm(k, 256, smem) != int(227 * 1024 / smem)) {
                        std::printf("device %d, %zu bytes: %d\n", dev, smem, tgtp::blocks_per_sm(k, 256, smem));
                        return 1;
                    }
        }
    return g_queries == 24 ? 0 : 2;  // the second round is answered from the record
}
"""


def test_limits_are_raised_on_every_device(tmp_path):
    src, exe = tmp_path / "fake.cpp", tmp_path / "fake"
    src.write_text(FAKE)
    csrc = os.path.join(ROOT, "tgtp_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I" + csrc, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), "-o", str(exe),
                    str(src), os.path.join(csrc, "occupancy.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
