"""What the library keeps for the process belongs to one device: the SM count and the kernels' shared-memory limits of a
second device are asked and set for that device. per_device.h is compiled against a fake runtime with two devices of
different sizes, and used from several threads."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "atsat_gb300", "csrc")

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <mutex>
#include <set>
#include <thread>
#include <tuple>
#include <vector>
#include "per_device.h"

static thread_local int device = 0;
static std::mutex m;
static std::multiset<std::tuple<int, const void*, int>> limits;    // device, kernel, bytes
static int queries = 0;
static bool no_device = false, refuse = false;

extern "C" {
cudaError_t cudaGetDevice(int* d) { if (no_device) return cudaErrorNoDevice; *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
    assert(a == cudaDevAttrMultiProcessorCount);
    std::lock_guard<std::mutex> l(m);
    queries++;
    *v = d == 0 ? 152 : 100 + d;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize);
    if (refuse) return cudaErrorInvalidValue;
    std::lock_guard<std::mutex> l(m);
    limits.insert({device, f, v});
    return cudaSuccess;
}
}

static char k1, k2;
static cudaError_t launch1() { static atsat::SharedMemory s; return s.allow(&k1, 73000); }
static cudaError_t launch2() { static atsat::SharedMemory s; return s.allow(&k2, 109000); }

int main() {
    refuse = true;
    assert(launch2() == cudaErrorInvalidValue);                    // not kept: set by the next launch
    refuse = false;
    for (int d : {0, 1, 0, 1, 70, 70}) {
        device = d;
        assert(launch1() == cudaSuccess && launch2() == cudaSuccess);
        assert(atsat::sm_count() == (d == 0 ? 152 : 100 + d));
    }
    for (int d : {0, 1}) assert(limits.count({d, &k1, 73000}) == 1 && limits.count({d, &k2, 109000}) == 1);
    assert(limits.count({70, &k1, 73000}) == 2);                   // beyond the kept devices: each time
    assert(queries == 4);
    std::vector<std::thread> t;
    for (int d = 2; d < 10; d++)
        t.emplace_back([d] {
            device = d;
            for (int n = 0; n < 1000; n++) assert(atsat::sm_count() == 100 + d && launch1() == cudaSuccess);
        });
    for (auto& x : t) x.join();
    for (int d = 2; d < 10; d++) assert(limits.count({d, &k1, 73000}) == 1);
    no_device = true;
    assert(atsat::sm_count() == 152 && launch1() == cudaSuccess);
    puts("ok");
}
"""


def include_dir():
    for nvcc in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if nvcc:
            d = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
            if os.path.exists(os.path.join(d, "cuda_runtime_api.h")):
                return d
    pytest.skip("no CUDA headers")


def test_two_devices(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", include_dir(), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "ok"


def test_no_launch_keeps_a_limit_by_itself():
    """The kernels' limits are set through per_device.h, or on every call; a flag of the launch's own would be the first
    device's."""
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read() if name.endswith((".cu", ".cuh")) else ""
        assert not re.search(r"\bstatic\s+(bool|int)\s+\w+\s*=", text), name
