"""The dynamic shared-memory limit of a kernel (capi.cu, configure_smem), compiled
against a recording CUDA runtime: a limit never falls, whatever the order and
number of sizes, kernels and devices, and one that suffices is not set again."""

import os
import subprocess

from frostspin_b200 import build

PROGRAM = r"""
#include <cuda_runtime.h>
#include <map>
#include <stdio.h>
#include <utility>

namespace fsb { int configure_smem(const void* func, int bytes); }

static int device = 0, sets = 0;
static bool fell = false, failing = false;
static std::map<std::pair<const void*, int>, int> limit;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes) {
    if (failing) return cudaErrorInvalidValue;
    int& now = limit[{f, device}];
    fell = fell || bytes < now;
    now = bytes;
    ++sets;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    a->maxDynamicSharedSizeBytes = limit[{f, device}];
    return cudaSuccess;
}
}

#define REQUIRE(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    static char kernels[600];
    // growing, then shrinking sizes of one kernel, on two devices
    for (device = 0; device < 2; ++device)
        for (int pass = 0; pass < 2; ++pass)
            for (int i = 0; i < 200; ++i) {
                const int bytes = 50000 + 100 * (pass ? 199 - i : i);
                REQUIRE(fsb::configure_smem(kernels, bytes) == 0);
                REQUIRE((limit[{kernels, device}] >= bytes));
            }
    REQUIRE(!fell && sets == 400);
    // more kernels than any table holds, largest size first
    device = 0;
    for (int bytes : {90000, 60000, 70000, 95000, 80000})
        for (char& k : kernels) {
            REQUIRE(fsb::configure_smem(&k, bytes) == 0);
            REQUIRE((limit[{&k, 0}] >= bytes));
        }
    REQUIRE(!fell && sets == 400 + 2 * 600);
    // a refused size is reported and does not count as set
    failing = true;
    REQUIRE(fsb::configure_smem(kernels, 200000) != 0);
    failing = false;
    REQUIRE(fsb::configure_smem(kernels, 150000) == 0);
    REQUIRE((limit[{kernels, 0}] == 150000));
    return 0;
}
"""


def test_limits_only_rise(tmp_path):
    # host code only: the device intrinsics of common.cuh are declared, never called
    (tmp_path / "device.h").write_text("unsigned __umulhi(unsigned, unsigned);\n"
                                       "int atomicCAS(int*, int, int);\n")
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = tmp_path / "limits"
    cuda = os.path.dirname(os.path.dirname(build._nvcc()))
    subprocess.run(["g++", "-std=c++17", "-x", "c++", "-include", str(tmp_path / "device.h"),
                    "-I", build.INCLUDE_DIR, "-I", os.path.join(cuda, "include"),
                    os.path.join(build.CSRC_DIR, "capi.cu"), str(tmp_path / "main.cpp"), "-o",
                    str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, check=False)
    assert res.returncode == 0, res.stdout
