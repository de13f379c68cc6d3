"""The table of tensor maps (csrc/wide_common.cuh) against a fake encoder: a weight tensor's map is encoded once, and calls on inputs at ever new addresses neither fill the table
nor push the weights' maps out of it."""
import importlib.util
import os
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "strix-halo-engine-lab_b200")

FAKES = r"""
#include <cuda.h>
#include <cuda_runtime_api.h>
int encodes = 0;
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { ++encodes; return CUDA_SUCCESS; }
extern "C" cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(&encode); *q = cudaDriverEntryPointSuccess; return cudaSuccess;
}
extern "C" cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
extern "C" void** __cudaRegisterFatBinary(void*) { return nullptr; }
extern "C" void __cudaRegisterFatBinaryEnd(void**) {}
extern "C" void __cudaUnregisterFatBinary(void**) {}
extern "C" char __cudaInitModule(void**) { return 0; }
"""
MAIN = r"""
#include "wide_common.cuh"
#include <cstdio>
extern int encodes;
namespace b200moe { int fail(int code, const char*, ...) { return code; } }
int main() {
    using namespace b200moe;
    CUtensorMap m;
    auto at = [](u64 n) { return reinterpret_cast<const u8*>(n << 12); };
    auto weights = [&] { const int before = encodes; return wide::rows_map(at(1), 1440, 64, 432, 32, &m) ? -1 : encodes - before; };
    const int first = weights(), again = weights();
    for (u64 i = 2; i < 3000; ++i)
        if (wide::pitched_map(at(i), 2048, 2048, 8, 784, 8, &m)) return 1;
    printf("%d %d %d\n", first, again, weights());
}
"""


def test_inputs_leave_the_weights_maps_alone(tmp_path):
    spec = importlib.util.spec_from_file_location("b200moe_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    (tmp_path / "fakes.cpp").write_text(FAKES)
    (tmp_path / "main.cu").write_text(MAIN)
    out = str(tmp_path / "table")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "none", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "main.cu"),
                    str(tmp_path / "fakes.cpp"), "-o", out], check=True)
    assert subprocess.run([out], capture_output=True, text=True, check=True).stdout.split() == ["1", "0", "0"]
