"""The resident level kernel's launch on several devices, without a GPU: its
object file linked against a stand-in for the CUDA runtime that keeps a
kernel's shared-memory limit per device, as the runtime does, and refuses a
launch that asks for more."""
import subprocess

import pytest

from amfls_solver_gb300 import build

SOURCE = r"""
#include <cuda_runtime.h>

#include <cstdio>
#include <map>
#include <set>
#include <utility>

#include "resident_levels.hpp"

static int device = 0, launches = 0;
static std::map<std::pair<int, const void*>, size_t> limit;
static std::set<const void*> kernels;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int value) {
    // another thread's launch may stand between its own call and this one
    size_t& v = limit[{device, f}];
    if ((size_t)value < v) return cudaErrorInvalidValue;
    v = (size_t)value;
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t shared,
                                        cudaStream_t) {
    const auto it = limit.find({device, f});
    if (shared > (it == limit.end() ? 48 * 1024 : it->second)) return cudaErrorInvalidValue;
    kernels.insert(f);
    ++launches;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
    return cudaSuccess;
}
}

int main() {
    const amfls_gpu::ResidentArgs args{};
    for (int d : {0, 1, 3, 0})
        for (int storage : {0, 1, 2})
            for (int k : {1, amfls_gpu::kResidentMaxBasis, 33}) {
                device = d;
                amfls_gpu::launch_resident_levels(args, 152, k, storage, nullptr);
            }
    std::printf("%d %d\n", launches, (int)kernels.size());
}
"""


def test_every_device_gets_the_shared_memory_limit(tmp_path):
    obj = build.OUT / "resident_levels.o"
    if not obj.exists():
        build.build(force=True)
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(SOURCE)
    include = build.Path(build._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++20", "-I", str(include), "-I", str(build.SRC), str(src),
                    str(obj), "-o", str(exe), "-pthread"], check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr
    assert run.stdout.split() == ["36", "3"]
