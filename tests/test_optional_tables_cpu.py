"""The sliced-row tables are an extra of a CSR operator, without a GPU: the
operator's object file linked against a stand-in for the CUDA runtime (memory on
the host, kernels that do nothing) and for the tables' construction, which runs
out of memory on either side or fails otherwise.  They are built when a solve
first asks for them, once."""
import subprocess

import pytest

from amfls_solver_gb300 import build

SOURCE = r"""
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <stdexcept>

#include "common.cuh"
#include "csr_operator.hpp"
#include "resident_levels.hpp"
#include "sliced_rows.cuh"

static int calls = 0, fail_at = 0, released = 0;
static cudaError_t failure = cudaSuccess, last = cudaSuccess;
static size_t free_bytes = 1ull << 38;

namespace amfls_gpu {
HostPage& host_page() {
    static unsigned char data[kPinnedBytes + 64];
    static HostPage page{data, reinterpret_cast<unsigned*>(data + kPinnedBytes), 0};
    return page;
}
void wait_flag(const HostPage&, unsigned, cudaStream_t) {}
namespace sliced {
void build(Store& s, const long long*, const int*, const double*, const int*, int, int,
           cudaStream_t) {
    if (++calls == fail_at) {
        last = failure;
        check_cuda(failure, "tables");
    }
    s.tasks = reinterpret_cast<int2*>(std::malloc(16));
}
void Store::release() {
    if (tasks) ++released;
    std::free(tasks);
    *this = Store{};
}
}  // namespace sliced
}  // namespace amfls_gpu

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 3
                                                                                              : 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = free_bytes; *t = 1ull << 38; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->binaryVersion = a->ptxVersion = 103;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
    *n = 2;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
    return cudaSuccess;
}
}

int main() {
    using namespace amfls_gpu;
    const long long off[4] = {0, 2, 4, 6}, idx[6] = {0, 1, 0, 1, 0, 1};
    const double val[6] = {1, 2, 3, 4, 5, 6};
    struct { int at; cudaError_t error; size_t free; } runs[] = {
        {0, cudaSuccess, 1ull << 38}, {0, cudaSuccess, 64}, {1, cudaErrorMemoryAllocation, 1ull << 38},
        {2, cudaErrorMemoryAllocation, 1ull << 38}, {2, cudaErrorLaunchFailure, 1ull << 38}};
    for (const auto& run : runs) {
        calls = released = 0;
        fail_at = run.at;
        failure = run.error;
        free_bytes = run.free;
        try {
            CsrOperator op(3, 2, off, idx, val, 6, nullptr);
            ResidentOperator view;
            const int sizes = op.resident(&view), early = calls;
            const int first = op.resident_tables(&view, nullptr);
            const int again = op.resident_tables(&view, nullptr);
            std::printf("%d %d %d%d %d %d %d\n", sizes, early, first, again, calls, released,
                        (int)last);
        } catch (const std::exception&) {
            std::printf("raised %d\n", released);
        }
    }
}
"""


@pytest.fixture(scope="module")
def outcomes(tmp_path_factory):
    obj = build.OUT / "csr_operator.o"
    if not obj.exists():
        build.build(force=True)
    tmp = tmp_path_factory.mktemp("tables")
    src, exe = tmp / "tables.cpp", tmp / "tables"
    src.write_text(SOURCE)
    include = build.Path(build._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++20", "-I", str(include), "-I", str(build.SRC), str(src),
                    str(obj), "-o", str(exe), "-pthread", "-ldl"], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr
    return run.stdout.splitlines()


def test_tables_are_built_once_and_when_asked_for(outcomes):
    """Sizes known, no table before the first request, two sides after it."""
    assert outcomes[0] == "1 0 11 2 0 0"


def test_tables_do_not_depend_on_the_free_memory(outcomes):
    assert outcomes[1] == outcomes[0]


def test_an_operator_without_memory_for_tables_does_without_them(outcomes):
    """No side's table is left, no further attempt, and no error for the next
    call to find."""
    assert outcomes[2:4] == ["1 0 00 1 0 0", "1 0 00 2 1 0"]


def test_other_failures_are_raised(outcomes):
    assert outcomes[4] == "raised 1"
