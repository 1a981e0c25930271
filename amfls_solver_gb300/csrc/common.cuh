// Shared device/host helpers for the GB300 AMFLS library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <string>

namespace amfls_gpu {

// Host-side CUDA error check that turns a failure into an exception; the
// C ABI layer converts it into an error code and a message.
struct CudaError : std::runtime_error {
    CudaError(const std::string& what, cudaError_t code) : std::runtime_error(what), code(code) {}
    cudaError_t code;
};

inline void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        throw CudaError(std::string(what) + ": " + cudaGetErrorString(e), e);
    }
}

#define AMFLS_CUDA(call) ::amfls_gpu::check_cuda((call), #call)

// Kernel launches made by this thread (reported per solve).  Launch sites
// use AMFLS_LAUNCHED() right after the <<<...>>> statement.
inline long long& launch_count() {
    static thread_local long long count = 0;
    return count;
}

#define AMFLS_LAUNCHED()                                             \
    do {                                                             \
        ::amfls_gpu::check_cuda(cudaGetLastError(), "kernel launch"); \
        ++::amfls_gpu::launch_count();                               \
    } while (0)

// Stream-ordered device allocation from the device's default memory pool.
// A solve allocates and frees its buffers on its own stream: unlike
// cudaFree, cudaFreeAsync does not synchronise the whole device, so solves
// running concurrently on different streams do not stall each other.
template <typename T>
inline void stream_alloc(T** p, size_t bytes, cudaStream_t s) {
    check_cuda(cudaMallocAsync(reinterpret_cast<void**>(p), bytes, s), "cudaMallocAsync");
}
inline void stream_free(const void* p, cudaStream_t s) {
    if (p) cudaFreeAsync(const_cast<void*>(p), s);
}

// Keeps freed blocks of the current device's default memory pool cached in
// the process (release threshold = unlimited) instead of returning them to
// the driver at every synchronisation, so consecutive solves reuse their
// buffers.  Called by each solve; takes effect once per device.
void keep_pool_memory();

// Small exchanges between a solve and its host thread.
//
// Copies of a few hundred bytes go through kernels, not through the copy
// engines: a device-to-host copy queued behind a long resident kernel holds
// its engine's queue, and with it the copies of every other solve that shares
// the queue.  Results land in pinned host memory that the GPU writes, followed
// by a sequence number the host polls, so that a wait costs neither a thread
// wake-up nor a driver call.

// Pinned host memory of the calling thread, freed with the thread: the
// landing place of small reads.  The first half belongs to reads that are
// waited for at once, the second half to values read after the next wait.
constexpr size_t kPinnedBytes = 1 << 16;
struct HostPage {
    unsigned char* data = nullptr;
    unsigned* flag = nullptr;  // last sequence number the GPU has reached
    unsigned seq = 0;
};
HostPage& host_page();

// Waits until the page's flag has reached seq: polls, then yields the core
// between polls, then sleeps between them (many solves on many host threads);
// a failed kernel ends the wait with its error.
void wait_flag(const HostPage& page, unsigned seq, cudaStream_t stream);

// Waits until the work enqueued on `stream` so far has finished.
void stream_wait(cudaStream_t stream);

#if defined(__CUDACC__)
static __global__ void copy_out_kernel(const unsigned* src, unsigned* dst, int words,
                                       unsigned* flag, unsigned seq) {
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    __threadfence_system();
    __syncthreads();
    if (flag && threadIdx.x == 0) *(volatile unsigned*)flag = seq;
}

// *dst = value, in stream order (values up to the size of a kernel argument).
template <typename T>
__global__ void put_kernel(T* dst, T value) {
    const unsigned* src = reinterpret_cast<const unsigned*>(&value);
    unsigned* out = reinterpret_cast<unsigned*>(dst);
    for (int i = threadIdx.x; i < (int)(sizeof(T) / sizeof(unsigned)); i += blockDim.x)
        out[i] = src[i];
}
template <typename T>
inline void put(T* dst, const T& value, cudaStream_t stream) {
    static_assert(sizeof(T) % sizeof(unsigned) == 0 && sizeof(T) <= 3072);
    put_kernel<T><<<1, 64, 0, stream>>>(dst, value);
    check_cuda(cudaGetLastError(), "kernel launch");
    ++launch_count();
}

// Device bytes (a multiple of 4, 4-byte aligned) into the page at `offset`;
// with `signal` the flag follows.
inline void copy_out(const void* device, size_t bytes, size_t offset, bool signal,
                     cudaStream_t stream) {
    HostPage& page = host_page();
    const int words = (int)(bytes / 4);
    copy_out_kernel<<<1, words > 128 ? 512 : 64, 0, stream>>>(
        static_cast<const unsigned*>(device), reinterpret_cast<unsigned*>(page.data + offset),
        words, signal ? page.flag : nullptr, signal ? ++page.seq : 0u);
    check_cuda(cudaGetLastError(), "kernel launch");
    ++launch_count();
}

// Copies a small device object to the host and waits for it.
template <typename T>
inline void read_back(T* host, const T* device, cudaStream_t stream, size_t count = 1) {
    const size_t bytes = sizeof(T) * count;
    if (bytes > kPinnedBytes / 2 || bytes % 4 != 0) {
        check_cuda(cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, stream),
                   "cudaMemcpyAsync");
        stream_wait(stream);
        return;
    }
    copy_out(device, bytes, 0, true, stream);
    const HostPage& page = host_page();
    wait_flag(page, page.seq, stream);
    std::memcpy(host, page.data, bytes);
}
#endif

// Streaming multiprocessors of the current device
// (cudaDevAttrMultiProcessorCount), queried once per device.
inline int sm_count() {
    static int cached[64] = {};
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    const int slot = dev >= 0 && dev < 64 ? dev : 0;
    int v = __atomic_load_n(&cached[slot], __ATOMIC_RELAXED);
    if (v == 0) {
        check_cuda(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev),
                   "cudaDeviceGetAttribute(MultiProcessorCount)");
        v = v > 0 ? v : 1;
        __atomic_store_n(&cached[slot], v, __ATOMIC_RELAXED);
    }
    return v;
}

// Grid cap of the grid-stride and reduction kernels: eight resident
// 256-thread blocks per SM.
inline int grid_cap() { return 8 * sm_count(); }

// Upper bound of grid_cap() (devices of up to 256 SMs), for sizing the
// per-block partial-sum scratch that is allocated once.
constexpr int kMaxGridCap = 8 * 256;

constexpr int kWarp = 32;
constexpr int kPanel = 32;  // columns per V panel (row-major n x 32 tiles)

__host__ __device__ inline long long ceil_div(long long a, long long b) {
    return (a + b - 1) / b;
}

#if defined(__CUDACC__)
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over all threads of a block (blockDim.x multiple of 32, <= 1024).
// Fixed reduction tree, so the result is deterministic for a fixed launch.
__device__ inline double block_sum(double v, double* scratch32) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch32[warp] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    double r = 0.0;
    if (warp == 0) {
        r = lane < nw ? scratch32[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;  // valid in warp 0
}

__device__ inline double block_max(double v, double* scratch32) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch32[warp] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    double r = 0.0;
    if (warp == 0) {
        r = lane < nw ? scratch32[lane] : 0.0;
        r = warp_max(r);
    }
    return r;
}

// "Last block done" pattern: every block writes its partial, the block that
// arrives last (by an atomic ticket) sees all partials after a fence.
// Returns true in the last block; the counter is reset for the next launch.
__device__ inline bool arrive_last(unsigned int* counter, unsigned int nblocks) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int ticket = atomicAdd(counter, 1u);
        last = (ticket == nblocks - 1);
        if (last) *counter = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}
#endif

}  // namespace amfls_gpu
