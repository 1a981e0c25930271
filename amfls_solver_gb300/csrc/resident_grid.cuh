// What the cooperative kernels with one block per SM share: the grid barrier
// and the sums over the grid (resident_levels.cu, resident_baselines.cu).
#pragma once

#include "common.cuh"
#include "resident_levels.hpp"

namespace amfls_gpu {
namespace resident {

constexpr int kT = kResidentThreads;
constexpr int kW = kT / 32;
constexpr unsigned kSpinLimit = 1u << 23;  // polls of about a microsecond

template <int N>
struct GridShared {
    unsigned arrived;  // barrier arrivals expected so far
    int failed;        // a wait gave up
    double lane[N][kT];  // values to be added over the block
};

// Grid barrier: the block's writes before it are visible to every block after
// it (the fences of thread 0 are cumulative over the block barriers around
// them, and the second one drops stale L1 lines).
template <typename Sh>
__device__ __forceinline__ void grid_barrier(Sh& s, unsigned* bar) {
    __syncthreads();
    if (threadIdx.x == 0) {
        s.arrived += gridDim.x;
        const unsigned want = s.arrived;
        __threadfence();
        atomicAdd(bar, 1u);
        unsigned seen, spins = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
            if (++spins > kSpinLimit) {
                s.failed = 1;
                break;
            }
        } while ((int)(seen - want) < 0);
        __threadfence();
    }
    __syncthreads();
}

// Block sums of N per-thread values, of which the first `warps` warps hold
// non-zero ones, into this block's entries of a slot: through shared memory
// and one warp per value.  FP64 operations are few (two lanes per SM clock)
// and slow one after the other, so only warps with something to add count.
template <int N, typename Sh>
__device__ __forceinline__ void block_partials(Sh& s, const double (&v)[N], int warps,
                                               double* red, int slot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < warps) {
#pragma unroll
        for (int i = 0; i < N; ++i) s.lane[i][threadIdx.x] = v[i];
    }
    __syncthreads();
    if (warp < N) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        for (int w = 0; w < warps; w += 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (w + i < warps) t[i] += s.lane[warp][(w + i) * 32 + lane];
        }
        const double a = warp_sum((t[0] + t[1]) + (t[2] + t[3]));
        if (lane == 0) red[((long long)slot * 4 + warp) * gridDim.x + blockIdx.x] = a;
    }
}

// After the barrier, one warp: the sum of entry i of a slot over the blocks,
// in a fixed order (every lane holds it).  Several values share the additions
// of one butterfly that halves the values a lane holds (three: six dependent
// FP64 additions over the lanes instead of fifteen).
template <int N>
__device__ __forceinline__ void reduce_slot(const double* red, int slot, double (&out)[N]) {
    constexpr int M = N <= 1 ? 1 : N <= 2 ? 2 : 4;
    const int lane = threadIdx.x & 31;
    const double* p = red + (long long)slot * 4 * gridDim.x;
    double v[M];
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __ldcg(p + (long long)i * gridDim.x + b);
    int have = M;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (have > 1) {
            const bool upper = (lane & o) != 0;
            have >>= 1;
#pragma unroll
            for (int j = 0; j < M / 2; ++j) {
                if (j < have) {
                    const double keep = upper ? v[j + have] : v[j];
                    const double send = upper ? v[j] : v[j + have];
                    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    // value i ended in the lanes whose top bits spell i
#pragma unroll
    for (int i = 0; i < N; ++i)
        out[i] = M == 1 ? v[0]
                        : __shfl_sync(0xffffffffu, v[0], M == 2 ? i * 16 : (i >> 1) * 16 + (i & 1) * 8);
}

// sqrt of each of N values, side by side in the lanes of a warp
template <int N>
__device__ __forceinline__ void warp_sqrt(double (&v)[N]) {
    const int lane = threadIdx.x & 31;
    double mine = v[0];
#pragma unroll
    for (int i = 1; i < N; ++i) mine = lane == i ? v[i] : mine;
    mine = sqrt(mine);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __shfl_sync(0xffffffffu, mine, i);
}

}  // namespace resident
}  // namespace amfls_gpu
