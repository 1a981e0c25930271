// Sliced-row copy of one side of a CSR operator, for the products inside the
// resident level kernel (resident_levels.cu).
//
// Rows are ordered by length, longest first (stable), and cut into warp tasks
// of 32 / g rows, g = 1 .. 32 lanes per row (a power of two, about 8 or 16
// elements per lane).  A task's elements are stored step by
// step: entry `step * 32 + lane` of the task is the element that lane reads
// at that step, so every load of values and indices is one coalesced warp
// access and a lane's place in the matrix needs no row offsets.  Lane `sub`
// of a row takes the elements sub, sub + g, sub + 2g, ...; the g sums are
// added by a fixed butterfly.  Tasks are dealt to the warps of the grid in
// snake order, longest first, so every sum's order is fixed by the table and
// the grid.
//
// Why a copy: the resident kernel runs both products of every level without a
// launch in between, so what counts is the chain of dependent memory rounds
// after each grid barrier.  Values, indices, row numbers and counts do not
// depend on the level, so a warp loads its first task's part of them before
// it waits at the barrier and only the gathers of x remain behind it.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace amfls_gpu {
namespace sliced {

constexpr int kUnroll = 8;         // steps in flight

struct Side {
    const int2* tasks = nullptr;   // {first step, steps}
    const int2* lanes = nullptr;   // 32 per task: {row or -1, elements of the lane}
    const int* idx = nullptr;      // 32 per step
    const double* val = nullptr;
    int ntasks = 0;
    int group_end[6] = {};         // tasks with 32, 16, 8, 4, 2, 1 lanes per row end here
};

// log2 of the lanes per row of a row of `len` elements, about `per_lane` each
__host__ __device__ inline int lane_shift(long long len, int per_lane) {
    int s = 0;
    while (s < 5 && len > (long long)per_lane << s) ++s;
    return s;
}

// Elements per lane aimed at: 8, one round of loads, while a row's sum is
// latency (few tasks per warp of the GPU); 16 for larger operators, where
// fewer and longer lane sums keep the cross-lane additions small.
inline int elements_per_lane(long long nonzeros) { return nonzeros <= (1LL << 20) ? 8 : 16; }

#if defined(__CUDACC__)
// Task of warp w among W in round k of the snake order.
__device__ __forceinline__ int snake(int k, int w, int W) {
    return k * W + ((k & 1) ? W - 1 - w : w);
}

struct Meta {
    int2 task, lane;
    int shift;
};

__device__ __forceinline__ Meta load_meta(const Side& s, int t) {
    Meta m;
    m.task = make_int2(0, 0);
    m.lane = make_int2(-1, 0);
    m.shift = 0;
    if (t < s.ntasks) {
        m.task = __ldg(s.tasks + t);
        m.lane = __ldg(s.lanes + (long long)t * 32 + (threadIdx.x & 31));
        int sh = 5;
#pragma unroll
        for (int i = 0; i < 5; ++i) sh -= t >= s.group_end[i] ? 1 : 0;
        m.shift = sh;
    }
    return m;
}

// The level-independent part of a task: what a warp may load before the
// vector it multiplies is complete.
struct Fetch {
    int row, count;  // of the lane
    int shift, steps, first;
    int idx[kUnroll];
    double val[kUnroll];
};

__device__ __forceinline__ void fetch_steps(const Side& s, Fetch& f, int j0) {
    const long long e = ((long long)f.first + j0) * 32 + (threadIdx.x & 31);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
        const bool in = j0 + u < f.count;
        f.idx[u] = in ? __ldg(s.idx + e + 32 * u) : 0;
        f.val[u] = in ? __ldg(s.val + e + 32 * u) : 0.0;
    }
}

__device__ __forceinline__ void start_fetch(const Side& s, const Meta& m, Fetch& f) {
    f.row = m.lane.x;
    f.count = m.lane.y;
    f.shift = m.shift;
    f.steps = m.task.y;
    f.first = m.task.x;
    fetch_steps(s, f, 0);
}

// A warp's walk over its tasks: the elements of the next task and the
// description of the one after it are on their way while one is summed.
struct Walk {
    Fetch cur, next;
    Meta after;
    int round;  // of `cur`
};

__device__ __forceinline__ void start_walk(const Side& s, Walk& k, int w, int W) {
    const Meta m0 = load_meta(s, snake(0, w, W)), m1 = load_meta(s, snake(1, w, W));
    k.after = load_meta(s, snake(2, w, W));
    start_fetch(s, m0, k.cur);
    start_fetch(s, m1, k.next);
    k.round = 0;
}

// Whether a further task was there.
__device__ __forceinline__ bool next_task(const Side& s, Walk& k, int w, int W) {
    ++k.round;
    if (snake(k.round, w, W) >= s.ntasks) return false;
    k.cur = k.next;
    start_fetch(s, k.after, k.next);
    k.after = load_meta(s, snake(k.round + 2, w, W));
    return true;
}

// The row sum of a fetched task against x (every lane of a row's group holds
// it).  x may have been written by other SMs earlier in the same kernel:
// plain loads, ordered by the grid barrier.  Two chains per lane, because a
// dependent FP64 operation takes far longer than one of the same warp's next.
__device__ __forceinline__ double task_sum(const Side& s, Fetch& f, const double* x) {
    double acc0 = 0.0, acc1 = 0.0;
    for (int j0 = 0; j0 < f.steps; j0 += kUnroll) {
        double xv[kUnroll], v[kUnroll];
        const int left = f.count - j0;
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            xv[u] = u < left ? x[f.idx[u]] : 0.0;
            v[u] = f.val[u];
        }
        if (j0 + kUnroll < f.steps) fetch_steps(s, f, j0 + kUnroll);
#pragma unroll
        for (int u = 0; u < kUnroll; u += 2) {
            if (u < left) acc0 = fma(v[u], xv[u], acc0);
            if (u + 1 < left) acc1 = fma(v[u + 1], xv[u + 1], acc1);
        }
    }
    double acc = acc0 + acc1;
    for (int o = (1 << f.shift) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}
#endif

// Owner of one side's arrays.
struct Store {
    Side side;
    int2* tasks = nullptr;
    int2* lanes = nullptr;
    int* idx = nullptr;
    double* val = nullptr;
    void release();
};

// Builds the table of a side from its CSR arrays (device), on `stream`;
// synchronises twice to size the copy.  `lens` holds the row lengths.
void build(Store& store, const long long* off, const int* idx, const double* val,
           const int* lens, int count, int per_lane, cudaStream_t stream);

}  // namespace sliced
}  // namespace amfls_gpu
