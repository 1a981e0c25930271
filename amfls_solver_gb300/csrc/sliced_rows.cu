// Construction of the sliced-row tables (see sliced_rows.cuh), on the device:
// a stable radix sort of the rows by descending length, a scan of the tasks'
// steps, and one pass that lays the elements out.
#include <cub/cub.cuh>

#include <algorithm>

#include "sliced_rows.cuh"

namespace amfls_gpu {
namespace sliced {
namespace {

// rows with 32, 16, 8, 4, 2, 1 lanes
__global__ void count_groups_kernel(const int* lens, int count, int per_lane, int* rows_of,
                                    int* counts) {
    __shared__ int local[6];
    if (threadIdx.x < 6) local[threadIdx.x] = 0;
    __syncthreads();
    // 64 bits: rows and tasks may end within a stride of 2^31
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < count;
         r += (long long)gridDim.x * blockDim.x) {
        atomicAdd(&local[5 - lane_shift(lens[r], per_lane)], 1);
        rows_of[r] = (int)r;
    }
    __syncthreads();
    if (threadIdx.x < 6 && local[threadIdx.x]) atomicAdd(&counts[threadIdx.x], local[threadIdx.x]);
}

struct Groups {
    int row_start[7];   // sorted rows of group i (32 >> i lanes per row)
    int task_start[7];  // its tasks
};

__global__ void task_steps_kernel(Groups g, const int* sorted_lens, int ntasks, int* steps) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t <= ntasks;
         t += (long long)gridDim.x * blockDim.x) {
        if (t == ntasks) {
            steps[t] = 0;
            continue;
        }
        int i = 0;
        while (t >= g.task_start[i + 1]) ++i;
        const int shift = 5 - i;
        const int first = g.row_start[i] + (int)(t - g.task_start[i]) * (32 >> shift);
        steps[t] = (sorted_lens[first] + (1 << shift) - 1) >> shift;
    }
}

__global__ void fill_kernel(Groups g, const int* rows, const int* sorted_lens, const int* first,
                            int ntasks, const long long* off, const int* idx, const double* val,
                            int2* tasks, int2* lanes, int* out_idx, double* out_val) {
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; t < ntasks;
         t += warps) {
        int i = 0;
        while (t >= g.task_start[i + 1]) ++i;
        const int shift = 5 - i, sub = lane & ((1 << shift) - 1);
        const long long pos =
            g.row_start[i] + (t - g.task_start[i]) * (32 >> shift) + (lane >> shift);
        const bool has = pos < g.row_start[i + 1];
        const int row = has ? rows[pos] : -1;
        const int len = has ? sorted_lens[pos] : 0;
        const int n = len > sub ? (len - sub + (1 << shift) - 1) >> shift : 0;
        const int s0 = first[t], steps = first[t + 1] - s0;
        if (lane == 0) tasks[t] = make_int2(s0, steps);
        lanes[t * 32 + lane] = make_int2(row, n);
        const long long e0 = has ? off[row] + sub : 0;
        for (int j = 0; j < steps; ++j) {
            const long long o = ((long long)s0 + j) * 32 + lane;
            const long long e = e0 + ((long long)j << shift);
            out_idx[o] = j < n ? idx[e] : 0;
            out_val[o] = j < n ? val[e] : 0.0;
        }
    }
}

int grid_for(long long items) {
    return (int)std::max<long long>(1, std::min<long long>((items + 255) / 256, 2 * grid_cap()));
}

}  // namespace

void Store::release() {
    cudaFree(val);  // the one allocation
    *this = Store{};
}

void build(Store& store, const long long* off, const int* idx, const double* val,
           const int* lens, int count, int per_lane, cudaStream_t stream) {
    int *rows = nullptr, *sorted = nullptr, *lens_out = nullptr, *counts = nullptr,
        *steps = nullptr, *first = nullptr;
    void* tmp = nullptr;
    auto free_all = [&] {
        for (void* p : {(void*)rows, (void*)sorted, (void*)lens_out, (void*)counts, (void*)steps,
                        (void*)first, tmp})
            stream_free(p, stream);
    };
    try {
        stream_alloc(&rows, sizeof(int) * count, stream);
        stream_alloc(&sorted, sizeof(int) * count, stream);
        stream_alloc(&lens_out, sizeof(int) * count, stream);
        stream_alloc(&counts, sizeof(int) * 8, stream);
        AMFLS_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * 8, stream));
        count_groups_kernel<<<grid_for(count), 256, 0, stream>>>(lens, count, per_lane, rows, counts);
        AMFLS_LAUNCHED();
        size_t bytes = 0, scan_bytes = 0;
        AMFLS_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, lens, lens_out, rows,
                                                             sorted, count, 0, 31, stream));
        // at most one partly filled task per group beyond count / 1 tasks
        AMFLS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, steps, first,
                                                 (int)std::min(count + 7LL, 0x7fffffffLL), stream));
        bytes = std::max({bytes, scan_bytes, (size_t)1});
        AMFLS_CUDA(cudaMallocAsync(&tmp, bytes, stream));
        AMFLS_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp, bytes, lens, lens_out, rows,
                                                             sorted, count, 0, 31, stream));
        int host[6] = {};
        AMFLS_CUDA(cudaMemcpyAsync(host, counts, sizeof(host), cudaMemcpyDeviceToHost, stream));
        AMFLS_CUDA(cudaStreamSynchronize(stream));
        Groups g{};
        for (int i = 0; i < 6; ++i) {
            const int per = 1 << i;  // rows per task: 32 / (32 >> i)
            g.row_start[i + 1] = g.row_start[i] + host[i];
            g.task_start[i + 1] = g.task_start[i] + (int)((host[i] + (long long)per - 1) / per);
        }
        const int ntasks = g.task_start[6];
        stream_alloc(&steps, sizeof(int) * (ntasks + 1LL), stream);
        stream_alloc(&first, sizeof(int) * (ntasks + 1LL), stream);
        task_steps_kernel<<<grid_for(ntasks + 1), 256, 0, stream>>>(g, lens_out, ntasks, steps);
        AMFLS_LAUNCHED();
        AMFLS_CUDA(cub::DeviceScan::ExclusiveSum(tmp, bytes, steps, first, ntasks + 1, stream));
        int total = 0;
        AMFLS_CUDA(cudaMemcpyAsync(&total, first + ntasks, sizeof(int), cudaMemcpyDeviceToHost,
                                   stream));
        AMFLS_CUDA(cudaStreamSynchronize(stream));
        const size_t entries = 32 * (size_t)std::max(1, total);
        // one allocation: val, lanes, idx and tasks are whole multiples of 128 bytes
        // but for the last
        const size_t slots = (size_t)std::max(1, ntasks);
        AMFLS_CUDA(cudaMalloc(&store.val, (sizeof(double) + sizeof(int)) * entries +
                                              sizeof(int2) * 33 * slots));
        store.lanes = reinterpret_cast<int2*>(store.val + entries);
        store.idx = reinterpret_cast<int*>(store.lanes + 32 * slots);
        store.tasks = reinterpret_cast<int2*>(store.idx + entries);
        fill_kernel<<<grid_for(32LL * ntasks), 256, 0, stream>>>(
            g, sorted, lens_out, first, ntasks, off, idx, val, store.tasks, store.lanes, store.idx,
            store.val);
        AMFLS_LAUNCHED();
        store.side.tasks = store.tasks;
        store.side.lanes = store.lanes;
        store.side.idx = store.idx;
        store.side.val = store.val;
        store.side.ntasks = ntasks;
        for (int i = 0; i < 6; ++i) store.side.group_end[i] = g.task_start[i + 1];
    } catch (...) {
        free_all();
        store.release();
        throw;
    }
    free_all();
}

}  // namespace sliced
}  // namespace amfls_gpu
