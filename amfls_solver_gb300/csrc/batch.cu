// Batched AMFLS: many independent least-squares problems solved
// concurrently on one GPU.  No counterpart in the reference (which solves
// one problem per call); each problem is the reference's solve_amfls.
//
// A pool of host worker threads, each with its own non-blocking CUDA
// stream, takes problems from a shared queue ordered by estimated cost
// (largest first, the LPT rule, so the last problems to start are the
// short ones).  The levels of a CSR problem run in the resident level kernel on
// a share of the SMs (sm_shares below), so that up to `workers` problems
// really run side by side: a small problem's level is a chain of latencies
// that leaves most of a whole GPU idle, and its work takes no longer on ten
// SMs than it waits anyway.  Sixteen CSR problems of up to 20000 x 4000, 16
// workers: 337 ms with the level kernels launched from the host, 261 ms with
// the waits of the validation taken out, 128 ms with the shares, 114 ms with
// shares that grow with the basis (Workspace::resident_interval_grid).  Other operators'
// levels are launched from the host when there is more than one worker
// (graphs of different streams ran one at a time: 48 problems, 16 workers,
// 12.5 s against 7.9 s).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <exception>
#include <mutex>
#include <numeric>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "batch.hpp"
#include "common.cuh"
#include "csr_operator.hpp"
#include "resident_levels.hpp"

namespace amfls_gpu {

namespace {

constexpr int kMinShare = 4;
// Resident solves that run side by side: the driver maps streams to
// CUDA_DEVICE_MAX_CONNECTIONS hardware queues, eight unless the process says
// otherwise, and kernels behind a resident one in the same queue wait for it.
// 1500-column problems on 8 SMs each: 8 in 50 ms, 9 in 75 ms, 16 in 171 ms; two
// rounds of eight on 17 SMs take 68 ms.
int resident_streams() {
    const char* v = std::getenv("CUDA_DEVICE_MAX_CONNECTIONS");
    const int n = v ? std::atoi(v) : 0;
    return n >= 1 && n <= 32 ? n : 8;
}

// Work of a problem's level, in FP64 operations of the resident kernel: the
// sweeps of a basis that grows with the columns (n k each, k about an eighth
// of n on average) and the products (a gather costs about two operations).
double cost_estimate(const DeviceOperator& op) {
    ResidentOperator view;
    const double n = op.cols();
    if (op.resident(&view)) return 0.25 * n * n + 4.0 * (double)view.nonzeros;
    if (const auto* csr = dynamic_cast<const CsrOperator*>(&op))
        return 0.25 * n * n + 4.0 * (double)csr->nonzeros();
    return 4.0 * op.rows() * n;
}

// The resident kernels' tables of all problems, before the first solve: their
// allocations would wait for the resident kernels of the others.
void build_tables(const std::vector<BatchItem>& items) {
    cudaStream_t s = nullptr;
    for (const BatchItem& it : items) {
        ResidentOperator view;
        if (!resident_levels(*it.op, &view)) continue;
        if (!s) AMFLS_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        try {
            it.op->resident_tables(&view, s);
        } catch (...) {
            cudaStreamDestroy(s);
            throw;
        }
    }
    if (s) cudaStreamDestroy(s);
}

// SMs of each problem in LPT order (0: it has no resident levels), from the
// batch alone (so that a repeat gives the same sums): of the `at_once` resident
// problems that run from position p on, each takes the part of the SMs that the
// square root of its work is of theirs (which makes the sum of work / SMs
// smallest; in proportion to the work the 16 problems took as long with 8 in
// flight, 128 ms, and 147 instead of 129 ms with 4).  A tenth of the SMs stays
// free for the checkpoints' kernels, which find no room beside a resident block.
std::vector<int> sm_shares(const std::vector<BatchItem>& items, const std::vector<int>& order,
                           int at_once) {
    const int sms = sm_count();
    std::vector<int> at;  // positions with resident levels
    std::vector<double> weight;
    for (int p = 0; p < (int)order.size(); ++p) {
        ResidentOperator view;
        const DeviceOperator& op = *items[order[p]].op;
        if (!resident_levels(op, &view)) continue;
        at.push_back(p);
        weight.push_back(std::sqrt(cost_estimate(op)));
    }
    const int count = (int)at.size();
    std::vector<int> share(order.size(), 0);
    for (int p = 0; p < count; ++p) {
        // the last `at_once` problems run beside each other to the end
        const int first = std::max(0, std::min(p, count - at_once));
        double sum = 0.0;
        for (int q = first; q < std::min(count, first + at_once); ++q) sum += weight[q];
        share[at[p]] = std::clamp((int)(0.9 * sms * weight[p] / sum), kMinShare, sms);
    }
    return share;
}

// The problems in LPT order; position -1: nothing is left for this worker.
class Queue {
public:
    explicit Queue(const std::vector<int>& share) : share_(share), taken_(share.size(), false) {}
    int take(bool resident_too) {
        std::lock_guard<std::mutex> lock(mu_);
        for (int p = 0; p < (int)share_.size(); ++p) {
            if (taken_[p] || (share_[p] > 0 && !resident_too)) continue;
            taken_[p] = true;
            return p;
        }
        return -1;
    }

private:
    const std::vector<int>& share_;
    std::vector<bool> taken_;
    std::mutex mu_;
};

}  // namespace

std::vector<BatchOutcome> solve_amfls_batch(const std::vector<BatchItem>& items, int workers,
                                            double* wall_seconds) {
    const int count = (int)items.size();
    std::vector<BatchOutcome> out(count);
    if (count == 0) {
        if (wall_seconds) *wall_seconds = 0.0;
        return out;
    }
    if (workers <= 0) throw std::invalid_argument("workers must be positive");
    for (const BatchItem& it : items)
        if (it.op == nullptr || it.b == nullptr || it.x == nullptr)
            throw std::invalid_argument("batch problems need an operator, b and a solution buffer");
    {
        // an operator's products use scratch it owns: concurrent solves need one each
        std::vector<const DeviceOperator*> ops;
        for (const BatchItem& it : items) ops.push_back(it.op);
        std::sort(ops.begin(), ops.end());
        if (std::adjacent_find(ops.begin(), ops.end()) != ops.end())
            throw std::invalid_argument("each problem of a batch needs its own operator");
    }
    workers = std::min(workers, count);
    std::vector<int> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return cost_estimate(*items[a].op) > cost_estimate(*items[b].op);
    });
    int device = 0;
    AMFLS_CUDA(cudaGetDevice(&device));
    const auto t0 = std::chrono::steady_clock::now();
    const int at_once = std::min(workers, resident_streams());
    build_tables(items);
    const std::vector<int> share = sm_shares(items, order, at_once);
    // workers beyond `at_once` take the other problems alone, on streams of
    // their own: the resident solves keep to as many streams as run at a time
    workers = std::min(workers, at_once + (int)std::count(share.begin(), share.end(), 0));
    Queue queue(share);
    auto work = [&](int w) {
        cudaStream_t s = nullptr;
        try {
            AMFLS_CUDA(cudaSetDevice(device));
            AMFLS_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        } catch (...) {
            // the remaining problems are left to the other workers
            return;
        }
        for (int k; (k = queue.take(w < at_once)) >= 0;) {
            const int i = order[k];
            BatchOutcome& o = out[i];
            o.worker = w;
            const auto ts = std::chrono::steady_clock::now();
            try {
                SolveOptions opts = items[i].options;
                if (workers > 1) {
                    opts.use_graphs = false;
                    opts.resident_sms = share[k];
                }
                o.result = solve_amfls(*items[i].op, items[i].b, opts, items[i].x, s);
                o.ok = true;
            } catch (const std::exception& e) {
                o.error = e.what();
            } catch (...) {
                o.error = "unknown error";
            }
            o.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - ts).count();
            o.finished = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        }
        cudaStreamDestroy(s);
    };
    std::vector<std::thread> pool;
    pool.reserve(workers);
    for (int w = 0; w < workers; ++w) pool.emplace_back(work, w);
    for (std::thread& t : pool) t.join();
    if (wall_seconds)
        *wall_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    for (int i = 0; i < count; ++i)
        if (!out[i].ok && out[i].error.empty()) out[i].error = "no worker could run the problem";
    return out;
}

}  // namespace amfls_gpu
