// Resident width-one levels: a whole checkpoint interval as one cooperative
// kernel (see resident_levels.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "sliced_rows.cuh"
#include "workspace_state.hpp"

namespace amfls_gpu {

// What the resident kernel needs of an operator: the sliced rows of A and of
// its transpose, and for [A; root I] the root of the appended rows.
struct ResidentOperator {
    sliced::Side a, t;
    int rows = 0;       // of A
    int cols = 0;
    long long nonzeros = 0;
    bool augmented = false;
    double root = 0.0;  // augmented: rows + i is root * x_i
};

struct ResidentArgs {
    DevState* st;
    sliced::Side a, t;
    int m;           // rows of A
    int ml;          // length of the left vectors (m, or m + n when augmented)
    int n;
    double root;
    const double* b;
    double* u;       // left vector, normalised at the start and the end
    double* y;       // left residual
    double* r;       // right residual
    double* v;       // newest right vector, contiguous
    double* const* panels;
    int npanels;     // panels allocated for the interval
    void* const* shadow;  // reduced copy's panels, or null
    double* alpha;
    double* beta;
    double* g;
    double* red;      // resident_red_doubles(grid)
    double* part;     // resident_part_doubles(grid, panels)
    unsigned* barrier;  // zero at launch
};

// Threads of a block; one block per SM.
constexpr int kResidentThreads = 384;
// Basis columns whose coefficients a block's shared memory holds.
constexpr int kResidentMaxBasis = 10240;

inline long long resident_red_doubles(int grid) { return 6LL * 4 * grid; }
inline long long resident_part_doubles(int grid, long long panels) {
    return (grid + panels + 1) * 32;
}

// Runs levels until st->target_depth or until the process stops; k_max bounds
// the basis at the end.  storage: 0, or the ReducedStorage of the shadow.
void launch_resident_levels(const ResidentArgs& args, int grid, int k_max, int storage,
                            cudaStream_t stream);

// SMs of the current device that resident kernels hold.  Every block of a
// resident kernel waits for the others at its grid barriers, so all of them
// have to be on the GPU at once: a solve leases the SMs of its grid before it
// launches and returns them when the interval has ended.  Leases are granted
// in the order of the requests; each thread holds at most one.
class SmLease {
public:
    SmLease() = default;
    ~SmLease() { release(); }
    SmLease(const SmLease&) = delete;
    SmLease& operator=(const SmLease&) = delete;
    void acquire(int sms);  // blocks the calling thread until they are free
    void release();
    bool held() const { return sms_ > 0; }

private:
    int sms_ = 0;
    int device_ = 0;
};

}  // namespace amfls_gpu
