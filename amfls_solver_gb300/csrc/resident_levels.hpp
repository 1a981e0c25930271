// Resident width-one levels: a whole checkpoint interval as one cooperative
// kernel (see resident_levels.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "device_operator.hpp"
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
    long long longest_row = 0, longest_col = 0;  // nonzeros, of A
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

// A row is one warp's, whatever its length, and the others wait for it at the
// grid barrier: with a dense row or column the kernel chain and the host path
// are faster, whose tiles slice such rows.  What counts is what a product's
// longest row holds beyond a warp's even share of the nonzeros, the two
// products of a level added up: 3 to 5 us per 1000.
inline long long resident_excess(const ResidentOperator& op) {
    const long long share = op.nonzeros / ((long long)sm_count() * (kResidentThreads / 32 - 1));
    const long long a = op.longest_row - share, t = op.longest_col - share;
    return (a > 0 ? a : 0) + (t > 0 ? t : 0);
}
// Excess up to which levels run in the resident kernel.  One column of L entries
// beside 10 or 20 per row, us per level, chain and resident: 60000 x 15000 with
// L = 15000 146 and 118, 30000 146 and 168; 200000 x 50000 (share 2400) 10000 255
// and 204, 30000 254 and 294; 1M x 250k (share 12000) 30000 710 and 664, 100000
// 709 and 1010.  Where both are equal the excess is 18000 to 23500.
constexpr long long kResidentLevelExcess = 18000;
// The same for LSQR and LSMR, whose general path waits for the host in every
// iteration (LSMR, us per iteration): 60000 x 15000 with L = 60000 246 and 224;
// 200000 x 50000 30000 295 and 221, 60000 299 and 357; 1M x 250k 30000 587 and 471,
// 100000 586 and 794.  Equal at 43000 to 66000.
constexpr long long kResidentIterationExcess = 42000;

// Whether the levels of `op` run in the resident kernel.
inline bool resident_levels(const DeviceOperator& op, ResidentOperator* view) {
    return op.resident(view) && resident_excess(*view) <= kResidentLevelExcess;
}
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
