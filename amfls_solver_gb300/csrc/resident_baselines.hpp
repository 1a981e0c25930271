// Resident LSQR and LSMR iterations: the iterations up to a checkpoint as one
// cooperative kernel (see resident_baselines.cu).
#pragma once

#include <cuda_runtime.h>

#include "resident_levels.hpp"

namespace amfls_gpu {

// The recurrences' scalars after `pos` half-steps (each iteration is A v, then
// A^T u), with the buffers that hold the vectors there.  LSQR keeps cs and sn of
// its rotation in cbar and sbar, phibar in zetabar.
struct BaselinePosition {
    double alpha, beta, rho, rhobar, cbar, sbar, alphabar, zetabar;
    long long pos;  // twice the iterations: past int for the largest limits
    int u, v;  // u's buffer; v's (and LSQR's w, LSMR's x, h, hbar); LSQR's x goes with u
};

struct BaselineState {
    BaselinePosition now;   // where the kernel stopped
    BaselinePosition back;  // the last unit's start, for a vector that was not finite
    long long target;       // half-steps to stop after
    int handed_back;        // `now` is a step that the general path has to take
    int nonfinite[2];       // a vector was not finite, of half-steps in turn
    int timeout;
    unsigned long long a_ns, at_ns;
};

struct BaselineArgs {
    BaselineState* st;
    sliced::Side a, t;
    int m, n;
    double damp;
    // current and next: [position's index], [1 - index]
    double *u[2], *v[2], *x[2], *w[2], *hbar[2];  // w: LSMR's h; hbar: LSMR alone
    double *left, *right;  // A v - alpha u and A^T u - beta v before normalisation
    double* red;           // 2 * 4 * grid doubles
    unsigned* barrier;     // zero at launch
};

void launch_resident_baseline(const BaselineArgs& args, bool lsmr, int grid, cudaStream_t stream);

}  // namespace amfls_gpu
