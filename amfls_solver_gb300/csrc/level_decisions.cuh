// Device-side decisions of a width-one level: the rank decisions of the right
// and left residuals, the DGKS test and the test whether a level may run.
// Shared by the kernel chain (workspace.cu) and the resident level kernel
// (resident_levels.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "workspace_state.hpp"

namespace amfls_gpu {

constexpr double kEps = 2.220446049250313e-16;

enum Hook { kHookNone = 0, kHookRightPass1 = 1, kHookRightPass2 = 2 };

__device__ inline bool dfinite(double v) { return isfinite(v); }

// Rank decision for the width-one right residual (krylov_workspace.cpp:197-310,
// scalar branch) after its final projection pass.
__device__ inline void decide_right(DevState* st, int m, int n) {
    const double scale = st->right_scale;
    const double after = st->norm_after;
    const int k = st->k;
    const int dim = max(max(1, m), max(n, max(k, 1)));
    const double cutoff = (scale >= 0.0 && dfinite(scale)) ? 64.0 * kEps * dim * scale
                                                           : __builtin_huge_val();
    const bool finite = dfinite(scale) && dfinite(after) && !st->coeff_nonfinite;
    const int max_rank = min(1, st->basis_limit - k);  // combined width is one
    StepAudit& a = st->audit;
    int rank = 0;
    double discarded = after, tracked = 0.0;
    bool positive = false;
    if (!finite) {
        discarded = __builtin_huge_val();
        tracked = __builtin_huge_val();  // tracked prefix = active width = 1
    } else if (max_rank == 0) {
        tracked = after;
    } else if (after > cutoff) {
        rank = 1;
        discarded = 0.0;
    } else if (after > 0.0) {
        positive = true;
        tracked = after;
    }
    a.retained_right_width = rank;
    a.right_rank_cutoff = cutoff;
    a.right_discarded_residual_norm = discarded;
    a.right_active_discarded_residual_norm = tracked;
    a.right_positive_finite_below_cutoff = positive;
    a.right_nonfinite_residual = !finite;
    a.right_rank_loss = rank < max_rank;
    a.right_basis_cap_truncation = max_rank < 1;
    const bool truncated = a.right_rank_loss && positive && tracked > 0.0;
    if (truncated || !finite) st->reliable = 0;
    st->right_rank = rank;
    if (rank == 0) {
        st->left_width = 0;
        st->active_first = st->rows_t;
        st->prev_right_first = k;
        st->prev_right_width = 0;
        st->coupling = 0.0;
        st->level_ok = 0;
        st->go = 0;
        return;
    }
    st->right_factor = after;
    st->inv_right = 1.0 / after;
    st->search_a_calls += 1;
    st->search_a_columns += 1;
}

// Rank decision of the left residual and the T / g update
// (krylov_workspace.cpp:736-830).
__device__ inline void decide_left(DevState* st, int m, int n, double* alpha, double* beta, double* g) {
    const double scale = st->left_scale;
    const double after = st->left_norm;
    const int dim = max(max(1, m), n);
    const double cutoff = (scale >= 0.0 && dfinite(scale)) ? 64.0 * kEps * dim * scale
                                                           : __builtin_huge_val();
    const bool finite = dfinite(scale) && dfinite(after) && dfinite(st->left_coeff);
    const int old_left = st->rows_t;
    const int max_rank = min(min(1, m - old_left), st->basis_limit + 1 - old_left);
    StepAudit& a = st->audit;
    int rank = 0;
    double discarded = after;
    bool positive = false;
    if (!finite) {
        discarded = __builtin_huge_val();
    } else if (max_rank <= 0) {
        // nothing retained, nothing tracked
    } else if (after > cutoff) {
        rank = 1;
        discarded = 0.0;
    } else if (after > 0.0) {
        positive = true;
    }
    a.retained_next_left_width = rank;
    a.left_rank_cutoff = cutoff;
    a.left_discarded_residual_norm = discarded;
    a.left_positive_finite_below_cutoff = positive;
    a.left_nonfinite_residual = !finite;
    a.left_rank_loss = rank < max_rank;
    a.left_basis_cap_truncation = max_rank < 1;
    const bool truncated = (a.left_rank_loss && positive);
    if (truncated || !finite) st->reliable = 0;
    if (!finite) {
        st->level_ok = 0;
        st->go = 0;
        return;
    }
    const int k_old = st->k;
    if (alpha) {  // the writer of T and g (every block of the resident kernel decides)
        alpha[k_old] = st->right_factor + st->left_coeff;  // active coupling + coefficient
        beta[k_old] = rank ? after : 0.0;
    }
    if (rank) {
        st->inv_left = 1.0 / after;
        if (alpha) g[old_left] = st->b_dot * st->inv_left;
    }
    st->left_rank = rank;
    st->k = k_old + 1;
    st->active_first = old_left;
    st->rows_t = old_left + rank;
    st->left_width = rank;
    st->prev_right_first = k_old;
    st->prev_right_width = 1;
    st->coupling = after;
    st->depth += 1;
    st->level_ok = 1;
    st->levels_run += 1;
    a.basis_rank_after = k_old + 1;
    if (!rank) st->go = 0;  // nothing to normalise; the process stops here
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool can_advance_dev(const DevState* st) {
    return st->reliable && (st->left_width + st->pending > 0) && st->k < st->basis_limit &&
           st->depth < st->target_depth;
}

// Start of a level: whether it runs, and its clean audit and flags
// (krylov_workspace.cpp:589-640).
__device__ inline void begin_level(DevState* st) {
    st->body_runs += 1;
    const bool go = can_advance_dev(st) && st->iterations_left > 0;
    st->iterations_left -= 1;
    st->go = go ? 1 : 0;
    if (!go) return;
    st->sub_col = st->prev_right_width > 0 ? st->prev_right_first : 0;
    st->t_mark = global_ns();
    StepAudit a;
    memset(&a, 0, sizeof(a));
    a.left_input_width = st->left_width + st->pending;
    a.basis_rank_before = st->k;
    a.basis_rank_after = st->k;
    st->audit = a;
    st->coupling_eff = (st->prev_right_width > 0 && st->left_width > 0) ? st->coupling : 0.0;
    st->second_pass = 0;
    st->right_rank = 0;
    st->left_rank = 0;
    st->coeff_nonfinite = 0;
    st->sweep_fp64 = 0;
    st->level_ok = 0;
    st->search_at_calls += 1;
    st->search_at_columns += st->left_width + st->pending;
}

// The DGKS test: whether a projection that took a norm from `before` to
// `after` is repeated.
__device__ inline bool dgks_again(double before, double after) {
    return isfinite(before) && isfinite(after) && after < 0.70710678118654757 * before;
}

// The DGKS test and rank decision after the right residual's norm is known
// (the hooks of v_c_kernel).
__device__ inline void finish_right_norm(DevState* st, int hook, double sumsq, int m, int n) {
    st->norm_after = sqrt(sumsq);
    if (hook == kHookRightPass1) {
        st->second_pass = dgks_again(st->norm_before, st->norm_after) ? 1 : 0;
        if (!st->second_pass) decide_right(st, m, n);
    } else if (hook == kHookRightPass2) {
        decide_right(st, m, n);
    }
}

constexpr double kReducedCoeffBound = 1e-3;

// Storage of the basis copy: FP32, or FP16 holding 2^8 v (the entries of a
// unit vector then stay in FP16's normal range down to 2.4e-7; products and
// sums run in FP32 and the results are scaled back by 2^-8, exactly).
template <typename S>
struct RedStore;
// kFlushSteps: steps (of 4 rows per lane) summed in FP32 before a lane's
// partial sums go into FP64.  Each fold costs FP64 instructions (this GPU
// retires two FP64 lanes per SM clock), which an FP16 copy, reading half the
// bytes per element, must amortise over more rows; its own rounding (2^-11)
// dwarfs the longer FP32 sums' (64 terms: about 2^-18).
template <>
struct RedStore<float> {
    static constexpr int kFlushSteps = 4;
    static constexpr float kInvScale = 1.0f;
    __device__ static void load8(const float* p, float v[8]) {
        const float4 a = __ldcs(reinterpret_cast<const float4*>(p));
        const float4 b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    __device__ static float store(double v) { return __double2float_rn(v); }
};
template <>
struct RedStore<__half> {
    static constexpr int kFlushSteps = 16;
    static constexpr float kInvScale = 1.0f / 256.0f;
    __device__ static void load8(const __half* p, float v[8]) {
        const uint4 u = __ldcs(reinterpret_cast<const uint4*>(p));
        const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    }
    __device__ static __half store(double v) { return __float2half_rn(__double2float_rn(v * 256.0)); }
};

}  // namespace amfls_gpu
