// Resident LSQR and LSMR.
//
// On the host path an iteration is 20 launches and four waits for norms
// (20000 x 5000, 10 nonzeros per row: 152 us, of which the products need 8).
// Here the iterations up to the next checkpoint run as one cooperative kernel
// with one block per SM and two grid barriers per iteration, 15 us.  As in
// resident_levels.cu the products gather from the vector before its
// normalisation and scale the finished row sum; every block adds the per-block
// sums itself and takes the recurrences on its own copy of the scalars.  The
// rotations (three square roots in a row for LSMR) run in warp 0 while the other
// warps sum the next product; the vectors that they update are elementwise and
// need no barrier.
//
// Vectors are double buffered and the scalars of the last two units (LSMR: an
// iteration, LSQR: a half-step) are kept, so a step that is out of the ordinary
// is undone and handed to the general path, which then takes it from the same
// vectors: a norm of zero or whose square leaves [1e-200, 1e200], a rotation out
// of range, a vector that is not finite.
#include <algorithm>

#include "common.cuh"
#include "level_decisions.cuh"
#include "resident_baselines.hpp"
#include "resident_grid.cuh"

namespace amfls_gpu {
namespace {

using namespace resident;

struct Shared : GridShared<1> {
    BaselinePosition now, cur, prev;  // cur, prev: starts of this unit and the last one
    double inv;      // 1 / norm of the newest raw vector
    double coef[3];  // of the pending vector updates
    int pending;     // half-step whose vectors are still to be written: 0 none, 1 A, 2 A^T
    int stop, bad;
    unsigned long long mark, ns[2];
};

__device__ __forceinline__ bool plain(double v) { return v > 1e-140 && v < 1e140; }

// a / r and b / r side by side in the lanes
__device__ __forceinline__ void divide_pair(double a, double b, double r, double& x, double& y) {
    const double q = ((threadIdx.x & 31) == 0 ? a : b) / r;
    x = __shfl_sync(0xffffffffu, q, 0);
    y = __shfl_sync(0xffffffffu, q, 1);
}

// The rotations of the half-step that has just ended (warp 0, every lane with
// the same values): `p` moves on and the vector updates' coefficients are
// set; false when a value leaves the range of the plain formulas.
template <bool kLsmr>
__device__ bool rotate(BaselinePosition& p, double damp, double (&coef)[3]) {
    if constexpr (kLsmr) {
        if (p.pos & 1) return true;  // all of it follows the second half-step
        const double dr = sqrt(fma(p.alphabar, p.alphabar, damp * damp));
        const double rho_old = p.rho, rhobar_old = p.rhobar;
        const double rho = sqrt(fma(dr, dr, p.beta * p.beta));
        double c, s;
        divide_pair(dr, p.beta, rho, c, s);
        const double theta_new = s * p.alpha;
        const double theta_bar = p.sbar * rho, rho_temp = p.cbar * rho;
        const double rhobar = sqrt(fma(rho_temp, rho_temp, theta_new * theta_new));
        double cbar, sbar;
        divide_pair(rho_temp, theta_new, rhobar, cbar, sbar);
        const double zeta = cbar * p.zetabar;
        const double hbar_den = rho_old * rhobar_old, sol_den = rho * rhobar;
        const int lane = threadIdx.x & 31;
        const double q = (lane == 0 ? theta_bar * rho : lane == 1 ? zeta : theta_new) /
                         (lane == 0 ? hbar_den : lane == 1 ? sol_den : rho);
#pragma unroll
        for (int i = 0; i < 3; ++i) coef[i] = __shfl_sync(0xffffffffu, q, i);
        p.alphabar = c * p.alpha;
        p.zetabar = -sbar * p.zetabar;
        p.rho = rho, p.rhobar = rhobar, p.cbar = cbar, p.sbar = sbar;
        return plain(dr) && plain(rho) && plain(rhobar) && isfinite(p.alphabar) &&
               isfinite(zeta) && isfinite(p.zetabar) && isfinite(hbar_den) && hbar_den != 0.0 &&
               isfinite(sol_den) && sol_den != 0.0 && isfinite(coef[0]) && isfinite(coef[1]) &&
               isfinite(coef[2]);
    } else if (p.pos & 1) {  // after A v: the update of x
        const double rhobar1 = sqrt(fma(p.rhobar, p.rhobar, damp * damp));
        const double phibar = p.rhobar / rhobar1 * p.zetabar;
        const double rho = sqrt(fma(rhobar1, rhobar1, p.beta * p.beta));
        double cs, sn;
        divide_pair(rhobar1, p.beta, rho, cs, sn);
        const double phi = cs * phibar;
        coef[0] = phi / rho;
        p.zetabar = sn * phibar;
        p.rho = rho, p.cbar = cs, p.sbar = sn;
        return plain(rhobar1) && plain(rho) && isfinite(phi) && isfinite(p.zetabar) &&
               isfinite(coef[0]);
    } else {  // after A^T u: the update of w
        const double theta = p.sbar * p.alpha;
        p.rhobar = -p.cbar * p.alpha;
        coef[0] = theta / p.rho;
        return isfinite(theta) && isfinite(p.rhobar) && isfinite(coef[0]);
    }
}

template <bool kLsmr>
__global__ void __launch_bounds__(kT, 1) resident_baseline_kernel(BaselineArgs a) {
    __shared__ Shared s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grid = gridDim.x;
    // product tasks go to warps 1 .. kW - 1, consecutive ones to different SMs
    const int W = grid * (kW - 1), w = warp > 0 ? (warp - 1) * grid + blockIdx.x : W;
    const bool writer = blockIdx.x == 0;
    const int r0 = (int)((long long)a.n * blockIdx.x / grid);
    const int r1 = (int)((long long)a.n * (blockIdx.x + 1) / grid);
    const int l0 = (int)((long long)a.m * blockIdx.x / grid);
    const int l1 = (int)((long long)a.m * (blockIdx.x + 1) / grid);
    if (tid == 0) {
        s.arrived = 0;
        s.failed = 0;
        s.now = a.st->now;
        s.cur = s.prev = s.now;
        s.inv = 1.0;
        s.pending = s.stop = s.bad = 0;
        s.ns[0] = s.ns[1] = 0;
        s.mark = global_ns();
    }
    __syncthreads();
    const long long target = a.st->target;
    // the rotations of the pending half-step (warp 0)
    auto settle_scalars = [&] {
        BaselinePosition p = s.now;
        double coef[3] = {0.0, 0.0, 0.0};
        const bool ok = rotate<kLsmr>(p, a.damp, coef);
        __syncwarp();
        if (lane == 0) {
            if (!ok) {
                s.bad = 1;
            } else {
                s.now = p;
                s.coef[0] = coef[0], s.coef[1] = coef[1], s.coef[2] = coef[2];
                if (!kLsmr || !(p.pos & 1)) {
                    s.prev = s.cur;
                    s.cur = p;
                }
            }
        }
    };
    // the vectors of the pending half-step, on the block's own rows
    auto commit = [&] {
        const double inv = s.inv, c0 = s.coef[0], c1 = s.coef[1], c2 = s.coef[2];
        const int un = s.now.u, vn = s.now.v;
        bool finite = true;
        if (s.pending == 1) {
            for (int i = l0 + tid; i < l1; i += kT) a.u[un][i] = a.left[i] * inv;
            if constexpr (!kLsmr) {
                for (int i = r0 + tid; i < r1; i += kT) {
                    const double x = fma(c0, a.w[vn][i], a.x[1 - un][i]);
                    a.x[un][i] = x;
                    finite = finite && isfinite(x);
                }
            }
        } else {
            for (int i = r0 + tid; i < r1; i += kT) {
                const double v = a.right[i] * inv, h = a.w[1 - vn][i];
                a.v[vn][i] = v;
                if constexpr (kLsmr) {
                    const double hb = fma(-c0, a.hbar[1 - vn][i], h);
                    const double x = fma(c1, hb, a.x[1 - vn][i]), nh = fma(-c2, h, v);
                    a.hbar[vn][i] = hb;
                    a.x[vn][i] = x;
                    a.w[vn][i] = nh;
                    finite = finite && isfinite(hb) && isfinite(x) && isfinite(nh);
                } else {
                    const double nw = fma(-c0, h, v);
                    a.w[vn][i] = nw;
                    finite = finite && isfinite(nw);
                }
            }
        }
        // the flags take turns: a block may set the next one while another still
        // reads this one behind the barrier
        if (!finite) atomicOr(&a.st->nonfinite[s.now.pos & 1], 1);
    };

    sliced::Walk walk;
    double x0 = 0.0;  // the first task's sum
    if (warp > 0 && s.now.pos < target) {
        const bool even = !(s.now.pos & 1);
        sliced::start_walk(even ? a.a : a.t, walk, w, W);
        x0 = sliced::task_sum(even ? a.a : a.t, walk.cur,
                              even ? a.v[s.now.v] : a.u[s.now.u]);
    }
    __syncthreads();
    while (s.now.pos < target) {
        const bool even = !(s.now.pos & 1);  // A v - alpha u, else A^T u - beta v
        double sq[1] = {0.0};
        {
            const sliced::Side& side = even ? a.a : a.t;
            const double* src = even ? (s.pending ? a.right : a.v[s.now.v])
                                     : (s.pending ? a.left : a.u[s.now.u]);
            const double* sub = even ? a.u[s.now.u] : a.v[s.now.v];
            double* out = even ? a.left : a.right;
            const double inv = s.pending ? s.inv : 1.0;
            const double coef = even ? s.now.alpha : s.now.beta;
            __syncthreads();  // warp 0 changes s.now
            if (warp == 0) {
                if (s.pending) settle_scalars();
            } else if (w < side.ntasks) {
                double x = x0;
                do {
                    if (walk.round > 0) x = sliced::task_sum(side, walk.cur, src);
                    const int row = walk.cur.row;
                    if (row >= 0 && (lane & ((1 << walk.cur.shift) - 1)) == 0) {
                        // rounded as the reference rounds: the product, the
                        // multiple and their difference (a fused one moves the
                        // iterates further from it once orthogonality is lost)
                        const double y = __dsub_rn(__dmul_rn(x, inv), __dmul_rn(coef, sub[row]));
                        out[row] = y;
                        sq[0] = fma(y, y, sq[0]);
                    }
                } while (sliced::next_task(side, walk, w, W));
            }
            __syncthreads();
            if (s.bad) break;
            if (s.pending) commit();
            block_partials(s, sq, min(kW, 1 + (side.ntasks + grid - 1) / grid), a.red, even ? 0 : 1);
        }
        const sliced::Side& next = even ? a.t : a.a;
        if (warp > 0) sliced::start_walk(next, walk, w, W);
        grid_barrier(s, a.barrier);
        if (s.failed) break;
        if (warp == 0) {
            double v[1];
            reduce_slot(a.red, even ? 0 : 1, v);
            const double norm = sqrt(v[0]);
            if (lane == 0) {
                if (writer) {
                    const unsigned long long t = global_ns();
                    s.ns[even ? 0 : 1] += t - s.mark;
                    s.mark = t;
                }
                if (__ldcg(&a.st->nonfinite[s.now.pos & 1])) {
                    s.now = s.prev;
                    s.stop = 1;
                } else if (!(v[0] > 1e-200 && v[0] < 1e200)) {
                    s.now = s.cur;
                    s.stop = 1;
                } else {
                    s.inv = 1.0 / norm;
                    if (even) {
                        s.now.beta = norm;
                        s.now.u ^= 1;
                    } else {
                        s.now.alpha = norm;
                        s.now.v ^= 1;
                    }
                    s.pending = even ? 1 : 2;
                    ++s.now.pos;
                }
            }
        } else {
            x0 = sliced::task_sum(next, walk.cur, even ? a.left : a.right);
        }
        __syncthreads();
        if (s.stop) break;
    }
    __syncthreads();
    const bool finish = !s.stop && !s.bad && !s.failed && s.pending;
    __syncthreads();  // warp 0 may set s.bad from here on
    if (finish) {
        if (warp == 0) settle_scalars();
        __syncthreads();
        if (!s.bad) commit();
    }
    __syncthreads();
    if (writer && tid == 0) {
        a.st->now = s.bad ? s.cur : s.now;
        a.st->back = s.prev;
        a.st->handed_back = s.bad || s.stop;
        a.st->timeout = s.failed;
        a.st->a_ns = s.ns[0];
        a.st->at_ns = s.ns[1];
    }
}

template <bool kLsmr>
void launch(const BaselineArgs& args, int grid, cudaStream_t stream) {
    BaselineArgs copy = args;
    void* params[] = {&copy};
    AMFLS_CUDA(cudaLaunchCooperativeKernel(
        reinterpret_cast<const void*>(resident_baseline_kernel<kLsmr>), dim3(grid), dim3(kT),
        params, 0, stream));
    AMFLS_LAUNCHED();
}

}  // namespace

void launch_resident_baseline(const BaselineArgs& args, bool lsmr, int grid, cudaStream_t stream) {
    if (lsmr) launch<true>(args, grid, stream);
    else launch<false>(args, grid, stream);
}

}  // namespace amfls_gpu
