// Device block Golub-Kahan workspace (see workspace.hpp for the layout).
//
// Width-one levels of CSR operators run in the resident level kernel
// (resident_levels.cu).  For every other operator, for bases beyond
// kResidentMaxBasis columns and with graphs switched off, one width-one level
// (krylov_workspace.cpp:589-831) is the kernel chain
//   begin        decide on the device whether the level runs (can_advance,
//                depth target); reset the step audit
//   A^T u        fused SpMV^T: r = A^T u - beta v_prev, ||A^T u||, ||r||
//   V^T r        c1: warp tasks (panel, row chunk), chunks added in order by
//                the warp that finishes a panel last
//   r -= V c1    warp tasks (row tile, panel group), with ||r||; the warp
//                that finishes the last tile takes the DGKS decision
//                (second pass only if ||r_after|| < sqrt(1/2) ||r_before||,
//                krylov_workspace.cpp:152-165) and, when no second pass is
//                needed, the rank decision against the cutoff
//                64 eps max(m,n,k,1) ||A^T u|| (krylov_workspace.cpp:63-80)
//   [V^T r, r -= V c2]   only when the device flag asks for it
//   normalise    v = r / ||r|| into V's new column and a contiguous copy
//   A v          fused SpMV: y = A v - ||r|| u, ||A v||, ||y||, u.y
//   left pass    y -= (u.y) u with ||y||, u.y, y.b; DGKS and rank decision,
//                T column (alpha = ||r|| + u.y, beta = ||y||), g = u'.b
//   [left pass]  second DGKS pass when flagged
//   normalise    u' = y / ||y||
// Every kernel reads the device flag `go` and does nothing once the level
// (or an earlier one) stopped, so a whole run of levels up to the next
// checkpoint is enqueued without a host round trip.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <thread>
#include <vector>

#include <cuda_fp16.h>

#include "common.cuh"
#include "level_decisions.cuh"
#include "vector_ops.hpp"
#include "workspace.hpp"

namespace amfls_gpu {

void keep_pool_memory() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    AMFLS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || done[dev]) return;
    cudaMemPool_t pool;
    AMFLS_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    unsigned long long threshold = ~0ULL;
    AMFLS_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold));
    done[dev] = true;
}

HostPage& host_page() {
    struct Owner {
        HostPage page;
        ~Owner() {
            if (page.data) cudaFreeHost(page.data);
        }
    };
    thread_local Owner owner;
    HostPage& page = owner.page;
    if (!page.data) {
        void* p = nullptr;
        AMFLS_CUDA(cudaHostAlloc(&p, kPinnedBytes + 64, cudaHostAllocPortable));
        page.data = static_cast<unsigned char*>(p);
        page.flag = reinterpret_cast<unsigned*>(page.data + kPinnedBytes);
        *page.flag = 0;
        page.seq = 0;
    }
    return page;
}

void wait_flag(const HostPage& page, unsigned seq, cudaStream_t stream) {
    const volatile unsigned* flag = page.flag;
    const auto reached = [&] { return (int)(*flag - seq) >= 0; };
    const auto t0 = std::chrono::steady_clock::now();
    auto checked = t0;
    while (!reached()) {
        const auto now = std::chrono::steady_clock::now();
        if (now - checked > std::chrono::milliseconds(2)) {
            // done without the flag: the kernel failed, or its last write is
            // on its way
            const cudaError_t e = cudaStreamQuery(stream);
            if (e != cudaSuccess && e != cudaErrorNotReady) check_cuda(e, "cudaStreamQuery");
            if (e == cudaSuccess && !reached()) AMFLS_CUDA(cudaStreamSynchronize(stream));
            checked = now;
        }
        if (now - t0 > std::chrono::milliseconds(20))
            std::this_thread::sleep_for(std::chrono::microseconds(20));
        else if (now - t0 > std::chrono::microseconds(100))
            std::this_thread::yield();
    }
    std::atomic_thread_fence(std::memory_order_acquire);
}

void stream_wait(cudaStream_t stream) {
    HostPage& page = host_page();
    copy_out_kernel<<<1, 32, 0, stream>>>(nullptr, nullptr, 0, page.flag, ++page.seq);
    AMFLS_CUDA(cudaGetLastError());
    wait_flag(page, page.seq, stream);
}

namespace {

constexpr int kThreads = 256;
// V^T r by blocks (vt_r_kernel) launches about 16 blocks per SM (panels x
// row chunks); kMaxGemvTargetBlocks bounds it for sizing the partials
inline int gemv_target_blocks() { return 16 * sm_count(); }
constexpr int kMaxGemvTargetBlocks = 16 * 256;

// Tall bases (n rows at least this) keep the block sweeps vt_r_kernel /
// v_c_kernel, which run closest to the FP64 roof there; shorter ones use the
// warp-task sweeps, whose grid does not shrink with n.
constexpr int kWarpSweepMaxRows = 1 << 17;

// Which sweeps a basis of n rows uses; AMFLS_GB300_WARP_SWEEPS=0 / 1 in the
// environment forces the block / warp-task kernels (for measurements).
bool use_warp_sweeps(long long n) {
    const char* v = std::getenv("AMFLS_GB300_WARP_SWEEPS");
    if (v && v[0] == '0') return false;
    if (v && v[0] == '1') return true;
    return n < kWarpSweepMaxRows;
}

__global__ void set_target_kernel(DevState* st, int target_depth, int iterations) {
    if (threadIdx.x != 0) return;
    st->target_depth = target_depth;
    st->iterations_left = iterations;
}

__global__ void level_begin_kernel(DevState* st) {
    if (threadIdx.x == 0) begin_level(st);
}

// after A^T u: scale and norm_before from the fused reduction
__global__ void right_scales_kernel(DevState* st, const RedResult* red, int m, int n) {
    if (threadIdx.x != 0 || !st->go) return;
    st->at_ns += global_ns() - st->t_mark;
    const bool no_projection = st->k == 0;
    st->right_scale = red->nonfinite ? __builtin_nan("") : sqrt(red->sq_t);
    st->norm_before = red->nonfinite ? __builtin_nan("") : sqrt(red->sq_out);
    if (no_projection) {  // empty basis: no pass, the norm is the block's norm
        st->norm_after = st->norm_before;
        decide_right(st, m, n);
    }
}

// c = V^T r, masked to k columns.  grid (panels, chunks); partials [P][C][32].
__global__ void __launch_bounds__(kThreads)
vt_r_kernel(double* const* __restrict__ panels, int n, int chunk_rows,
            const double* __restrict__ r, double* __restrict__ c, double* partials,
            unsigned* panel_tickets, DevState* st, int pass, int only_fp64 = 0) {
    if (!st->go || (pass == 2 && !st->second_pass) || (only_fp64 && !st->sweep_fp64)) return;
    const int k = st->k;  // k == 0: no projection (decided in right_scales_kernel)
    const int p = blockIdx.x, chunk = blockIdx.y, nchunks = gridDim.y;
    if (p * 32 >= k) return;  // panel beyond the current basis
    const double* __restrict__ vp = panels[p];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, rsub = lane >> 2;
    const long long row0 = (long long)chunk * chunk_rows;
    const long long row1 = min((long long)n, row0 + chunk_rows);
    double acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0;
    for (long long base = row0 + warp * 8; base < row1; base += 64) {
        const long long row = base + rsub;
        if (row < row1) {
            const double2* src = reinterpret_cast<const double2*>(vp + row * 32 + q * 8);
            const double2 a0 = __ldg(src), a1 = __ldg(src + 1), a2 = __ldg(src + 2),
                          a3 = __ldg(src + 3);
            const double rv = __ldg(r + row);
            acc[0] = fma(a0.x, rv, acc[0]);
            acc[1] = fma(a0.y, rv, acc[1]);
            acc[2] = fma(a1.x, rv, acc[2]);
            acc[3] = fma(a1.y, rv, acc[3]);
            acc[4] = fma(a2.x, rv, acc[4]);
            acc[5] = fma(a2.y, rv, acc[5]);
            acc[6] = fma(a3.x, rv, acc[6]);
            acc[7] = fma(a3.y, rv, acc[7]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 4);
        acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 8);
        acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
    }
    __shared__ double sm[8][32];
    __shared__ bool last;
    if (lane < 4) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sm[warp][lane * 8 + i] = acc[i];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += sm[w][threadIdx.x];
        partials[((long long)p * nchunks + chunk) * 32 + threadIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(&panel_tickets[p], 1u);
        last = (t == (unsigned)nchunks - 1);
        if (last) panel_tickets[p] = 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int ch = 0; ch < nchunks; ++ch)
            s += partials[((long long)p * nchunks + ch) * 32 + threadIdx.x];
        const int col = p * 32 + threadIdx.x;
        if (col < k) {
            c[col] = s;
            if (!isfinite(s)) st->coeff_nonfinite = 1;
        }
    }
}

// out = r - V c (subtract) or out = V c; 32-row tiles, warps split the
// panels; a block takes tiles blockIdx.x, blockIdx.x + gridDim.x, ... (one
// tile per block when the grid covers them, fewer blocks for launches that
// usually find their guard off).  Sum of squares of out reduced by the last
// block, then `hook`.
// guarded: 0 always runs, 1 runs when the level (and pass) runs, 2 as 1 but
// only when a reduced-basis level redoes its projection in FP64.
__global__ void __launch_bounds__(kThreads)
v_c_kernel(double* const* __restrict__ panels, int n, int k_arg, const double* __restrict__ c,
           const double* r_in, double* out, int subtract, double* partials, unsigned* ticket,
           DevState* st, int hook, int m_rows, int guarded, int pass) {
    if (guarded && (!st->go || (pass == 2 && !st->second_pass) || st->k == 0 ||
                    (guarded == 2 && !st->sweep_fp64)))
        return;
    const int k = k_arg >= 0 ? k_arg : st->k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, rsub = lane >> 2;
    const int P = (k + 31) / 32;
    const long long tiles = ((long long)n + 31) / 32;
    __shared__ double sm[8][32];
    __shared__ double red[32];
    double sq = 0.0;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long row0 = tile * 32;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int p = warp; p < P; p += 8) {
            const double* __restrict__ vp = panels[p];
            double cv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int col = p * 32 + q * 8 + i;
                cv[i] = col < k ? c[col] : 0.0;
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const long long row = row0 + s * 8 + rsub;
                if (row < n) {
                    const double2* src = reinterpret_cast<const double2*>(vp + row * 32 + q * 8);
                    const double2 a0 = __ldg(src), a1 = __ldg(src + 1), a2 = __ldg(src + 2),
                                  a3 = __ldg(src + 3);
                    double t = acc[s];
                    t = fma(a0.x, cv[0], t);
                    t = fma(a0.y, cv[1], t);
                    t = fma(a1.x, cv[2], t);
                    t = fma(a1.y, cv[3], t);
                    t = fma(a2.x, cv[4], t);
                    t = fma(a2.y, cv[5], t);
                    t = fma(a3.x, cv[6], t);
                    t = fma(a3.y, cv[7], t);
                    acc[s] = t;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 1);
            acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 2);
        }
        if (q == 0) {
#pragma unroll
            for (int s = 0; s < 4; ++s) sm[warp][s * 8 + rsub] = acc[s];
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const long long row = row0 + threadIdx.x;
            double y = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) y += sm[w][threadIdx.x];
            if (row < n) {
                const double o = subtract ? r_in[row] - y : y;
                out[row] = o;
                sq = fma(o, o, sq);
            }
        }
        __syncthreads();  // sm is reused by the next tile
    }
    if (hook == kHookNone) return;
    const double bs = block_sum(sq, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (arrive_last(ticket, gridDim.x)) {
        double a = 0.0;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) a += partials[b];
        a = block_sum(a, red);
        if (threadIdx.x == 0) {
            st->norm_after = sqrt(a);
            if (hook == kHookRightPass1) {
                const double before = st->norm_before, after = st->norm_after;
                const bool again = isfinite(before) && isfinite(after) &&
                                   after < 0.70710678118654757 * before;
                st->second_pass = again ? 1 : 0;
                if (!again) decide_right(st, m_rows, n);
            } else {
                decide_right(st, m_rows, n);
            }
        }
    }
}

// ----------------------------------------------------------------------------
// Reduced-basis sweeps: width-one levels that keep a reduced copy V~ of V
// (FP32, or FP16 holding 2^8 v; see RedStore) run their first projection
// pass on it,
//   c  = V~^T r~          r~ = fl32(r); FP32 products, FP32 sums over runs of
//                         16 (FP32 copy) or 64 (FP16) rows per lane, FP64
//                         above that
//   r <- r - fl64(V~ c~)  c~ = fl32(c); FP32 products and sums, the
//                         subtraction in FP64
// At width one the recurrence has already removed the previous column in
// FP64 (the fused A^T u - beta v product), so the pass-one coefficients only
// measure the loss of orthogonality of r against V.  Rounding V to the copy
// (unit roundoff u: 2^-24 FP32, 2^-11 FP16) and r to FP32 perturbs each
// coefficient by about u ||r|| / sqrt(n_eff) (n_eff the rows the vectors
// spread over), which is the level of orthogonality V keeps instead of
// FP64's; the sum V~ c~ perturbs r itself by about u ||V c|| (at most
// 5e-7 ||r|| for FP16 while ||c|| <= kReducedCoeffBound ||r||).  A level
// whose coefficients exceed that bound (or are not finite) redoes the pass
// with the FP64 kernels, and the DGKS second pass is always FP64, so FP64
// stays on the recurrence, the correction of large components, the norms and
// every rank decision.  The sweeps then read 4 or 2 bytes per basis element
// on the FP32 pipe (HBM-bound) instead of 8 bytes on the FP64 pipe (two FMA
// lanes per SM clock on this GPU).
// The orthogonality this keeps suits the restart cycles of the mixed form,
// whose corrections need a few digits each: with one-sided
// reorthogonalisation the left basis U inherits V's orthogonality level
// amplified by about cond(A), so a single solve of an ill-conditioned
// problem to FP64 accuracy stalls on it (the certificate then reports the
// failure; it never certifies a wrong x).
// r~ = fl32(r) for the reduced pass (only when the level projects).
__global__ void round_residual_kernel(const double* __restrict__ r, float* __restrict__ r32, int n,
                                      const DevState* st) {
    if (!st->go || st->k == 0) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        r32[i] = __double2float_rn(r[i]);
}

// Row chunks per panel of vt_r32_kernel on `grid` blocks: about four
// (panel, chunk) tasks per block, at least 256 rows per chunk.
__host__ __device__ inline int reduced_chunks(long long n, int panels, int grid) {
    const long long want = (4LL * grid + panels - 1) / panels;
    const long long most = (n + 255) / 256;
    return (int)(want < 1 ? 1 : (want < most ? want : (most < 1 ? 1 : most)));
}

// Partial-sum doubles vt_r32_kernel needs for up to `panels` panels.
inline long long reduced_part_doubles(int grid, long long panels) {
    return (4LL * grid + panels + 1) * 32;
}

// c = V~^T r~ over the (panel, row chunk) tasks of the current basis, taken
// by the blocks in a fixed round robin.  The chunks of a panel are added in
// chunk order by the block that finishes the panel last; the block that
// finishes the last panel adds the panels' sums of c^2 in panel order and
// decides whether the level redoes the pass in FP64.  Deterministic for a
// fixed grid.
template <typename S>
__global__ void __launch_bounds__(kThreads)
vt_r32_kernel(const S* const* __restrict__ panels, int n, const float* __restrict__ r,
              double* __restrict__ c, float* __restrict__ c32, double* part, double* panel_sq,
              unsigned* panel_tickets, unsigned* all_ticket, DevState* st) {
    if (!st->go) return;
    const int k = st->k;
    if (k == 0) return;
    const int P = (k + 31) / 32;
    const int chunks = reduced_chunks(n, P, gridDim.x);
    const long long chunk_rows = ((long long)n + chunks - 1) / chunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, rsub = lane >> 2;
    __shared__ double sm[8][32];
    __shared__ int last;
    for (int t = blockIdx.x; t < P * chunks; t += gridDim.x) {
        const int p = t / chunks, chunk = t - p * chunks;
        const S* __restrict__ vp = panels[p];
        const long long row0 = (long long)chunk * chunk_rows;
        const long long row1 = min((long long)n, row0 + chunk_rows);
        double acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.0;
        // a warp covers 32 rows per step (rows base + 8j + rsub), a block 256
        long long base = row0 + warp * 32;
        while (base < row1) {
            float s8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) s8[i] = 0.f;
            for (int step = 0; step < RedStore<S>::kFlushSteps && base < row1;
                 ++step, base += 256) {
                float a[4][8];
                float rv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const long long row = base + j * 8 + rsub;
                    if (row < row1) {
                        RedStore<S>::load8(vp + row * 32 + q * 8, a[j]);
                        rv[j] = __ldg(r + row);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) a[j][i] = 0.f;
                        rv[j] = 0.f;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) s8[i] = fmaf(a[j][i], rv[j], s8[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] += (double)s8[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 4);
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 8);
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
        }
        if (lane < 4) {
#pragma unroll
            for (int i = 0; i < 8; ++i) sm[warp][lane * 8 + i] = acc[i];
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) v += sm[w][threadIdx.x];
            part[((long long)p * chunks + chunk) * 32 + threadIdx.x] = v;
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned tk = atomicAdd(&panel_tickets[p], 1u);
            last = tk == (unsigned)chunks - 1;
            if (last) panel_tickets[p] = 0u;
        }
        __syncthreads();
        if (last && threadIdx.x < 32) {  // warp 0 closes the panel
            __threadfence();
            double v = 0.0;
            for (int ch = 0; ch < chunks; ++ch)
                v += __ldcg(&part[((long long)p * chunks + ch) * 32 + threadIdx.x]);
            v *= (double)RedStore<S>::kInvScale;  // exact: a power of two
            const int col = p * 32 + threadIdx.x;
            double sq = 0.0;
            if (col < k) {
                c[col] = v;
                c32[col] = __double2float_rn(v);
                sq = v * v;
            }
            sq = warp_sum(sq);
            if (threadIdx.x == 0) {
                panel_sq[p] = sq;
                __threadfence();
                const unsigned a = atomicAdd(all_ticket, 1u);
                if (a == (unsigned)P - 1) {
                    *all_ticket = 0u;
                    __threadfence();
                    double tot = 0.0;
                    for (int pp = 0; pp < P; ++pp) tot += __ldcg(&panel_sq[pp]);
                    const double before = st->norm_before;
                    const double bound = kReducedCoeffBound * before;
                    const bool redo = !(isfinite(tot) && isfinite(before)) || tot > bound * bound;
                    st->sweep_fp64 = redo ? 1 : 0;
                    st->reduced_levels += 1;
                    if (redo) st->reduced_fallbacks += 1;
                }
            }
        }
        __syncthreads();  // sm and `last` are reused by the next task
    }
}

// r <- r - fl64(V~ c~) with ||r||^2 and the DGKS decision of the first pass
// (as v_c_kernel's kHookRightPass1); 32 rows per block, warps split the
// panels.  Skipped when the level redoes the pass in FP64.
template <typename S>
__global__ void __launch_bounds__(kThreads)
v_c32_kernel(const S* const* __restrict__ panels, int n, const float* __restrict__ c,
             double* r, double* partials, unsigned* ticket, DevState* st, int m_rows) {
    if (!st->go || st->k == 0 || st->sweep_fp64) return;
    const int k = st->k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, rsub = lane >> 2;
    const long long row0 = (long long)blockIdx.x * 32;
    const int P = (k + 31) / 32;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int p = warp; p < P; p += 8) {
        const S* __restrict__ vp = panels[p];
        float cv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int col = p * 32 + q * 8 + i;
            cv[i] = col < k ? c[col] : 0.f;
        }
        float a[4][8];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const long long row = row0 + s * 8 + rsub;
            if (row < n) {
                RedStore<S>::load8(vp + row * 32 + q * 8, a[s]);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) a[s][i] = 0.f;
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            float t = acc[s];
#pragma unroll
            for (int i = 0; i < 8; ++i) t = fmaf(a[s][i], cv[i], t);
            acc[s] = t;
        }
    }
    // V~ c~ is small (the pass-one coefficients are): its cross-lane and
    // cross-warp sums stay in FP32, only the subtraction from r is FP64
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 1);
        acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 2);
    }
    __shared__ float sm[8][32];
    __shared__ double red[32];
    if (q == 0) {
#pragma unroll
        for (int s = 0; s < 4; ++s) sm[warp][s * 8 + rsub] = acc[s];
    }
    __syncthreads();
    double sq = 0.0;
    if (threadIdx.x < 32) {
        const long long row = row0 + threadIdx.x;
        float y32 = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) y32 += sm[w][threadIdx.x];
        const double y = (double)y32 * (double)RedStore<S>::kInvScale;
        if (row < n) {
            const double o = r[row] - y;
            r[row] = o;
            sq = o * o;
        }
    }
    const double bs = block_sum(sq, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    if (arrive_last(ticket, gridDim.x)) {
        double a = 0.0;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) a += partials[b];
        a = block_sum(a, red);
        if (threadIdx.x == 0) {
            st->norm_after = sqrt(a);
            const double before = st->norm_before, after = st->norm_after;
            const bool again = isfinite(before) && isfinite(after) &&
                               after < 0.70710678118654757 * before;
            st->second_pass = again ? 1 : 0;
            if (!again) decide_right(st, m_rows, n);
        }
    }
}

// Blocks of vt_r32_kernel: as many as are resident at once.
int reduced_sweep_grid() {
    static int cached[64] = {};
    int dev = 0;
    AMFLS_CUDA(cudaGetDevice(&dev));
    const int slot = dev >= 0 && dev < 64 ? dev : 0;
    int g = __atomic_load_n(&cached[slot], __ATOMIC_RELAXED);
    if (g == 0) {  // concurrent first callers compute the same value
        int a = 0;
        int b = 0;
        AMFLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, vt_r32_kernel<float>,
                                                                 kThreads, 0));
        AMFLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, vt_r32_kernel<__half>,
                                                                 kThreads, 0));
        a = std::min(a, b);
        g = std::max(1, a) * sm_count();
        __atomic_store_n(&cached[slot], g, __ATOMIC_RELAXED);
    }
    return g;
}

// ----------------------------------------------------------------------------
// Basis sweeps of the width-one levels as warp tasks.  Every V element costs
// one FP64 FMA and this GPU retires two lanes' FP64 FMAs per SM clock, so a
// sweep is bound by the FP64 pipe (about 5 TB/s of V), not by HBM; the layout
// keeps FP64 instructions to the FMAs themselves:
//   * V^T r: a warp task is (panel p, chunk of rows); lane l owns column
//     p*32 + l and sums V[row][l] r[row] down the chunk as one FMA chain (a
//     warp load reads one whole 256-byte panel row); the chunks of a panel
//     are added in chunk order by the warp that finishes the panel last
//     (atomic ticket per panel);
//   * r - V c: a warp task is (tile of 32 rows, group of panels); lane l owns
//     row t*32 + l and sums V[row][col] c[col] along the row as one FMA
//     chain; a tile's groups are added in group order by the warp that
//     finishes the tile last, which also writes the tile's sum of squares;
//     the warp that finishes the last tile adds those in tile order and
//     takes the DGKS decision.
// Tasks are dealt to warps in contiguous balanced ranges, and every sum runs
// in an order fixed by (n, k, grid), so results are deterministic.
constexpr int kSweepTargetTasksPerWarp = 8;

struct SweepShape {
    int P;       // panels in use
    int chunks;  // V^T r: row chunks per panel
    int chunk_rows;
    int T;       // r - V c: row tiles
    int G;       // r - V c: panel groups per tile
    int Pg;      // panels per group
};

__device__ inline SweepShape sweep_shape(int n, int k, int warps) {
    SweepShape sh;
    sh.P = (k + 31) / 32;
    const long long target = (long long)kSweepTargetTasksPerWarp * warps;
    int chunks = sh.P > 0 ? (int)min((target + sh.P - 1) / sh.P, ((long long)n + 127) / 128) : 1;
    chunks = max(1, chunks);
    int rows = (int)(((long long)n + chunks - 1) / chunks);
    rows = (rows + 31) / 32 * 32;
    sh.chunk_rows = rows;
    sh.chunks = (n + rows - 1) / rows;
    sh.T = (n + 31) / 32;
    const int gmax = max(1, sh.P / 4);  // at least four panels per task
    int G = (int)min(max(1LL, (target + sh.T - 1) / sh.T), (long long)gmax);
    sh.Pg = sh.P > 0 ? (sh.P + G - 1) / G : 1;
    sh.G = sh.P > 0 ? (sh.P + sh.Pg - 1) / sh.Pg : 1;
    return sh;
}

// the contiguous range of tasks of warp w among W warps
__device__ inline void warp_range(long long tasks, int w, int W, long long& t0, long long& t1) {
    t0 = tasks * w / W;
    t1 = tasks * (w + 1) / W;
}

// the warp that takes the last ticket: sum `count` partials spaced `stride`
// apart, in index order, with eight loads in flight (L2 reads; the writers
// were other SMs)
__device__ inline double ordered_sum(const double* p, int count, long long stride) {
    double s = 0.0;
    int j = 0;
    for (; j + 8 <= count; j += 8) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldcg(p + (long long)(j + u) * stride);
#pragma unroll
        for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; j < count; ++j) s += __ldcg(p + (long long)j * stride);
    return s;
}

__global__ void __launch_bounds__(kThreads)
sweep_vt_kernel(double* const* __restrict__ panels, int n, const double* __restrict__ r,
                double* __restrict__ c, double* __restrict__ part, unsigned* panel_tickets,
                DevState* st, int pass) {
    if (!st->go || (pass == 2 && !st->second_pass)) return;
    const int k = st->k;
    const int lane = threadIdx.x & 31;
    const int W = gridDim.x * (blockDim.x >> 5);
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const SweepShape sh = sweep_shape(n, k, W);
    long long t0, t1;
    warp_range((long long)sh.P * sh.chunks, w, W, t0, t1);
    for (long long t = t0; t < t1; ++t) {
        const int p = (int)(t / sh.chunks), ch = (int)(t - (long long)p * sh.chunks);
        const double* __restrict__ vp = panels[p] + lane;
        const int row0 = ch * sh.chunk_rows, row1 = min(n, row0 + sh.chunk_rows);
        double acc = 0.0;
        for (int base = row0; base < row1; base += 32) {
            const int cnt = min(32, row1 - base);
            const double rv = lane < cnt ? __ldg(r + base + lane) : 0.0;
            if (cnt == 32) {
#pragma unroll
                for (int j0 = 0; j0 < 32; j0 += 16) {
                    double v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __ldg(vp + (long long)(base + j0 + j) * 32);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc = fma(v[j], __shfl_sync(0xffffffffu, rv, j0 + j), acc);
                }
            } else {
                for (int j = 0; j < cnt; ++j)
                    acc = fma(__ldg(vp + (long long)(base + j) * 32),
                              __shfl_sync(0xffffffffu, rv, j), acc);
            }
        }
        part[((long long)p * sh.chunks + ch) * 32 + lane] = acc;
        __threadfence();
        __syncwarp();
        unsigned ticket = 0;
        if (lane == 0) ticket = atomicAdd(&panel_tickets[p], 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket != (unsigned)sh.chunks - 1) continue;
        __threadfence();
        const double s = ordered_sum(part + (long long)p * sh.chunks * 32 + lane, sh.chunks, 32);
        const int col = p * 32 + lane;
        if (col < k) {
            c[col] = s;
            if (!isfinite(s)) st->coeff_nonfinite = 1;
        }
        if (lane == 0) panel_tickets[p] = 0u;
    }
}

// out = r_in - V c (subtract) or V c over the current basis, its sum of
// squares, then `hook`.
__global__ void __launch_bounds__(kThreads)
sweep_vc_kernel(double* const* __restrict__ panels, int n, const double* __restrict__ c,
                const double* r_in, double* out, int subtract, double* __restrict__ part,
                double* __restrict__ tile_sq, unsigned* tile_tickets, unsigned* done, DevState* st,
                int hook, int m_rows, int pass) {
    if (!st->go || (pass == 2 && !st->second_pass) || st->k == 0) return;
    const int k = st->k;
    const int lane = threadIdx.x & 31;
    const int W = gridDim.x * (blockDim.x >> 5);
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const SweepShape sh = sweep_shape(n, k, W);
    long long t0, t1;
    warp_range((long long)sh.T * sh.G, w, W, t0, t1);
    for (long long t = t0; t < t1; ++t) {
        const int tile = (int)(t / sh.G), g = (int)(t - (long long)tile * sh.G);
        const int row = tile * 32 + lane;
        const int p0 = g * sh.Pg, p1 = min(sh.P, p0 + sh.Pg);
        double acc = 0.0;
        if (row < n) {
            for (int p = p0; p < p1; ++p) {
                const double2* __restrict__ src =
                    reinterpret_cast<const double2*>(panels[p] + (long long)row * 32);
                const double* cp = c + p * 32;
                const int valid = min(32, k - p * 32);
                double2 v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __ldg(src + j);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const double c0 = 2 * j < valid ? cp[2 * j] : 0.0;
                    const double c1 = 2 * j + 1 < valid ? cp[2 * j + 1] : 0.0;
                    acc = fma(v[j].x, c0, acc);
                    acc = fma(v[j].y, c1, acc);
                }
            }
        }
        double y = acc;
        if (sh.G > 1) {
            part[((long long)tile * sh.G + g) * 32 + lane] = acc;
            __threadfence();
            __syncwarp();
            unsigned ticket = 0;
            if (lane == 0) ticket = atomicAdd(&tile_tickets[tile], 1u);
            ticket = __shfl_sync(0xffffffffu, ticket, 0);
            if (ticket != (unsigned)sh.G - 1) continue;
            __threadfence();
            y = ordered_sum(part + (long long)tile * sh.G * 32 + lane, sh.G, 32);
            if (lane == 0) tile_tickets[tile] = 0u;
        }
        double sq = 0.0;
        if (row < n) {
            const double o = subtract ? r_in[row] - y : y;
            out[row] = o;
            sq = o * o;
        }
        if (hook == kHookNone) continue;
        sq = warp_sum(sq);
        if (lane == 0) tile_sq[tile] = sq;
        __threadfence();
        __syncwarp();
        unsigned fin = 0;
        if (lane == 0) fin = atomicAdd(done, 1u);
        fin = __shfl_sync(0xffffffffu, fin, 0);
        if (fin != (unsigned)sh.T - 1) continue;
        __threadfence();
        double a = 0.0;
        for (int j = lane; j < sh.T; j += 32) a += __ldcg(tile_sq + j);
        a = warp_sum(a);
        if (lane == 0) {
            *done = 0u;
            finish_right_norm(st, hook, a, m_rows, n);
        }
    }
}

// Grid of the sweep kernels: every block resident at once (so the balanced
// task ranges are balanced per SM), set up once per device.
int sweep_grid() {
    // AMFLS_GB300_SWEEP_BLOCKS (measurements): a fixed grid instead
    if (const char* v = std::getenv("AMFLS_GB300_SWEEP_BLOCKS")) {
        const int g = std::atoi(v);
        if (g > 0) return g;
    }
    static int cached[64] = {};
    int dev = 0;
    AMFLS_CUDA(cudaGetDevice(&dev));
    const int slot = dev >= 0 && dev < 64 ? dev : 0;
    int g = __atomic_load_n(&cached[slot], __ATOMIC_RELAXED);
    if (g == 0) {
        int a = 0, b = 0;
        AMFLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, sweep_vt_kernel, kThreads, 0));
        AMFLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, sweep_vc_kernel, kThreads, 0));
        g = std::max(1, std::min(a, b)) * sm_count();
        __atomic_store_n(&cached[slot], g, __ATOMIC_RELAXED);
    }
    return g;
}

// Partial-sum doubles the sweeps need for n rows and up to `panels` panels
// on a grid of `grid` blocks (the task bounds of sweep_shape).
long long sweep_part_doubles(int n, long long panels, int grid) {
    const long long W = (long long)grid * (kThreads / 32);
    const long long tiles = (n + 31) / 32;
    return (kSweepTargetTasksPerWarp * W + std::max(panels, tiles) + 1) * 32;
}

// v = r / ||r|| into V's new column (and the reduced copy's, when kept) and a
// contiguous copy.
template <typename S = float>
__global__ void normalize_right_kernel(const double* r, int n, double* const* panels,
                                       double* vnew, DevState* st,
                                       S* const* shadow = nullptr) {
    if (!st->go || !st->right_rank) return;
    const double inv = st->inv_right;
    const int k = st->k;
    double* vcol = panels[k >> 5] + (k & 31);
    S* vcol_s = shadow ? shadow[k >> 5] + (k & 31) : nullptr;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->t_mark = global_ns();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double v = r[i] * inv;
        vcol[i * 32] = v;
        vnew[i] = v;
        if (vcol_s) vcol_s[i * 32] = RedStore<S>::store(v);
    }
}

// Left DGKS pass: y -= c u with reductions ||y||^2, u.y, y.b.
__global__ void __launch_bounds__(kThreads)
left_pass_kernel(double* y, const double* u, const double* b, int m, const RedResult* spmv_red,
                 double* partials, unsigned* ticket, DevState* st, int pass, int n_cols,
                 double* alpha, double* beta, double* g) {
    if (!st->go || (pass == 2 && !st->second_pass)) return;
    if (pass == 1 && blockIdx.x == 0 && threadIdx.x == 0) st->a_ns += global_ns() - st->t_mark;
    const double c = pass == 1 ? spmv_red->dot : st->pass_coeff;
    double sq = 0.0, du = 0.0, db = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m;
         i += (long long)gridDim.x * blockDim.x) {
        const double ui = u[i];
        const double v = y[i] - c * ui;
        y[i] = v;
        sq = fma(v, v, sq);
        du = fma(v, ui, du);
        db = fma(v, b[i], db);
    }
    __shared__ double red[32];
    const double s0 = block_sum(sq, red);
    const double s1 = block_sum(du, red);
    const double s2 = block_sum(db, red);
    if (threadIdx.x == 0) {
        partials[3 * blockIdx.x] = s0;
        partials[3 * blockIdx.x + 1] = s1;
        partials[3 * blockIdx.x + 2] = s2;
    }
    if (!arrive_last(ticket, gridDim.x)) return;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (unsigned blk = threadIdx.x; blk < gridDim.x; blk += blockDim.x) {
        a0 += partials[3 * blk];
        a1 += partials[3 * blk + 1];
        a2 += partials[3 * blk + 2];
    }
    a0 = block_sum(a0, red);
    a1 = block_sum(a1, red);
    a2 = block_sum(a2, red);
    if (threadIdx.x != 0) return;
    const double after = sqrt(a0);
    st->b_dot = a2;
    if (pass == 1) {
        st->left_scale = spmv_red->nonfinite ? __builtin_nan("") : sqrt(spmv_red->sq_t);
        st->norm_before = spmv_red->nonfinite ? __builtin_nan("") : sqrt(spmv_red->sq_out);
        st->left_coeff = c;
        st->left_norm = after;
        st->pass_coeff = a1;
        const double before = st->norm_before;
        const bool again = isfinite(before) && isfinite(after) &&
                           after < 0.70710678118654757 * before;
        st->second_pass = again ? 1 : 0;
        if (!again) decide_left(st, m, n_cols, alpha, beta, g);
    } else {
        st->left_coeff += c;
        st->left_norm = after;
        decide_left(st, m, n_cols, alpha, beta, g);
    }
}

__global__ void normalize_left_kernel(const double* y, double* u, int m, const DevState* st) {
    if (!st->go || !st->left_rank) return;
    const double inv = st->inv_left;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m;
         i += (long long)gridDim.x * blockDim.x)
        u[i] = y[i] * inv;
}

// Loop control of the captured level: continue while the next level can run.
__global__ void level_end_kernel(DevState* st, cudaGraphConditionalHandle handle) {
    if (threadIdx.x != 0) return;
    const bool more = st->go && can_advance_dev(st) && st->iterations_left > 0;
    cudaGraphSetConditional(handle, more ? 1u : 0u);
}

__global__ void scale_copy_kernel(const double* src, double* dst, long long n, double s) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i] * s;
}

// Incremental Givens QR of the lower-bidiagonal T, with sqrt(lambda) I rows
// folded in by one extra rotation per column (the damped LSQR recurrence of
// Paige and Saunders), then back substitution for y.  qr = [rho | theta |
// phi | y] (4 x cap); state = [c, s, phibar, processed, largest row sum of R,
// flags, |z|, ||z||^2] (row sum and z belong to the rank estimate).
//
// What bounds it: dependent FP64 operations of 64 clocks and more, one column
// after the other (one thread doing everything took 6 us per new column and
// 0.4 us per column of the back substitution: 8.6 ms of a 79 ms solve with
// 1368 levels and 21 evaluations).  Only what a column needs of its neighbour
// stays in order, one or two operations; square roots and quotients are formed
// for a tile of columns at once:
//   q_j = rhobar_j^2:  q_{j+1} = alpha_{j+1}^2 (q_j + lambda) / (q_j + lambda + beta_j^2),
//     every term positive, kept as a ratio X / Y so that no division is in the
//     chain (rescaled by a power of two every eight columns); for lambda = 0 as
//     1 / q_{j+1} = 1 / alpha_{j+1}^2 + (beta_j / alpha_{j+1})^2 / q_j;
//   phibar_{j+1} = (-s_j c1_j) phibar_j + c_j g_{j+1}   (c1: damping rotation);
//   y_j = phi_j / rho_j - (theta_{j+1} / rho_j) y_{j+1};
//   |z_j| = 1 / |rho_j| + |theta_j / rho_j| |z_{j-1}|.
// rhobar takes the sign of alpha's product so far (a damping rotation makes it
// positive first).  Tiles with an entry outside 1e-15 .. 1e15 (a zero beta
// apart) could leave FP64's range in the ratio, and for lambda = 0 tiles whose 1 / q
// passes 1e300 have left it: they are rotated one by one.
constexpr int kProjThreads = 128;
constexpr int kProjTile = 512;

__device__ inline bool ratio_safe(double v) {
    const double a = fabs(v);
    return a > 1e-15 && a < 1e15;
}

__global__ void __launch_bounds__(kProjThreads)
projected_solve_kernel(const double* alpha, const double* beta, const double* g, int k, int rows_t,
                       double lambda, double* qr, int cap, double* state, double rcond) {
    __shared__ double X[kProjTile], Y[kProjTile], A[kProjTile], B[kProjTile];
    __shared__ signed char negative[kProjTile];
    __shared__ double c_s, s_s, phibar_s, zmag_s, red[32];
    __shared__ int flags_s;
    const int tid = threadIdx.x;
    double* rho = qr;
    double* theta = qr + cap;
    double* phi = qr + 2 * (long long)cap;
    double* y = qr + 3 * (long long)cap;
    const int done = (int)state[3];
    double rmax = done > 0 ? state[4] : 0.0, zsq = 0.0;
    if (tid == 0) {
        c_s = done > 0 ? state[0] : 1.0;
        s_s = done > 0 ? state[1] : 0.0;
        phibar_s = done > 0 ? state[2] : g[0];
        zmag_s = done > 0 ? state[6] : 0.0;
        zsq = done > 0 ? state[7] : 0.0;
        flags_s = 0;
    }
    __syncthreads();
    for (int j0 = done; j0 < k; j0 += kProjTile) {
        const int nt = min(kProjTile, k - j0);
        // rhobar of the tile's first column before damping
        const double rhobar0 = c_s * alpha[j0];
        int unsafe = tid == 0 && (!ratio_safe(rhobar0) ||
                                  (lambda > 0.0 && !(lambda > 1e-30 && lambda < 1e30)));
        for (int i = tid; i < nt; i += kProjThreads) {
            const int j = j0 + i;
            const double b = j + 1 < rows_t ? beta[j] : 0.0;
            const double an = i + 1 < nt ? alpha[j + 1] : 1.0;
            if (!ratio_safe(an) || !(b == 0.0 || ratio_safe(b))) unsafe = 1;
            const double b2 = b * b, a2 = an * an;
            A[i] = lambda > 0.0 ? lambda + b2 : b2 / a2;
            B[i] = lambda > 0.0 ? a2 : 1.0 / a2;
            negative[i] = alpha[j] < 0.0 ? 1 : 0;
        }
        bool chained = !__syncthreads_or(unsafe);
        if (chained) {
            if (tid == 0) {  // the chain of q
                if (lambda > 0.0) {
                    double x = rhobar0 * rhobar0, w = 1.0;
                    for (int i0 = 0; i0 < nt; i0 += 8) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            if (i0 + u < nt) {
                                X[i0 + u] = x;
                                Y[i0 + u] = w;
                                const double nx = B[i0 + u] * fma(lambda, w, x);
                                w = fma(A[i0 + u], w, x);
                                x = nx;
                            }
                        }
                        // both by 2^-exponent(w), exactly
                        const int e = (int)((__double_as_longlong(w) >> 52) & 0x7ff);
                        const double f = __longlong_as_double((long long)(2046 - e) << 52);
                        x *= f;
                        w *= f;
                    }
                } else {
                    double p = 1.0 / (rhobar0 * rhobar0);
#pragma unroll 8
                    for (int i = 0; i < nt; ++i) {
                        X[i] = p;
                        p = fma(A[i], p, B[i]);
                    }
                }
            } else if (tid == 32) {  // signs of rhobar
                int neg = rhobar0 < 0.0 ? 1 : 0;
                negative[0] = (signed char)neg;
                if (!(lambda > 0.0))
                    for (int i = 1; i < nt; ++i) {
                        neg ^= negative[i];
                        negative[i] = (signed char)neg;
                    }
            }
            // 1 / q of columns whose beta exceeds alpha again and again grows past
            // FP64's range: then rhobar, its root, is taken column by column
            int spilled = 0;
            __syncthreads();
            if (!(lambda > 0.0))
                for (int i = tid; i < nt; i += kProjThreads)
                    if (!(X[i] < 1e300)) spilled = 1;
            chained = !__syncthreads_or(spilled);
        }
        if (!chained) {  // one thread, rotation by rotation
            if (tid == 0) {
                double c = c_s, s = s_s, phibar = phibar_s;
                const double root = sqrt(lambda);
                for (int j = j0; j < j0 + nt; ++j) {
                    // the rotation of column j-1 acting on rows (j-1, j) meets column j
                    theta[j] = s * alpha[j];
                    double rhobar = c * alpha[j];
                    if (lambda > 0.0) {
                        const double r = hypot(rhobar, root);
                        phibar = rhobar / r * phibar;
                        rhobar = r;
                    }
                    c = 1.0;
                    s = 0.0;
                    rho[j] = rhobar;
                    phi[j] = phibar;
                    if (j + 1 < rows_t) {
                        const double b = beta[j];
                        const double r = hypot(rhobar, b);
                        c = rhobar / r;
                        s = b / r;
                        rho[j] = r;
                        phi[j] = c * phibar + s * g[j + 1];
                        phibar = -s * phibar + c * g[j + 1];
                    }
                }
                c_s = c;
                s_s = s;
                phibar_s = phibar;
            }
            __syncthreads();
        } else {
            for (int i = tid; i < nt; i += kProjThreads) {
                const int j = j0 + i;
                const double sign = negative[i] ? -1.0 : 1.0;
                const double q = lambda > 0.0 ? X[i] / Y[i] : 1.0 / X[i];
                const double d = q + lambda;
                const double rhobar = lambda > 0.0 ? sqrt(d) : sign * sqrt(q);
                const double c1 = lambda > 0.0 ? sign * sqrt(q / d) : 1.0;
                double c = 1.0, s = 0.0, r = rhobar, gn = 0.0;
                if (j + 1 < rows_t) {
                    const double b = beta[j];
                    r = sqrt(fma(b, b, d));
                    c = rhobar / r;
                    s = b / r;
                    gn = g[j + 1];
                }
                rho[j] = r;
                if (i + 1 < nt) theta[j + 1] = s * alpha[j + 1];
                if (i == 0) theta[j] = s_s * alpha[j];
                // phi_j = (c c1) phibar_j + s g_{j+1}
                phi[j] = s * gn;
                y[j] = c * c1;
                A[i] = -s * c1;
                B[i] = c * gn;
                Y[i] = c;  // of the last column, for the next tile
                X[i] = s;
            }
            __syncthreads();
            if (tid == 0) {
                c_s = Y[nt - 1];
                s_s = X[nt - 1];
            }
            __syncthreads();
            if (tid == 0) {
                double p = phibar_s;
#pragma unroll 8
                for (int i = 0; i < nt; ++i) {
                    X[i] = p;
                    p = fma(A[i], p, B[i]);
                }
                phibar_s = p;
            }
            __syncthreads();
            for (int i = tid; i < nt; i += kProjThreads)
                phi[j0 + i] = fma(y[j0 + i], X[i], phi[j0 + i]);
            __syncthreads();
        }
        // LINPACK-style estimate of ||R^{-1}|| for the rank test the reference
        // makes with dgelsy (rcond = min(1/2, 64 eps max(rows, cols))): solve
        // R^T z = e with e_j = +-1 chosen to grow |z|
        if (lambda == 0.0) {
            for (int i = tid; i < nt; i += kProjThreads) {
                const double r = fabs(rho[j0 + i]);
                const double off = j0 + i > 0 ? fabs(theta[j0 + i]) : 0.0;
                A[i] = off / r;
                B[i] = 1.0 / r;
                rmax = fmax(rmax, r + off);
            }
            __syncthreads();
            if (tid == 0) {
                double z = zmag_s;
#pragma unroll 8
                for (int i = 0; i < nt; ++i) {
                    z = fma(A[i], z, B[i]);
                    X[i] = z;
                }
                zmag_s = z;
            }
            __syncthreads();
            for (int i = tid; i < nt; i += kProjThreads) zsq = fma(X[i], X[i], zsq);
            __syncthreads();
        }
    }
    // back substitution R y = phi, the last tile first
    double ynext = 0.0;
    for (int j1 = k; j1 > 0; j1 -= kProjTile) {
        const int j0 = max(0, j1 - kProjTile), nt = j1 - j0;
        for (int i = tid; i < nt; i += kProjThreads) {
            const int j = j0 + i;
            const double r = rho[j];
            if (!(r != 0.0)) flags_s = 1;
            A[i] = j + 1 < k ? -theta[j + 1] / r : 0.0;
            B[i] = phi[j] / r;
        }
        __syncthreads();
        if (tid == 0) {
#pragma unroll 8
            for (int i = nt - 1; i >= 0; --i) {
                ynext = j0 + i + 1 < k ? fma(A[i], ynext, B[i]) : B[i];
                X[i] = ynext;
            }
        }
        __syncthreads();
        for (int i = tid; i < nt; i += kProjThreads) y[j0 + i] = X[i];
        __syncthreads();
    }
    zsq = block_sum(zsq, red);
    rmax = block_max(rmax, red);
    if (tid != 0) return;
    int flags = flags_s;
    if (lambda == 0.0 && k > 0) {
        // ||R^{-1}|| >= ||z|| / ||e|| with ||e|| = sqrt(k)
        const double cond = rmax * sqrt(zsq / (double)k);
        if (!(cond * rcond < 1.0)) flags |= 2;
    }
    state[0] = c_s;
    state[1] = s_s;
    state[2] = phibar_s;
    state[3] = (double)k;
    state[4] = rmax;
    state[5] = (double)flags;
    state[6] = zmag_s;
    state[7] = zsq;
}

}  // namespace

// ------------------------------------------------------------ panels ----

namespace {
template <typename T>
struct PointerChunk {
    T* p[64];
};
template <typename T>
__global__ void put_pointers_kernel(T** table, PointerChunk<T> c, int count) {
    if ((int)threadIdx.x < count) table[threadIdx.x] = c.p[threadIdx.x];
}
}  // namespace

template <typename T>
PanelStoreT<T>::PanelStoreT(int n, int max_panels, cudaStream_t stream)
    : n_(n), stream_(stream), table_cap_(std::max(1, max_panels)) {
    // fixed-capacity device table: its address never changes, so captured
    // kernels may keep it
    stream_alloc(&table_, sizeof(T*) * table_cap_, stream_);
    host_.reserve(table_cap_);
}

template <typename T>
PanelStoreT<T>::~PanelStoreT() {
    for (T* p : host_) stream_free(p, stream_);
    stream_free(table_, stream_);
}

template <typename T>
void PanelStoreT<T>::ensure_columns(int cols) {
    const int need = (cols + 31) / 32;
    if (need <= panels()) return;
    if (need > table_cap_) throw std::length_error("basis exceeds the panel table capacity");
    const int first = panels();
    while (panels() < need) {
        T* p = nullptr;
        // zeroed: the sweeps read whole panels and mask columns beyond k by
        // their coefficients, which needs finite (zero) entries there
        stream_alloc(&p, sizeof(T) * 32 * static_cast<size_t>(n_), stream_);
        AMFLS_CUDA(cudaMemsetAsync(p, 0, sizeof(T) * 32 * static_cast<size_t>(n_), stream_));
        host_.push_back(p);
    }
    for (int i = first; i < need; i += 64) {
        PointerChunk<T> c{};
        const int count = std::min(64, need - i);
        std::copy_n(host_.data() + i, count, c.p);
        put_pointers_kernel<<<1, 64, 0, stream_>>>(table_ + i, c, count);
        AMFLS_LAUNCHED();
    }
}

template class PanelStoreT<double>;
template class PanelStoreT<float>;
template class PanelStoreT<__half>;

// --------------------------------------------------------- workspace ----

Workspace::Workspace(const DeviceOperator& op, const double* d_b, double regularization,
                     int maximum_basis_size, cudaStream_t stream, bool time_operators,
                     bool use_graphs, int reduced_basis, int resident_sms)
    : op_(op), stream_(stream), m_(op.rows()), n_(op.cols()), reg_(regularization),
      time_ops_(time_operators), use_graphs_(use_graphs), b_(d_b) {
    if (m_ <= 0 || n_ <= 0) throw std::invalid_argument("block Golub-Kahan operator dimensions must be positive");
    if (d_b == nullptr) throw std::invalid_argument("block Golub-Kahan right-hand side must not be null");
    if (!std::isfinite(regularization) || regularization < 0.0)
        throw std::invalid_argument("block Golub-Kahan regularization must be finite and nonnegative");
    if (maximum_basis_size < 0) throw std::invalid_argument("block Golub-Kahan basis limit must be nonnegative");
    if (reduced_basis != kReducedOff && reduced_basis != kReducedFp32 &&
        reduced_basis != kReducedFp16)
        throw std::invalid_argument("reduced_basis must be 0 (off), 1 (FP32) or 2 (FP16)");
    keep_pool_memory();
    try {
        const int mn = std::min(m_, n_);
        basis_limit_ = maximum_basis_size > 0 ? std::min(maximum_basis_size, mn) : mn;
        stream_alloc(&dstate_, sizeof(DevState), stream_);
        stream_alloc(&red_, sizeof(RedResult) * 4, stream_);
        // scratch: V^T r partials ((target blocks + panels) x 32), then the
        // per-block norm partials of the V c sweep (n/32 + slack)
        const long long max_panels = basis_limit_ / 32 + 2;
        vc_partials_offset_ = (kMaxGemvTargetBlocks + max_panels) * 32 + 6 * kMaxGridCap;
        const long long pcount = vc_partials_offset_ + (n_ + 31) / 32 + 1024;
        stream_alloc(&partials_, sizeof(double) * pcount, stream_);
        sweep_grid_ = sweep_grid();
        warp_sweeps_ = use_warp_sweeps(n_);
        sweep_panels_ = max_panels;
        const long long tiles = (n_ + 31) / 32;
        stream_alloc(&sweep_part_, sizeof(double) * sweep_part_doubles(n_, max_panels, sweep_grid_),
                     stream_);
        stream_alloc(&sweep_sq_, sizeof(double) * tiles, stream_);
        stream_alloc(&sweep_tickets_, sizeof(unsigned) * (max_panels + tiles + 1), stream_);
        AMFLS_CUDA(cudaMemsetAsync(sweep_tickets_, 0, sizeof(unsigned) * (max_panels + tiles + 1),
                                   stream_));
        const long long ncounters = 64 + max_panels + 64;
        stream_alloc(&counter_, sizeof(unsigned) * ncounters, stream_);
        AMFLS_CUDA(cudaMemsetAsync(counter_, 0, sizeof(unsigned) * ncounters, stream_));
        stream_alloc(&R_, sizeof(double) * n_, stream_);
        stream_alloc(&vnew_, sizeof(double) * n_, stream_);
        stream_alloc(&Y_, sizeof(double) * m_, stream_);
        ucap_ = 1;
        stream_alloc(&U_, sizeof(double) * m_ * ucap_, stream_);
        V_ = std::make_unique<PanelStore>(n_, static_cast<int>(max_panels), stream_);
        V_->ensure_columns(1);  // panel 0 exists (zeroed) before any level runs
        reduced_storage_ = reduced_basis;
        reduced_basis_ = reduced_basis != kReducedOff;
        if (reduced_basis_) {
            if (reduced_storage_ == kReducedFp16) {
                V16_ = std::make_unique<PanelStore16>(n_, static_cast<int>(max_panels), stream_);
                V16_->ensure_columns(1);
            } else {
                V32_ = std::make_unique<PanelStore32>(n_, static_cast<int>(max_panels), stream_);
                V32_->ensure_columns(1);
            }
            red_grid_ = reduced_sweep_grid();
            stream_alloc(&r32_, sizeof(float) * n_, stream_);
            stream_alloc(&panel_sq_, sizeof(double) * max_panels, stream_);
            stream_alloc(&red_part_, sizeof(double) * reduced_part_doubles(red_grid_, max_panels),
                         stream_);
            stream_alloc(&red_tickets_, sizeof(unsigned) * (max_panels + 1), stream_);
            AMFLS_CUDA(cudaMemsetAsync(red_tickets_, 0, sizeof(unsigned) * (max_panels + 1),
                                       stream_));
        }
        if (resident_sms > 0 && resident_levels(op_, &resident_op_)) {
            resident_grid_ = std::min(resident_sms, sm_count());
            // sized for the largest grid of an interval
            stream_alloc(&resident_red_, sizeof(double) * resident_red_doubles(sm_count()),
                         stream_);
            stream_alloc(&resident_part_,
                         sizeof(double) * resident_part_doubles(sm_count(), max_panels),
                         stream_);
            stream_alloc(&resident_barrier_, sizeof(unsigned), stream_);
        }
        std::memset(&host_, 0, sizeof(host_));
        host_.reliable = 1;
        host_.basis_limit = basis_limit_;
        put(dstate_, host_, stream_);
    } catch (...) {  // e.g. out of device memory part way: free what was allocated
        release();
        throw;
    }
}

Workspace::~Workspace() { release(); }

void Workspace::release() noexcept {
    cudaStreamSynchronize(stream_);
    lease_.release();
    stream_free(resident_red_, stream_);
    stream_free(resident_part_, stream_);
    stream_free(resident_barrier_, stream_);
    if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
    if (graph_) cudaGraphDestroy(graph_);
    if (capture_stream_) cudaStreamDestroy(capture_stream_);
    stream_free(dstate_, stream_);
    stream_free(red_, stream_);
    stream_free(partials_, stream_);
    stream_free(sweep_part_, stream_);
    stream_free(sweep_sq_, stream_);
    stream_free(sweep_tickets_, stream_);
    stream_free(counter_, stream_);
    stream_free(R_, stream_);
    stream_free(vnew_, stream_);
    stream_free(Y_, stream_);
    stream_free(U_, stream_);
    stream_free(P_, stream_);
    stream_free(c1_, stream_);
    stream_free(c2_, stream_);
    stream_free(c32_, stream_);
    stream_free(r32_, stream_);
    stream_free(panel_sq_, stream_);
    stream_free(red_part_, stream_);
    stream_free(red_tickets_, stream_);
    stream_free(alpha_, stream_);
    stream_free(beta_, stream_);
    stream_free(g_, stream_);
    stream_free(qr_, stream_);
    stream_free(qr_state_, stream_);
    stream_free(U2_, stream_);
    stream_free(BR_, stream_);
    stream_free(BL_, stream_);
    stream_free(BQ_, stream_);
    stream_free(BT_, stream_);
    stream_free(small_, stream_);
    stream_free(coefs_, stream_);
    stream_free(bpart_, stream_);
    stream_free(tsqr_, stream_);
    stream_free(dflags_, stream_);
    stream_free(dnorm_, stream_);
    stream_free(d_meta_, stream_);
    stream_free(d_vals_, stream_);
    stream_free(d_pstate_, stream_);
    stream_free(d_carry_, stream_);
    stream_free(d_pwork_, stream_);
    stream_free(d_y_, stream_);
    stream_free(level_, stream_);
    for (cudaEvent_t e : ev_)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : nev_)
        if (e) cudaEventDestroy(e);
}

void Workspace::ensure_t_capacity(int cols) {
    if (cols + 2 <= tcap_ && cols <= ccap_) return;
    int cap = std::max(1024, tcap_);
    while (cap < cols + 2) cap *= 2;
    stream_wait(stream_);
    auto grow = [&](double*& p, size_t old_count, size_t new_count) {
        double* q = nullptr;
        stream_alloc(&q, sizeof(double) * new_count, stream_);
        AMFLS_CUDA(cudaMemsetAsync(q, 0, sizeof(double) * new_count, stream_));
        if (p) {
            AMFLS_CUDA(cudaMemcpyAsync(q, p, sizeof(double) * old_count, cudaMemcpyDeviceToDevice,
                                       stream_));
            stream_wait(stream_);
            stream_free(p, stream_);
        }
        p = q;
    };
    const size_t old = tcap_;
    grow(alpha_, old, cap);
    grow(beta_, old, cap);
    grow(g_, old, cap);
    grow(c1_, old, cap);
    grow(c2_, old, cap);
    if (reduced_basis_) {  // rewritten by every level before use: no copy
        stream_free(c32_, stream_);
        c32_ = nullptr;
        stream_alloc(&c32_, sizeof(float) * cap, stream_);
        AMFLS_CUDA(cudaMemsetAsync(c32_, 0, sizeof(float) * cap, stream_));
    }
    // the QR arrays are laid out by capacity: rebuild them from scratch
    stream_free(qr_, stream_);
    qr_ = nullptr;
    stream_alloc(&qr_, sizeof(double) * 4 * cap, stream_);
    if (!qr_state_) stream_alloc(&qr_state_, sizeof(double) * 8, stream_);
    AMFLS_CUDA(cudaMemsetAsync(qr_state_, 0, sizeof(double) * 8, stream_));
    tcap_ = cap;
    ccap_ = cap;
    invalidate_graph();  // captured kernels hold the old buffer addresses
}

void Workspace::invalidate_graph() {
    if (graph_exec_) {
        stream_wait(stream_);
        cudaGraphExecDestroy(graph_exec_);
        graph_exec_ = nullptr;
    }
    if (graph_) {
        cudaGraphDestroy(graph_);
        graph_ = nullptr;
    }
    graph_pcap_ = 0;
}

void Workspace::initialize(const double* d_aux, int aux_cols) {
    if (initialized_) throw std::logic_error("block Golub-Kahan workspace is already initialized");
    initialized_ = true;
    // ||b|| (scaled two-pass, stands in for dnrm2)
    NormResult* nr = nullptr;
    AMFLS_CUDA(cudaMallocAsync(&nr, sizeof(NormResult), stream_));
    VectorSet set{};
    set.v[0] = b_;
    set.n[0] = m_;
    set.count = 1;
    norm_passes(set, nr, partials_, counter_ + 1, stream_);
    NormResult h{};
    read_back(&h, nr, stream_);
    AMFLS_CUDA(cudaFreeAsync(nr, stream_));
    if (h.nonfinite[0]) throw std::invalid_argument("block Golub-Kahan right-hand side must be finite");
    b_norm_ = euclid_from(h, 0);
    ensure_t_capacity(64);
    if (std::isfinite(b_norm_) && b_norm_ > 0.0 && basis_limit_ > 0) {
        const double inv = 1.0 / b_norm_;
        scale_copy_kernel<<<std::max<long long>(1, std::min<long long>(grid_cap(), (m_ + 255) / 256)), 256, 0,
                            stream_>>>(b_, U_, m_, inv);
        AMFLS_LAUNCHED();
        put(g_, b_norm_, stream_);
        host_.left_width = 1;
        host_.rows_t = 1;
        host_.active_first = 0;
    }
    std::memset(&host_.audit, 0, sizeof(host_.audit));
    put(dstate_, host_, stream_);
    if (b_norm_ > 0.0 && aux_cols > 0) append_left_seed(d_aux, aux_cols);
}

// The kernels of one width-one level.  Every per-level value (k, the
// previous right column, the depth target) is read from DevState, so the
// same launches serve every level and can be captured once.
void Workspace::enqueue_level_kernels(cudaStream_t s, int pcap) {
    level_begin_kernel<<<1, 32, 0, s>>>(dstate_);
    AMFLS_LAUNCHED();
    // A^T u - beta v_prev
    Epilogue ep;
    ep.out = R_;
    ep.sub_table = V_->device_table();
    ep.sub_col = &dstate_->sub_col;
    ep.coef = &dstate_->coupling_eff;
    ep.red = &red_[0];
    ep.guard = &dstate_->go;
    ep.level = true;
    ep.partials = partials_;
    ep.counter = counter_ + 2;
    if (!op_.product1(true, U_, ep, s)) throw std::runtime_error("operator has no fused device product");
    right_scales_kernel<<<1, 32, 0, s>>>(dstate_, &red_[0], m_, n_);
    AMFLS_LAUNCHED();
    const long long tiles = (n_ + 31) / 32;
    unsigned* panel_tickets = sweep_tickets_;
    unsigned* tile_tickets = sweep_tickets_ + sweep_panels_;
    unsigned* done = tile_tickets + tiles;
    const int max_chunks = (int)std::max<long long>(1, (n_ + 255) / 256);
    const int chunks = std::max(1, std::min(max_chunks, (gemv_target_blocks() + pcap - 1) / pcap));
    const int chunk_rows = (int)(((long long)n_ + chunks - 1) / chunks);
    const bool reduced = reduced_basis_ && !block_mode_;
    // grid of the sweeps that usually find their guard off (DGKS second
    // pass, FP64 redo of a reduced pass): a few blocks per SM
    const int rare_grid = (int)std::min<long long>(tiles, 2LL * sm_count());
    if (reduced) {
        // first pass on the reduced copy of V; the FP64 kernels after it run
        // only when the coefficients were too large for it (sweep_fp64)
        round_residual_kernel<<<(int)std::min<long long>(grid_cap(), (n_ + 255) / 256), 256, 0,
                                s>>>(R_, r32_, n_, dstate_);
        AMFLS_LAUNCHED();
        if (V16_)
            vt_r32_kernel<__half><<<red_grid_, kThreads, 0, s>>>(
                V16_->device_table(), n_, r32_, c1_, c32_, red_part_, panel_sq_, red_tickets_,
                red_tickets_ + sweep_panels_, dstate_);
        else
            vt_r32_kernel<float><<<red_grid_, kThreads, 0, s>>>(
                V32_->device_table(), n_, r32_, c1_, c32_, red_part_, panel_sq_, red_tickets_,
                red_tickets_ + sweep_panels_, dstate_);
        AMFLS_LAUNCHED();
        vt_r_kernel<<<dim3(pcap, chunks), kThreads, 0, s>>>(V_->device_table(), n_, chunk_rows,
                                                            R_, c1_, partials_, counter_ + 64,
                                                            dstate_, 1, 1);
        AMFLS_LAUNCHED();
        if (V16_)
            v_c32_kernel<__half><<<(int)tiles, kThreads, 0, s>>>(
                V16_->device_table(), n_, c32_, R_, partials_ + vc_partials_offset_, counter_ + 3,
                dstate_, m_);
        else
            v_c32_kernel<float><<<(int)tiles, kThreads, 0, s>>>(
                V32_->device_table(), n_, c32_, R_, partials_ + vc_partials_offset_, counter_ + 3,
                dstate_, m_);
        AMFLS_LAUNCHED();
        v_c_kernel<<<rare_grid, kThreads, 0, s>>>(
            V_->device_table(), n_, -1, c1_, R_, R_, 1, partials_ + vc_partials_offset_,
            counter_ + 3, dstate_, kHookRightPass1, m_, 2, 1);
        AMFLS_LAUNCHED();
    }
    for (int pass = reduced ? 2 : 1; pass <= 2; ++pass) {
        double* c = pass == 1 ? c1_ : c2_;
        const int hook = pass == 1 ? kHookRightPass1 : kHookRightPass2;
        if (warp_sweeps_ && !reduced) {
            sweep_vt_kernel<<<sweep_grid_, kThreads, 0, s>>>(V_->device_table(), n_, R_, c,
                                                             sweep_part_, panel_tickets, dstate_,
                                                             pass);
            AMFLS_LAUNCHED();
            sweep_vc_kernel<<<sweep_grid_, kThreads, 0, s>>>(
                V_->device_table(), n_, c, R_, R_, 1, sweep_part_, sweep_sq_, tile_tickets, done,
                dstate_, hook, m_, pass);
            AMFLS_LAUNCHED();
        } else {
            vt_r_kernel<<<dim3(pcap, chunks), kThreads, 0, s>>>(V_->device_table(), n_, chunk_rows,
                                                                R_, c, partials_, counter_ + 64,
                                                                dstate_, pass);
            AMFLS_LAUNCHED();
            // the second pass rarely runs: a grid that is cheap to skip
            v_c_kernel<<<pass == 1 ? (int)tiles : rare_grid, kThreads, 0, s>>>(
                V_->device_table(), n_, -1, c, R_, R_, 1, partials_ + vc_partials_offset_,
                counter_ + 3, dstate_, hook, m_, 1, pass);
            AMFLS_LAUNCHED();
        }
    }
    const int ngrid = (int)std::min<long long>(grid_cap(), (n_ + 255) / 256);
    if (reduced && V16_)
        normalize_right_kernel<__half><<<ngrid, 256, 0, s>>>(R_, n_, V_->device_table(), vnew_,
                                                            dstate_, V16_->device_table());
    else
        normalize_right_kernel<float><<<ngrid, 256, 0, s>>>(
            R_, n_, V_->device_table(), vnew_, dstate_, reduced ? V32_->device_table() : nullptr);
    AMFLS_LAUNCHED();
    // y = A v - ||r|| u, with ||A v||, ||y||, u.y
    Epilogue el;
    el.out = Y_;
    el.sub = U_;
    el.sub_stride = 1;
    el.coef = &dstate_->right_factor;
    el.dot_vec = U_;
    el.red = &red_[1];
    el.guard = &dstate_->go;
    el.level = true;
    el.partials = partials_;
    el.counter = counter_ + 2;
    op_.product1(false, vnew_, el, s);
    const int lgrid = (int)std::max<long long>(1, std::min<long long>(grid_cap(), (m_ + 1023) / 1024));
    for (int pass = 1; pass <= 2; ++pass) {
        // the second pass rarely runs: a grid that is cheap to skip
        left_pass_kernel<<<pass == 1 ? lgrid : std::min(lgrid, rare_grid), kThreads, 0, s>>>(
            Y_, U_, b_, m_, &red_[1], partials_, counter_ + 4, dstate_, pass, n_, alpha_, beta_,
            g_);
        AMFLS_LAUNCHED();
    }
    normalize_left_kernel<<<(int)std::min<long long>(grid_cap(), (m_ + 255) / 256), 256, 0, s>>>(
        Y_, U_, m_, dstate_);
    AMFLS_LAUNCHED();
}

void Workspace::build_graph(int pcap) {
    invalidate_graph();
    if (!capture_stream_)
        AMFLS_CUDA(cudaStreamCreateWithFlags(&capture_stream_, cudaStreamNonBlocking));
    AMFLS_CUDA(cudaGraphCreate(&graph_, 0));
    cudaGraphConditionalHandle handle;
    AMFLS_CUDA(cudaGraphConditionalHandleCreate(&handle, graph_, 1, cudaGraphCondAssignDefault));
    // the params union has no default constructor: build it in zeroed storage
    alignas(cudaGraphNodeParams) unsigned char storage[sizeof(cudaGraphNodeParams)] = {};
    auto* params = reinterpret_cast<cudaGraphNodeParams*>(storage);
    params->type = cudaGraphNodeTypeConditional;
    params->conditional.handle = handle;
    params->conditional.type = cudaGraphCondTypeWhile;
    params->conditional.size = 1;
    cudaGraphNode_t node;
    AMFLS_CUDA(cudaGraphAddNode(&node, graph_, nullptr, nullptr, 0, params));
    cudaGraph_t body = params->conditional.phGraph_out[0];
    AMFLS_CUDA(cudaStreamBeginCaptureToGraph(capture_stream_, body, nullptr, nullptr, 0,
                                             cudaStreamCaptureModeRelaxed));
    const long long launches_before = launch_count();
    try {
        enqueue_level_kernels(capture_stream_, pcap);
        level_end_kernel<<<1, 32, 0, capture_stream_>>>(dstate_, handle);
        AMFLS_LAUNCHED();
    } catch (...) {
        cudaGraph_t dummy;
        cudaStreamEndCapture(capture_stream_, &dummy);
        throw;
    }
    // captured launches run once per loop iteration, counted from body_runs
    body_kernels_ = launch_count() - launches_before;
    launch_count() = launches_before;
    cudaGraph_t captured;
    AMFLS_CUDA(cudaStreamEndCapture(capture_stream_, &captured));
    AMFLS_CUDA(cudaGraphInstantiate(&graph_exec_, graph_, 0));
    graph_pcap_ = pcap;
}

void Workspace::advance_to(int target_depth) {
    if (!initialized_) throw std::logic_error("block Golub-Kahan workspace is not initialized");
    if (block_mode_) {
        while (can_advance() && host_.depth < target_depth) {
            if (!block_level()) break;
        }
        return;
    }
    int levels = target_depth - host_.depth;
    levels = std::min(levels, basis_limit_ - host_.k);
    if (levels <= 0 || !can_advance()) return;
    // all allocations for the run happen before the launch, so the device
    // runs the whole interval without the host
    ensure_t_capacity(host_.k + levels + 2);
    V_->ensure_columns(host_.k + levels + 1);
    if (V32_) V32_->ensure_columns(host_.k + levels + 1);
    if (V16_) V16_->ensure_columns(host_.k + levels + 1);
    interval_graph_ = false;
    if (resident_grid_ > 0 && host_.k + levels <= kResidentMaxBasis && resident_ready()) {
        run_resident(levels, target_depth);
        return;
    }
    const int pneed = (host_.k + levels + 31) / 32;
    int pcap = 4;
    while (pcap < pneed) pcap *= 2;
    set_target_kernel<<<1, 32, 0, stream_>>>(dstate_, target_depth, levels);
    AMFLS_LAUNCHED();
    if (!use_graphs_) {  // same kernels, launched one by one
        for (int i = 0; i < levels; ++i) enqueue_level_kernels(stream_, pcap);
        return;
    }
    if (!graph_exec_ || pcap > graph_pcap_) build_graph(pcap);
    AMFLS_CUDA(cudaGraphLaunch(graph_exec_, stream_));
    ++graph_launches_;
    interval_graph_ = true;
}

// SMs of the next interval: the solve's share, doubled when the basis reaches
// kGrowBasis columns and at each doubling from there.  A share is chosen
// before the solve's depth is known; once the basis is long the sweeps are bound
// by their FP64 operations, so more SMs are well used and the longest solve of
// a batch does not end on its small share alone (48 uneven problems, 16 workers:
// 10.4 s with fixed shares, 7.0 s with this; 16 of 5000 to 20000 rows 129 -> 114 ms, and 144 when
// the growth starts at 256 columns).  The rule depends on the basis alone: a
// solve's sums keep their order from run to run.
int Workspace::resident_interval_grid() const {
    constexpr int kGrowBasis = 512;
    int grid = resident_grid_;
    for (long long k = kGrowBasis; k <= host_.k && grid < sm_count(); k *= 2) grid *= 2;
    return std::min(grid, sm_count());
}

// The operator's tables are there: the first solve with an interval of
// width-one levels builds them.
bool Workspace::resident_ready() {
    if (!resident_op_.a.tasks && !op_.resident_tables(&resident_op_, stream_)) resident_grid_ = 0;
    return resident_grid_ > 0;
}

void Workspace::run_resident(int levels, int target_depth) {
    const int grid = resident_interval_grid();
    ResidentArgs a{};
    a.st = dstate_;
    a.a = resident_op_.a;
    a.t = resident_op_.t;
    a.m = resident_op_.rows;
    a.ml = m_;
    a.n = n_;
    a.root = resident_op_.root;
    a.b = b_;
    a.u = U_;
    a.y = Y_;
    a.r = R_;
    a.v = vnew_;
    a.panels = V_->device_table();
    a.npanels = (host_.k + levels + 31) / 32;
    if (V16_) a.shadow = reinterpret_cast<void* const*>(V16_->device_table());
    else if (V32_) a.shadow = reinterpret_cast<void* const*>(V32_->device_table());
    a.alpha = alpha_;
    a.beta = beta_;
    a.g = g_;
    a.red = resident_red_;
    a.part = resident_part_;
    a.barrier = resident_barrier_;
    lease_.acquire(grid);
    AMFLS_CUDA(cudaMemsetAsync(resident_barrier_, 0, sizeof(unsigned), stream_));
    set_target_kernel<<<1, 32, 0, stream_>>>(dstate_, target_depth, levels);
    AMFLS_LAUNCHED();
    launch_resident_levels(a, grid, host_.k + levels, reduced_storage_, stream_);
}

bool Workspace::advance_level() {
    if (!initialized_) throw std::logic_error("block Golub-Kahan workspace is not initialized");
    if (block_mode_) return block_level();
    const int before = host_.depth;
    advance_to(host_.depth + 1);
    sync();
    return host_.depth > before && host_.level_ok;
}

void Workspace::sync() {
    read_back(&host_, dstate_, stream_);
    lease_.release();
    if (host_.barrier_timeout)
        throw std::runtime_error("resident level kernel: a grid barrier timed out");
    if (interval_graph_) {  // kernels the device ran inside graph-launched intervals
        launch_count() += body_kernels_ * (host_.body_runs - counted_body_runs_);
    }
    counted_body_runs_ = host_.body_runs;
}

void Workspace::take_operator_seconds(double& a_seconds, double& at_seconds) {
    a_seconds = static_cast<double>(host_.a_ns - seen_a_ns_) * 1e-9;
    at_seconds = static_cast<double>(host_.at_ns - seen_at_ns_) * 1e-9;
    seen_a_ns_ = host_.a_ns;
    seen_at_ns_ = host_.at_ns;
}

void Workspace::solve_projected(double* d_x) {
    const int k = host_.k;
    projected_flags_ = 0;
    pending_flags_ = nullptr;
    if (k == 0) {
        AMFLS_CUDA(cudaMemsetAsync(d_x, 0, sizeof(double) * n_, stream_));
        return;
    }
    if (block_mode_) {
        int flags = 0;
        const double* y = block_projected_y(&flags);
        v_c_kernel<<<(int)((n_ + 31) / 32), kThreads, 0, stream_>>>(
            V_->device_table(), n_, k, y, nullptr, d_x, 0, partials_, counter_ + 5, dstate_,
            kHookNone, m_, 0, 1);
        AMFLS_LAUNCHED();
        projected_flags_ = flags;
        return;
    }
    const double rcond = std::min(0.5, 64.0 * kEps * std::max(host_.rows_t, k));
    projected_solve_kernel<<<1, kProjThreads, 0, stream_>>>(alpha_, beta_, g_, k, host_.rows_t, reg_, qr_,
                                                  tcap_, qr_state_, rcond);
    AMFLS_LAUNCHED();
    const double* y = qr_ + 3 * (long long)tcap_;
    v_c_kernel<<<(int)((n_ + 31) / 32), kThreads, 0, stream_>>>(
        V_->device_table(), n_, k, y, nullptr, d_x, 0, partials_, counter_ + 5, dstate_, kHookNone,
        m_, 0, 1);
    AMFLS_LAUNCHED();
    // the flags arrive with the next wait on the stream
    copy_out(qr_state_ + 5, sizeof(double), kPinnedBytes / 2, false, stream_);
    pending_flags_ = reinterpret_cast<const double*>(host_page().data + kPinnedBytes / 2);
}

int Workspace::projected_flags() {
    if (pending_flags_) {
        projected_flags_ = (int)*pending_flags_;
        pending_flags_ = nullptr;
    }
    return projected_flags_;
}

namespace {

__global__ void probe_fill_kernel(double* const* panels, int n, int k, double* r) {
    const long long total = (long long)n * 32;
    const int P = (k + 31) / 32;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total * P;
         i += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(i / total);
        const long long e = i - (long long)p * total;
        const long long row = e / 32;
        const int col = p * 32 + (int)(e % 32);
        panels[p][e] = col < k ? (double)((row * 7 + col * 13) % 17 - 8) * 1e-3 : 0.0;
        if (p == 0 && e % 32 == 0) r[row] = (double)((row * 5) % 11 - 5) * 1e-2;
    }
}

template <typename S>
__global__ void probe_round_kernel(double* const* panels, S* const* shadow, int n, int k,
                                   const double* r, float* r32) {
    const long long total = (long long)n * 32;
    const int P = (k + 31) / 32;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total * P;
         i += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(i / total);
        const long long e = i - (long long)p * total;
        shadow[p][e] = RedStore<S>::store(panels[p][e]);
        if (p == 0 && e % 32 == 0) r32[e / 32] = __double2float_rn(r[e / 32]);
    }
}

template <typename S>
void probe_reduced(int n, int k, int reps, cudaStream_t s, double seconds[2],
                   double* max_rel_error) {
    const int P = (k + 31) / 32;
    PanelStore V(n, P, s);
    PanelStoreT<S> V32(n, P, s);
    V.ensure_columns(k);
    V32.ensure_columns(k);
    const int grid = reduced_sweep_grid();
    const long long tiles = (n + 31) / 32;
    double *r = nullptr, *c = nullptr, *c64 = nullptr, *part = nullptr, *psq = nullptr,
           *vcpart = nullptr;
    float *r32 = nullptr, *c32 = nullptr;
    unsigned* tickets = nullptr;
    DevState* st = nullptr;
    stream_alloc(&r, sizeof(double) * n, s);
    stream_alloc(&r32, sizeof(float) * n, s);
    stream_alloc(&c, sizeof(double) * 32 * P, s);
    stream_alloc(&c64, sizeof(double) * 32 * P, s);
    stream_alloc(&c32, sizeof(float) * 32 * P, s);
    // partial sums of the reduced pass ([P][chunks][32], reduced_chunks) and
    // of the FP64 reference pass ([P][chunks64][32]) share one buffer
    const int chunks64 = std::max(1, std::min((int)std::max<long long>(1, (n + 255) / 256),
                                              (gemv_target_blocks() + P - 1) / P));
    stream_alloc(&part,
                 sizeof(double) * std::max<long long>(reduced_part_doubles(grid, P),
                                                      32LL * P * chunks64),
                 s);
    stream_alloc(&psq, sizeof(double) * P, s);
    stream_alloc(&vcpart, sizeof(double) * (tiles + 1), s);
    stream_alloc(&tickets, sizeof(unsigned) * (2 * P + 2), s);
    stream_alloc(&st, sizeof(DevState), s);
    AMFLS_CUDA(cudaMemsetAsync(tickets, 0, sizeof(unsigned) * (2 * P + 2), s));
    DevState h;
    std::memset(&h, 0, sizeof(h));
    h.k = k;
    h.go = 1;
    h.reliable = 1;
    h.basis_limit = k + 1;
    h.right_scale = 1.0;
    h.norm_before = 1e300;  // the pass never decides the level: state stays as set
    AMFLS_CUDA(cudaMemcpyAsync(st, &h, sizeof(DevState), cudaMemcpyHostToDevice, s));
    probe_fill_kernel<<<grid_cap(), 256, 0, s>>>(V.device_table(), n, k, r);
    AMFLS_LAUNCHED();
    probe_round_kernel<S><<<grid_cap(), 256, 0, s>>>(V.device_table(), V32.device_table(), n, k,
                                                     r, r32);
    AMFLS_LAUNCHED();
    // the FP64 projection of the same basis, for the error
    {
        const int chunk_rows = (int)(((long long)n + chunks64 - 1) / chunks64);
        vt_r_kernel<<<dim3(P, chunks64), kThreads, 0, s>>>(V.device_table(), n, chunk_rows, r,
                                                           c64, part, tickets, st, 1);
        AMFLS_LAUNCHED();
    }
    auto vt = [&] {
        vt_r32_kernel<S><<<grid, kThreads, 0, s>>>(V32.device_table(), n, r32, c, c32, part, psq,
                                                   tickets, tickets + 2 * P + 1, st);
        AMFLS_LAUNCHED();
    };
    // r is restored by the caller's pattern only once; the subtraction of
    // the tiny probe coefficients leaves it finite, which is all timing needs
    auto vc = [&] {
        v_c32_kernel<S><<<(int)tiles, kThreads, 0, s>>>(V32.device_table(), n, c32, r, vcpart,
                                                        tickets + P, st, n);
        AMFLS_LAUNCHED();
    };
    vt();
    std::vector<double> hc(k), hc64(k), hr(n);
    AMFLS_CUDA(cudaMemcpyAsync(hc.data(), c, sizeof(double) * k, cudaMemcpyDeviceToHost, s));
    AMFLS_CUDA(cudaMemcpyAsync(hc64.data(), c64, sizeof(double) * k, cudaMemcpyDeviceToHost, s));
    AMFLS_CUDA(cudaMemcpyAsync(hr.data(), r, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    stream_wait(s);
    double rn = 0.0, worst = 0.0;
    for (double v : hr) rn += v * v;
    rn = std::sqrt(rn);
    for (int j = 0; j < k; ++j) worst = std::max(worst, std::fabs(hc[j] - hc64[j]));
    if (max_rel_error) *max_rel_error = rn > 0.0 ? worst / rn : worst;
    cudaEvent_t e[3];
    for (auto& ev : e) AMFLS_CUDA(cudaEventCreate(&ev));
    for (int i = 0; i < 3; ++i) {  // warm-up
        vt();
        vc();
    }
    AMFLS_CUDA(cudaEventRecord(e[0], s));
    for (int i = 0; i < reps; ++i) vt();
    AMFLS_CUDA(cudaEventRecord(e[1], s));
    for (int i = 0; i < reps; ++i) vc();
    AMFLS_CUDA(cudaEventRecord(e[2], s));
    AMFLS_CUDA(cudaEventSynchronize(e[2]));
    float ms0 = 0.f, ms1 = 0.f;
    AMFLS_CUDA(cudaEventElapsedTime(&ms0, e[0], e[1]));
    AMFLS_CUDA(cudaEventElapsedTime(&ms1, e[1], e[2]));
    for (auto& ev : e) cudaEventDestroy(ev);
    seconds[0] = ms0 * 1e-3 / reps;
    seconds[1] = ms1 * 1e-3 / reps;
    stream_free(r, s);
    stream_free(r32, s);
    stream_free(c, s);
    stream_free(c64, s);
    stream_free(c32, s);
    stream_free(part, s);
    stream_free(psq, s);
    stream_free(vcpart, s);
    stream_free(tickets, s);
    stream_free(st, s);
    stream_wait(s);
}

}  // namespace

void probe_reorthogonalization_reduced(int n, int k, int reps, int storage, cudaStream_t s,
                                       double seconds[2], double* max_rel_error) {
    if (n <= 0 || k <= 0 || reps <= 0) throw std::invalid_argument("probe sizes must be positive");
    if (storage == kReducedFp16)
        probe_reduced<__half>(n, k, reps, s, seconds, max_rel_error);
    else if (storage == kReducedFp32)
        probe_reduced<float>(n, k, reps, s, seconds, max_rel_error);
    else
        throw std::invalid_argument("probe storage must be 1 (FP32) or 2 (FP16)");
}

void probe_reorthogonalization(int n, int k, int reps, cudaStream_t s, double seconds[2]) {
    if (n <= 0 || k <= 0 || reps <= 0) throw std::invalid_argument("probe sizes must be positive");
    const int P = (k + 31) / 32;
    PanelStore V(n, P, s);
    V.ensure_columns(k);
    const int grid = sweep_grid();
    const long long tiles = (n + 31) / 32;
    double *r = nullptr, *w = nullptr, *c = nullptr, *part = nullptr, *sq = nullptr;
    unsigned* tickets = nullptr;
    DevState* st = nullptr;
    stream_alloc(&r, sizeof(double) * n, s);
    stream_alloc(&w, sizeof(double) * n, s);
    stream_alloc(&c, sizeof(double) * 32 * P, s);
    stream_alloc(&part, sizeof(double) * sweep_part_doubles(n, P, grid), s);
    stream_alloc(&sq, sizeof(double) * tiles, s);
    stream_alloc(&tickets, sizeof(unsigned) * (P + tiles + 1), s);
    stream_alloc(&st, sizeof(DevState), s);
    AMFLS_CUDA(cudaMemsetAsync(tickets, 0, sizeof(unsigned) * (P + tiles + 1), s));
    DevState h;
    std::memset(&h, 0, sizeof(h));
    h.k = k;
    h.go = 1;
    h.reliable = 1;
    h.basis_limit = k + 1;
    h.right_scale = 1.0;
    h.norm_before = 1e300;  // the pass never decides the level: state stays as set
    AMFLS_CUDA(cudaMemcpyAsync(st, &h, sizeof(DevState), cudaMemcpyHostToDevice, s));
    probe_fill_kernel<<<grid_cap(), 256, 0, s>>>(V.device_table(), n, k, r);
    AMFLS_LAUNCHED();
    const bool warp_sweeps = use_warp_sweeps(n);  // as the workspace chooses
    int pcap = 4;
    while (pcap < P) pcap *= 2;
    const int max_chunks = (int)std::max<long long>(1, (n + 255) / 256);
    const int chunks = std::max(1, std::min(max_chunks, (gemv_target_blocks() + pcap - 1) / pcap));
    const int chunk_rows = (int)(((long long)n + chunks - 1) / chunks);
    auto vt = [&] {
        if (warp_sweeps)
            sweep_vt_kernel<<<grid, kThreads, 0, s>>>(V.device_table(), n, r, c, part, tickets, st,
                                                      1);
        else
            vt_r_kernel<<<dim3(P, chunks), kThreads, 0, s>>>(V.device_table(), n, chunk_rows, r, c,
                                                             part, tickets, st, 1);
        AMFLS_LAUNCHED();
    };
    auto vc = [&] {
        if (warp_sweeps)
            sweep_vc_kernel<<<grid, kThreads, 0, s>>>(V.device_table(), n, c, r, w, 0, part, sq,
                                                      tickets + P, tickets + P + tiles, st,
                                                      kHookRightPass1, n, 1);
        else
            v_c_kernel<<<(int)tiles, kThreads, 0, s>>>(V.device_table(), n, -1, c, r, w, 0, part,
                                                       tickets + P, st, kHookRightPass1, n, 1, 1);
        AMFLS_LAUNCHED();
    };
    cudaEvent_t e[3];
    for (auto& ev : e) AMFLS_CUDA(cudaEventCreate(&ev));
    for (int i = 0; i < 3; ++i) {  // warm-up
        vt();
        vc();
    }
    AMFLS_CUDA(cudaEventRecord(e[0], s));
    for (int i = 0; i < reps; ++i) vt();
    AMFLS_CUDA(cudaEventRecord(e[1], s));
    for (int i = 0; i < reps; ++i) vc();
    AMFLS_CUDA(cudaEventRecord(e[2], s));
    AMFLS_CUDA(cudaEventSynchronize(e[2]));
    float ms0 = 0.f, ms1 = 0.f;
    AMFLS_CUDA(cudaEventElapsedTime(&ms0, e[0], e[1]));
    AMFLS_CUDA(cudaEventElapsedTime(&ms1, e[1], e[2]));
    for (auto& ev : e) cudaEventDestroy(ev);
    seconds[0] = ms0 * 1e-3 / reps;
    seconds[1] = ms1 * 1e-3 / reps;
    stream_free(r, s);
    stream_free(w, s);
    stream_free(c, s);
    stream_free(part, s);
    stream_free(sq, s);
    stream_free(tickets, s);
    stream_free(st, s);
    stream_wait(s);
}

}  // namespace amfls_gpu
