// Resident width-one levels.
//
// The kernel chain of workspace.cu spends 13 to 18 launches on a level; on
// problems whose level takes tens of microseconds the launches, not the work,
// set the time (20000 x 5000, 10 nonzeros per row: 104 us per level, of which
// the FP64 pipe needs 11).  Here a whole checkpoint interval is one
// cooperative kernel with one block of 384 threads on each SM of its grid (512
// threads spill registers and 256 leave too few gathers in flight: 129 us per
// level of a 200000 x 50000 power-law problem against 139 and 148).
// Whole solves, kernel chain -> now: 2000 x 500 28.7 -> 10.0 ms, 20000 x 5000 142 ->
// 65 ms, 60000 x 15000 274 -> 160 ms, the mixed form on 200000 x 50000 565 -> 242 ms.  It
// stays ahead up to the 2M x 500k matrix (500 levels: 1253 -> 1207 us per level FP64,
// 967 -> 780 us on the FP16 copy), so operators that have the tables use it but for
// those with rows far longer than the others (resident_excess).
// A level (krylov_workspace.cpp:589-831) is five phases with a grid barrier
// after each:
//   1  u = y / ||y|| (the previous level's), r = A^T u - beta v
//   2  c = V^T r
//   3  r -= V c, then the DGKS test and the right rank decision (phases 2 and
//      3 repeat when the test asks for the second pass)
//   4  v = r / ||r||, appended to V; y = A v - ||r|| u
//   5  y -= (u . y) u, then the left test and decision
// Products gather from the unnormalised vector and scale the finished row
// sum, so no phase is spent on a normalisation.  Every block reduces the
// per-block partial sums itself, in block order, and takes the decisions on
// its own copy of the state (the same numbers in every block); block 0 keeps
// T, g and, at the end, the state.  All sums run in an order fixed by the
// tables and the grid.
//
// Work is split so that every SM gets the same number of FP64 operations,
// which bound the sweeps (two lanes' FMAs per SM clock): V^T r in 4 KB units
// of the panels, r - V c in groups of rows, both in equal contiguous shares per
// block.  In both a warp multiplies two 256-byte panel rows at a time, 16 lanes
// a row, so that few partial sums per lane have to be added across lanes.
//
// Every wait is bounded (kSpinLimit polls); a barrier that gives up sets
// barrier_timeout, which the host reports as an error.
#include <algorithm>
#include <cstddef>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <type_traits>

#include "common.cuh"
#include "level_decisions.cuh"
#include "resident_grid.cuh"
#include "resident_levels.hpp"

namespace amfls_gpu {
namespace {

using namespace resident;

enum Slot { kRedRight = 0, kRedNorm = 1, kRedNorm2 = 2, kRedA = 3, kRedLeft = 4, kRedLeft2 = 5 };
constexpr int kMaxPanels = kResidentMaxBasis / 32 + 1;
constexpr int kSlots = 2;           // ring slots of a warp
constexpr int kSlotBytes = 4096;
constexpr int kSegs = 4;  // panels of V^T r whose partial sums are added together

struct Shared : GridShared<3> {
    DevState st;
    int left_raw;
    double val[4];      // reduced values
    // shares of the V^T r units for the current number of panels
    int P, upp, p0;     // panels, units per panel, panel of the first unit
    long long u0, u1;   // this block's units
    unsigned long long full[kW][kSlots];  // mbarriers of the warps' ring slots
    short seg_first[kMaxPanels], seg_last[kMaxPanels];  // blocks with units of a panel
    double* panels[kMaxPanels];
    alignas(16) double seg[kSegs][kW][32];  // stored and read in pairs
};

constexpr size_t kSharedBytes = (sizeof(Shared) + 127) / 128 * 128;
constexpr size_t kRingBytes = (size_t)kW * kSlots * kSlotBytes;
static_assert(offsetof(Shared, seg) % 16 == 0 && kW <= 16);

// ---- the rings through which a warp reads the basis ----
//
// Each warp owns kSlots slots of 4 KB and is its own producer: bulk copies
// bring the next pieces of the basis while the current one is multiplied, and
// the first pieces of a sweep before the grid barrier in front of it (V does
// not change while r or c is formed).  The 96 KB on their way per SM cover the
// memory's latency at the FP64 pipe's rate without holding registers.

struct Ring {
    unsigned char* base;
    unsigned bars;   // shared address of the warp's mbarriers
    int issued, taken;
};

__device__ __forceinline__ unsigned shared_address(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void expect_bytes(const Ring& k, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     k.bars + 8 * (k.issued & (kSlots - 1))),
                 "r"(bytes)
                 : "memory");
}

// Copies `bytes` (a multiple of 16, both ends 16-byte aligned) to the slot
// being filled, at `offset`.
__device__ __forceinline__ void copy_bytes(const Ring& k, unsigned offset, const void* src,
                                           unsigned bytes) {
    const int slot = k.issued & (kSlots - 1);
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(shared_address(k.base + slot * kSlotBytes + offset)),
        "l"(src), "r"(bytes), "r"(k.bars + 8 * slot)
        : "memory");
}

// Waits for the oldest slot; false when it gave up (s.failed is then set).
__device__ __forceinline__ const unsigned char* take_slot(Shared& s, Ring& k) {
    const int slot = k.taken & (kSlots - 1);
    const unsigned parity = (unsigned)(k.taken / kSlots) & 1u, bar = k.bars + 8 * slot;
    ++k.taken;
    unsigned done = 0;
    for (unsigned spins = 0; spins < kSpinLimit; ++spins) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) break;
    }
    if (!done) s.failed = 1;
    return k.base + slot * kSlotBytes;
}

// ---- V^T r in 4 KB units of the panels, equal shares per block ----

// Shares for a basis of k columns: block b of the first `used` (all of them
// unless there are fewer than four units for each) takes units
// [total b / used, total (b+1) / used).  Four units are one for each SM quarter,
// so more blocks would not finish sooner, and every block adds the segments of
// all (2000 x 500, V^T r to the norm test: 20.7 -> 16.5 us per level with the
// shared butterflies of reduce_slot).
__device__ __forceinline__ void set_shares(Shared& s, int n, int k, int unit_rows) {
    const int P = (k + 31) >> 5;
    const int upp = (n + unit_rows - 1) / unit_rows;
    if (P == s.P && upp == s.upp) return;  // uniform: they change only between block barriers
    const long long total = (long long)P * upp;
    const int used = (int)min((total + 3) / 4, (long long)gridDim.x);
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += kT) {
        // the block of unit u: the largest b with total b / used <= u
        const long long f = (long long)p * upp, l = f + upp - 1;
        s.seg_first[p] = (short)(((f + 1) * used - 1) / total);
        s.seg_last[p] = (short)(((l + 1) * used - 1) / total);
    }
    if (threadIdx.x == 0) {
        const long long b = min((int)blockIdx.x, used);
        s.u0 = total * b / used;
        s.u1 = total * min(b + 1, (long long)used) / used;
        s.p0 = (int)(s.u0 / upp);
        s.upp = upp;
        s.P = P;
    }
    __syncthreads();
}

// Where a warp stands among its units: unit, first unit of the next panel.
struct Unit {
    long long u, end_of_panel;
    int p;
};

__device__ __forceinline__ void settle(const Shared& s, Unit& t) {
    while (t.u >= t.end_of_panel) {
        ++t.p;
        t.end_of_panel += s.upp;
    }
}

__device__ __forceinline__ Unit first_unit(const Shared& s) {
    Unit t;
    t.u = s.u0 + (threadIdx.x >> 5);
    t.p = s.p0;
    t.end_of_panel = (long long)(s.p0 + 1) * s.upp;
    settle(s, t);
    return t;
}

template <int kRows>  // rows of a unit
__device__ __forceinline__ int unit_row(const Shared& s, const Unit& t) {
    return (int)(t.u - (t.end_of_panel - s.upp)) * kRows;
}

// Starts the copy of unit t and moves it on (nothing beyond the share).
template <typename T>
__device__ __forceinline__ void issue_unit(const Shared& s, Ring& k, T* const* panels, int n,
                                           Unit& t) {
    constexpr int kRows = kSlotBytes / (32 * (int)sizeof(T));
    if (t.u >= s.u1) return;
    if ((threadIdx.x & 31) == 0) {
        const int row0 = unit_row<kRows>(s, t);
        const unsigned bytes = min(kRows, n - row0) * 32 * (unsigned)sizeof(T);
        expect_bytes(k, bytes);
        copy_bytes(k, 0, panels[t.p] + (long long)row0 * 32, bytes);
    }
    ++k.issued;
    t.u += kW;
    settle(s, t);
}

// Partial sums of this block's units; segment (panel p, block b) goes to
// part[(b + p) * 32], a place of its own.  `ahead`: the next unit to copy.
__device__ __forceinline__ void sweep_vt(Shared& s, const ResidentArgs& a, Ring& k, Unit ahead) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, q = lane & 15;
    Unit t = first_unit(s);
    auto load_r = [&](const Unit& x) {
        const int row = unit_row<16>(s, x) + q;
        return row < a.n ? a.r[row] : 0.0;
    };
    double rv = t.u < s.u1 ? load_r(t) : 0.0;
    for (int pb = s.p0; (long long)pb * s.upp < s.u1; pb += kSegs) {
        const long long ue = min(s.u1, (long long)(pb + kSegs) * s.upp);
#pragma unroll
        for (int i = 0; i < kSegs; ++i) s.seg[i][warp][lane] = 0.0;
        __syncwarp();
        double c0 = 0.0, c1 = 0.0;
        while (t.u < ue) {
            Unit nx = t;
            nx.u += kW;
            settle(s, nx);
            const double rn = nx.u < s.u1 ? load_r(nx) : 0.0;
            const double2* v = reinterpret_cast<const double2*>(take_slot(s, k)) + lane;
            if (unit_row<16>(s, t) + 16 <= a.n) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const double2 e = v[32 * i];
                    const double x = __shfl_sync(0xffffffffu, rv, 2 * i + half);
                    c0 = fma(e.x, x, c0);
                    c1 = fma(e.y, x, c1);
                }
            } else {  // rows beyond n were not copied
                const int rows = a.n - unit_row<16>(s, t);
                for (int i = 0; 2 * i < rows; ++i) {
                    const double x = __shfl_sync(0xffffffffu, rv, 2 * i + half);
                    if (2 * i + half < rows) {
                        const double2 e = v[32 * i];
                        c0 = fma(e.x, x, c0);
                        c1 = fma(e.y, x, c1);
                    }
                }
            }
            __syncwarp();
            issue_unit(s, k, s.panels, a.n, ahead);
            if (nx.p != t.p || nx.u >= ue) {
                c0 += __shfl_xor_sync(0xffffffffu, c0, 16);
                c1 += __shfl_xor_sync(0xffffffffu, c1, 16);
                if (half == 0)
                    *reinterpret_cast<double2*>(&s.seg[t.p - pb][warp][2 * q]) =
                        make_double2(c0, c1);
                c0 = c1 = 0.0;
            }
            t = nx;
            rv = rn;
        }
        __syncthreads();
        const int p = pb + warp;
        if (warp < kSegs && (long long)p * s.upp < ue) {
            double x[4] = {0.0, 0.0, 0.0, 0.0};
            const int warps = (int)min((long long)kW, s.u1 - s.u0);  // the others' are zero
            for (int w = 0; w < warps; w += 4)
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] += s.seg[warp][w + i][lane];
            a.part[((long long)blockIdx.x + p) * 32 + lane] = (x[0] + x[1]) + (x[2] + x[3]);
        }
        if ((long long)(pb + kSegs) * s.upp < s.u1) __syncthreads();  // seg is reused
    }
}

// The coefficients of the whole basis from the segments, summed in block order
// into shared memory (zero up to the end of the last panel); a non-finite one
// sets coeff_nonfinite.
__device__ __forceinline__ void gather_coefficients(Shared& s, const ResidentArgs& a, int k,
                                                    double* c, double scale) {
    for (int j = threadIdx.x; j < s.P * 32; j += kT) {
        const int p = j >> 5;
        const int b1 = s.seg_last[p];
        const double* src = a.part + (long long)p * 32 + (j & 31);
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = s.seg_first[p]; b <= b1; b += 8) {
            double v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = b + i <= b1 ? __ldcg(src + (long long)(b + i) * 32) : 0.0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (b + i <= b1) x[i & 3] += v[i];
        }
        double t = (x[0] + x[1]) + (x[2] + x[3]);
        t *= scale;
        if (j >= k) t = 0.0;
        c[j] = t;
        if (!isfinite(t)) s.st.coeff_nonfinite = 1;
    }
    __syncthreads();
}

// ---- r - V c in groups of rows (512 bytes of a panel), the rows in equal
// shares per block; a piece is a group's rows in eight panels ----

struct Piece {
    int row, chunk;  // first row of the group, chunk of eight panels
};

template <typename T>
__device__ __forceinline__ void issue_piece(const Shared& s, Ring& k, T* const* panels, int row1,
                                            Piece& t) {
    constexpr int kRows = 512 / (32 * (int)sizeof(T));
    if (t.row >= row1) return;
    const int lane = threadIdx.x & 31;
    const unsigned bytes = min(kRows, row1 - t.row) * 32 * (unsigned)sizeof(T);
    const int count = min(8, s.P - t.chunk * 8);
    if (lane == 0) expect_bytes(k, bytes * count);
    if (lane < count)
        copy_bytes(k, lane * 512, panels[t.chunk * 8 + lane] + (long long)t.row * 32, bytes);
    ++k.issued;
    if (++t.chunk * 8 >= s.P) {
        t.chunk = 0;
        t.row += kRows * kW;
    }
}

// r -= V c on this block's rows (c in shared memory); returns the thread's
// part of ||r||^2.  `ahead`: the next piece to copy.
__device__ __forceinline__ double sweep_vc(Shared& s, const ResidentArgs& a, Ring& k, int row0,
                                           int row1, const double* c, Piece ahead) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, q = lane & 15;
    double sq = 0.0;
    for (int row = row0 + 2 * warp; row < row1; row += 2 * kW) {
        const bool in = row + half < row1;
        const double old = q == 0 && in ? a.r[row + half] : 0.0;
        double t0 = 0.0, t1 = 0.0;
        for (int p = 0; p < s.P; p += 8) {
            const double2* v = reinterpret_cast<const double2*>(take_slot(s, k)) + lane;
            const double2* cp = reinterpret_cast<const double2*>(c) + p * 16 + q;
            if (p + 8 <= s.P) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const double2 e = v[32 * i], cv = cp[16 * i];
                    t0 = fma(e.x, cv.x, t0);
                    t1 = fma(e.y, cv.y, t1);
                }
            } else {
                for (int i = 0; p + i < s.P; ++i) {
                    const double2 e = v[32 * i], cv = cp[16 * i];
                    t0 = fma(e.x, cv.x, t0);
                    t1 = fma(e.y, cv.y, t1);
                }
            }
            __syncwarp();
            issue_piece(s, k, s.panels, row1, ahead);
        }
        // a row beyond the share holds whatever the slot held: it stays in its
        // own sixteen lanes and is not stored
        double y = t0 + t1;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (q == 0 && in) {
            const double x = old - y;
            a.r[row + half] = x;
            sq = fma(x, x, sq);
        }
    }
    return sq;
}

// Block sum of the values that lanes 0, g, 2g, ... of every warp hold.
template <int kStep>
__device__ __forceinline__ void sparse_partial(Shared& s, double v, double* red, int slot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= kStep; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) s.lane[0][warp] = v;
    __syncthreads();
    if (warp == 0) {
        double t = lane < kW ? s.lane[0][lane] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[(long long)slot * 4 * gridDim.x + blockIdx.x] = t;
    }
}

// ---- the same on the reduced copy (FP32, or FP16 holding 2^8 v) ----

template <typename S>
struct Copy {
    static constexpr int kLanes = 32 * (int)sizeof(S) / 16;  // lanes of one panel row
    static constexpr int kCols = 16 / (int)sizeof(S);        // columns of a lane
    static constexpr int kRows = 32 / kLanes;                // rows of one warp load
    static constexpr int kRun = 4 * RedStore<S>::kFlushSteps;  // rows summed in FP32
};

// sixteen bytes of a slot as FP32
__device__ __forceinline__ void widen(const unsigned char* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void widen(const unsigned char* p, float (&v)[8]) {
    const uint4 x = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&x);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// Partial sums of V~^T fl32(r): FP32 over runs of at most kRun rows (of one
// lane, or of lanes added while their runs together stay within it), FP64
// above that.  `fold` holds kW * kRows * 32 floats.
template <typename S>
__device__ __forceinline__ void sweep_vt_copy(Shared& s, const ResidentArgs& a, Ring& k,
                                              S* const* panels, Unit ahead, float* fold) {
    using C = Copy<S>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & (C::kLanes - 1), sub = lane / C::kLanes;
    constexpr int kUnit = kSlotBytes / (32 * (int)sizeof(S));  // rows of a unit
    constexpr int kLoads = kUnit / C::kRows;                   // rows per lane
    constexpr int kR = kUnit / 32;
    Unit t = first_unit(s);
    auto load_r = [&](const Unit& x, float (&v)[kR]) {
        const int row = unit_row<kUnit>(s, x) + lane;
#pragma unroll
        for (int i = 0; i < kR; ++i)
            v[i] = x.u < s.u1 && row + 32 * i < a.n ? __double2float_rn(a.r[row + 32 * i]) : 0.f;
    };
    float rv[kR];
    load_r(t, rv);
    int p = s.p0;
    for (long long base = s.u0; base < s.u1; ++p) {
        const long long end = min(s.u1, (long long)(p + 1) * s.upp);
        double acc[C::kCols];
        float f[C::kCols];
#pragma unroll
        for (int c = 0; c < C::kCols; ++c) acc[c] = 0.0, f[c] = 0.f;
        int run = 0;
        // a segment longer than one run per lane folds into FP64 as it goes
        const int longest = (int)((end - base + kW - 1) / kW) * kLoads;
        const bool longer = longest > C::kRun;
        while (t.u < end) {
            Unit nx = t;
            nx.u += kW;
            settle(s, nx);
            float rn[kR];
            load_r(nx, rn);
            const unsigned char* slot = take_slot(s, k) + lane * 16;
            const int rows = a.n - unit_row<kUnit>(s, t);
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const int row = i * C::kRows + sub;
                const float x = __shfl_sync(0xffffffffu, rv[i * C::kRows / 32], row & 31);
                float v[C::kCols];
                widen(slot + 512 * i, v);
                if (row < rows) {  // rows beyond n were not copied
#pragma unroll
                    for (int c = 0; c < C::kCols; ++c) f[c] = fmaf(v[c], x, f[c]);
                }
            }
            __syncwarp();
            issue_unit(s, k, panels, a.n, ahead);
            run += kLoads;
            if (longer && run + kLoads > C::kRun) {
#pragma unroll
                for (int c = 0; c < C::kCols; ++c) acc[c] += (double)f[c], f[c] = 0.f;
                run = 0;
            }
            t = nx;
#pragma unroll
            for (int i = 0; i < kR; ++i) rv[i] = rn[i];
        }
        if (longer) {
#pragma unroll
            for (int c = 0; c < C::kCols; ++c) {
                acc[c] += (double)f[c];
#pragma unroll
                for (int o = 16; o >= C::kLanes; o >>= 1)
                    acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                if (sub == 0) s.seg[0][warp][q * C::kCols + c] = acc[c];
            }
        } else {
            // the longest run of any warp decides how far lanes are added in FP32
            run = longest;
            int left = C::kRows;
#pragma unroll
            for (int o = 16; o >= C::kLanes; o >>= 1) {
                if (2 * run > C::kRun) break;
#pragma unroll
                for (int c = 0; c < C::kCols; ++c) f[c] += __shfl_xor_sync(0xffffffffu, f[c], o);
                run *= 2;
                left >>= 1;
            }
            if (sub < left) {
#pragma unroll
                for (int c = 0; c < C::kCols; ++c)
                    fold[(warp * left + sub) * 32 + q * C::kCols + c] = f[c];
            }
            __syncwarp();
            double sum = 0.0;
            for (int i = 0; i < left; ++i) sum += (double)fold[(warp * left + i) * 32 + lane];
            s.seg[0][warp][lane] = sum;
        }
        __syncthreads();
        if (warp == 0) {
            double x[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int w = 0; w < kW; ++w) x[w & 3] += s.seg[0][w][lane];
            a.part[((long long)blockIdx.x + p) * 32 + lane] = (x[0] + x[1]) + (x[2] + x[3]);
        }
        __syncthreads();
        base = end;
    }
}

// r -= fl64(V~ c~) on this block's rows.
template <typename S>
__device__ __forceinline__ double sweep_vc_copy(Shared& s, const ResidentArgs& a, Ring& k,
                                                S* const* panels, int row0, int row1,
                                                const float* c, Piece ahead) {
    using C = Copy<S>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & (C::kLanes - 1), sub = lane / C::kLanes;
    double sq = 0.0;
    for (int first = row0 + C::kRows * warp; first < row1; first += C::kRows * kW) {
        const int row = first + sub;
        const bool in = row < row1;
        const double old = q == 0 && in ? a.r[row] : 0.0;
        float f[C::kCols];
#pragma unroll
        for (int i = 0; i < C::kCols; ++i) f[i] = 0.f;
        for (int p = 0; p < s.P; p += 8) {
            const unsigned char* slot = take_slot(s, k) + lane * 16;
            const float* cp = c + p * 32 + q * C::kCols;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (p + j < s.P) {
                    float v[C::kCols], cv[C::kCols];
                    widen(slot + 512 * j, v);
#pragma unroll
                    for (int i = 0; i < C::kCols; i += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(cp + 32 * j + i);
                        cv[i] = x.x, cv[i + 1] = x.y, cv[i + 2] = x.z, cv[i + 3] = x.w;
                    }
#pragma unroll
                    for (int i = 0; i < C::kCols; ++i) f[i] = fmaf(v[i], cv[i], f[i]);
                }
            }
            __syncwarp();
            issue_piece(s, k, panels, row1, ahead);
        }
#pragma unroll
        for (int w = C::kCols / 2; w > 0; w >>= 1)
#pragma unroll
            for (int i = 0; i < w; ++i) f[i] += f[i + w];
#pragma unroll
        for (int o = C::kLanes / 2; o > 0; o >>= 1) f[0] += __shfl_xor_sync(0xffffffffu, f[0], o);
        if (q == 0 && in) {
            const double x = old - (double)f[0] * (double)RedStore<S>::kInvScale;
            a.r[row] = x;
            sq = fma(x, x, sq);
        }
    }
    return sq;
}

template <int kStorage>
__host__ __device__ constexpr size_t fold_bytes() {
    return kStorage == 0 ? 0
                         : sizeof(float) * kW * 32 *
                               (kStorage == 2 ? Copy<__half>::kRows : Copy<float>::kRows);
}

static_assert(kSharedBytes + kRingBytes + fold_bytes<2>() + 8 * kResidentMaxBasis <= 227 * 1024);

// kStorage: 0 FP64 sweeps, 1 / 2 first pass on the FP32 / FP16 copy
template <int kStorage>
__global__ void __launch_bounds__(kT, 1) resident_levels_kernel(ResidentArgs a) {
    using S = std::conditional_t<kStorage == 2, __half, float>;
    extern __shared__ __align__(16) unsigned char shared_raw[];
    Shared& s = *reinterpret_cast<Shared*>(shared_raw);
    unsigned char* rings = shared_raw + kSharedBytes;
    float* fold = reinterpret_cast<float*>(rings + kRingBytes);
    double* coeff = reinterpret_cast<double*>(rings + kRingBytes + fold_bytes<kStorage>());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grid = gridDim.x;
    // product tasks go to warps 1 .. kW - 1 (warp 0 takes the decisions
    // meanwhile), consecutive tasks to different SMs
    const int W = grid * (kW - 1), w = warp > 0 ? (warp - 1) * grid + blockIdx.x : W;
    const bool writer = blockIdx.x == 0;
    const int n = a.n;
    // this block's shares of the right and the left vectors' rows
    const int r0 = (int)((long long)n * blockIdx.x / grid);
    const int r1 = (int)((long long)n * (blockIdx.x + 1) / grid);
    const int l0 = (int)((long long)a.ml * blockIdx.x / grid);
    const int l1 = (int)((long long)a.ml * (blockIdx.x + 1) / grid);
    const int warps_left = min(kW, (l1 - l0 + 31) >> 5);
    // warps that hold terms of a product's sums
    auto product_warps = [&](int ntasks) { return min(kW, 1 + (ntasks + grid - 1) / grid); };
    const int warps_t = product_warps(a.t.ntasks);
    const int warps_a =
        max(product_warps(a.a.ntasks), a.ml > a.m ? min(kW, (r1 - r0 + 31) >> 5) : 0);
    {
        const int* src = reinterpret_cast<const int*>(a.st);
        int* dst = reinterpret_cast<int*>(&s.st);
        for (int i = tid; i < (int)(sizeof(DevState) / sizeof(int)); i += kT) dst[i] = src[i];
        for (int p = tid; p < a.npanels; p += kT) s.panels[p] = a.panels[p];
        if (lane < kSlots)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                             shared_address(&s.full[warp][lane]))
                         : "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
        if (tid == 0) {
            s.arrived = 0;
            s.failed = 0;
            s.left_raw = 0;
            s.P = 0;
            s.upp = 0;
        }
    }
    __syncthreads();
    Ring ring{rings + (size_t)warp * kSlots * kSlotBytes, shared_address(&s.full[warp][0]), 0, 0};
    S* const* shadow = reinterpret_cast<S* const*>(a.shadow);
    constexpr int kUnitRows = kSlotBytes / (32 * (kStorage ? (int)sizeof(S) : 8));
    bool left_raw = false;  // the left vector is y / ||y||, not yet written to u
    sliced::Walk walk;
    if (warp > 0) sliced::start_walk(a.t, walk, w, W);
    if (tid == 0) begin_level(&s.st);
    __syncthreads();
    double x0 = 0.0;  // the first task's sum
    if (s.st.go && warp > 0) x0 = sliced::task_sum(a.t, walk.cur, a.u);
    while (s.st.go && !s.failed) {
        const int k = s.st.k;
        asm volatile("fence.proxy.async;" ::: "memory");
        set_shares(s, n, k, kUnitRows);
        // the first units of V^T r are on their way during phase 1
        Unit ahead = first_unit(s);
        if (k > 0) {
            for (int i = 0; i < kSlots; ++i) {
                if constexpr (kStorage != 0) issue_unit(s, ring, shadow, n, ahead);
                else issue_unit(s, ring, s.panels, n, ahead);
            }
        }

        // 1: r = A^T u - coupling v (the first task's sum is there)
        {
            const double* src = left_raw ? a.y : a.u;
            const double inv = left_raw ? s.st.inv_left : 1.0;
            const double coupling = s.st.coupling_eff;
            double sums[2] = {0.0, 0.0};
            if (warp > 0 && walk.round * W + w < a.t.ntasks) {
                double x = x0;
                do {
                    const sliced::Fetch& f = walk.cur;
                    if (walk.round > 0) x = sliced::task_sum(a.t, walk.cur, src);
                    if (f.row >= 0 && (lane & ((1 << f.shift) - 1)) == 0) {
                        if (a.ml > a.m) x = fma(a.root, src[a.m + f.row], x);
                        x *= inv;
                        const double out = coupling != 0.0 ? x - coupling * a.v[f.row] : x;
                        a.r[f.row] = out;
                        sums[0] = fma(x, x, sums[0]);
                        sums[1] = fma(out, out, sums[1]);
                    }
                } while (sliced::next_task(a.t, walk, w, W));
            }
            if (left_raw)
                for (int i = l0 + tid; i < l1; i += kT) a.u[i] = a.y[i] * inv;
            left_raw = false;
            block_partials(s, sums, warps_t, a.red, kRedRight);
        }
        grid_barrier(s, a.barrier);
        if (s.failed) break;
        if (writer && tid == 0) s.st.at_ns += global_ns() - s.st.t_mark;
        // 2, 3: projection passes; pass 0 (reduced copy) or 1 first, 2 when
        // the DGKS test asks for it.  After the last barrier warp 0 decides
        // while the other warps sum their first task of the next product.
        int pass = kStorage == 0 ? 1 : 0;
        bool failed = false;
        while (true) {
            bool copy = false;
            if (k > 0) {
                double part = 0.0;
                if constexpr (kStorage != 0) {
                    if (pass == 0) {
                        sweep_vt_copy<S>(s, a, ring, shadow, ahead, fold);
                        Piece piece{r0 + Copy<S>::kRows * warp, 0};
                        for (int i = 0; i < kSlots; ++i)
                            issue_piece(s, ring, shadow, r1, piece);
                        grid_barrier(s, a.barrier);
                        if (s.failed) {
                            failed = true;
                            break;
                        }
                        gather_coefficients(s, a, k, coeff, (double)RedStore<S>::kInvScale);
                        if (warp == 0) {
                            double nb[2];
                            reduce_slot(a.red, kRedRight, nb);
                            double q2 = 0.0;
                            for (int j = lane; j < k; j += 32) q2 = fma(coeff[j], coeff[j], q2);
                            q2 = warp_sum(q2);
                            warp_sqrt(nb);
                            if (lane == 0) {
                                const double before = nb[1];
                                s.st.right_scale = nb[0];
                                s.st.norm_before = before;
                                const double bound = kReducedCoeffBound * before;
                                const bool redo =
                                    !(isfinite(q2) && isfinite(before)) || q2 > bound * bound;
                                s.st.sweep_fp64 = redo ? 1 : 0;
                                s.st.coeff_nonfinite = 0;  // the FP64 pass finds them again
                                s.st.reduced_levels += 1;
                                if (redo) s.st.reduced_fallbacks += 1;
                            }
                        }
                        __syncthreads();
                        copy = !s.st.sweep_fp64;
                        pass = 1;
                        if (!copy) {  // the copy's pieces are not used
                            while (ring.taken < ring.issued) take_slot(s, ring);
                            // the FP64 pass writes its sums to a.part, from which
                            // other blocks may still be reading the copy's
                            grid_barrier(s, a.barrier);
                            if (s.failed) {
                                failed = true;
                                break;
                            }
                        } else {
                            // narrow in place: element j's float lies before its double
                            float* c32 = reinterpret_cast<float*>(coeff);
                            const int kp = s.P * 32;
                            for (int j0 = 0; j0 < kp; j0 += kT) {
                                const float c =
                                    j0 + tid < kp ? __double2float_rn(coeff[j0 + tid]) : 0.f;
                                __syncthreads();
                                if (j0 + tid < kp) c32[j0 + tid] = c;
                                __syncthreads();
                            }
                            part = sweep_vc_copy<S>(s, a, ring, shadow, r0, r1, c32, piece);
                            sparse_partial<Copy<S>::kLanes>(s, part, a.red, kRedNorm);
                        }
                    }
                }
                if (!copy) {
                    if (kStorage != 0 || pass == 2) {
                        set_shares(s, n, k, 16);
                        ahead = first_unit(s);
                        for (int i = 0; i < kSlots; ++i)
                            issue_unit(s, ring, s.panels, n, ahead);
                    }
                    sweep_vt(s, a, ring, ahead);
                    Piece piece{r0 + 2 * warp, 0};
                    for (int i = 0; i < kSlots; ++i) issue_piece(s, ring, s.panels, r1, piece);
                    grid_barrier(s, a.barrier);
                    if (s.failed) {
                        failed = true;
                        break;
                    }
                    if (pass == 1 && warp == kW - 1) {
                        // a warp with few coefficients: off the decision's path
                        double nb[2];
                        reduce_slot(a.red, kRedRight, nb);
                        warp_sqrt(nb);
                        if (lane == 0) {
                            s.st.right_scale = nb[0];
                            s.st.norm_before = nb[1];
                        }
                    }
                    gather_coefficients(s, a, k, coeff, 1.0);
                    part = sweep_vc(s, a, ring, r0, r1, coeff, piece);
                    sparse_partial<16>(s, part, a.red, pass == 1 ? kRedNorm : kRedNorm2);
                }
            }
            if (warp > 0) sliced::start_walk(a.a, walk, w, W);
            if (k > 0) {
                grid_barrier(s, a.barrier);
                if (s.failed) {
                    failed = true;
                    break;
                }
            }
            if (warp == 0) {
                double v[2] = {0.0, 0.0};
                if (k > 0) {
                    double after[1];
                    reduce_slot(a.red, pass == 1 ? kRedNorm : kRedNorm2, after);
                    v[1] = sqrt(after[0]);
                } else {
                    reduce_slot(a.red, kRedRight, v);
                    warp_sqrt(v);
                }
                if (lane == 0) {
                    if (k == 0) {
                        s.st.right_scale = v[0];
                        s.st.norm_before = v[1];
                    }
                    s.st.norm_after = v[1];
                    s.st.second_pass = k > 0 && pass < 2 && dgks_again(s.st.norm_before, v[1]) ? 1 : 0;
                    if (!s.st.second_pass) decide_right(&s.st, a.ml, n);
                    if (writer) s.st.t_mark = global_ns();
                }
            } else {
                x0 = sliced::task_sum(a.a, walk.cur, a.r);
            }
            __syncthreads();
            if (!s.st.second_pass) break;
            pass = 2;
        }
        if (failed || !s.st.go) break;  // no right vector kept

        // 4: v = r / ||r||, y = A v - ||r|| u
        double ub = 0.0, bb = 0.0;
        {
            const double inv = s.st.inv_right, factor = s.st.right_factor;
            double* vcol = s.panels[k >> 5] + (k & 31);
            S* vcopy = kStorage ? reinterpret_cast<S*>(a.shadow[k >> 5]) + (k & 31) : nullptr;
            double sums[3] = {0.0, 0.0, 0.0};
            auto row_term = [&](int row, double x) {
                const double ui = a.u[row];
                const double out = x - factor * ui;
                a.y[row] = out;
                sums[0] = fma(x, x, sums[0]);
                sums[1] = fma(out, out, sums[1]);
                sums[2] = fma(out, ui, sums[2]);
            };
            if (warp > 0 && w < a.a.ntasks) {
                double x = x0;
                do {
                    if (walk.round > 0) x = sliced::task_sum(a.a, walk.cur, a.r);
                    if (walk.cur.row >= 0 && (lane & ((1 << walk.cur.shift) - 1)) == 0)
                        row_term(walk.cur.row, x * inv);
                } while (sliced::next_task(a.a, walk, w, W));
            }
            for (int i = r0 + tid; i < r1; i += kT) {
                const double v = a.r[i] * inv;
                vcol[(long long)i * 32] = v;
                a.v[i] = v;
                if constexpr (kStorage != 0) vcopy[(long long)i * 32] = RedStore<S>::store(v);
                if (a.ml > a.m) row_term(a.m + i, a.root * v);  // the appended rows
            }
            // the new column is read by bulk copies after the barrier
            asm volatile("fence.proxy.async;" ::: "memory");
            block_partials(s, sums, warps_a, a.red, kRedA);
            if (l0 + tid < l1) {
                ub = a.u[l0 + tid];
                bb = a.b[l0 + tid];
            }
        }
        grid_barrier(s, a.barrier);
        if (s.failed) break;
        // 5: y -= (u . y) u, with ||y||, u . y and b . y; a second time when
        // the DGKS test asks for it
        double yb = l0 + tid < l1 ? a.y[l0 + tid] : 0.0;
        if (warp == 0) {
            double v[3];
            reduce_slot(a.red, kRedA, v);
            if (lane == 0) {
                s.st.pass_coeff = v[2];
                s.val[0] = v[0];
                s.val[1] = v[1];
                s.st.left_coeff = 0.0;
                if (writer) s.st.a_ns += global_ns() - s.st.t_mark;
            }
        }
        __syncthreads();
        for (int lp = 1; lp <= 2; ++lp) {
            const double c = s.st.pass_coeff;
            double sums[3] = {0.0, 0.0, 0.0};
            for (int i = l0 + tid; i < l1; i += kT) {
                if (i != l0 + tid || lp == 2) {
                    ub = a.u[i];
                    yb = a.y[i];
                    bb = a.b[i];
                }
                const double y = yb - c * ub;
                a.y[i] = y;
                sums[0] = fma(y, y, sums[0]);
                sums[1] = fma(y, ub, sums[1]);
                sums[2] = fma(y, bb, sums[2]);
            }
            block_partials(s, sums, warps_left, a.red, lp == 1 ? kRedLeft : kRedLeft2);
            if (warp > 0) sliced::start_walk(a.t, walk, w, W);
            grid_barrier(s, a.barrier);
            if (s.failed) break;
            if (warp == 0) {
                double v[3];
                reduce_slot(a.red, lp == 1 ? kRedLeft : kRedLeft2, v);
                double r[3] = {lp == 1 ? s.val[0] : 0.0, lp == 1 ? s.val[1] : 0.0, v[0]};
                warp_sqrt(r);
                if (lane == 0) {
                    DevState& st = s.st;
                    if (lp == 1) {
                        st.left_scale = r[0];
                        st.norm_before = r[1];
                    }
                    st.left_norm = r[2];
                    st.left_coeff += c;
                    st.pass_coeff = v[1];
                    st.b_dot = v[2];
                    st.second_pass = lp == 1 && dgks_again(r[1], r[2]) ? 1 : 0;
                    if (!st.second_pass) {
                        decide_left(&st, a.ml, n, writer ? a.alpha : nullptr, a.beta, a.g);
                        s.left_raw = st.go && st.left_rank > 0;
                        // the next level starts here: its first product is
                        // already being summed
                        if (st.go) begin_level(&st);
                    }
                }
            } else {
                x0 = sliced::task_sum(a.t, walk.cur, a.y);
            }
            __syncthreads();
            if (!s.st.second_pass) break;
        }
        left_raw = s.left_raw;
    }
    // the newest left vector, for the next interval or the block levels
    if (left_raw && !s.failed) {
        const double inv = s.st.inv_left;
        for (int i = l0 + tid; i < l1; i += kT) a.u[i] = a.y[i] * inv;
    }
    // nothing is left in flight, whichever way the loop ended
    while (ring.taken < ring.issued) take_slot(s, ring);
    if (writer) {
        __syncthreads();
        if (tid == 0) s.st.barrier_timeout = s.failed;
        __syncthreads();
        const int* src = reinterpret_cast<const int*>(&s.st);
        int* dst = reinterpret_cast<int*>(a.st);
        for (int i = tid; i < (int)(sizeof(DevState) / sizeof(int)); i += kT) dst[i] = src[i];
    }
}

template <int kStorage>
void launch(const ResidentArgs& args, int grid, int k_max, cudaStream_t stream) {
    const size_t fixed = kSharedBytes + kRingBytes + fold_bytes<kStorage>();
    const size_t smem = fixed + sizeof(double) * 32 * (size_t)((k_max + 31) / 32);
    auto kernel = resident_levels_kernel<kStorage>;
    // the limit is the current device's: set at every launch, to the same value
    // by every thread
    AMFLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(fixed + sizeof(double) * kResidentMaxBasis)));
    ResidentArgs copy = args;
    void* params[] = {&copy};
    AMFLS_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(grid),
                                           dim3(kT), params, smem, stream));
    AMFLS_LAUNCHED();
}

struct Budget {
    std::mutex mu;
    std::condition_variable cv;
    int used = 0;
    std::uint64_t next = 0, serving = 0;  // requests are granted in order
};

Budget& budget(int device) {
    static Budget b[64];
    return b[device >= 0 && device < 64 ? device : 0];
}

}  // namespace

void launch_resident_levels(const ResidentArgs& args, int grid, int k_max, int storage,
                            cudaStream_t stream) {
    if (storage == 2) launch<2>(args, grid, k_max, stream);
    else if (storage == 1) launch<1>(args, grid, k_max, stream);
    else launch<0>(args, grid, k_max, stream);
}

void SmLease::acquire(int sms) {
    release();
    AMFLS_CUDA(cudaGetDevice(&device_));
    const int total = sm_count();
    sms = std::max(1, std::min(sms, total));
    Budget& b = budget(device_);
    std::unique_lock<std::mutex> lock(b.mu);
    const std::uint64_t ticket = b.next++;
    b.cv.wait(lock, [&] { return b.serving == ticket && b.used + sms <= total; });
    ++b.serving;
    b.used += sms;
    sms_ = sms;
    b.cv.notify_all();
}

void SmLease::release() {
    if (sms_ == 0) return;
    Budget& b = budget(device_);
    {
        std::lock_guard<std::mutex> lock(b.mu);
        b.used -= sms_;
    }
    sms_ = 0;
    b.cv.notify_all();
}

}  // namespace amfls_gpu
