// Block levels of up to sixteen columns without host decisions.
//
// The block path read every singular value back before it went on: some 25
// waits and 40 launches a level, among them a one-block Jacobi SVD (163 us for
// 8 columns), a Householder TSQR (82 us) and product kernels that computed 32
// columns for 8 (5000 x 1200, 8 columns: 2.4 ms a level).  As long as a residual
// block is safely of full rank the singular vectors are not needed: any
// orthonormal basis of its span continues the same block Krylov space
// (krylov_workspace.cpp:263-307 takes the left singular vectors), and Cholesky
// QR with a second pass gives one to working accuracy while the block's
// condition stays below 1e6.  So a level is enqueued as a whole, and the host
// reads one LevelResult; where the factorisation says that the block is near
// the rank cutoff (its smallest singular value is at least 1 / ||R^{-1}||_F),
// ill conditioned or not finite, the host goes on from the projected residual
// with the rank-revealing path.  A solve of 128 such levels and its checkpoints
// went from 331 to 49 ms, one of 4 columns on a dense 16384 x 512 matrix from 302
// to 50 ms.
//
// FP64 operations bound the projections (one multiply-add per basis element and
// column at two lanes per SM clock); the kernels carry exactly the columns
// there are (a predicated-off FP64 instruction takes its slot all the same) and
// give every SM quarter a warp.  The small factorisations are chains of
// dependent FP64 operations in one warp.
#include <algorithm>
#include <stdexcept>

#include "narrow_block.hpp"

namespace amfls_gpu {
namespace narrow {
namespace {

constexpr int kThreads = 256;
constexpr int kTileRows = 64;
constexpr int kNnThreads = 128;
constexpr int kApplyThreads = 128;

template <typename F>
void with_padded(int c, F&& f) {
    switch (padded(c)) {
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        default: f(std::integral_constant<int, 16>{}); break;
    }
}

__global__ void frobenius2_kernel(const double* x, long long count, double* sum, double* partials,
                                  unsigned* ticket) {
    __shared__ double red[32];
    double s0 = 0.0, s1 = 0.0;
    const long long step = (long long)gridDim.x * blockDim.x;
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (; i + step < count; i += 2 * step) {
        s0 = fma(x[i], x[i], s0);
        s1 = fma(x[i + step], x[i + step], s1);
    }
    if (i < count) s0 = fma(x[i], x[i], s0);
    const double t = block_sum(s0 + s1, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = t;
    if (!arrive_last(ticket, gridDim.x)) return;
    double a = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) a += partials[b];
    a = block_sum(a, red);
    if (threadIdx.x == 0) *sum = a;
}

// grid (panels, chunks of rows).  A warp multiplies two panel rows at a time,
// 16 lanes a row and two basis columns a lane, by the rows' block entries; the
// last block of a panel adds the chunks in order.
template <int C>
__global__ void __launch_bounds__(kThreads)
panel_tn_kernel(double* const* panels, int n, int k, const double* B, int c, int chunk_rows,
                double* out, double* partials, unsigned* tickets, int* nonfinite) {
    __shared__ __align__(16) double bs[kTileRows][C];
    __shared__ double red[kThreads / 32][C][32];
    const int p = blockIdx.x, chunk = blockIdx.y, chunks = gridDim.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int half = lane >> 4, q = lane & 15;
    const int row0 = chunk * chunk_rows, row1 = min(n, row0 + chunk_rows);
    const double2* vp = reinterpret_cast<const double2*>(panels[p]);
    double a0[C], a1[C];
#pragma unroll
    for (int j = 0; j < C; ++j) a0[j] = a1[j] = 0.0;
    for (int base = row0; base < row1; base += kTileRows) {
        double2 v[kTileRows / 16];
#pragma unroll
        for (int i = 0; i < kTileRows / 16; ++i) {
            const int row = base + warp * (kTileRows / 8) + 2 * i + half;
            v[i] = row < row1 ? vp[(long long)row * 16 + q] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int t = threadIdx.x; t < kTileRows * C; t += kThreads) {
            const int i = t % kTileRows, j = t / kTileRows;
            bs[i][j] = j < c && base + i < row1 ? B[base + i + (long long)j * n] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kTileRows / 16; ++i) {
            const double* x = bs[warp * (kTileRows / 8) + 2 * i + half];
#pragma unroll
            for (int j = 0; j < C; ++j) {
                a0[j] = fma(v[i].x, x[j], a0[j]);
                a1[j] = fma(v[i].y, x[j], a1[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < C; ++j) {
        a0[j] += __shfl_xor_sync(0xffffffffu, a0[j], 16);
        a1[j] += __shfl_xor_sync(0xffffffffu, a1[j], 16);
        if (half == 0) {
            red[warp][j][2 * q] = a0[j];
            red[warp][j][2 * q + 1] = a1[j];
        }
    }
    __syncthreads();
    double* part = partials + ((long long)p * chunks + chunk) * C * 32;
    for (int t = threadIdx.x; t < C * 32; t += kThreads) {
        const double* s = &red[0][0][0] + t;
        part[t] = ((s[0] + s[C * 32]) + (s[2 * C * 32] + s[3 * C * 32])) +
                  ((s[4 * C * 32] + s[5 * C * 32]) + (s[6 * C * 32] + s[7 * C * 32]));
    }
    if (!arrive_last(&tickets[p], chunks)) return;
    for (int t = threadIdx.x; t < C * 32; t += kThreads) {
        const double* s = partials + (long long)p * chunks * C * 32 + t;
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        for (int ch = 0; ch < chunks; ch += 8) {  // eight loads on their way
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = ch + u < chunks ? __ldcg(s + (long long)(ch + u) * C * 32) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u & 3] += v[u];
        }
        double v = (x[0] + x[1]) + (x[2] + x[3]);
        if (p * 32 + (t & 31) >= k) v = 0.0;
        out[(long long)p * C * 32 + t] = v;
        if (!isfinite(v)) *nonfinite = 1;
    }
}

// B -= V C: a warp takes R pairs of rows over all panels, 16 lanes a row; the
// lanes' sums are added by a butterfly that halves the columns a lane holds.
// Four warps a block, one for each SM quarter: with eight, 1200 rows kept half of
// the SMs busy (25 -> 20 us at 480 columns and 8 block columns).
template <int C, int R>
__global__ void __launch_bounds__(kNnThreads)
panel_nn_kernel(double* const* panels, int n, int p0, int p1, const double* __restrict__ coeff,
                int c, double* B) {
    const int lane = threadIdx.x & 31, half = lane >> 4, q = lane & 15;
    const int warp = blockIdx.x * (kNnThreads / 32) + (threadIdx.x >> 5);
    const int first = warp * 2 * R;
    if (first >= n) return;
    double acc[R][C];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < C; ++j) acc[r][j] = 0.0;
    // several panels' loads in flight: a quarter has one warp to hide them
#pragma unroll(C* R <= 8 ? 4 : 2)
    for (int p = p0; p < p1; ++p) {
        const double2* vp = reinterpret_cast<const double2*>(panels[p]);
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = min(first + 2 * r + half, n - 1);
            v[r] = vp[(long long)row * 16 + q];
        }
        const double2* cp = reinterpret_cast<const double2*>(coeff + (long long)(p - p0) * C * 32) + q;
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const double2 x = __ldg(cp + 16 * j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                acc[r][j] = fma(v[r].x, x.x, acc[r][j]);
                acc[r][j] = fma(v[r].y, x.y, acc[r][j]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int col = 0, have = C;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            if (have > 1) {
                const bool upper = (q & o) != 0;
                have >>= 1;
#pragma unroll
                for (int j = 0; j < C / 2; ++j) {
                    if (j < have) {
                        const double keep = upper ? acc[r][j + have] : acc[r][j];
                        const double send = upper ? acc[r][j] : acc[r][j + have];
                        acc[r][j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                col = 2 * col + (upper ? 1 : 0);
            } else {
                acc[r][0] += __shfl_xor_sync(0xffffffffu, acc[r][0], o);
            }
        }
        // lanes that differ only below the bits used hold the same column
        constexpr int kSame = 16 / C;
        const int row = first + 2 * r + half;
        // bits were taken from the top: col's most significant bit is o = 8
        if ((q & (kSame - 1)) == 0 && col < c && row < n)
            B[row + (long long)col * n] -= acc[r][0];
    }
}

__global__ void spread_kernel(Small m, int first, int w, int c, int C, int p0, int panels,
                              double* out) {
    for (int t = threadIdx.x; t < panels * C * 32; t += blockDim.x) {
        const int col = (p0 + t / (C * 32)) * 32 + (t & 31), j = (t / 32) % C;
        const int l = col - first;
        out[t] = l >= 0 && l < w && j < c ? m.v[j + l * c] : 0.0;
    }
}

// One warp: upper Cholesky factor of the c x c matrix in G (row-major, ld
// kNarrowMax, both triangles), its inverse, in place in R and I; false when a
// pivot is not positive.
__device__ bool warp_cholesky(double (*G)[kNarrowMax + 1], double (*R)[kNarrowMax + 1],
                              double (*I)[kNarrowMax + 1], double* pivot_inv, int c) {
    const int lane = threadIdx.x & 31;
    bool ok = true;
    for (int j = 0; j < c; ++j) {
        const double d = G[j][j];
        const bool good = d > 0.0 && isfinite(d);
        ok = ok && good;
        const double inv = good ? rsqrt(d) : 1.0;
        if (lane == 0) pivot_inv[j] = inv;
        // lane j: the pivot's root (d / sqrt(d))
        if (lane < c) R[j][lane] = lane < j ? 0.0 : good ? G[j][lane] * inv : lane == j ? 1.0 : G[j][lane];
        __syncwarp();
        for (int t = lane; t < c * c; t += 32) {
            const int i = t / c, l = t % c;
            if (i > j && l > j) G[i][l] = fma(-R[j][i], R[j][l], G[i][l]);
        }
        __syncwarp();
    }
    if (lane < c) {  // column `lane` of R^{-1}
        for (int i = c - 1; i >= 0; --i) {
            double s = i == lane ? 1.0 : 0.0;
            for (int l = i + 1; l <= lane; ++l) s = fma(-R[i][l], I[l][lane], s);
            I[i][lane] = i <= lane ? s * pivot_inv[i] : 0.0;
        }
    }
    __syncwarp();
    return ok;
}

enum GramEnd { kGramStore = 0, kGramFirst = 1, kGramSecond = 2 };

// X^T Y: warps take 32-row tiles, lanes outputs; the last block adds the
// blocks' sums and, for a Cholesky pass, factorises.
template <int A, int B>
__global__ void __launch_bounds__(128)
gram_kernel(const double* X, const double* Y, long long m, int a, int b, int end, double* C,
            double* sum, Factorisation* f, double cutoff_unit, double* partials, unsigned* ticket,
            int* nonfinite) {
    constexpr int kOut = A * B, kPer = (kOut + 31) / 32, kWarps = 4;
    __shared__ double xs[kWarps][32][A + 1], ys[kWarps][32][B + 1];
    __shared__ double red[kWarps][kOut];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) acc[u] = 0.0;
    const long long stride = (long long)gridDim.x * kWarps * 32;
    for (long long base = ((long long)blockIdx.x * kWarps + warp) * 32; base < m; base += stride) {
        const bool in = base + lane < m;
#pragma unroll
        for (int j = 0; j < A; ++j) xs[warp][lane][j] = in && j < a ? X[base + lane + j * m] : 0.0;
#pragma unroll
        for (int j = 0; j < B; ++j) ys[warp][lane][j] = in && j < b ? Y[base + lane + j * m] : 0.0;
        __syncwarp();
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int o = min(lane + 32 * u, kOut - 1);
                acc[u] = fma(xs[warp][i][o % A], ys[warp][i][o / A], acc[u]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u)
        if (lane + 32 * u < kOut) red[warp][lane + 32 * u] = acc[u];
    __syncthreads();
    for (int o = threadIdx.x; o < kOut; o += 128)
        partials[(long long)blockIdx.x * kOut + o] =
            (red[0][o] + red[1][o]) + (red[2][o] + red[3][o]);
    if (!arrive_last(ticket, gridDim.x)) return;
    // warp w adds every fourth block, four chains each
    for (int o = lane; o < kOut; o += 32) {
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        for (int g = warp; g < (int)gridDim.x; g += 4 * kWarps) {
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = g + u * kWarps < (int)gridDim.x
                           ? __ldcg(partials + (long long)(g + u * kWarps) * kOut + o)
                           : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] += v[u];
        }
        red[warp][o] = (x[0] + x[1]) + (x[2] + x[3]);
    }
    __syncthreads();
    for (int o = threadIdx.x; o < kOut; o += 128) {
        const int i = o % A, j = o / A;
        const double v = (red[0][o] + red[1][o]) + (red[2][o] + red[3][o]);
        red[0][o] = v;
        if (end == kGramStore && i < a && j < b) {
            C[i + j * a] = v;
            if (sum) sum[i + j * a] += v;
            if (nonfinite && !isfinite(v)) *nonfinite = 1;
        }
    }
    if (end == kGramStore) return;
    if constexpr (A == B) {
        __shared__ double G[kNarrowMax][kNarrowMax + 1], R[kNarrowMax][kNarrowMax + 1],
            I[kNarrowMax][kNarrowMax + 1], old[kNarrowMax][kNarrowMax + 1], pinv[kNarrowMax];
        __syncthreads();
        const int c = a;
        for (int t = threadIdx.x; t < c * c; t += 128) {
            const int i = t % c, j = t / c;
            G[i][j] = red[0][i + j * A];
            if (end == kGramSecond) old[i][j] = f->factor[i + j * c];
        }
        __syncthreads();
        if (warp != 0) return;
        double trace = 0.0;
        for (int j = 0; j < c; ++j) trace += G[j][j];
        bool ok = warp_cholesky(G, R, I, pinv, c);
        double fr = 0.0, fi = 0.0;
        for (int t = lane; t < c * c; t += 32) {
            const double r = R[t % c][t / c], v = I[t % c][t / c];
            fr = fma(r, r, fr);
            fi = fma(v, v, fi);
            f->inverse[t] = v;
            if (end == kGramFirst) {
                f->factor[t] = r;
            } else {
                double s = 0.0;
                const int i = t % c, j = t / c;
                for (int l = i; l <= j; ++l) s = fma(R[i][l], old[l][j], s);
                f->factor[t] = s;
            }
        }
        fr = warp_sum(fr);
        fi = warp_sum(fi);
        if (lane == 0) {
            if (end == kGramFirst) {
                f->resid2 = trace;
                // smallest singular value >= 1 / ||R^{-1}||_F, condition <=
                // ||R||_F ||R^{-1}||_F
                const double unit = 1.01 * cutoff_unit;
                ok = ok && isfinite(trace) && isfinite(fi) && isfinite(f->scale2) &&
                     !f->nonfinite && fr * fi < 1e12 && 1.0 > unit * unit * f->scale2 * fi;
                f->ok = ok ? 1 : 0;
            } else {
                f->ok = f->ok && ok && isfinite(fi) ? 1 : 0;
            }
        }
    }
}

template <int A, int B>
void gram_launch(const double* X, const double* Y, long long m, int a, int b, int end, double* C,
                 double* sum, Factorisation* f, double cutoff_unit, double* partials,
                 unsigned* ticket, int* nonfinite, cudaStream_t s) {
    const int grid = (int)std::max<long long>(1, std::min<long long>(sm_count(), (m + 127) / 128));
    gram_kernel<A, B><<<grid, 128, 0, s>>>(X, Y, m, a, b, end, C, sum, f, cutoff_unit, partials,
                                          ticket, nonfinite);
    AMFLS_LAUNCHED();
}

// A thread takes one row and J of the b columns (blockIdx.y chooses them):
// with all of them in one thread, 5000 rows of 8 columns gave 20 blocks of 512 FP64
// operations a thread (12.6 -> 5.9 us).
template <int J>
__global__ void __launch_bounds__(kApplyThreads)
apply_kernel(const double* X, const double* C, int transposed, int ldc, long long m, int a, int b,
             double* Y, double alpha, double beta) {
    __shared__ double cs[kNarrowMax][J];
    const int j0 = blockIdx.y * J;
    for (int t = threadIdx.x; t < a * J; t += kApplyThreads) {
        const int i = t / J, j = j0 + t % J;
        cs[i][t % J] = j < b ? (transposed ? C[j + i * ldc] : C[i + j * ldc]) : 0.0;
    }
    __syncthreads();
    for (long long r = blockIdx.x * (long long)kApplyThreads + threadIdx.x; r < m;
         r += (long long)gridDim.x * kApplyThreads) {
        double old[J], acc[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            old[j] = beta != 0.0 && j0 + j < b ? Y[r + (long long)(j0 + j) * m] : 0.0;
            acc[j] = 0.0;
        }
#pragma unroll 4
        for (int i = 0; i < a; ++i) {
            const double x = X[r + (long long)i * m];
#pragma unroll
            for (int j = 0; j < J; ++j) acc[j] = fma(x, cs[i][j], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (j0 + j < b)
                Y[r + (long long)(j0 + j) * m] =
                    beta == 0.0 ? alpha * acc[j] : fma(alpha, acc[j], beta * old[j]);
        }
    }
}

__global__ void append_kernel(double* const* panels, long long n, int k0, const double* Q, int r,
                              const LevelResult* level) {
    if (!level->right.ok || !level->left.ok) return;
    const long long total = n * r;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long i = t / r;
        const int j = (int)(t - i * r), col = k0 + j;
        panels[col >> 5][i * 32 + (col & 31)] = Q[i + (long long)j * n];
    }
}

int grid_1d(long long items) {
    return (int)std::max<long long>(1, std::min<long long>((items + 255) / 256, grid_cap()));
}

// rows per block: about two blocks per SM over all panels, whole tiles
int chunk_rows(long long n, int P) {
    const long long want = std::max<long long>(1, (2LL * sm_count() + P - 1) / P);
    long long rows = (n + want - 1) / want;
    rows = (rows + kTileRows - 1) / kTileRows * kTileRows;
    return (int)std::max<long long>(rows, kTileRows);
}

}  // namespace

long long panel_tn_partial_doubles(long long n, int k, int c) {
    const int P = (std::max(k, 1) + 31) / 32;
    const int rows = chunk_rows(n, P);
    return (long long)P * ((n + rows - 1) / rows) * padded(c) * 32;
}

void frobenius2(const double* X, long long count, double* sum, double* partials, unsigned* ticket,
                cudaStream_t s) {
    const int grid = (int)std::max<long long>(1, std::min<long long>(2 * sm_count(), (count + 511) / 512));
    frobenius2_kernel<<<grid, kThreads, 0, s>>>(X, count, sum, partials, ticket);
    AMFLS_LAUNCHED();
}

void panel_tn(double* const* panels, long long n, int k, const double* B, int c, double* C,
              double* partials, unsigned* tickets, int* nonfinite, cudaStream_t s) {
    const int P = (k + 31) / 32, rows = chunk_rows(n, P);
    const dim3 grid(P, (unsigned)((n + rows - 1) / rows));
    with_padded(c, [&](auto w) {
        panel_tn_kernel<w()><<<grid, kThreads, 0, s>>>(panels, (int)n, k, B, c, rows, C, partials,
                                                      tickets, nonfinite);
    });
    AMFLS_LAUNCHED();
}

void panel_nn(double* const* panels, long long n, int p0, int p1, const double* C, int c,
              double* B, cudaStream_t s) {
    if (p1 <= p0) return;
    // four row pairs per warp share the loads of the coefficients once there
    // are enough rows for every SM quarter to have a warp all the same
    const bool many = n >= 32LL * sm_count();
    with_padded(c, [&](auto w) {
        constexpr int W = w(), R = W <= 8 ? 4 : 2;
        if (many) {
            const long long warps = (n + 2 * R - 1) / (2 * R);
            panel_nn_kernel<W, R><<<(unsigned)((warps + 3) / 4), kNnThreads, 0, s>>>(
                panels, (int)n, p0, p1, C, c, B);
        } else {
            const long long warps = (n + 1) / 2;
            panel_nn_kernel<W, 1><<<(unsigned)((warps + 3) / 4), kNnThreads, 0, s>>>(
                panels, (int)n, p0, p1, C, c, B);
        }
    });
    AMFLS_LAUNCHED();
}

void spread_coefficients(const Small& m, int first, int w, int c, double* C, cudaStream_t s) {
    const int p0 = first / 32, p1 = (first + w + 31) / 32;
    spread_kernel<<<1, kThreads, 0, s>>>(m, first, w, c, padded(c), p0, p1 - p0, C);
    AMFLS_LAUNCHED();
}

void gram(const double* X, const double* Y, long long m, int a, int b, double* C, double* sum,
          double* partials, unsigned* ticket, int* nonfinite, cudaStream_t s) {
    with_padded(a, [&](auto A) {
        with_padded(b, [&](auto B) {
            gram_launch<A(), B()>(X, Y, m, a, b, kGramStore, C, sum, nullptr, 0.0, partials, ticket,
                                  nonfinite, s);
        });
    });
}

void apply(const double* X, const double* C, bool transposed, int ldc, long long m, int a, int b,
           double* Y, double alpha, double beta, cudaStream_t s) {
    // one column a thread while that does not give every SM quarter several
    // warps; beyond, four share the loads of X
    const int J = m * b <= 32LL * 32 * sm_count() || b < 4 ? 1 : 4;
    const long long rows = (m + kApplyThreads - 1) / kApplyThreads;
    const dim3 grid((unsigned)std::max<long long>(1, std::min<long long>(rows, 4LL * grid_cap())),
                    (unsigned)((b + J - 1) / J));
    (J == 1 ? apply_kernel<1> : apply_kernel<4>)<<<grid, kApplyThreads, 0, s>>>(
        X, C, transposed ? 1 : 0, ldc, m, a, b, Y, alpha, beta);
    AMFLS_LAUNCHED();
}

void cholesky_pass(const double* B, long long m, int c, int pass, double cutoff_unit,
                   Factorisation* f, double* partials, unsigned* ticket, cudaStream_t s) {
    with_padded(c, [&](auto C) {
        gram_launch<C(), C()>(B, B, m, c, c, pass == 1 ? kGramFirst : kGramSecond, nullptr, nullptr,
                              f, cutoff_unit, partials, ticket, nullptr, s);
    });
}

void append(double* const* panels, long long n, int k0, const double* Q, int r,
            const LevelResult* level, cudaStream_t s) {
    append_kernel<<<grid_1d(n * r), 256, 0, s>>>(panels, n, k0, Q, r, level);
    AMFLS_LAUNCHED();
}

}  // namespace narrow
}  // namespace amfls_gpu
