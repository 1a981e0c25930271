// Block levels of up to kNarrowMax columns: the products, projections and
// factorisations of block_level.cu as device work that needs no decision of
// the host (see narrow_block.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace amfls_gpu {
namespace narrow {

constexpr int kNarrowMax = 16;
constexpr int kSquare = kNarrowMax * kNarrowMax;

// What one orthogonalisation leaves behind, read by the host once per level.
struct Factorisation {
    double scale2;   // squared Frobenius norm before the projection
    double resid2;   // and after it
    int ok;          // full rank beyond doubt: factor and q are valid
    int nonfinite;   // a projection coefficient was not finite
    double factor[kSquare];  // c x c upper triangular, column-major, ld c
    double inverse[kSquare]; // of the current triangular factor
};
struct LevelResult {
    Factorisation right, left;
    double coefficients[kSquare];  // U^T B summed over both passes, aw x r
    double g[kNarrowMax];          // new left block's U^T b
};

struct Small {  // a small matrix handed to a kernel by value
    double v[kSquare];
};

// columns padded to a power of two (2, 4, 8, 16)
inline int padded(int c) { return c <= 2 ? 2 : c <= 4 ? 4 : c <= 8 ? 8 : 16; }

// Doubles of the panel coefficients ([panel][padded(c)][32]) of k columns, and
// of the partial sums panel_tn needs; tickets: one per panel.
inline long long panel_coefficient_doubles(int k, int c) {
    return (long long)((k + 31) / 32) * padded(c) * 32;
}
long long panel_tn_partial_doubles(long long n, int k, int c);

// *sum = ||X||_F^2 of `count` doubles (partials: kMaxGridCap doubles).
void frobenius2(const double* X, long long count, double* sum, double* partials, unsigned* ticket,
                cudaStream_t s);

// C = V[:, 0:k]^T B (B n x c, ld n).
void panel_tn(double* const* panels, long long n, int k, const double* B, int c, double* C,
              double* partials, unsigned* tickets, int* nonfinite, cudaStream_t s);

// B -= V[:, panels p0 .. p1) C, with C as panel_tn leaves it, panel p0 first.
void panel_nn(double* const* panels, long long n, int p0, int p1, const double* C, int c,
              double* B, cudaStream_t s);

// The panel layout of a w x c block of coefficients for columns
// first .. first + w of the basis (zero elsewhere): C[w][c] from `m`, stored
// transposed (m.v[j + l * c] multiplies basis column first + l and block
// column j).
void spread_coefficients(const Small& m, int first, int w, int c, double* C, cudaStream_t s);

// C (a x b, ld a) = X^T Y, optionally added to `sum`.
void gram(const double* X, const double* Y, long long m, int a, int b, double* C, double* sum,
          double* partials, unsigned* ticket, int* nonfinite, cudaStream_t s);

// Y = beta Y + alpha X C (X m x a, C a x b with ld a, or its transpose with
// ld ldc: C(i, j) = c[j + i * ldc]).
void apply(const double* X, const double* C, bool transposed, int ldc, long long m, int a, int b,
           double* Y, double alpha, double beta, cudaStream_t s);

// First and second Cholesky QR pass of the block B (m x c): the Gram matrix of
// B, its factor R and R^{-1} into f.  The first pass decides f.ok (cutoff_unit
// times the norm before the projection is the rank cutoff); the second one
// multiplies its factor onto the first's.
void cholesky_pass(const double* B, long long m, int c, int pass, double cutoff_unit,
                   Factorisation* f, double* partials, unsigned* ticket, cudaStream_t s);

// V[:, k0 + j] = Q[:, j] where *right_ok and *left_ok (both set by the
// factorisations of the level) say that the level stands.
void append(double* const* panels, long long n, int k0, const double* Q, int r,
            const LevelResult* level, cudaStream_t s);

}  // namespace narrow
}  // namespace amfls_gpu
