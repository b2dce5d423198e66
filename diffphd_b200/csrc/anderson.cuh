// The Type-II Anderson system (forward_gpu.cpp:1340-1379), solved by one thread.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace dphd {

constexpr int kAaVals = 2 * kMaxWindow + 2;  // new Gram column, right-hand side, |g|^2, |x_raw|^2

// tot: the new difference's Gram column (j < m) and, from kMaxWindow on, dG^T g; gram by ring slot.  Sets `accept` with
// gamma, or `restart`.
__device__ __forceinline__ void aa_solve(const double* tot, int m, int head, int W, double (*gram)[kMaxWindow],
                                         double* gamma, int* accept, int* restart) {
    // Extend the stored Gram matrix by the new difference's column, then solve
    // (dG^T dG + reg I) gamma = dG^T g, reg = max(1e-6 |dG|_F^2 / m, 1e-12), by Cholesky.  All loops run to
    // kMaxWindow with guards so that the small arrays stay in registers; the stored entries are loaded
    // independently (one round trip) rather than inside the factorisation.
    const int snew = (head + m - 1) % W;
    double A[kMaxWindow][kMaxWindow], b[kMaxWindow];
#pragma unroll
    for (int i = 0; i < kMaxWindow; ++i)
#pragma unroll
        for (int j = 0; j < kMaxWindow; ++j)
            if (i < m && j < m)
                A[i][j] = (i == m - 1) ? tot[j] : (j == m - 1) ? tot[i] : gram[(head + i) % W][(head + j) % W];
#pragma unroll
    for (int j = 0; j < kMaxWindow; ++j)
        if (j < m) {
            const int sj = (head + j) % W;
            gram[snew][sj] = tot[j];
            gram[sj][snew] = tot[j];
        }
    double fro = 0;
#pragma unroll
    for (int j = 0; j < kMaxWindow; ++j)
        if (j < m) fro += A[j][j];
    const double reg = fmax(1e-6 * fro / m, 1e-12);
#pragma unroll
    for (int i = 0; i < kMaxWindow; ++i)
        if (i < m) {
            A[i][i] += reg;
            b[i] = tot[kMaxWindow + i];
        }
    // one reciprocal per column (a single thread runs this: FP64 divisions dominate its latency)
    double inv_diag[kMaxWindow];
#pragma unroll
    for (int j = 0; j < kMaxWindow; ++j) {
        inv_diag[j] = 0.0;
        if (j < m) {
            double d = A[j][j];
#pragma unroll
            for (int k = 0; k < kMaxWindow; ++k)
                if (k < j) d -= A[j][k] * A[j][k];
            d = sqrt(fmax(d, 1e-300));
            A[j][j] = d;
            const double inv = 1.0 / d;
            inv_diag[j] = inv;
#pragma unroll
            for (int i = 0; i < kMaxWindow; ++i)
                if (i > j && i < m) {
                    double t = A[i][j];
#pragma unroll
                    for (int k = 0; k < kMaxWindow; ++k)
                        if (k < j) t -= A[i][k] * A[j][k];
                    A[i][j] = t * inv;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < kMaxWindow; ++i)
        if (i < m) {
            double t = b[i];
#pragma unroll
            for (int k = 0; k < kMaxWindow; ++k)
                if (k < i) t -= A[i][k] * b[k];
            b[i] = t * inv_diag[i];
        }
#pragma unroll
    for (int i = kMaxWindow - 1; i >= 0; --i)
        if (i < m) {
            double t = b[i];
#pragma unroll
            for (int k = 0; k < kMaxWindow; ++k)
                if (k > i && k < m) t -= A[k][i] * b[k];
            b[i] = t * inv_diag[i];
        }
    double gn = 0;
#pragma unroll
    for (int i = 0; i < kMaxWindow; ++i)
        if (i < m) gn += b[i] * b[i];
    gn = sqrt(gn);
    if (!(gn < 10.0)) {
        *restart = 1;
    } else {
        *accept = 1;
#pragma unroll
        for (int i = 0; i < kMaxWindow; ++i)
            if (i < m) gamma[i] = b[i];
    }
}

}  // namespace dphd
