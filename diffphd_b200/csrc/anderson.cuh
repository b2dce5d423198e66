// The Type-II Anderson system (forward_gpu.cpp:1340-1379), solved by one warp.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace dphd {

constexpr int kAaVals = 2 * kMaxWindow + 2;  // sums of an iteration, at most
// Shared memory of the solve.  tot: the new difference's Gram column (m entries), dG^T g (m), |g|^2, |x_raw|^2.
struct AaSystem {
    double tot[kAaVals];
    double A[kMaxWindow][kMaxWindow + 1], b[kMaxWindow], inv[kMaxWindow], gamma[kMaxWindow];
    int accept, restart;
};

// Extends the Gram matrix (by ring slot) by the new difference's column, then solves (dG^T dG + reg I) gamma = dG^T g,
// reg = max(1e-6 |dG|_F^2 / m, 1e-12), by Cholesky, lane i on row i: sets `accept` with gamma, or `restart`.  The loops
// stay rolled: this runs once per iteration, so its code comes from the outer instruction caches, and unrolled to the
// largest window it took a single thread 128 registers and 9 us.
__device__ __forceinline__ void aa_solve_warp(AaSystem& s, double (*gram)[kMaxWindow], int m, int head, int W, int lane) {
    const int snew = (head + m - 1) % W, si = (head + lane) % W;
    if (lane < m) {
#pragma unroll 1
        for (int j = 0; j < m; ++j)
            s.A[lane][j] = (lane == m - 1) ? s.tot[j] : (j == m - 1) ? s.tot[lane] : gram[si][(head + j) % W];
        s.b[lane] = s.tot[m + lane];
    }
    __syncwarp();
    if (lane < m) {
        gram[snew][si] = s.tot[lane];
        gram[si][snew] = s.tot[lane];
    }
    double fro = 0;
#pragma unroll 1
    for (int j = 0; j < m; ++j) fro += s.A[j][j];
    const double reg = fmax(1e-6 * fro / m, 1e-12);
    __syncwarp();
    if (lane < m) s.A[lane][lane] += reg;
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < m; ++j) {
        double t = 0.0;
        if (lane >= j && lane < m) {
            t = s.A[lane][j];
#pragma unroll 1
            for (int k = 0; k < j; ++k) t -= s.A[lane][k] * s.A[j][k];
        }
        const double d = sqrt(fmax(__shfl_sync(0xffffffffu, t, j), 1e-300));
        const double inv = 1.0 / d;
        if (lane == j) {
            s.A[j][j] = d;
            s.inv[j] = inv;
        } else if (lane > j && lane < m) {
            s.A[lane][j] = t * inv;
        }
        __syncwarp();
    }
    double t = lane < m ? s.b[lane] : 0.0;
#pragma unroll 1
    for (int k = 0; k < m; ++k) {  // L y = b
        if (lane == k) t *= s.inv[k];
        const double yk = __shfl_sync(0xffffffffu, t, k);
        if (lane > k && lane < m) t -= s.A[lane][k] * yk;
    }
    if (lane < m) s.b[lane] = t;
    __syncwarp();
    if (lane == 0) {
#pragma unroll 1
        for (int i = m - 1; i >= 0; --i) {  // L^T x = y
            double x = s.b[i];
#pragma unroll 1
            for (int k = i + 1; k < m; ++k) x -= s.A[k][i] * s.b[k];
            s.b[i] = x * s.inv[i];
        }
        double gn = 0;
#pragma unroll 1
        for (int i = 0; i < m; ++i) gn += s.b[i] * s.b[i];
        gn = sqrt(gn);
        if (!(gn < 10.0)) {
            s.restart = 1;
        } else {
            s.accept = 1;
#pragma unroll 1
            for (int i = 0; i < m; ++i) s.gamma[i] = s.b[i];
        }
    }
}

}  // namespace dphd
