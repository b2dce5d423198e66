// Signorini–Coulomb contact for a planar frictional boundary, inside the PD iteration
// (ForwardProjectiveDynamicsAlgPhd, cpp/core/src/fem/deformable_projective_dynamics_forward_gpu.cpp:461-528,
// 849-1061, 1116-1321, 1483-1545).
//
// Delassus operator.  With one node-level A for all axes, (A^-1 (n_j e_j))_i = G_ij n_j with G the node block
// of A^-1 = S^T S at the candidates, so W_ij = (n_i . n_j) G_ij and the tangential 2x2 blocks are G_ii I.  A does
// not change between frames, so G is formed once per factor build: G_ij is the dot product of two S columns,
// whose nonzeros are the etree paths of the two columns, i.e. a dot product over the shared root-first prefix.
//
// Each PD iteration: (1) delta_j = n . q_j + offset for every candidate; candidates with lambda_j = 0 and
// delta_j > 0 have omega_j = 0, E_j = r_j, phi_j = 0, so their rows and columns of M = Omega W Omega + E
// decouple with Delta lambda_j = 0 exactly — only the others (the active set) enter the dense solve;
// (2) A^-1 b at active nodes from y = S b through the S column paths; (3) M Delta lambda = h - J A^-1 g by a
// dense Cholesky factorisation, clamp lambda to [0, 1e8], Coulomb cone per contact; (4) the contact impulse
// J^T f is written as a sparse right-hand side so that y += S J^T f before the single S^T pass.
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "launch.cuh"
#include "ncp_common.cuh"

namespace dphd {

namespace {

__device__ __forceinline__ double warp_sum_d(double v) { return ncp_warp_sum(v); }

// G_ij for i <= j, one warp per pair (prefix of matching rows from the root).
__global__ void __launch_bounds__(256) k_delassus(int K, const int64_t* __restrict__ off, const int* __restrict__ prow,
                                                  const double* __restrict__ pval, double* __restrict__ G) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long npairs = (long long)K * (K + 1) / 2;
    if (w >= npairs) return;
    // w -> (i, j) with i <= j, row-major over the upper triangle
    long long i = (long long)((sqrt(8.0 * (double)w + 1.0) - 1.0) / 2.0);  // j index in tri ordering
    while ((i + 1) * (i + 2) / 2 <= w) ++i;
    while (i * (i + 1) / 2 > w) --i;
    const int j = (int)i;
    const int ii = (int)(w - i * (i + 1) / 2);  // ii <= j
    const int64_t oa = off[ii], ob = off[j];
    const int la = (int)(off[ii + 1] - oa), lb = (int)(off[j + 1] - ob);
    const int L = min(la, lb);
    double s = 0.0;
    bool matching = true;
    for (int base = 0; base < L && matching; base += 32) {
        const int d = base + lane;
        const bool in = d < L;
        const bool eq = in && prow[oa + d] == prow[ob + d];
        const unsigned mism = __ballot_sync(0xffffffffu, in && !eq);
        const int first_bad = mism ? __ffs(mism) - 1 : 32;
        if (lane < first_bad && in) s += pval[oa + d] * pval[ob + d];
        if (mism) matching = false;
    }
    s = warp_sum_d(s);
    if (lane == 0) {
        G[(size_t)ii * K + j] = s;
        G[(size_t)j * K + ii] = s;
    }
}

// Fischer-Burmeister terms of every candidate, the active flags and the ordered active list.  The candidates are
// spread over the grid (one flag bit each, a word per warp); the block that arrives last compacts the bit words in
// order.  Candidates outside the active set carry no friction and no contact force: their tangential multipliers are
// cleared and their S-pass input becomes r64 (or 0).  One CTA took 15 us over 4,913 candidates and 42 us over 15,625
// (three block barriers per 1,024 candidates in series).
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads) k_ncp_prepare(ContactDev c, const double* __restrict__ x,
                                                              const double* __restrict__ r64, Ctrl* ctrl) {
    pdl_enter();
    if (ctrl->done) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = blockIdx.x * kPrepThreads + threadIdx.x;
    int act = 0;
    if (k < c.K) {
        const int node = c.cand[k];
        const double dj = c.n[0] * x[3 * node] + c.n[1] * x[3 * node + 1] + c.n[2] * x[3 * node + 2] + c.offset;
        const double lj = c.lam[k], rj = c.rprec[k];
        double den = sqrt(dj * dj + rj * rj * lj * lj);
        if (den < 1e-14) den = 1e-14;
        const double om = 1.0 - dj / den;
        const double E = (1.0 - rj * lj / den) * rj;
        const double phi = dj + rj * lj - den;
        const double Hq = dj - c.offset;
        c.omega[k] = om;
        c.Ediag[k] = E;
        c.hvec[k] = -phi + om * Hq;
        act = (lj > 0.0 || dj <= 0.0) ? 1 : 0;
        if (!act) {
            c.lt1[k] = c.lt2[k] = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) c.vc[3 * (size_t)k + d] = r64 ? r64[3 * node + d] : 0.0;
        }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, act);
    if (lane == 0 && k < c.K) c.act_mask[k >> 5] = bal;
    // last block: ordered compaction of the bit words
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(reinterpret_cast<unsigned int*>(c.ncp_flags) + 4, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __shared__ int warp_tot[kPrepThreads / 32];
    const int nw = (c.K + 31) >> 5;
    int base = 0;
    for (int w0 = 0; w0 < nw; w0 += kPrepThreads) {
        const int w = w0 + threadIdx.x;
        unsigned bits = w < nw ? __ldcg(c.act_mask + w) : 0u;
        const int cnt = __popc(bits);
        int pre = cnt;  // inclusive scan over the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += t;
        }
        if (lane == 31) warp_tot[wid] = pre;
        __syncthreads();
        int woff = 0, tot = 0;
#pragma unroll
        for (int v = 0; v < kPrepThreads / 32; ++v) {
            if (v < wid) woff += warp_tot[v];
            tot += warp_tot[v];
        }
        int o = base + woff + pre - cnt;
        while (bits) {
            c.act[o++] = 32 * w + __ffs(bits) - 1;
            bits &= bits - 1;
        }
        base += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        c.kact[0] = base;
        c.ncp_flags[4] = 0;
    }
}

// A^-1 b at active candidate nodes: dot of the node's S column path with y = S b (3 right-hand sides), one CTA per
// active candidate (a path of a thousand rows is a chain of dependent row and y loads: one warp took 16 us for it).
constexpr int kDotThreads = 256;
__global__ void __launch_bounds__(kDotThreads) k_ncp_ainvb(ContactDev c, const double* __restrict__ y, int npad,
                                                           const double* __restrict__ x_base, const Ctrl* ctrl) {
    pdl_enter();
    if (ctrl->done) return;
    __shared__ double sh[3][kDotThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ka = c.kact[0];
    for (int a = blockIdx.x; a < ka; a += gridDim.x) {
        const int k = c.act[a];
        const int64_t o = c.off[k];
        const int L = (int)(c.off[k + 1] - o);
        double s0 = 0, s1 = 0, s2 = 0;
        for (int d = threadIdx.x; d < L; d += kDotThreads) {
            const int r = c.prow[o + d];
            const double v = c.pval[o + d];
            s0 += v * y[r];
            s1 += v * y[npad + r];
            s2 += v * y[2 * (size_t)npad + r];
        }
        s0 = warp_sum_d(s0);
        s1 = warp_sum_d(s1);
        s2 = warp_sum_d(s2);
        if (lane == 0) {
            sh[0][wid] = s0;
            sh[1][wid] = s1;
            sh[2][wid] = s2;
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kDotThreads / 32; ++w) s += sh[threadIdx.x][w];
            c.ainvb[3 * a + threadIdx.x] = s + (x_base ? x_base[3 * c.cand[k] + threadIdx.x] : 0.0);
        }
        __syncthreads();
    }
}

// ---- Dense solve of the active NCP system (multi-CTA, one cooperative launch per PD iteration) -------------
//
// M = Omega G Omega + E over the ka active candidates (ka <= K, known only on the device) is factored by a
// blocked right-looking Cholesky in 64 x 64 tiles, and M dlambda = h - J A^-1 g solved, by every CTA of one
// cooperative grid (all CTAs co-resident) with grid-wide barriers between the dependent phases:
//   A  assemble M (lower triangle, padded to a multiple of 64 with identity rows) and the right-hand side;
//   B  per block column kb: factor the 64 x 64 diagonal block (redundantly in every CTA that needs it) and
//      solve its panel tiles; barrier; update the trailing lower tiles and the right-hand side; barrier;
//   C  backward substitution by block rows, one barrier per block;
//   D  clamp lambda to [0, 1e8]; barrier; Coulomb cone per active contact and the contact right-hand side.
// The barrier is a counter + generation word with a bounded spin: a CTA that waits too long sets
// kStatusBarrierTimeout and `done` in the control block and every later barrier returns at once, so the
// kernel always ends (the host turns the status into an error).
constexpr int kNcpTile = 64;
constexpr int kNcpThreads = 256;
constexpr int kNcpLd = kNcpTile + 1;  // padded smem row (doubles) for the row-major 64 x 64 tiles
constexpr long long kBarrierSpins = 1ll << 24;

// Returns false when the grid is aborting (a barrier timed out somewhere): the caller returns.
__device__ __forceinline__ bool ncp_grid_sync(unsigned int* bar, Ctrl* ctrl) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned int* vbar = bar;
        int ok = vbar[2] == 0u;
        if (ok) {
            const unsigned int gen = vbar[1];
            __threadfence();
            const unsigned int arrived = atomicAdd(bar, 1u);
            if (arrived == gridDim.x - 1) {
                vbar[0] = 0u;
                __threadfence();
                atomicAdd(bar + 1, 1u);
            } else {
                long long spins = 0;
                while (vbar[1] == gen) {
                    if (vbar[2] != 0u || ++spins > kBarrierSpins) {
                        ok = 0;
                        break;
                    }
                    __nanosleep(64);
                }
                if (!ok && vbar[2] == 0u) {
                    atomicExch(bar + 2, 1u);
                    atomicOr(&ctrl->status, (int)kStatusBarrierTimeout);
                    ctrl->done = 1;
                }
            }
            __threadfence();
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Cholesky of the 64 x 64 lower block sD (row-major, ld kNcpLd) in place, the reference's pivot guard
// (sqrt(max(d, 1e-300))); all threads of the CTA take part.
__device__ void ncp_tile_cholesky(double* sD) {
    __shared__ double piv;
    for (int j = 0; j < kNcpTile; ++j) {
        if (threadIdx.x == 0) {
            const double d = sD[j * kNcpLd + j];
            piv = sqrt(d > 1e-300 ? d : 1e-300);
            sD[j * kNcpLd + j] = piv;
        }
        __syncthreads();
        const double inv = 1.0 / piv;
        for (int r = j + 1 + (int)threadIdx.x; r < kNcpTile; r += blockDim.x) sD[r * kNcpLd + j] *= inv;
        __syncthreads();
        const int rem = kNcpTile - j - 1;
        for (int t = threadIdx.x; t < rem * rem; t += blockDim.x) {
            const int r = j + 1 + t / rem, l = j + 1 + t % rem;
            if (l <= r) sD[r * kNcpLd + l] -= sD[r * kNcpLd + j] * sD[l * kNcpLd + j];
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kNcpThreads, 1)
k_ncp_block_solve(ContactDev c, const double* __restrict__ q0, const double* __restrict__ r64, Ctrl* ctrl) {
    extern __shared__ double smem[];
    double* sA = smem;                           // 64 x kNcpLd: diagonal block / k-major panel i
    double* sB = smem + kNcpTile * kNcpLd;       // 64 x kNcpLd: panel tile / k-major panel j
    double* sy = smem + 2 * kNcpTile * kNcpLd;   // 64: the block's right-hand side / solution
    if (ctrl->done) return;  // every CTA reads the same value: no CTA reaches a barrier the others skip
    const int ka = c.kact[0];
    const int tid = threadIdx.x, nt = blockDim.x, G = gridDim.x, bid = blockIdx.x;
    const int gt = bid * nt + tid, nthr = G * nt;
    const int lane = tid & 31, gw = gt >> 5, nwarps = nthr >> 5;
    if (ka == 0) return;
    const int nb = (ka + kNcpTile - 1) / kNcpTile, ld = nb * kNcpTile;
    double* M = c.Mwork;  // ld x ld, row-major, lower triangle used
    double* rhs = c.rhs;  // ld
    // ---- A: M and the right-hand side h - J A^-1 g (one warp per row) ----
    for (int a = gw; a < ld; a += nwarps) {
        double* Ma = M + (size_t)a * ld;
        if (a >= ka) {  // identity padding row
            for (int b = lane; b <= a; b += 32) Ma[b] = (a == b) ? 1.0 : 0.0;
            if (lane == 0) rhs[a] = 0.0;
            continue;
        }
        const double h = ncp_row(c, a, ka, lane, [&](int b, double m) {
            if (b <= a) Ma[b] = m;
        });
        if (lane == 0) rhs[a] = h;
    }
    if (!ncp_grid_sync(c.bar, ctrl)) return;
    // ---- B: blocked factorisation with the forward substitution folded in ----
    for (int kb = 0; kb < nb; ++kb) {
        const int below = nb - kb - 1;
        if (bid == 0 || bid < below) {
            const double* Dg = M + (size_t)kb * kNcpTile * ld + kb * kNcpTile;
            for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                const int r = t / kNcpTile, l = t % kNcpTile;
                if (l <= r) sA[r * kNcpLd + l] = Dg[(size_t)r * ld + l];
            }
            if (bid == 0 && tid < kNcpTile) sy[tid] = rhs[kb * kNcpTile + tid];
            __syncthreads();
            ncp_tile_cholesky(sA);
            if (bid == 0) {  // y_kb = L_kk^-1 rhs_kb (one warp, column-oriented); L_kk goes back after the barrier
                if (tid < 32) {
                    for (int j = 0; j < kNcpTile; ++j) {
                        double yj = 0.0;
                        if (lane == 0) sy[j] /= sA[j * kNcpLd + j];
                        __syncwarp();
                        yj = sy[j];
                        for (int r = j + 1 + lane; r < kNcpTile; r += 32) sy[r] -= sA[r * kNcpLd + j] * yj;
                        __syncwarp();
                    }
                }
                __syncthreads();
                if (tid < kNcpTile) rhs[kb * kNcpTile + tid] = sy[tid];  // no other CTA reads rhs_kb in this phase
            }
            // panel tiles L[i, kb] = M[i, kb] L_kk^-T
            for (int i = kb + 1 + bid; i < nb; i += G) {
                double* Pg = M + (size_t)i * kNcpTile * ld + kb * kNcpTile;
                __syncthreads();
                for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                    const int r = t / kNcpTile, l = t % kNcpTile;
                    sB[r * kNcpLd + l] = Pg[(size_t)r * ld + l];
                }
                __syncthreads();
                if (tid < kNcpTile) {  // row tid: x L_kk^T = m, four independent partial sums per dot
                    double* row = sB + tid * kNcpLd;
                    for (int j = 0; j < kNcpTile; ++j) {
                        const double* Lj = sA + j * kNcpLd;
                        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                        int l = 0;
                        for (; l + 4 <= j; l += 4) {
                            s0 += row[l] * Lj[l];
                            s1 += row[l + 1] * Lj[l + 1];
                            s2 += row[l + 2] * Lj[l + 2];
                            s3 += row[l + 3] * Lj[l + 3];
                        }
                        for (; l < j; ++l) s0 += row[l] * Lj[l];
                        row[j] = (row[j] - ((s0 + s1) + (s2 + s3))) / Lj[j];
                    }
                }
                __syncthreads();
                for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                    const int r = t / kNcpTile, l = t % kNcpTile;
                    Pg[(size_t)r * ld + l] = sB[r * kNcpLd + l];
                }
            }
        }
        if (!ncp_grid_sync(c.bar, ctrl)) return;
        // every CTA has now read M[kb][kb]: CTA 0 stores L_kk (still in its sA) in its place
        if (bid == 0) {
            double* Dw = M + (size_t)kb * kNcpTile * ld + kb * kNcpTile;
            for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                const int r = t / kNcpTile, l = t % kNcpTile;
                if (l <= r) Dw[(size_t)r * ld + l] = sA[r * kNcpLd + l];
            }
        }
        // trailing update M[i][j] -= L[i,kb] L[j,kb]^T for kb < j <= i, and rhs_i -= L[i,kb] y_kb
        const int ntri = below * (below + 1) / 2;
        const int ty = tid >> 4, tx = tid & 15;
        for (int w = bid; w < ntri + below; w += G) {
            __syncthreads();
            if (w < ntri) {
                int ii = (int)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
                while ((ii + 1) * (ii + 2) / 2 <= w) ++ii;
                while (ii * (ii + 1) / 2 > w) --ii;
                const int jj = w - ii * (ii + 1) / 2;
                const int i = kb + 1 + ii, j = kb + 1 + jj;
                const double* Pi = M + (size_t)i * kNcpTile * ld + kb * kNcpTile;
                const double* Pj = M + (size_t)j * kNcpTile * ld + kb * kNcpTile;
                // k-major copies: sA[k][r] = L[i*64 + r, kb*64 + k]
                for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                    const int r = t / kNcpTile, k = t % kNcpTile;
                    sA[k * kNcpLd + r] = Pi[(size_t)r * ld + k];
                    sB[k * kNcpLd + r] = Pj[(size_t)r * ld + k];
                }
                __syncthreads();
                double acc[4][4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] = 0.0;
#pragma unroll 4
                for (int k = 0; k < kNcpTile; ++k) {
                    double av[4], bv[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) av[u] = sA[k * kNcpLd + ty * 4 + u];
#pragma unroll
                    for (int v = 0; v < 4; ++v) bv[v] = sB[k * kNcpLd + tx * 4 + v];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * bv[v];
                }
                double* Cg = M + (size_t)i * kNcpTile * ld + j * kNcpTile;
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) Cg[(size_t)(ty * 4 + u) * ld + tx * 4 + v] -= acc[u][v];
            } else {
                const int i = kb + 1 + (w - ntri);
                if (tid < kNcpTile) {
                    const double* Li = M + (size_t)(i * kNcpTile + tid) * ld + kb * kNcpTile;
                    const double* y = rhs + kb * kNcpTile;
                    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                    for (int k = 0; k < kNcpTile; k += 4) {
                        s0 += Li[k] * y[k];
                        s1 += Li[k + 1] * y[k + 1];
                        s2 += Li[k + 2] * y[k + 2];
                        s3 += Li[k + 3] * y[k + 3];
                    }
                    rhs[i * kNcpTile + tid] -= (s0 + s1) + (s2 + s3);
                }
            }
        }
        if (!ncp_grid_sync(c.bar, ctrl)) return;
    }
    // ---- C: backward substitution L^T x = y by block rows ----
    for (int kb = nb - 1; kb >= 0; --kb) {
        if (bid == 0 || bid < kb) {
            const double* Dg = M + (size_t)kb * kNcpTile * ld + kb * kNcpTile;
            __syncthreads();
            for (int t = tid; t < kNcpTile * kNcpTile; t += nt) {
                const int r = t / kNcpTile, l = t % kNcpTile;
                if (l <= r) sA[r * kNcpLd + l] = Dg[(size_t)r * ld + l];
            }
            if (tid < kNcpTile) sy[tid] = rhs[kb * kNcpTile + tid];
            __syncthreads();
            if (tid < 32) {
                for (int j = kNcpTile - 1; j >= 0; --j) {
                    if (lane == 0) sy[j] /= sA[j * kNcpLd + j];
                    __syncwarp();
                    const double xj = sy[j];
                    for (int l = lane; l < j; l += 32) sy[l] -= sA[j * kNcpLd + l] * xj;
                    __syncwarp();
                }
            }
            __syncthreads();
            if (bid == 0 && tid < kNcpTile) c.xsol[kb * kNcpTile + tid] = sy[tid];
            // rhs_p -= L[kb, p]^T x_kb for the block rows p < kb (rhs_kb itself is only read in this phase)
            for (int p = bid; p < kb; p += G) {
                if (tid < kNcpTile) {
                    const double* Lkp = M + (size_t)kb * kNcpTile * ld + p * kNcpTile + tid;
                    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                    for (int i = 0; i < kNcpTile; i += 4) {
                        s0 += Lkp[(size_t)i * ld] * sy[i];
                        s1 += Lkp[(size_t)(i + 1) * ld] * sy[i + 1];
                        s2 += Lkp[(size_t)(i + 2) * ld] * sy[i + 2];
                        s3 += Lkp[(size_t)(i + 3) * ld] * sy[i + 3];
                    }
                    rhs[p * kNcpTile + tid] -= (s0 + s1) + (s2 + s3);
                }
            }
        }
        if (!ncp_grid_sync(c.bar, ctrl)) return;
    }
    // ---- D: multipliers, Coulomb cone, contact right-hand side ----
    for (int a = gt; a < ka; a += nthr) ncp_clamp_row(c, c.act[a], c.xsol[a]);
    if (!ncp_grid_sync(c.bar, ctrl)) return;
    for (int a = gw; a < ka; a += nwarps) ncp_finish_row(c, a, ka, lane, q0, r64);
}

// Restitution (forward_gpu.cpp:1483-1531), planar boundary.
__global__ void k_restitution(ContactDev c, double* __restrict__ q, const double* __restrict__ q0,
                              const double* __restrict__ v0, double h, double e, double slop) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.K || !(c.lam[k] > 0.0)) return;
    const int node = c.cand[k];
    const double* n = c.n;
    const double sd = n[0] * q[3 * node] + n[1] * q[3 * node + 1] + n[2] * q[3 * node + 2] + c.offset;
    if (sd > slop) return;
    const double vin = v0[3 * node] * n[0] + v0[3 * node + 1] * n[1] + v0[3 * node + 2] * n[2];
    if (!(vin < 0)) return;
    double vo = 0;
    for (int d = 0; d < 3; ++d) vo += (q[3 * node + d] - q0[3 * node + d]) / h * n[d];
    const double dv = -e * vin - vo;
    if (dv > 0)
        for (int d = 0; d < 3; ++d) q[3 * node + d] += h * dv * n[d];
}

}  // namespace

int ncp_grid() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}

size_t ncp_matrix_capacity(int K) {
    const size_t kp = ((size_t)K + kNcpTile - 1) / kNcpTile * kNcpTile;
    return kp;
}

void launch_delassus(int K, const int64_t* off, const int* prow, const double* pval, double* G, cudaStream_t st) {
    const long long npairs = (long long)K * (K + 1) / 2;
    const long long blocks = (npairs * 32 + 255) / 256;
    if (npairs > 0) k_delassus<<<(unsigned)blocks, 256, 0, st>>>(K, off, prow, pval, G);
}

void launch_ncp_iteration(const ContactDev& c, const double* x, const double* y, int npad, const double* x_base,
                          const double* q0, const double* r64, Ctrl* ctrl, cudaStream_t st) {
    launch_k(k_ncp_prepare, (c.K + kPrepThreads - 1) / kPrepThreads, kPrepThreads, 0, st, c, x, r64, ctrl);
    launch_k(k_ncp_ainvb, c.K < 4 * ncp_grid() ? c.K : 4 * ncp_grid(), kDotThreads, 0, st, c, y, npad, x_base,
             (const Ctrl*)ctrl);
    if (c.cached) {
        launch_ncp_cached_solve(c, q0, r64, ctrl, st);
        return;
    }
    // one cooperative grid of one CTA per SM (the barrier needs every CTA resident)
    const size_t smem = (size_t)(2 * kNcpTile * kNcpLd + kNcpTile) * sizeof(double);
    cudaFuncSetAttribute(k_ncp_block_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncp_grid());
    cfg.blockDim = dim3(kNcpThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_ncp_block_solve, c, q0, r64, ctrl);
}

namespace {
// One warp per row of U.  v supported on few candidates (`list`): a lane per candidate looks its path up at the row's
// depth -- the row lies on the path of candidate k exactly when the path's entry at that depth is the row -- so a row
// costs `count` look-ups instead of a pass over every candidate below it.  With every node of a block a candidate and
// 3 to 9 of them in contact the row lists hold all of S (24^3: 249 us per apply; the look-ups 6 us).  A look-up is a
// 32-byte sector where a list entry is 12 streamed bytes and a 24-byte gather, hence the factor in the rule.
constexpr int kPathLookupCost = 4;
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) k_path_apply(ContactDev c, const double* __restrict__ vsrc, int from_nodes,
                                                    const int* __restrict__ list, const int* __restrict__ count,
                                                    const TI* yin, TO* yout, int npad, const Ctrl* ctrl) {
    pdl_enter();
    if (ctrl->done) return;
    const int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (u >= c.nU) return;
    const int row = c.tp_row[u];
    const int cnt = list ? *count : 0;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (list && (long long)cnt * c.nU * kPathLookupCost <= c.tp_entries) {
        const int depth = c.tp_depth[u];
        for (int a = lane; a < cnt; a += 32) {
            const int k = list[a];
            const int64_t o = c.off[k] + depth;
            if (o < c.off[k + 1] && c.prow[o] == row) {
                const double v = c.pval[o];
                const double* src = vsrc + 3 * (size_t)(from_nodes ? c.cand[k] : k);
                s0 += v * src[0];
                s1 += v * src[1];
                s2 += v * src[2];
            }
        }
    } else {
        const int64_t e0 = c.tp_ptr[u], e1 = c.tp_ptr[u + 1];
        for (int64_t e = e0 + lane; e < e1; e += 32) {
            const int k = c.tp_k[e];
            const double v = c.tp_val[e];
            const double* src = vsrc + 3 * (size_t)(from_nodes ? c.cand[k] : k);
            s0 += v * src[0];
            s1 += v * src[1];
            s2 += v * src[2];
        }
    }
    s0 = warp_sum_d(s0);
    s1 = warp_sum_d(s1);
    s2 = warp_sum_d(s2);
    if (lane == 0) {
        const double a0 = (double)yin[row], a1 = (double)yin[npad + row], a2 = (double)yin[2 * (size_t)npad + row];
        yout[row] = (TO)(a0 + s0);
        yout[npad + row] = (TO)(a1 + s1);
        yout[2 * (size_t)npad + row] = (TO)(a2 + s2);
    }
}

__global__ void k_cand_zero(ContactDev c, const int* __restrict__ iperm, float* __restrict__ v, int npad,
                            const Ctrl* ctrl) {
    pdl_enter();
    if (ctrl->done) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.K) return;
    const int j = iperm[c.cand[k]];
    v[j] = 0.0f;
    v[npad + j] = 0.0f;
    v[2 * (size_t)npad + j] = 0.0f;
}

__global__ void k_path_gather_vals(long long E, const int64_t* __restrict__ src_e, const double* __restrict__ pval,
                                   double* __restrict__ tp_val) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < E) tp_val[i] = pval[src_e[i]];
}
}  // namespace

template <typename TI, typename TO>
void launch_path_apply(const ContactDev& c, const double* v_src, int from_nodes, const TI* y_in, TO* y_out, int npad,
                       const Ctrl* ctrl, cudaStream_t st, const int* list, const int* count) {
    if (c.nU <= 0) return;
    launch_k(k_path_apply<TI, TO>, (unsigned)(((long long)c.nU * 32 + 255) / 256), 256, 0, st, c, v_src, from_nodes,
             list, count, y_in, y_out, npad, ctrl);
}
template void launch_path_apply<double, double>(const ContactDev&, const double*, int, const double*, double*, int,
    const Ctrl*, cudaStream_t, const int*, const int*);
template void launch_path_apply<double, float>(const ContactDev&, const double*, int, const double*, float*, int,
    const Ctrl*, cudaStream_t, const int*, const int*);
template void launch_path_apply<float, double>(const ContactDev&, const double*, int, const float*, double*, int,
    const Ctrl*, cudaStream_t, const int*, const int*);
template void launch_path_apply<float, float>(const ContactDev&, const double*, int, const float*, float*, int,
    const Ctrl*, cudaStream_t, const int*, const int*);

void launch_cand_zero(const ContactDev& c, const int* iperm, float* v, int npad, const Ctrl* ctrl, cudaStream_t st) {
    if (c.K > 0) launch_k(k_cand_zero, (c.K + 255) / 256, 256, 0, st, c, iperm, v, npad, ctrl);
}

void launch_path_gather_vals(long long E, const int64_t* src_e, const double* pval, double* tp_val, cudaStream_t st) {
    if (E > 0) k_path_gather_vals<<<(unsigned)((E + 255) / 256), 256, 0, st>>>(E, src_e, pval, tp_val);
}

void launch_restitution(const ContactDev& c, double* q, const double* q0, const double* v0, double h, double e,
                        double slop, cudaStream_t st) {
    if (c.K > 0) k_restitution<<<(c.K + 255) / 256, 256, 0, st>>>(c, q, q0, v0, h, e, slop);
}

}  // namespace dphd
