// The NCP's dense solve M dlambda = rhs (M = Omega G Omega + E over the ka active candidates) with a cached
// factor: the reference factors M at every PD iteration (forward_gpu.cpp:1238-1240).  Here one cooperative
// launch per PD iteration
//   A  assembles M (full rows, identity-padded to a multiple of 64) and the right-hand side, and counts the active
//      candidates that are not in the list act_ref the cached factor was built for;
//   B  when a cached factor X = L_ref^-1 of an earlier M_ref of this frame exists and the two lists differ in at
//      most kNcpMaxListChange candidates: conjugate gradients on M to |r| <= tol |rhs| (option ncp_cg_tol, 1e-13
//      by default: looser steps leave multipliers just above 0 and change the active list more often),
//      preconditioned by D^-1 X^T X D^-1 on the candidates in both lists (D = Omega Omega_ref^-1, see phase B)
//      and diag(M)^-1 on the others.  X^T X restricted to a subset of its list is the inverse of a Schur
//      complement of M_ref, so P M differs from I by the change of E between the PD iterations plus a term of
//      rank <= (dropped + 2 x new candidates); near the fixed point a few iterations suffice.  X is applied from
//      FP32 copies (the preconditioner only has to be symmetric positive definite; the residual and the iterate
//      are FP64);
//   C  otherwise (no factor, a large change of the list, or CG not converged): the blocked Cholesky of M with the
//      triangular solve of the identity folded in (X = L^-1, only the lower blocks, kept as the new cached factor),
//      then dlambda = X^T (X rhs);
//   D  clamp, Coulomb cone and the contact right-hand side, as k_ncp_block_solve.
// Both paths solve the same system (to the CG tolerance), so the iterates match the refactor-every-iteration
// solve (option ncp_solver = 0) to that level.
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "ncp_common.cuh"

namespace dphd {

namespace {

constexpr int kT = 64;
constexpr int kLd = kT + 1;
constexpr int kThr = 256;
constexpr int kNcpPcgIters = 40;       // CG iteration cap for an unchanged list; + 2 per changed candidate
constexpr int kNcpMaxListChange = 32;  // larger changes of the active list refactor at once
constexpr double kOmegaMin = 1e-6;     // |omega| below this: the candidate's row is decoupled (E only)
constexpr double kEDrift = 0.1;        // |E - (omega / omega_ref)^2 E_ref| above this fraction of M_kk: diagonal
constexpr long long kSpins = 1ll << 24;
static_assert(kNcpSmall <= kT, "a small system fits one tile of shared memory");

__device__ __forceinline__ double wsum(double v) { return ncp_warp_sum(v); }

__device__ __forceinline__ bool gsync(unsigned int* bar, Ctrl* ctrl) {
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
                    if (vbar[2] != 0u || ++spins > kSpins) {
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

// Sum of one value per CTA (part[0 .. G)), the same in every CTA: each CTA sums the partials in block order.
__device__ double grid_total(const double* part) {
    __shared__ double sh[32];
    __shared__ double tot;
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += __ldcg(part + b);
    v = wsum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
        tot = s;
    }
    __syncthreads();
    return tot;
}

// CTA partial of a value that each warp accumulated in `v` (lane 0 holds the warp's share): written to part[bid].
__device__ void cta_partial(double v, double* part) {
    __shared__ double sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
        part[blockIdx.x] = s;
    }
    __syncthreads();
}

// 64x64 Cholesky of sD (row-major, ld kLd) in place; the reference's pivot guard.
__device__ void tile_chol(double* sD) {
    __shared__ double piv;
    for (int j = 0; j < kT; ++j) {
        if (threadIdx.x == 0) {
            const double d = sD[j * kLd + j];
            piv = sqrt(d > 1e-300 ? d : 1e-300);
            sD[j * kLd + j] = piv;
        }
        __syncthreads();
        const double inv = 1.0 / piv;
        for (int r = j + 1 + (int)threadIdx.x; r < kT; r += blockDim.x) sD[r * kLd + j] *= inv;
        __syncthreads();
        const int rem = kT - j - 1;
        for (int t = threadIdx.x; t < rem * rem; t += blockDim.x) {
            const int r = j + 1 + t / rem, l = j + 1 + t % rem;
            if (l <= r) sD[r * kLd + l] -= sD[r * kLd + j] * sD[l * kLd + j];
        }
        __syncthreads();
    }
}

// acc -= A B^T for 64x64 tiles given k-major in shared memory.
__device__ __forceinline__ void tile_fma(const double* sA, const double* sB, double (&acc)[4][4]) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll 4
    for (int k = 0; k < kT; ++k) {
        double av[4], bv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) av[u] = sA[k * kLd + ty * 4 + u];
#pragma unroll
        for (int v = 0; v < 4; ++v) bv[v] = sB[k * kLd + tx * 4 + v];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * bv[v];
    }
}

// An active system of at most kNcpSmall candidates, by one CTA: M in shared memory, Cholesky, two triangular solves by
// one warp, then the multipliers and the cone.  The grid's phases below cost about 5 us per grid barrier (67 us for
// 3 to 6 active candidates); here a column costs three block barriers (kNcpSmall: where the two meet).  The cached factor
// and its list are untouched.
__device__ void small_solve(const ContactDev& c, int ka, const double* __restrict__ q0, const double* __restrict__ r64,
                            double* sM) {
    __shared__ double sx[kNcpSmall];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    for (int a = wid; a < ka; a += nw) {
        const double h = ncp_row(c, a, ka, lane, [&](int b, double m) { sM[a * kLd + b] = m; });
        if (lane == 0) sx[a] = h;
    }
    __syncthreads();
    for (int j = 0; j < ka; ++j) {
        const double d = sM[j * kLd + j];
        const double piv = sqrt(d > 1e-300 ? d : 1e-300), inv = 1.0 / piv;
        __syncthreads();  // every thread holds the pivot before column j is scaled
        for (int r = j + tid; r < ka; r += blockDim.x) sM[r * kLd + j] = r == j ? piv : sM[r * kLd + j] * inv;
        __syncthreads();
        const int rem = ka - j - 1;
        for (int t = tid; t < rem * rem; t += blockDim.x) {
            const int r = j + 1 + t / rem, l = j + 1 + t % rem;
            if (l <= r) sM[r * kLd + l] -= sM[r * kLd + j] * sM[l * kLd + j];
        }
        __syncthreads();
    }
    if (wid == 0) {
        for (int j = 0; j < ka; ++j) {  // L y = rhs
            if (lane == 0) sx[j] /= sM[j * kLd + j];
            __syncwarp();
            const double xj = sx[j];
            for (int r = j + 1 + lane; r < ka; r += 32) sx[r] -= sM[r * kLd + j] * xj;
            __syncwarp();
        }
        for (int j = ka - 1; j >= 0; --j) {  // L^T x = y
            if (lane == 0) sx[j] /= sM[j * kLd + j];
            __syncwarp();
            const double xj = sx[j];
            for (int l = lane; l < j; l += 32) sx[l] -= sM[j * kLd + l] * xj;
            __syncwarp();
        }
    }
    __syncthreads();
    if (tid < ka) ncp_clamp_row(c, c.act[tid], sx[tid]);
    __syncthreads();
    for (int a = wid; a < ka; a += nw) ncp_finish_row(c, a, ka, lane, q0, r64);
}

__global__ void __launch_bounds__(kThr, 1)
k_ncp_cached_solve(ContactDev c, const double* __restrict__ q0, const double* __restrict__ r64, Ctrl* ctrl) {
    extern __shared__ double smem[];
    double* sD = smem;
    double* sA = smem + kT * kLd;
    double* sB = smem + 2 * kT * kLd;
    if (ctrl->done) return;
    const int ka = c.kact[0];
    const int tid = threadIdx.x, nt = blockDim.x, G = gridDim.x, bid = blockIdx.x;
    const int gt = bid * nt + tid, nthr = G * nt;
    const int lane = tid & 31, gw = gt >> 5, nwarps = nthr >> 5;
    const int ldx = (int)c.kcap;
    if (ka == 0) return;
    if (ka <= kNcpSmall) {  // the same in every CTA: no grid barrier is reached
        if (bid == 0) {
            small_solve(c, ka, q0, r64, smem);
            if (tid == 0) c.ncp_stats[1] += 1;
        }
        return;
    }
    const int nb = (ka + kT - 1) / kT, ld = nb * kT;
    double* M = c.Mwork;
    double* rhs = c.rhs;
    double* x = c.xsol;
    double* dg = c.pcg + 5 * (size_t)ldx;    // diag(M)
    double* part = c.pcg + 9 * (size_t)ldx;  // per-CTA partial sums (omega_ref and E_ref, kept with the factor,
                                             // at 7 ldx and 8 ldx)
    double* part_r = part + G;               // those of r.r: no barrier lies between the total of p.w and their stores
    // [0] cached factor valid, [1] its ka, [2] candidates not in its list (this launch), [3] the last CG fell back
    int* flags = c.ncp_flags;
    const bool have = flags[0] != 0;
    const int ka_ref = have ? flags[1] : 0;
    const int ld_ref = (ka_ref + kT - 1) / kT * kT;
    // ---- A: M (full rows), diag(M), rhs, and the active candidates that are new to the cached factor's list ----
    for (int a = gt; a < ka_ref; a += nthr) c.ref_inv[a] = -1;
    int n_new_w = 0;
    for (int a = gw; a < ld; a += nwarps) {
        double* Ma = M + (size_t)a * ld;
        if (a >= ka) {
            for (int b = lane; b < ld; b += 32) Ma[b] = (a == b) ? 1.0 : 0.0;
            if (lane == 0) {
                rhs[a] = 0.0;
                dg[a] = 1.0;
            }
            continue;
        }
        const int k = c.act[a];
        if (have && lane == 0 && c.ref_pos[k] < 0) ++n_new_w;
        const double h = ncp_row(c, a, ka, lane, [&](int b, double m) {
            Ma[b] = m;
            if (a == b) dg[a] = m;
        });
        for (int b = ka + lane; b < ld; b += 32) Ma[b] = 0.0;
        if (lane == 0) rhs[a] = h;
    }
    if (n_new_w) atomicAdd(flags + 2, n_new_w);
    if (!gsync(c.bar, ctrl)) return;
    // candidates whose positions changed: new to the list, or dropped from it
    const int n_new = have ? __ldcg(flags + 2) : 0;
    const int n_chg = n_new + (ka_ref - (ka - n_new));
    bool solved = false;
    if (have && n_chg <= kNcpMaxListChange) {
        // ---- B: CG on M, preconditioned by the cached factor on the common candidates, diag(M) on the others ----
        // M = Omega G Omega + E and M_ref = Omega_r G Omega_r + E_r, so with D = Omega Omega_r^-1 (diagonal)
        // M = D M_ref D + (E - D^2 E_r): the preconditioner D^-1 X^T X D^-1 follows the change of Omega between PD
        // iterations exactly and leaves only the diagonal change of E (small for resting contacts) to CG.
        // Candidates with omega or omega_ref near 0 (decoupled rows E only), or whose E moved away from D^2 E_r by
        // more than kEDrift of their diagonal (a contact opening or closing), take the diagonal preconditioner.
        double* r = c.pcg;
        double* p = c.pcg + ldx;
        double* w = c.pcg + 2 * (size_t)ldx;
        double* t = c.pcg + 3 * (size_t)ldx;
        double* zr = c.pcg + 4 * (size_t)ldx;  // X^T X (D^-1 r) over the cached list
        double* sc = c.pcg + 6 * (size_t)ldx;  // omega_ref / omega at a scaled common candidate, else 0
        const double* om_ref = c.pcg + 7 * (size_t)ldx;
        const double* e_ref = c.pcg + 8 * (size_t)ldx;
        for (int a = gt; a < ld; a += nthr) {
            double f = 0.0;
            if (a < ka) {
                const int k = c.act[a];
                const int pr = c.ref_pos[k];
                const double om = c.omega[k];
                if (pr >= 0 && fabs(om) >= kOmegaMin && fabs(om_ref[pr]) >= kOmegaMin) {
                    const double g = om / om_ref[pr];
                    if (fabs(c.Ediag[k] - g * g * e_ref[pr]) <= kEDrift * dg[a]) {
                        f = 1.0 / g;
                        c.ref_inv[pr] = a;
                    }
                }
            }
            sc[a] = f;
        }
        if (!gsync(c.bar, ctrl)) return;
        // r = rhs, x = 0, |rhs|^2
        double acc = 0.0;
        for (int a = gt; a < ld; a += nthr) {
            const double v = a < ka ? rhs[a] : 0.0;
            r[a] = v;
            x[a] = 0.0;
            acc += v * v;
        }
        cta_partial(wsum(acc), part);
        if (!gsync(c.bar, ctrl)) return;
        const double rhs2 = grid_total(part);
        if (!gsync(c.bar, ctrl)) return;
        double rz = 0.0;
        int it = 0;
        bool conv = rhs2 == 0.0;
        // after an attempt that fell back, the next one gets a quarter of the cap (a system far from the cached one)
        const int cap = (__ldcg(flags + 3) != 0 ? kNcpPcgIters / 4 : kNcpPcgIters) + 2 * n_chg;
        while (!conv && it < cap) {
            // t = X (D^-1 r)_ref over the cached list (one warp per row; 0 at dropped or unscaled candidates)
            for (int a = gw; a < ld_ref; a += nwarps) {
                const float* Xa = c.X32 + (size_t)a * ldx;
                double s = 0.0;
                for (int b = lane; b <= a && b < ka_ref; b += 32) {
                    const int nb_ = __ldcg(c.ref_inv + b);
                    if (nb_ >= 0) s += (double)Xa[b] * (__ldcg(r + nb_) * __ldcg(sc + nb_));
                }
                s = wsum(s);
                if (lane == 0) t[a] = s;
            }
            if (!gsync(c.bar, ctrl)) return;
            // zr = X^T t (one warp per row of the stored transpose)
            for (int b = gw; b < ld_ref; b += nwarps) {
                const float* Xb = c.Xt32 + (size_t)b * ldx;
                double s = 0.0;
                for (int a = b + lane; a < ld_ref; a += 32) s += (double)Xb[a] * __ldcg(t + a);
                s = wsum(s);
                if (lane == 0) zr[b] = s;
            }
            if (!gsync(c.bar, ctrl)) return;
            // z on the current list (kept in w): D^-1 zr at the scaled candidates, r / M_aa elsewhere; rz = r . z
            acc = 0.0;
            for (int a = gt; a < ld; a += nthr) {
                const double ra = __ldcg(r + a);
                double z = ra;
                if (a < ka) {
                    const double f = __ldcg(sc + a);
                    z = f != 0.0 ? __ldcg(zr + c.ref_pos[c.act[a]]) * f : (dg[a] > 0.0 ? ra / dg[a] : ra);
                }
                w[a] = z;
                acc += ra * z;
            }
            cta_partial(wsum(acc), part);
            if (!gsync(c.bar, ctrl)) return;
            const double rz_new = grid_total(part);
            const double beta = it == 0 ? 0.0 : rz_new / rz;
            rz = rz_new;
            for (int a = gt; a < ld; a += nthr) p[a] = __ldcg(w + a) + beta * (it == 0 ? 0.0 : __ldcg(p + a));
            if (!gsync(c.bar, ctrl)) return;
            // w = M p (one warp per row), p . w
            acc = 0.0;
            for (int a = gw; a < ld; a += nwarps) {
                const double* Ma = M + (size_t)a * ld;
                double s = 0.0;
                for (int b = lane; b < ld; b += 32) s += Ma[b] * __ldcg(p + b);
                s = wsum(s);
                if (lane == 0) {
                    w[a] = s;
                    acc += s * __ldcg(p + a);
                }
            }
            cta_partial(wsum(acc), part);
            if (!gsync(c.bar, ctrl)) return;
            const double pw = grid_total(part);
            const double alpha = pw > 0.0 ? rz / pw : 0.0;
            acc = 0.0;
            for (int a = gt; a < ld; a += nthr) {
                x[a] += alpha * __ldcg(p + a);
                const double rv = __ldcg(r + a) - alpha * __ldcg(w + a);
                r[a] = rv;
                acc += rv * rv;
            }
            cta_partial(wsum(acc), part_r);
            if (!gsync(c.bar, ctrl)) return;
            const double rr = grid_total(part_r);
            ++it;
            conv = pw > 0.0 && rr <= c.cg_tol * c.cg_tol * rhs2;
            if (!gsync(c.bar, ctrl)) return;
        }
        solved = conv;
        if (gt == 0) {
            c.ncp_stats[2] += it;         // CG iterations
            if (!conv) c.ncp_stats[3] += 1;  // CG attempts that fall back to a factorisation
            flags[3] = conv ? 0 : 1;
        }
    }
    if (!solved) {
        // ---- C: blocked Cholesky of M with X = L^-1 (identity solved in place), then x = X^T X rhs ----
        double* X = c.Xinv;
        for (int k = gt; k < c.K; k += nthr) c.ref_pos[k] = -1;  // read no more in this launch (after its CG)
        for (size_t e = (size_t)gt; e < (size_t)ld * ld; e += (size_t)nthr) {
            const int a = (int)(e / ld), b = (int)(e % ld);
            X[(size_t)a * ldx + b] = a == b ? 1.0 : 0.0;
        }
        if (!gsync(c.bar, ctrl)) return;
        for (int kb = 0; kb < nb; ++kb) {
            const int below = nb - kb - 1;
            // every CTA with a panel tile or an X chunk of this block row factors the diagonal block
            const int n_items = below + (kb + 1);  // panels, then X_kb chunks of block columns 0..kb
            if (bid < n_items) {
                const double* Dg = M + (size_t)kb * kT * ld + kb * kT;
                for (int e = tid; e < kT * kT; e += nt) {
                    const int rr = e / kT, ll = e % kT;
                    if (ll <= rr) sD[rr * kLd + ll] = Dg[(size_t)rr * ld + ll];
                }
                __syncthreads();
                tile_chol(sD);
            }
            for (int item = bid; item < n_items; item += G) {
                __syncthreads();
                if (item < below) {  // panel L[i, kb] = M[i, kb] L_kk^-T
                    double* Pg = M + (size_t)(kb + 1 + item) * kT * ld + kb * kT;
                    for (int e = tid; e < kT * kT; e += nt) sA[(e / kT) * kLd + e % kT] = Pg[(size_t)(e / kT) * ld + e % kT];
                    __syncthreads();
                    if (tid < kT) {
                        double* row = sA + tid * kLd;
                        for (int j = 0; j < kT; ++j) {
                            const double* Lj = sD + j * kLd;
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
                    for (int e = tid; e < kT * kT; e += nt) Pg[(size_t)(e / kT) * ld + e % kT] = sA[(e / kT) * kLd + e % kT];
                } else {  // X_kb[:, block column cc] <- L_kk^-1 X_kb[:, cc] (cc <= kb; blocks right of kb stay 0)
                    const int cc = item - below;
                    double* Xg = X + (size_t)kb * kT * ldx + cc * kT;
                    for (int e = tid; e < kT * kT; e += nt) sA[(e / kT) * kLd + e % kT] = Xg[(size_t)(e / kT) * ldx + e % kT];
                    __syncthreads();
                    if (tid < kT) {
                        for (int rr = 0; rr < kT; ++rr) {
                            const double* Lr = sD + rr * kLd;
                            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                            int l = 0;
                            for (; l + 4 <= rr; l += 4) {
                                s0 += Lr[l] * sA[l * kLd + tid];
                                s1 += Lr[l + 1] * sA[(l + 1) * kLd + tid];
                                s2 += Lr[l + 2] * sA[(l + 2) * kLd + tid];
                                s3 += Lr[l + 3] * sA[(l + 3) * kLd + tid];
                            }
                            for (; l < rr; ++l) s0 += Lr[l] * sA[l * kLd + tid];
                            sA[rr * kLd + tid] = (sA[rr * kLd + tid] - ((s0 + s1) + (s2 + s3))) / Lr[rr];
                        }
                    }
                    __syncthreads();
                    for (int e = tid; e < kT * kT; e += nt) Xg[(size_t)(e / kT) * ldx + e % kT] = sA[(e / kT) * kLd + e % kT];
                }
            }
            if (!gsync(c.bar, ctrl)) return;
            if (bid == 0) {  // every CTA has read M[kb][kb]: store L_kk (the trailing updates read only panels)
                double* Dw = M + (size_t)kb * kT * ld + kb * kT;
                for (int e = tid; e < kT * kT; e += nt) {
                    const int rr = e / kT, ll = e % kT;
                    if (ll <= rr) Dw[(size_t)rr * ld + ll] = sD[rr * kLd + ll];
                }
            }
            // trailing updates: M[i][j] -= L[i,kb] L[j,kb]^T (kb < j <= i); X[i][cc] -= L[i,kb] X[kb][cc] (cc <= kb)
            const int ntri = below * (below + 1) / 2, nx = below * (kb + 1);
            const int ty = tid >> 4, tx = tid & 15;
            for (int item = bid; item < ntri + nx; item += G) {
                __syncthreads();
                int i, j = -1, cc = 0;
                if (item < ntri) {
                    int ii = (int)((sqrt(8.0 * (double)item + 1.0) - 1.0) * 0.5);
                    while ((ii + 1) * (ii + 2) / 2 <= item) ++ii;
                    while (ii * (ii + 1) / 2 > item) --ii;
                    i = kb + 1 + ii;
                    j = kb + 1 + (item - ii * (ii + 1) / 2);
                } else {
                    const int q = item - ntri;
                    i = kb + 1 + q / (kb + 1);
                    cc = q % (kb + 1);
                }
                const double* Pi = M + (size_t)i * kT * ld + kb * kT;
                for (int e = tid; e < kT * kT; e += nt) {
                    const int rr = e / kT, k = e % kT;
                    sA[k * kLd + rr] = Pi[(size_t)rr * ld + k];
                }
                if (j >= 0) {
                    const double* Pj = M + (size_t)j * kT * ld + kb * kT;
                    for (int e = tid; e < kT * kT; e += nt) {
                        const int rr = e / kT, k = e % kT;
                        sB[k * kLd + rr] = Pj[(size_t)rr * ld + k];
                    }
                } else {
                    const double* Yg = X + (size_t)kb * kT * ldx + cc * kT;
                    for (int e = tid; e < kT * kT; e += nt) {
                        const int k = e / kT, cl = e % kT;
                        sB[k * kLd + cl] = Yg[(size_t)k * ldx + cl];
                    }
                }
                __syncthreads();
                double acc4[4][4] = {};
                tile_fma(sA, sB, acc4);
                if (j >= 0) {
                    double* Cg = M + (size_t)i * kT * ld + j * kT;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int v = 0; v < 4; ++v) Cg[(size_t)(ty * 4 + u) * ld + tx * 4 + v] -= acc4[u][v];
                } else {
                    double* Xi = X + (size_t)i * kT * ldx + cc * kT;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int v = 0; v < 4; ++v) Xi[(size_t)(ty * 4 + u) * ldx + tx * 4 + v] -= acc4[u][v];
                }
            }
            if (!gsync(c.bar, ctrl)) return;
        }
        // the transpose of X (its lower triangle), for row-wise X^T products; then x = X^T (X rhs)
        for (size_t e = (size_t)gt; e < (size_t)ld * ld; e += (size_t)nthr) {
            const int a = (int)(e / ld), b = (int)(e % ld);
            if (b <= a) {
                const double v = X[(size_t)a * ldx + b];
                c.Xt[(size_t)b * ldx + a] = v;
                c.X32[(size_t)a * ldx + b] = (float)v;
                c.Xt32[(size_t)b * ldx + a] = (float)v;
            }
        }
        double* t = c.pcg + 3 * (size_t)ldx;
        for (int a = gw; a < ld; a += nwarps) {
            const double* Xa = X + (size_t)a * ldx;
            double s = 0.0;
            for (int b = lane; b <= a; b += 32) s += Xa[b] * rhs[b];
            s = wsum(s);
            if (lane == 0) t[a] = s;
        }
        if (!gsync(c.bar, ctrl)) return;
        for (int b = gw; b < ld; b += nwarps) {
            const double* Xb = c.Xt + (size_t)b * ldx;
            double s = 0.0;
            for (int a = b + lane; a < ld; a += 32) s += Xb[a] * __ldcg(t + a);
            s = wsum(s);
            if (lane == 0) x[b] = s;
        }
        // the new cached factor: its active list, the candidates' positions in it and their omega
        for (int a = gt; a < ka; a += nthr) {
            c.act_ref[a] = c.act[a];
            c.ref_pos[c.act[a]] = a;
            c.pcg[7 * (size_t)ldx + a] = c.omega[c.act[a]];
            c.pcg[8 * (size_t)ldx + a] = c.Ediag[c.act[a]];
        }
        if (gt == 0) {
            flags[0] = 1;
            flags[1] = ka;
            c.ncp_stats[1] += 1;  // fresh factorisations
        }
    } else if (gt == 0) {
        c.ncp_stats[0] += 1;  // solves by the cached factor
    }
    if (!gsync(c.bar, ctrl)) return;
    if (gt == 0) flags[2] = 0;  // re-armed for the next launch
    // ---- D: multipliers, Coulomb cone, contact right-hand side ----
    for (int a = gt; a < ka; a += nthr) ncp_clamp_row(c, c.act[a], x[a]);
    if (!gsync(c.bar, ctrl)) return;
    for (int a = gw; a < ka; a += nwarps) ncp_finish_row(c, a, ka, lane, q0, r64);
}

}  // namespace

void launch_ncp_cached_solve(const ContactDev& c, const double* q0, const double* r64, Ctrl* ctrl, cudaStream_t st) {
    const size_t smem = (size_t)(3 * kT * kLd) * sizeof(double);
    cudaFuncSetAttribute(k_ncp_cached_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncp_grid());
    cfg.blockDim = dim3(kThr);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_ncp_cached_solve, c, q0, r64, ctrl);
}

}  // namespace dphd
