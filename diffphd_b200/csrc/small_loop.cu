// The FP64 fixed-point loops (forward PD without contact, and the backbone adjoint) of small meshes in one kernel.
//
// A mesh of a few hundred nodes gives the iteration's eight launches almost nothing to do: on 425 nodes an iteration
// took 49 us (forward) and 42 us (adjoint), nearly all of it launch and drain of grids of 5 to 64 CTAs.  Here one
// cluster of 16 CTAs x 256 threads runs every iteration of the solve; the phases are separated by cluster barriers
// (hardware, a few hundred ns), the Anderson history stays in shared memory and registers, and every CTA takes the
// stop decision itself from the same sums.  What bounds it now is latency: the SVD's dependent divisions and roots (10
// of 30 us forward), each phase's chain of L2 loads, and fetching each phase's code anew in every iteration.
//
// Phases: element terms | node gather to the permuted right-hand side | y = S v by row groups | S^T column chunks |
// x_raw, Anderson sums | extrapolation, gate.  Every value is formed by the expressions and in the order of the kernels
// of the launched loop (kernels.cu), so both give the same bits; only the gate's sum of the projection change runs over
// other blocks.  Data that another CTA wrote is read from L2 (__ldcg): the read-only path is not coherent within a
// kernel.
#include <cuda_runtime.h>

#include "anderson.cuh"
#include "element.cuh"
#include "kernels.cuh"

namespace dphd {

namespace {

constexpr int kCtas = 16, kThr = 256;  // the launched loop's block of the Anderson sums and of the S^T chunks

struct Smem {
    double hist[2 * kMaxWindow][kThr];  // differences dG, dX by ring slot, of this CTA's block of degrees of freedom
    double red[8][3][kTileCols];        // S^T chunk sums by warp
    int2 cl[kSmallChunk];
    long long off[kSmallChunk];
    int slot[kSmallChunk];
    double y[3][kSmallChunk];
    double sh[kAaVals][32];   // per-warp sums: Gram column (m), right-hand side (m), |g|^2, |x_raw|^2
    double tot2[5];
    double gram[kMaxWindow][kMaxWindow];
    AaSystem aa;
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double gsum8(double v) {
#pragma unroll
    for (int o = kGatherLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the first `n` (<= 32) entries of a partial-sum array with stride `ld`, in every lane.
__device__ __forceinline__ double total_of(const double* part, int n, int ld, int lane) {
    return wsum(lane < n ? __ldcg(part + (size_t)lane * ld) : 0.0);
}

// y of 4 rows of a unit (k_spmv_S_units' order); every row here is a single item, its partial is y.
__device__ __forceinline__ void s_rows(const SpmvPlan<double>& p, const double* v, int w, int lane) {
    constexpr int R = kWarpRows, kParts = kUnitRows / R;
    const int4 ud = __ldg(p.unit_desc + w / kParts);
    const int r0 = (w % kParts) * R;
    const int nr = min(R, ud.y - r0), first = ud.x + r0, ncmax = ud.w;
    if (nr <= 0) return;
    const double* sp[R];
    int nc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        sp[r] = p.vals;
        nc[r] = 0;
        if (r < nr) {
            const int4 d = __ldg(p.unit_item_desc + first + r);
            sp[r] = p.vals + ((int64_t)(uint32_t)d.x | ((int64_t)d.y << 32));
            nc[r] = d.w;
        }
    }
    const double* vd[3] = {v + ud.z, v + p.npad + ud.z, v + 2 * (size_t)p.npad + ud.z};
    double acc[R][3];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = acc[r][2] = 0.0;
    for (int c = lane * 4; c < ncmax; c += 128) {
        double x[3][4], s[R][4];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double2 a = __ldcg(reinterpret_cast<const double2*>(vd[d] + c));
            const double2 b = __ldcg(reinterpret_cast<const double2*>(vd[d] + c) + 1);
            x[d][0] = a.x; x[d][1] = a.y; x[d][2] = b.x; x[d][3] = b.y;
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (c < nc[r]) {
                const double2 a = __ldg(reinterpret_cast<const double2*>(sp[r] + c));
                const double2 b = __ldg(reinterpret_cast<const double2*>(sp[r] + c) + 1);
                s[r][0] = a.x; s[r][1] = a.y; s[r][2] = b.x; s[r][3] = b.y;
            }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (c < nc[r])
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[r][0] += s[r][q] * x[0][q];
                    acc[r][1] += s[r][q] * x[1][q];
                    acc[r][2] += s[r][q] * x[2][q];
                }
    }
    // Totals of the 12 sums: each step hands the half of the values that the partner keeps to it, so a lane ends with one
    // value (the pairs and their order are those of the butterfly over each value).
    double t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = i < 3 * R ? acc[i < 3 * R ? i / 3 : 0][i % 3] : 0.0;
    int idx = 0;
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double keep = up ? t[i + h] : t[i], give = up ? t[i] : t[i + h];
            t[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
        if (up) idx += h;
    }
    const double tot = t[0] + __shfl_xor_sync(0xffffffffu, t[0], 1);
    if ((lane & 1) == 0 && idx < 3 * nr)
        p.ypart[(size_t)__ldg(p.unit_item_slot + first + idx / 3) * 3 + idx % 3] = tot;
}

template <int K, int S, int MODE>
__global__ void __launch_bounds__(kThr, 1) k_small_loop(SmallLoop a, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int cta = blockIdx.x;
    const int gw = wid * kCtas + cta;  // warps are dealt to the CTAs in turn, so that few warps' work uses every SM
    constexpr int kThreads = kCtas * kThr, kWarps = kThreads / 32;
    const int n = a.n, n3 = 3 * n, npad = a.p.npad;
    const int samples = a.m * S, sample_span = (samples + 31) / 32 * 32;
    const int nblk = (n3 + kThr - 1) / kThr;  // <= kCtas
    Ctrl* const ctrl = a.ctrl;
    const int W = ctrl->window, max_iter = ctrl->max_iter;
    const double rel_tol = ctrl->rel_tol, abs_tol = ctrl->abs_tol, clip = ctrl->clip;
    int count = 0, head = 0, iter = 0, converged = 0, status = 0, loops = 0;
    const int r = cta * kThr + tid;  // this thread's degree of freedom
    const bool own = r < n3;
    double xp = 0.0, lg = 0.0, lx = 0.0, fv = 0.0;
    bool fx = false;
    int c0 = 0, c1 = 0, col = 0;
    if (own) {
        xp = a.x[r];
        fx = a.fixed_dof[r] != 0;
        if (MODE == 0) fv = a.fixed_val[r];
        const int j = a.iperm[r / 3], tile = j / kTileCols;
        c0 = a.p.tile_chunk_ptr[tile];
        c1 = a.p.tile_chunk_ptr[tile + 1];
        col = (r % 3) * kTileCols + j % kTileCols;
    }
    double err = 0.0, xraw_norm = 0.0, dq = 0.0, rn = 0.0, pdc = 0.0, pdr = 0.0;
    bool done = false;
    while (!done) {
        // ---- element terms ----
        for (int t = gw * 32 + lane; t < sample_span; t += kThreads) {  // whole warps: sample_span is a multiple of 32
            if constexpr (MODE == 0)
                elem_fwd_sample<double, K, S>(t, a.m, a.E, LdL2{a.x}, a.qb, a.elem_dir, a.grad, a.vol_over_s, a.ep,
                                              a.elem_out, &ctrl->status);
            else
                kpd_sample<K, S>(t, a.m, a.E, LdL2{a.x}, a.grad, a.J, a.elem_out);
        }
        cluster_sync();
        // ---- node gather ----
        double g0 = 0.0, g1 = 0.0;
        for (int base = gw * (32 / kGatherLanes); base < n; base += kThreads / kGatherLanes) {
            const int i = base + lane / kGatherLanes, gl = lane & (kGatherLanes - 1);
            const bool valid = i < n, out = valid && gl < 3;  // lane d of a node's group finishes component d
            const int o = 3 * i + gl;
            double p[3] = {0.0, 0.0, 0.0}, pr = 0.0, rhs = 0.0;
            int j = 0;
            bool fix = false;
            if (out) {  // in flight together with the sums' loads
                j = a.iperm[i];
                fix = a.fixed_node[i] != 0;
                rhs = a.rhs[o];
                if (MODE == 0) pr = a.prev[o];
            }
            if (valid) {
                const int e = a.node_ptr[i + 1];
#pragma unroll 1
                for (int idx = a.node_ptr[i] + gl; idx < e; idx += 4 * kGatherLanes) {
                    int k[4];
                    double c[4][3];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        k[u] = idx + u * kGatherLanes < e ? __ldg(a.node_inc + idx + u * kGatherLanes) : -1;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (k[u] >= 0)
#pragma unroll
                            for (int d = 0; d < 3; ++d) c[u][d] = __ldcg(a.elem_out + (size_t)k[u] * 3 + d);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (k[u] >= 0)
#pragma unroll
                            for (int d = 0; d < 3; ++d) p[d] += c[u][d];
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) p[d] = gsum8(p[d]);
            if (out) {
                const double pd = gl == 0 ? p[0] : gl == 1 ? p[1] : p[2];
                double val;
                if (MODE == 0) {
                    g0 += (pd - pr) * (pd - pr);
                    g1 += pr * pr;
                    a.prev[o] = pd;
                    val = fix ? 0.0 : a.inv_h2m * rhs + pd;
                } else {
                    val = fix ? 0.0 : rhs + pd;
                }
                a.v[(size_t)gl * npad + j] = val;
            }
        }
        if (MODE == 0) {  // |d pd|^2, |pd|^2 of this CTA
            g0 = wsum(g0);
            g1 = wsum(g1);
            if (lane == 0) {
                s.sh[0][wid] = g0;
                s.sh[1][wid] = g1;
            }
            __syncthreads();
            if (wid < 2) {
                const double t = wsum(lane < kThr / 32 ? s.sh[wid][lane] : 0.0);
                if (lane == 0) a.part_gate[2 * cta + wid] = t;
            }
        }
        cluster_sync();
        // ---- y = S v ----
        for (int w = gw; w < a.p.n_units * (kUnitRows / kWarpRows); w += kWarps) s_rows(a.p, a.v, w, lane);
        cluster_sync();
        // ---- S^T chunks: one per CTA (k_spmv_ST_part's order) ----
        for (int ch = cta; ch < a.p.n_chunks; ch += kCtas) {
            const int p0 = __ldg(a.p.chunk_p0 + ch), cnt = __ldg(a.p.chunk_p1 + ch) - p0;
            const int c = __ldg(a.p.chunk_tile + ch) * kTileCols + lane * 4;
            for (int t = tid; t < cnt; t += kThr) {
                if (loops == 0 || a.p.n_chunks > kCtas) {  // one chunk a CTA: its rows stay in place
                    const int4 dd = __ldg(a.p.trow_desc + p0 + t);
                    s.cl[t] = make_int2(dd.x, dd.y);
                    s.off[t] = __ldg(a.p.trow_off + p0 + t);
                    s.slot[t] = dd.z;
                }
                const double* y = a.p.ypart + 3 * (size_t)s.slot[t];
#pragma unroll
                for (int d = 0; d < 3; ++d) s.y[d][t] = __ldcg(y + d);
            }
            __syncthreads();
            double acc[3][4];
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[d][q] = 0.0;
            for (int b = wid; b < cnt; b += 32) {
                double sv[4][4];
                bool in[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int t = b + 8 * u;
                    in[u] = false;
                    if (t < cnt) {
                        const int2 cl = s.cl[t];
                        in[u] = cl.y > 0 && c >= cl.x && c + 4 <= cl.x + cl.y;
                        if (in[u]) {
                            const double2* q = reinterpret_cast<const double2*>(a.p.vals + s.off[t] + (c - cl.x));
                            const double2 x0 = __ldg(q), x1 = __ldg(q + 1);
                            sv[u][0] = x0.x; sv[u][1] = x0.y; sv[u][2] = x1.x; sv[u][3] = x1.y;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (in[u]) {
                        const int t = b + 8 * u;
                        const double y0 = s.y[0][t], y1 = s.y[1][t], y2 = s.y[2][t];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            acc[0][q] += sv[u][q] * y0;
                            acc[1][q] += sv[u][q] * y1;
                            acc[2][q] += sv[u][q] * y2;
                        }
                    }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int q = 0; q < 4; ++q) s.red[wid][d][lane * 4 + q] = acc[d][q];
            __syncthreads();
            for (int t = tid; t < 3 * kTileCols; t += kThr) {
                const int d = t / kTileCols, cc = t % kTileCols;
                double sum = 0.0;
#pragma unroll
                for (int w = 0; w < 8; ++w) sum += s.red[w][d][cc];
                a.p.xpart[(size_t)ch * 3 * kTileCols + t] = sum;
            }
            __syncthreads();
        }
        cluster_sync();
        // ---- x_raw (ordered chunk sums) and the Anderson sums (k_aa_reduce's blocks) ----
        const int m = W > 0 ? count : 0;
        const int nv = 2 * m + 2;
        double xv = 0.0, g = 0.0, gnew = 0.0;
        if (own) {
#pragma unroll 1
            for (int ch = c0; ch < c1; ch += 8) {
                double t8[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    t8[u] = ch + u < c1 ? __ldcg(a.p.xpart + (size_t)(ch + u) * 3 * kTileCols + col) : 0.0;
#pragma unroll
                for (int u = 0; u < 8; ++u) xv += t8[u];
            }
            if (fx) xv = fv;  // 0 in the adjoint
            g = xv - xp;
            if (W > 0) {
                if (count >= 1) {
                    const int sl = (head + count - 1) % W;
                    gnew = g - lg;
                    s.hist[sl][tid] = gnew;
                    s.hist[kMaxWindow + sl][tid] = xp - lx;
                }
                lg = g;
                lx = xp;
            }
        }
        if (cta < nblk) {
#pragma unroll 1
            for (int j = 0; j < m; ++j) {
                const double dgj = own ? s.hist[(head + j) % W][tid] : 0.0;
                const double t0 = wsum(gnew * dgj), t1 = wsum(dgj * g);
                if (lane == 0) {
                    s.sh[j][wid] = t0;
                    s.sh[m + j][wid] = t1;
                }
            }
            const double t0 = wsum(g * g), t1 = wsum(xv * xv);
            if (lane == 0) {
                s.sh[2 * m][wid] = t0;
                s.sh[2 * m + 1][wid] = t1;
            }
            __syncthreads();
#pragma unroll 1
            for (int i = wid; i < nv; i += kThr / 32) {
                const double t = wsum(lane < kThr / 32 ? s.sh[i][lane] : 0.0);
                if (lane == 0) a.part_aa[(size_t)cta * kAaVals + i] = t;
            }
        }
        cluster_sync();
#pragma unroll 1
        for (int i = wid; i < nv; i += kThr / 32) {
            const double t = total_of(a.part_aa + i, nblk, kAaVals, lane);
            if (lane == 0) s.aa.tot[i] = t;
        }
        __syncthreads();
        err = sqrt(s.aa.tot[2 * m]);
        xraw_norm = sqrt(s.aa.tot[2 * m + 1]);
        const bool diverged = MODE == 1 && (!(xraw_norm == xraw_norm) || xraw_norm > 1e300 ||
                                            (clip > 0 && xraw_norm > clip));
        if (diverged)
            status |= (xraw_norm == xraw_norm && xraw_norm <= 1e300) ? (int)kStatusDiverged
                                                                     : (int)(kStatusDiverged | kStatusNonFinite);
        if (wid == 0) {
            if (lane == 0) s.aa.accept = s.aa.restart = 0;
            __syncwarp();
            if (!diverged && m >= 1) aa_solve_warp(s.aa, s.gram, m, head, W, lane);
        }
        __syncthreads();
        // ---- extrapolation, Dirichlet values, gate (k_aa_update's blocks) ----
        const int accept = s.aa.accept, restart = s.aa.restart;
        double u3[3] = {0.0, 0.0, 0.0};
        if (own) {
            double xn = xv;
            if (accept) {
#pragma unroll 1
                for (int j = 0; j < m; ++j) {
                    const int sl = (head + j) % W;
                    xn -= (s.hist[kMaxWindow + sl][tid] + s.hist[sl][tid]) * s.aa.gamma[j];
                }
                if (fx) xn = fv;
            }
            a.x[r] = xn;
            u3[0] += (xn - xp) * (xn - xp);
            u3[1] += xp * xp;
            u3[2] += xn * xn;
            xp = xn;
        }
        if (cta < nblk) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double t = wsum(u3[i]);
                if (lane == 0) s.sh[i][wid] = t;
            }
            __syncthreads();
            if (wid < 3) {
                const double t = wsum(lane < kThr / 32 ? s.sh[wid][lane] : 0.0);
                if (lane == 0) a.part_upd[3 * cta + wid] = t;
            }
        }
        cluster_sync();
        if (wid < 3) {
            const double t = total_of(a.part_upd + wid, nblk, 3, lane);
            if (lane == 0) s.tot2[wid] = t;
        } else if (wid < 5 && MODE == 0) {
            const double t = total_of(a.part_gate + (wid - 3), kCtas, 2, lane);
            if (lane == 0) s.tot2[wid] = t;
        }
        __syncthreads();
        dq = sqrt(s.tot2[0]);
        const double xnorm = sqrt(s.tot2[2]);
        bool conv;
        if (MODE == 0) {
            rn = sqrt(s.tot2[1]);
            pdc = sqrt(s.tot2[3]);
            pdr = sqrt(s.tot2[4]);
            conv = iter > 0 && dq <= rel_tol * rn + abs_tol && pdc <= rel_tol * pdr + abs_tol;
            if (!(dq == dq) || !(pdc == pdc)) status |= kStatusNonFinite;
        } else {
            rn = xnorm;
            conv = iter > 0 && err < rel_tol * xnorm + abs_tol;
            if (!(xnorm == xnorm)) status |= kStatusNonFinite | kStatusDiverged;
            else if (clip > 0 && xnorm > clip) status |= kStatusDiverged;
        }
        if (W > 0) {
            if (restart) {
                count = 0;
                head = 0;
            } else if (++count > W) {
                count = W;
                head = (head + 1) % W;
            }
        }
        ++iter;
        ++loops;
        if (conv) converged = 1;
        done = conv || iter >= max_iter || (status & (kStatusNonFinite | kStatusDiverged)) || loops >= cap;
        __syncthreads();  // the shared sums are read before the next iteration writes them
    }
    if (cta == 0 && tid == 0) {
        ctrl->iter = iter;
        ctrl->converged = converged;
        ctrl->count = count;
        ctrl->head = head;
        ctrl->dq = dq;
        ctrl->rn = rn;
        ctrl->pdc = pdc;
        ctrl->pdr = pdr;
        ctrl->err = err;
        ctrl->xn = xraw_norm;
        ctrl->loops = loops;
        ctrl->done = 1;
        if (status) atomicOr(&ctrl->status, status);
    }
}

using Kernel = void (*)(SmallLoop, int);
Kernel kernel_of(bool hex, int mode) {
    if (hex) return mode == 0 ? k_small_loop<8, 8, 0> : k_small_loop<8, 8, 1>;
    return mode == 0 ? k_small_loop<4, 1, 0> : k_small_loop<4, 1, 1>;
}

cudaLaunchConfig_t config(cudaLaunchAttribute* attr, cudaStream_t st) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCtas);
    cfg.blockDim = dim3(kThr);
    cfg.dynamicSmemBytes = sizeof(Smem);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

// Whether a 16-CTA cluster of the kernel fits the current device (non-portable cluster size).
bool small_loop_supported(bool hex) {
    for (int mode = 0; mode < 2; ++mode) {
        const void* f = reinterpret_cast<const void*>(kernel_of(hex, mode));
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = config(attr, nullptr);
        int clusters = 0;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            return false;
        }
    }
    return true;
}

void launch_small_loop(const SmallLoop& a, bool hex, int mode, int cap, cudaStream_t st) {
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = config(attr, st);
    cudaLaunchKernelEx(&cfg, kernel_of(hex, mode), a, cap);
}

}  // namespace dphd
