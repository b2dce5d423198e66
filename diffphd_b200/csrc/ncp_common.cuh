// Parts of the NCP step shared by its solves (contact.cu, ncp_cached.cu).
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace dphd {

__device__ __forceinline__ double ncp_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// lambda_k of active row a after the dense solve: clamped to [0, 1e8] (forward_gpu.cpp:1255-1262).
__device__ __forceinline__ void ncp_clamp_row(const ContactDev& c, int k, double dlam) {
    const double l = c.lam[k] + dlam;
    c.lam[k] = l < 0.0 ? 0.0 : (l > 1e8 ? 1e8 : l);
}

// Right-hand side of active row a, h - J A^-1 g, and its row of M = Omega G Omega + E at columns b = lane, lane + 32,
// ... (one warp): `put(b, M_ab)` takes the entries; the value returned is valid in every lane.
template <typename Put>
__device__ __forceinline__ double ncp_row(const ContactDev& c, int a, int ka, int lane, Put put) {
    const int k = c.act[a];
    const double om = c.omega[k];
    const double* Gk = c.G + (size_t)k * c.K;
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    for (int b = lane; b < ka; b += 32) {
        const int kb = c.act[b];
        const double Gab = Gk[kb];
        const double fn = c.omega[kb] * c.lam[kb];
        const double f1 = c.lt1[kb], f2 = c.lt2[kb];
        g0 += Gab * (fn * c.n[0] + f1 * c.t1[0] + f2 * c.t2[0]);
        g1 += Gab * (fn * c.n[1] + f1 * c.t1[1] + f2 * c.t2[1]);
        g2 += Gab * (fn * c.n[2] + f1 * c.t1[2] + f2 * c.t2[2]);
        put(b, om * Gab * c.omega[kb] + (a == b ? c.Ediag[k] : 0.0));
    }
    g0 = ncp_warp_sum(g0) + c.ainvb[3 * a];
    g1 = ncp_warp_sum(g1) + c.ainvb[3 * a + 1];
    g2 = ncp_warp_sum(g2) + c.ainvb[3 * a + 2];
    return c.hvec[k] - om * (c.n[0] * g0 + c.n[1] * g1 + c.n[2] * g2);
}

// Coulomb cone of active row a (one warp; forward_gpu.cpp:1263-1302) and the contact right-hand side at its node,
// J^T f (plus r64 at the node): omega from this iteration times the new multipliers, written to c.vc.
__device__ __forceinline__ void ncp_finish_row(const ContactDev& c, int a, int ka, int lane,
                                               const double* __restrict__ q0, const double* __restrict__ r64) {
    const int k = c.act[a];
    const double n0 = c.n[0], n1 = c.n[1], n2 = c.n[2];
    double t1v = 0.0, t2v = 0.0;
    const int node = c.cand[k];
    if (c.mu > 0.0 && c.lam[k] > 0.0) {
        const double* Gk = c.G + (size_t)k * c.K;
        double f = 0.0;
        for (int b = lane; b < ka; b += 32) {
            const int kb = c.act[b];
            f += c.omega[kb] * c.lam[kb] * Gk[kb];
        }
        f = ncp_warp_sum(f);
        const double qn0 = c.ainvb[3 * a] + f * n0, qn1 = c.ainvb[3 * a + 1] + f * n1,
                     qn2 = c.ainvb[3 * a + 2] + f * n2;
        const double s0 = qn0 - q0[3 * node], s1 = qn1 - q0[3 * node + 1], s2 = qn2 - q0[3 * node + 2];
        const double sn = s0 * n0 + s1 * n1 + s2 * n2;
        const double u0 = s0 - sn * n0, u1 = s1 - sn * n1, u2 = s2 - sn * n2;
        const double ut1 = u0 * c.t1[0] + u1 * c.t1[1] + u2 * c.t1[2];
        const double ut2 = u0 * c.t2[0] + u1 * c.t2[1] + u2 * c.t2[2];
        const double Gkk = Gk[k];
        double st1 = 0.0, st2 = 0.0;
        if (fabs(Gkk * Gkk) > 1e-20) {
            st1 = -ut1 / Gkk;
            st2 = -ut2 / Gkk;
        }
        const double cone = c.mu * c.lam[k];
        if (sqrt(st1 * st1 + st2 * st2) <= cone + 1e-14) {
            t1v = st1;
            t2v = st2;
        } else {
            const double um = sqrt(ut1 * ut1 + ut2 * ut2);
            if (um > 1e-14) {
                t1v = -cone * ut1 / um;
                t2v = -cone * ut2 / um;
            }
        }
    }
    if (lane == 0) {
        c.lt1[k] = t1v;
        c.lt2[k] = t2v;
        const double fn = c.omega[k] * c.lam[k];
        const double r0 = r64 ? r64[3 * node] : 0.0, r1 = r64 ? r64[3 * node + 1] : 0.0,
                     r2 = r64 ? r64[3 * node + 2] : 0.0;
        c.vc[3 * (size_t)k] = r0 + fn * n0 + t1v * c.t1[0] + t2v * c.t2[0];
        c.vc[3 * (size_t)k + 1] = r1 + fn * n1 + t1v * c.t1[1] + t2v * c.t2[1];
        c.vc[3 * (size_t)k + 2] = r2 + fn * n2 + t1v * c.t1[2] + t2v * c.t2[2];
    }
}

}  // namespace dphd
