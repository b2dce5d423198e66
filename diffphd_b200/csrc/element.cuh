// Per-sample element work shared by the kernels of the iteration (kernels.cu) and the small-mesh loop (small_loop.cu):
// the same expressions in the same order, so that both give the same bits.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace dphd {

// How node values are read: ordinary loads, or loads from L2 where another CTA of the running kernel wrote them.
struct LdPlain {
    const double* __restrict__ p;
    __device__ __forceinline__ double operator()(int i) const { return p[i]; }
};
struct LdL2 {
    const double* p;
    __device__ __forceinline__ double operator()(int i) const { return __ldcg(p + i); }
};

template <typename T>
__device__ __forceinline__ T ld_weight(const ElemEnergyDev& en, int e);
template <>
__device__ __forceinline__ double ld_weight<double>(const ElemEnergyDev& en, int e) {
    return en.per_element ? __ldg(en.w + e) : en.w_mean;
}
template <>
__device__ __forceinline__ float ld_weight<float>(const ElemEnergyDev& en, int e) {
    return en.per_element ? __ldg(en.w32 + e) : (float)en.w_mean;
}

// Deformation gradient F(i,j) = sum_a x_a[i] grad_a[j] over the element's nodes (FP64 accumulation).
template <int K, class Ld>
__device__ __forceinline__ void def_grad(const int* __restrict__ E, int e, Ld x, const double* __restrict__ g,
                                         double* F) {
#pragma unroll
    for (int i = 0; i < 9; ++i) F[i] = 0.0;
#pragma unroll
    for (int a = 0; a < K; ++a) {
        const int node = __ldg(E + (size_t)e * K + a);
        const double x0 = x(3 * node), x1 = x(3 * node + 1), x2 = x(3 * node + 2);
        const double g0 = __ldg(g + a * 3), g1 = __ldg(g + a * 3 + 1), g2 = __ldg(g + a * 3 + 2);
        F[0] += x0 * g0; F[1] += x1 * g0; F[2] += x2 * g0;
        F[3] += x0 * g1; F[4] += x1 * g1; F[5] += x2 * g1;
        F[6] += x0 * g2; F[7] += x1 * g2; F[8] += x2 * g2;
    }
}

// Contribution P g_a of a sample's corner a.
__device__ __forceinline__ void corner(const double* P, const double* __restrict__ g, int a, double* c) {
    const double g0 = __ldg(g + a * 3), g1 = __ldg(g + a * 3 + 1), g2 = __ldg(g + a * 3 + 2);
#pragma unroll
    for (int i = 0; i < 3; ++i) c[i] = P[i] * g0 + P[i + 3] * g1 + P[i + 6] * g2;
}

// The 8 corners' contributions of the 8 consecutive lanes (samples) of a hex, summed over the lanes; lane l is left with
// corner l in acc.  Each step hands the half of the corners that the partner keeps to it and adds the partner's: the same
// pairs, in the same order, as a butterfly over all corners, with 21 exchanges instead of 72, and the corners are formed
// as the first step hands them over (12 live values instead of 24).
__device__ __forceinline__ void sum_samples(const double* P, const double* __restrict__ g, int smp, double* acc) {
    double c[4][3];
    const int up4 = smp & 4;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        double give[3];
        corner(P, g, a + up4, c[a]);
        corner(P, g, a + (up4 ^ 4), give);
#pragma unroll
        for (int i = 0; i < 3; ++i) c[a][i] += __shfl_xor_sync(0xffffffffu, give[i], 4);
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
        const bool up = (smp & o) != 0;
#pragma unroll
        for (int a = 0; a < o; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double keep = up ? c[a + o][i] : c[a][i], give = up ? c[a][i] : c[a + o][i];
                c[a][i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
    }
    acc[0] = c[0][0]; acc[1] = c[0][1]; acc[2] = c[0][2];
}

// Writes the sample's corner contributions P g_a to the element's slots (hexes: summed over the samples first; every lane
// of the warp calls this).
template <int K, int S>
__device__ __forceinline__ void scatter_corners(const double* P, const double* __restrict__ g, int e, int smp, bool valid,
                                                double* __restrict__ out) {
    if constexpr (S == 8) {
        double c[3];
        sum_samples(P, g, smp, c);
        if (valid) {
            double* o = out + ((size_t)e * K + smp) * 3;
            o[0] = c[0]; o[1] = c[1]; o[2] = c[2];
        }
    } else if (valid) {
#pragma unroll
        for (int a = 0; a < K; ++a) corner(P, g, a, out + ((size_t)e * K + a) * 3);
    }
}

// Node contributions of one (element, sample): sum_en w (Bp - F_bound) through the sample's gradients; the 8 samples of
// a hex (8 consecutive lanes) are summed by shuffles, so every lane of the warp calls this.
template <typename T, int K, int S, class Ld>
__device__ __forceinline__ void elem_fwd_sample(int t, int m, const int* __restrict__ E, Ld x,
                                                const double* __restrict__ qb,
                                                const unsigned char* __restrict__ elem_dir,
                                                const double* __restrict__ grad, double vol_over_s,
                                                const EnergyPack& ep, double* __restrict__ out, int* status) {
    const int e = t / S, smp = t % S;
    const bool valid = e < m;
    const double* g = (S == 8) ? grad + smp * 24 : grad + (size_t)e * 12;
    double P[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = 0.0;
    if (valid) {
        double Fd[9], Fbd[9];
        def_grad<K>(E, e, x, g, Fd);
        if (elem_dir[e]) def_grad<K>(E, e, LdPlain{qb}, g, Fbd);
        else {
#pragma unroll
            for (int i = 0; i < 9; ++i) Fbd[i] = 0.0;
        }
        T F[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i] = (T)Fd[i];
        T U[9], V[9], sig[3];
        svd3<T>(F, U, sig, V);
        bool ok = true;
        for (int k = 0; k < ep.count; ++k) {
            const ElemEnergyDev& en = ep.en[k];
            if (en.mask && !en.mask[e]) continue;
            const double w = ld_weight<double>(en, e) * vol_over_s;
            T Bp[9];
            if (sizeof(T) == 8) {
                ok = project<T>(en.type, (T)en.mu, (T)en.la, (T)en.w_mean, U, sig, V, Bp) && ok;
#pragma unroll
                for (int i = 0; i < 9; ++i) P[i] += w * ((double)Bp[i] - Fbd[i]);
            } else {
                ok = project_delta<T>(en.type, (T)en.mu, (T)en.la, (T)en.w_mean, U, sig, V, Bp) && ok;
#pragma unroll
                for (int i = 0; i < 9; ++i) P[i] += w * ((Fd[i] - Fbd[i]) + (double)Bp[i]);
            }
        }
        if (!ok) atomicOr(status, (int)kStatusSingularF);
    }
    scatter_corners<K, S>(P, g, e, smp, valid, out);
}

// The cached Jacobians are stored by blocks of 32 samples, entry by entry within a block (entry k of sample t at
// ((t / 32) 81 + k) 32 + t % 32), so that the lanes of a warp -- consecutive samples -- read and write consecutive
// addresses.  (With a sample's 81 values together, each access of a warp touched 32 lines; entry by entry over all
// samples, a warp's 81 streams lay megabytes apart.)
constexpr int kJStride = 32;
__device__ __forceinline__ size_t j_base(int t, int entries) { return (size_t)(t >> 5) * (entries * 32) + (t & 31); }

// K_pd u of one (element, sample) from its cached Jacobian; every lane of the warp calls this.
template <int K, int S, class Ld>
__device__ __forceinline__ void kpd_sample(int t, int m, const int* __restrict__ E, Ld x,
                                           const double* __restrict__ grad, const double* __restrict__ J,
                                           double* __restrict__ out) {
    const int e = t / S, smp = t % S;
    const bool valid = e < m;
    const double* g = (S == 8) ? grad + smp * 24 : grad + (size_t)e * 12;
    double P[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = 0.0;
    if (valid) {
        double dF[9];
        def_grad<K>(E, e, x, g, dF);
        constexpr int N = kJStride;
        const double* Jt = J + j_base(t, 81);
#pragma unroll
        for (int col = 0; col < 9; ++col) {
            const double f = dF[col];
#pragma unroll
            for (int i = 0; i < 9; ++i) P[i] += __ldg(Jt + (col * 9 + i) * N) * f;
        }
    }
    scatter_corners<K, S>(P, g, e, smp, valid, out);
}

}  // namespace dphd
