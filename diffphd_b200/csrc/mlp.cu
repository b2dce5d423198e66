// Learned warm start of the PD fixed point: a per-node MLP 15 -> 128 -> 128 -> 3 (GELU), BF16 weights and
// activations on the tensor cores (mma.sync m16n8k16, FP32 accumulation), FP32 master weights and AdamW.
//
// Layout.  Rows are nodes (one sample = one node at one time step); a CTA owns 128 rows, in groups of 16.  In
// k_mlp_forward a warp owns a group and the three layers are chained in registers: the FP32 accumulator fragment of one
// layer is the BF16 A-operand fragment of the next (columns 16kk..16kk+15 of the next layer's K are the n-tiles
// 2kk, 2kk+1 of the previous layer's output).  Weight matrices live in shared memory in the "col" layout the
// B operand wants (W^T, i.e. [out][in] with `in` contiguous).
//
// Training step (k_mlp_train): two warps share a group; each layer's rows are staged in shared memory, where the next
// one and the weight-gradient partials (x^T dz1, a1^T dz2, a2^T dz3: tensor-core MMAs over the 128 rows) read
// them; k_mlp_adamw sums the CTA
// partials in a fixed order (deterministic), applies AdamW to the FP32 master weights and re-packs the BF16
// copies.  Features are built on the device by k_mlp_features.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"

namespace dphd {

constexpr int kIn = 16, kHid = 128, kOut = 8, kOutUsed = 4;
constexpr int kRowsPerCta = 128;
// per-CTA gradient partial: W1 [16][128], W2 [128][128], W3 [128][8], b1, b2 [128], b3 [8], loss
constexpr int kPartW1 = 0, kPartW2 = kPartW1 + kIn * kHid, kPartW3 = kPartW2 + kHid * kHid;
constexpr int kPartB1 = kPartW3 + kHid * kOut, kPartB2 = kPartB1 + kHid, kPartB3 = kPartB2 + kHid;
constexpr int kPartLoss = kPartB3 + kOut, kPartSize = kPartLoss + 8;

struct MlpParams {
    // FP32 masters (row-major [in][out]) and biases
    float* W1;  // 16 x 128
    float* W2;  // 128 x 128
    float* W3;  // 128 x 8
    float* b1;
    float* b2;
    float* b3;
    // BF16 operand copies
    __nv_bfloat16* W1T;  // [128][16]  forward layer 1 (B, col)
    __nv_bfloat16* W2T;  // [128][128] forward layer 2
    __nv_bfloat16* W3T;  // [8][128]   forward layer 3
    __nv_bfloat16* W2b;  // [128][128] backward through layer 2 ([in][out])
    __nv_bfloat16* W3b;  // [128][16]  backward through layer 3 ([hidden][out], out padded to 16)
};

namespace {

__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint32_t pair16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// Shared-memory tiles of 128 BF16 columns: the eight-column chunk c of row r is stored at chunk c ^ (r & 7), so that the
// fragment loads below (the same chunk of eight consecutive rows, 256 bytes apart) touch all banks instead of four.
__device__ __forceinline__ int swz(int row, int col) { return row * 128 + (((col >> 3) ^ (row & 7)) << 3) + (col & 7); }

// Four (two) 8x8 BF16 matrices; `p`: this lane's 16-byte row (lanes 8 i .. 8 i + 7: the rows of matrix i).  Lane (g, t)
// receives elements (g, 2t), (g, 2t + 1) of each, or with trans (2t, g), (2t + 1, g).
__device__ __forceinline__ void ldsm4(const __nv_bfloat16* p, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm4t(const __nv_bfloat16* p, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm2t(const __nv_bfloat16* p, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * expf(-0.5f * x * x);
}

struct Smem {
    __align__(16) __nv_bfloat16 W1T[kHid * kIn];
    __align__(16) __nv_bfloat16 W2T[kHid * kHid];  // swizzled
    __align__(16) __nv_bfloat16 W3T[kOut * kHid];  // swizzled
    float b1[kHid], b2[kHid], b3[kOut];
};
struct SmemTrain {
    Smem f;
    __align__(16) __nv_bfloat16 W2b[kHid * kHid];  // swizzled
    __align__(16) __nv_bfloat16 W3b[kHid * 16];
    // staged CTA rows for the weight gradients (128-column tiles swizzled)
    __align__(16) __nv_bfloat16 x[kRowsPerCta * kIn];
    __align__(16) __nv_bfloat16 a1[kRowsPerCta * kHid];
    __align__(16) __nv_bfloat16 a2[kRowsPerCta * kHid];
    __align__(16) __nv_bfloat16 dz1[kRowsPerCta * kHid];
    __align__(16) __nv_bfloat16 dz2[kRowsPerCta * kHid];
    __align__(16) __nv_bfloat16 dz3[kRowsPerCta * 16];
    float red[8][kHid * 2 + kOut + 1];
};

// Eight BF16 of the packed weights: one load where they lie on a 16-byte boundary (the caller's array may not).
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* src) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) return *reinterpret_cast<const uint4*>(src);
    return make_uint4(pair16(src[0], src[1]), pair16(src[2], src[3]), pair16(src[4], src[5]), pair16(src[6], src[7]));
}
// `rows` x 128 BF16 into a swizzled tile, and `count` of them as they are.
__device__ __forceinline__ void copy_swz(__nv_bfloat16* dst, const __nv_bfloat16* src, int rows) {
    for (int i = threadIdx.x; i < rows * 16; i += blockDim.x)
        *reinterpret_cast<uint4*>(dst + swz(i >> 4, (i & 15) * 8)) = load8(src + 8 * i);
}
__device__ __forceinline__ void copy_plain(__nv_bfloat16* dst, const __nv_bfloat16* src, int count) {
    for (int i = threadIdx.x; i < count / 8; i += blockDim.x) *reinterpret_cast<uint4*>(dst + 8 * i) = load8(src + 8 * i);
}

__device__ void load_weights(Smem& s, const MlpParams& p) {
    copy_plain(s.W1T, p.W1T, kHid * kIn);
    copy_swz(s.W2T, p.W2T, kHid);
    copy_swz(s.W3T, p.W3T, kOut);
    for (int i = threadIdx.x; i < kHid; i += blockDim.x) {
        s.b1[i] = p.b1[i];
        s.b2[i] = p.b2[i];
    }
    if (threadIdx.x < kOut) s.b3[threadIdx.x] = p.b3[threadIdx.x];
}

// A fragment of the 16-row input tile (rows r0.., 16 features, row stride kIn), zero rows beyond n.
__device__ __forceinline__ void load_x(const __nv_bfloat16* X, int r0, int n, uint32_t* a) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int ra = r0 + g, rb = r0 + g + 8;
    a[0] = ra < n ? ld32(X + (size_t)ra * kIn + 2 * t) : 0u;
    a[1] = rb < n ? ld32(X + (size_t)rb * kIn + 2 * t) : 0u;
    a[2] = ra < n ? ld32(X + (size_t)ra * kIn + 2 * t + 8) : 0u;
    a[3] = rb < n ? ld32(X + (size_t)rb * kIn + 2 * t + 8) : 0u;
}

// Layer 1 pre-activations (16 rows, NJ 8-column tiles from tile j0) for one warp.
template <int NJ>
__device__ __forceinline__ void layer1(const Smem& s, const uint32_t* ax, float (*z)[4], int j0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int jj = 0; jj < NJ; ++jj) {
        const int j = j0 + jj;
        const uint32_t b[2] = {ld32(&s.W1T[(8 * j + g) * kIn + 2 * t]), ld32(&s.W1T[(8 * j + g) * kIn + 2 * t + 8])};
        z[jj][0] = s.b1[8 * j + 2 * t];
        z[jj][1] = s.b1[8 * j + 2 * t + 1];
        z[jj][2] = z[jj][0];
        z[jj][3] = z[jj][1];
        mma16816(z[jj], ax, b);
    }
}

// 16x128 activation (FP32 fragments) -> 8 BF16 A fragments.
__device__ __forceinline__ void to_afrag(float (*c)[4], uint32_t (*a)[4]) {
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
        a[kk][0] = pack_bf16(c[2 * kk][0], c[2 * kk][1]);
        a[kk][1] = pack_bf16(c[2 * kk][2], c[2 * kk][3]);
        a[kk][2] = pack_bf16(c[2 * kk + 1][0], c[2 * kk + 1][1]);
        a[kk][3] = pack_bf16(c[2 * kk + 1][2], c[2 * kk + 1][3]);
    }
}

// C (16 x 128) = A (16 x 128, 8 k-steps) * B, B from swizzled [n][k] storage, plus bias.  The k-steps are the outer loop:
// the sixteen accumulators are independent, and each still adds its k-steps in order.
__device__ __forceinline__ void layer_hh(const __nv_bfloat16* BT, const float* bias, uint32_t (*a)[4],
                                         float (*c)[4]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const int mat = lane >> 3, mr = lane & 7;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        c[j][0] = bias ? bias[8 * j + 2 * t] : 0.f;
        c[j][1] = bias ? bias[8 * j + 2 * t + 1] : 0.f;
        c[j][2] = c[j][0];
        c[j][3] = c[j][1];
    }
#pragma unroll
    for (int kk = 0; kk < 8; kk += 2)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            uint32_t b[4];  // two k-steps
            ldsm4(BT + swz(8 * j + mr, 16 * kk + 8 * mat), b);
            mma16816(c[j], a[kk], b);
            mma16816(c[j], a[kk + 1], b + 2);
        }
}

// A fragment (16 rows from r0, k-step kk) of a swizzled row tile.
__device__ __forceinline__ void ld_afrag(const __nv_bfloat16* tile, int r0, int kk, uint32_t* a) {
    const int lane = threadIdx.x & 31, mat = lane >> 3, mr = lane & 7;
    ldsm4(tile + swz(r0 + (mat & 1) * 8 + mr, 16 * kk + (mat >> 1) * 8), a);
}

// layer_hh with A from a swizzled row tile (rows r0..r0+15), for the eight 8-column tiles from j0.
__device__ __forceinline__ void layer_tile(const __nv_bfloat16* BT, const float* bias, const __nv_bfloat16* rows, int r0,
                                           int j0, float (*c)[4]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const int mat = lane >> 3, mr = lane & 7;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
        c[jj][0] = bias ? bias[8 * (j0 + jj) + 2 * t] : 0.f;
        c[jj][1] = bias ? bias[8 * (j0 + jj) + 2 * t + 1] : 0.f;
        c[jj][2] = c[jj][0];
        c[jj][3] = c[jj][1];
    }
#pragma unroll 2  // fully unrolled, the hoisted loads spill
    for (int kk = 0; kk < 8; kk += 2) {
        uint32_t a[2][4];
        ld_afrag(rows, r0, kk, a[0]);
        ld_afrag(rows, r0, kk + 1, a[1]);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            uint32_t b[4];  // two k-steps
            ldsm4(BT + swz(8 * (j0 + jj) + mr, 16 * kk + 8 * mat), b);
            mma16816(c[jj], a[0], b);
            mma16816(c[jj], a[1], b + 2);
        }
    }
}

// Output layer of one warp's 16 rows; afrag(kk, a): the A fragment of k-step kk.
template <class AFrag>
__device__ __forceinline__ void layer3(const Smem& s, AFrag afrag, float* c) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const int mat = lane >> 3, mr = lane & 7;
    c[0] = s.b3[2 * t];
    c[1] = s.b3[2 * t + 1];
    c[2] = c[0];
    c[3] = c[1];
#pragma unroll
    for (int kk = 0; kk < 8; kk += 2) {
        uint32_t b[4], a[2][4];
        afrag(kk, a[0]);
        afrag(kk + 1, a[1]);
        ldsm4(s.W3T + swz(mr, 16 * kk + 8 * mat), b);
        mma16816(c, a[0], b);
        mma16816(c, a[1], b + 2);
    }
}

__global__ void __launch_bounds__(256) k_mlp_forward(MlpParams p, const __nv_bfloat16* __restrict__ X, int n,
                                                     float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    load_weights(s, p);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * kRowsPerCta + warp * 16;
    if (r0 >= n) return;
    uint32_t ax[4];
    load_x(X, r0, n, ax);
    float z[16][4];
    layer1<16>(s, ax, z, 0);
#pragma unroll
    for (int j = 0; j < 16; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) z[j][e] = gelu(z[j][e]);
    uint32_t a[8][4];
    to_afrag(z, a);
    layer_hh(s.W2T, s.b2, a, z);
#pragma unroll
    for (int j = 0; j < 16; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) z[j][e] = gelu(z[j][e]);
    to_afrag(z, a);
    float o[4];
    layer3(s, [&](int kk, uint32_t* f) {
        for (int e = 0; e < 4; ++e) f[e] = a[kk][e];
    }, o);
    const int ra = r0 + g, rb = r0 + g + 8;
    if (ra < n) { out[(size_t)ra * kOut + 2 * t] = o[0]; out[(size_t)ra * kOut + 2 * t + 1] = o[1]; }
    if (rb < n) { out[(size_t)rb * kOut + 2 * t] = o[2]; out[(size_t)rb * kOut + 2 * t + 1] = o[3]; }
}

// Column sums over the warp's 16 rows of a 16x8 FP32 fragment (valid in lanes 0..3: cols 2t, 2t+1).
__device__ __forceinline__ void colsum(const float* c, float& s0, float& s1) {
    s0 = c[0] + c[2];
    s1 = c[1] + c[3];
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
}

// One training step, a tile of 128 rows after another: MSE(out[:, :3], Y) / n_total, a gradient partial per tile.
// Bound by the erf / exp arithmetic of the activations and its latency; the staged rows and both weight orders fill the
// SM's shared memory, so one CTA an SM.  Two warps share 16 rows, each with half of every layer's columns, and hand the
// halves over through the staged row tiles: sixteen warps hide what eight (one per 16 rows, activations chained in
// registers) left exposed.  A step on 65,536 rows (this kernel and the AdamW one): 157 us with eight, 116 with sixteen;
// 104 with one CTA an SM that keeps the weights for all its tiles and loads the next tile's rows ahead.
constexpr int kTrainThreads = 512;
__global__ void __launch_bounds__(kTrainThreads) k_mlp_train(MlpParams p, const __nv_bfloat16* __restrict__ X,
                                                             const float* __restrict__ Y, int n, float inv_n,
                                                             float* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemTrain& s = *reinterpret_cast<SmemTrain*>(smem_raw);
    load_weights(s.f, p);
    copy_swz(s.W2b, p.W2b, kHid);
    copy_plain(s.W3b, p.W3b, kHid * 16);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rw = warp & 7, half = warp >> 3, j0 = 8 * half;  // 16-row group, column half, its first 8-column tile
    const int rl = rw * 16;                                    // local row base
    // the two warps of a row group have written their halves of a row tile
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + rw) : "memory"); };
    auto put = [&](__nv_bfloat16* at, uint32_t v) { *reinterpret_cast<uint32_t*>(at) = v; };
    // one 8-column accumulator tile of the warp's rows, as BF16
    auto stage = [&](__nv_bfloat16* dst, int j, uint32_t lo, uint32_t hi) {
        put(dst + swz(rl + g, 8 * j + 2 * t), lo);
        put(dst + swz(rl + g + 8, 8 * j + 2 * t), hi);
    };
    auto stage16 = [&](__nv_bfloat16* dst, const uint32_t* fr) {  // 16 columns
        put(dst + (rl + g) * 16 + 2 * t, fr[0]);
        put(dst + (rl + g + 8) * 16 + 2 * t, fr[1]);
        put(dst + (rl + g) * 16 + 2 * t + 8, fr[2]);
        put(dst + (rl + g + 8) * 16 + 2 * t + 8, fr[3]);
    };
    // gelu'(z) is parked (BF16) in the tile of dz, which each thread later overwrites at the same positions
    auto activate = [&](float (*c)[4], __nv_bfloat16* act, __nv_bfloat16* dz) {
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            float* z = c[jj];
            stage(dz, j0 + jj, pack_bf16(gelu_d(z[0]), gelu_d(z[1])), pack_bf16(gelu_d(z[2]), gelu_d(z[3])));
            stage(act, j0 + jj, pack_bf16(gelu(z[0]), gelu(z[1])), pack_bf16(gelu(z[2]), gelu(z[3])));
        }
    };
    const int tiles = (n + kRowsPerCta - 1) / kRowsPerCta;
    uint32_t ax[4];
    load_x(X, blockIdx.x * kRowsPerCta + rl, n, ax);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int r0 = tile * kRowsPerCta + rl;
        // ---- forward ----
        if (half == 0) stage16(s.x, ax);
        float c[8][4];
        layer1<8>(s.f, ax, c, j0);  // z1
        activate(c, s.a1, s.dz1);
        pair_sync();
        layer_tile(s.f.W2T, s.f.b2, s.a1, rl, j0, c);  // z2
        activate(c, s.a2, s.dz2);
        pair_sync();
        float o[4];  // both warps of the pair
        layer3(s.f, [&](int kk, uint32_t* a) { ld_afrag(s.a2, rl, kk, a); }, o);
        // ---- loss gradient dz3 = 2 (pred - y) / n (3 used outputs), and the loss ----
        const int ra = r0 + g, rb = r0 + g + 8;
        float dz3[4] = {0.f, 0.f, 0.f, 0.f}, lsum = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = e < 2 ? ra : rb, col = 2 * t + (e & 1);
            if (row < n && col < kOutUsed) {
                const float d = o[e] - Y[(size_t)row * kOutUsed + col];
                dz3[e] = 2.f * d * inv_n;
                lsum += d * d;
            }
        }
        // ---- backward ----
        const uint32_t adz3[4] = {pack_bf16(dz3[0], dz3[1]), pack_bf16(dz3[2], dz3[3]), 0u, 0u};
        float bs[2];
        if (half == 0) {
            stage16(s.dz3, adz3);
            colsum(dz3, bs[0], bs[1]);
            if (lane < 4) {
                s.red[rw][2 * kHid + 2 * lane] = bs[0];
                s.red[rw][2 * kHid + 2 * lane + 1] = bs[1];
            }
            float ls = lsum;
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, of);
            if (lane == 0) s.red[rw][2 * kHid + kOut] = ls;
        }
        // times the parked gelu', column sums for the bias gradient, and the tile itself
        auto finish = [&](float* cj, __nv_bfloat16* dz, int j, int red0) {
            const float2 lo =
                __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dz + swz(rl + g, 8 * j + 2 * t)));
            const float2 hi =
                __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dz + swz(rl + g + 8, 8 * j + 2 * t)));
            cj[0] *= lo.x;
            cj[1] *= lo.y;
            cj[2] *= hi.x;
            cj[3] *= hi.y;
            colsum(cj, bs[0], bs[1]);
            if (lane < 4) {
                s.red[rw][red0 + 8 * j + 2 * lane] = bs[0];
                s.red[rw][red0 + 8 * j + 2 * lane + 1] = bs[1];
            }
            stage(dz, j, pack_bf16(cj[0], cj[1]), pack_bf16(cj[2], cj[3]));
        };
        // da2 = dz3 W3^T  (K = outputs padded to 16); dz2 = da2 * gelu'(z2)
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            const int j = j0 + jj;
            c[jj][0] = c[jj][1] = c[jj][2] = c[jj][3] = 0.f;
            const uint32_t b[2] = {ld32(&s.W3b[(8 * j + g) * 16 + 2 * t]), ld32(&s.W3b[(8 * j + g) * 16 + 2 * t + 8])};
            mma16816(c[jj], adz3, b);
            finish(c[jj], s.dz2, j, kHid);
        }
        pair_sync();
        // da1 = dz2 W2^T, B from W2b ([in][out]); dz1 = da1 * gelu'(z1)
        layer_tile(s.W2b, nullptr, s.dz2, rl, j0, c);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) finish(c[jj], s.dz1, j0 + jj, 0);
        __syncthreads();
        float* P = part + (size_t)tile * kPartSize;
        if (tile + (int)gridDim.x < tiles) load_x(X, r0 + (int)gridDim.x * kRowsPerCta, n, ax);  // the next tile's rows
        // biases and loss (fixed order of the row groups)
        for (int i = threadIdx.x; i < 2 * kHid + kOut + 1; i += blockDim.x) {
            float v = 0.f;
            for (int w = 0; w < 8; ++w) v += s.red[w][i];
            if (i < kHid) P[kPartB1 + i] = v;
            else if (i < 2 * kHid) P[kPartB2 + i - kHid] = v;
            else if (i < 2 * kHid + kOut) P[kPartB3 + i - 2 * kHid] = v;
            else P[kPartLoss] = v;
        }
        // ---- weight gradients over the CTA's 128 rows: D[m][n] = sum_r L[r][m] R[r][n] ----
        // A[m][k] = L[k][m] and B[k][n] = R[k][n] are both transposed loads of row-major tiles; a warp keeps the
        // fragments of its 16 rows of A over all its column tiles.
        constexpr int kSteps = kRowsPerCta / 16;
        const int mat = lane >> 3, mr = lane & 7;
        auto store = [&](float* dst, int ld, int m0, int n0, const float* acc) {
            dst[(m0 + g) * ld + n0 + 2 * t] = acc[0];
            dst[(m0 + g) * ld + n0 + 2 * t + 1] = acc[1];
            dst[(m0 + g + 8) * ld + n0 + 2 * t] = acc[2];
            dst[(m0 + g + 8) * ld + n0 + 2 * t + 1] = acc[3];
        };
        uint32_t A[kSteps][4];
        // dW2 [in][out] = a1^T dz2: warp owns input rows [16 rw, 16 rw + 16) and its half of the columns
#pragma unroll
        for (int kk = 0; kk < kSteps; ++kk)
            ldsm4t(s.a1 + swz(16 * kk + (mat >> 1) * 8 + mr, 16 * rw + (mat & 1) * 8), A[kk]);
#pragma unroll 2
        for (int j = j0; j < j0 + 8; j += 2) {
            float acc[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk) {
                uint32_t B[4];  // two n-tiles
                ldsm4t(s.dz2 + swz(16 * kk + (mat & 1) * 8 + mr, 8 * (j + (mat >> 1))), B);
                mma16816(acc[0], A[kk], B);
                mma16816(acc[1], A[kk], B + 2);
            }
            store(P + kPartW2, kHid, 16 * rw, 8 * j, acc[0]);
            store(P + kPartW2, kHid, 16 * rw, 8 * (j + 1), acc[1]);
        }
        if (half == 0) {
            // dW3 [hidden][out=8] = a2^T dz3: warp owns hidden rows [16 rw, 16 rw + 16)
            float acc[4] = {};
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk) {
                uint32_t B[2];
                ldsm4t(s.a2 + swz(16 * kk + (mat >> 1) * 8 + mr, 16 * rw + (mat & 1) * 8), A[kk]);
                ldsm2t(s.dz3 + (16 * kk + (mat & 1) * 8 + mr) * 16, B);
                mma16816(acc, A[kk], B);
            }
            store(P + kPartW3, kOut, 16 * rw, 0, acc);
        } else {
            // dW1 [in=16][out] = x^T dz1: warp owns output n-tiles 2 rw, 2 rw + 1
            float acc[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk) {
                uint32_t B[4];
                ldsm4t(s.x + (16 * kk + (mat >> 1) * 8 + mr) * 16 + (mat & 1) * 8, A[kk]);
                ldsm4t(s.dz1 + swz(16 * kk + (mat & 1) * 8 + mr, 8 * (2 * rw + (mat >> 1))), B);
                mma16816(acc[0], A[kk], B);
                mma16816(acc[1], A[kk], B + 2);
            }
            store(P + kPartW1, kHid, 0, 8 * (2 * rw), acc[0]);
            store(P + kPartW1, kHid, 0, 8 * (2 * rw + 1), acc[1]);
        }
        __syncthreads();  // the next tile's rows replace these
    }
}

// BF16 operand copies of parameter i (a weight; the biases have none), whose master is w.
__device__ __forceinline__ void pack_param(const MlpParams& p, int i, float w) {
    if (i < kPartW2) {  // W1 [in][out] -> W1T [out][in]
        const int in = i / kHid, o = i % kHid;
        p.W1T[o * kIn + in] = __float2bfloat16_rn(in < 15 ? w : 0.f);
    } else if (i < kPartW3) {  // W2 [in][out] -> W2T [out][in] and W2b = W2
        const int k = i - kPartW2, in = k / kHid, o = k % kHid;
        const __nv_bfloat16 v = __float2bfloat16_rn(w);
        p.W2T[o * kHid + in] = v;
        p.W2b[k] = v;
    } else if (i < kPartB1) {  // W3 [hidden][out] -> W3T [out][hidden], W3b [hidden][16]
        const int k = i - kPartW3, h = k / kOut, o = k % kOut;
        const __nv_bfloat16 v = __float2bfloat16_rn(o < kOutUsed ? w : 0.f);
        p.W3T[o * kHid + h] = v;
        p.W3b[h * 16 + o] = v;
        p.W3b[h * 16 + o + 8] = __float2bfloat16_rn(0.f);
    }
}

// Sum of the CTA partials, AdamW on the FP32 masters, BF16 re-pack: a block takes 32 consecutive parameters and its eight
// warps an eighth of the partials each (in order; the eight sums are added in warp order).  One thread per parameter over
// all partials took 44 us for 512 of them (42 MB): 78 blocks with a serial chain of additions.  The loss's
// running sum takes its partials 256 at a time (one chain of loads and additions per 32 was the kernel's longest path)
// and each parameter's BF16 copies are written here: with both, a step of 65,536 rows went from 104 to 95 us.
constexpr int kAdamWarps = 8;
__global__ void __launch_bounds__(32 * kAdamWarps) k_mlp_adamw(MlpParams p, const float* __restrict__ part, int nblocks,
                                                               float lr, float beta1, float beta2, float eps, float wd,
                                                               int step, float* __restrict__ m, float* __restrict__ v,
                                                               float* __restrict__ grad_out,
                                                               float* __restrict__ loss_out) {
    __shared__ float sums[kAdamWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    if (blockIdx.x == gridDim.x - 1) {  // the loss: one running sum over the partials in order
        if (w != 0 || !loss_out) return;
        float l = 0.f;
        for (int b = 0; b < nblocks; b += 256) {
            float t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int at = b + 32 * k + lane;
                t[k] = at < nblocks ? part[(size_t)at * kPartSize + kPartLoss] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int left = nblocks - b - 32 * k;
                if (left >= 32) {
#pragma unroll
                    for (int u = 0; u < 32; ++u) l += __shfl_sync(0xffffffffu, t[k], u);
                } else {
                    for (int u = 0; u < left; ++u) l += __shfl_sync(0xffffffffu, t[k], u);
                }
            }
        }
        if (lane == 0) *loss_out = l;
        return;
    }
    const int b0 = (int)((long long)nblocks * w / kAdamWarps), b1 = (int)((long long)nblocks * (w + 1) / kAdamWarps);
    float acc = 0.f;
    if (i < kPartLoss) {
        int b = b0;
        for (; b + 8 <= b1; b += 8) {
            float t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) t[u] = __ldcs(part + (size_t)(b + u) * kPartSize + i);
#pragma unroll
            for (int u = 0; u < 8; ++u) acc += t[u];
        }
        for (; b < b1; ++b) acc += __ldcs(part + (size_t)b * kPartSize + i);
    }
    sums[w][lane] = acc;
    __syncthreads();
    if (w != 0 || i >= kPartLoss) return;
    float gsum = 0.f;
#pragma unroll
    for (int u = 0; u < kAdamWarps; ++u) gsum += sums[u][lane];
    // masked entries: the unused input column 15, unused outputs 3..7
    bool used = true;
    float* wp = nullptr;
    bool decay = true;
    if (i < kPartW2) {
        const int in = i / kHid;
        used = in < 15;
        wp = p.W1 + i;
    } else if (i < kPartW3) {
        wp = p.W2 + (i - kPartW2);
    } else if (i < kPartB1) {
        const int o = (i - kPartW3) % kOut;
        used = o < kOutUsed;
        wp = p.W3 + (i - kPartW3);
    } else if (i < kPartB2) {
        wp = p.b1 + (i - kPartB1);
        decay = false;
    } else if (i < kPartB3) {
        wp = p.b2 + (i - kPartB2);
        decay = false;
    } else {
        const int o = i - kPartB3;
        used = o < kOutUsed;
        wp = p.b3 + o;
        decay = false;
    }
    if (grad_out) grad_out[i] = used ? gsum : 0.f;
    if (!used || lr == 0.f) {
        pack_param(p, i, *wp);
        return;
    }
    const float b1c = 1.f - powf(beta1, (float)step), b2c = 1.f - powf(beta2, (float)step);
    m[i] = beta1 * m[i] + (1.f - beta1) * gsum;
    v[i] = beta2 * v[i] + (1.f - beta2) * gsum * gsum;
    const float mh = m[i] / b1c, vh = v[i] / b2c;
    float wv = *wp;
    if (decay) wv -= lr * wd * wv;
    wv -= lr * mh / (sqrtf(vh) + eps);
    *wp = wv;
    pack_param(p, i, wv);
}

__global__ void k_mlp_pack(MlpParams p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kPartW2) pack_param(p, i, p.W1[i]);
    else if (i < kPartW3) pack_param(p, i, p.W2[i - kPartW2]);
    else if (i < kPartB1) pack_param(p, i, p.W3[i - kPartW3]);
}

}  // namespace

static_assert(sizeof(SmemTrain) <= 227 * 1024, "shared memory of the training kernel");
size_t mlp_forward_smem() { return sizeof(Smem); }
size_t mlp_train_smem() { return sizeof(SmemTrain); }

void launch_mlp_forward(const MlpParams& p, const void* X, int n, float* out, cudaStream_t st) {
    // per device and cheap: set on every call
    cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
    const int blocks = (n + kRowsPerCta - 1) / kRowsPerCta;
    if (blocks > 0)
        k_mlp_forward<<<blocks, 256, sizeof(Smem), st>>>(p, reinterpret_cast<const __nv_bfloat16*>(X), n, out);
}

int launch_mlp_train(const MlpParams& p, const void* X, const float* Y, int n, float* part, cudaStream_t st) {
    cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemTrain));
    const int blocks = (n + kRowsPerCta - 1) / kRowsPerCta;
    if (blocks > 0)
        k_mlp_train<<<std::min(blocks, device_sms()), kTrainThreads, sizeof(SmemTrain), st>>>(
            p, reinterpret_cast<const __nv_bfloat16*>(X), Y, n, 1.f / (float)n, part);
    return blocks;
}

void launch_mlp_adamw(const MlpParams& p, const float* part, int nblocks, float lr, float b1, float b2, float eps,
                      float wd, int step, float* m, float* v, float* grad_out, float* loss_out, cudaStream_t st) {
    k_mlp_adamw<<<(kPartLoss + 31) / 32 + 1, 32 * kAdamWarps, 0, st>>>(p, part, nblocks, lr, b1, b2, eps, wd, step, m, v,
                                                                       grad_out, loss_out);
}

void launch_mlp_pack(const MlpParams& p, cudaStream_t st) { k_mlp_pack<<<(kPartB1 + 255) / 256, 256, 0, st>>>(p); }

int mlp_part_size() { return kPartSize; }
int mlp_param_count() { return kPartLoss; }
int mlp_rows_per_block() { return kRowsPerCta; }
int mlp_packed_count() { return kHid * kIn + kHid * kHid + kOut * kHid + kHid * kHid + kHid * 16; }

static MlpParams flat_params(float* master, void* packed) {
    MlpParams p;
    p.W1 = master + kPartW1;
    p.W2 = master + kPartW2;
    p.W3 = master + kPartW3;
    p.b1 = master + kPartB1;
    p.b2 = master + kPartB2;
    p.b3 = master + kPartB3;
    __nv_bfloat16* b = reinterpret_cast<__nv_bfloat16*>(packed);
    p.W1T = b;
    p.W2T = p.W1T + kHid * kIn;
    p.W3T = p.W2T + kHid * kHid;
    p.W2b = p.W3T + kOut * kHid;
    p.W3b = p.W2b + kHid * kHid;
    return p;
}

void mlp_pack_flat(float* master, void* packed, cudaStream_t st) { launch_mlp_pack(flat_params(master, packed), st); }
void mlp_forward_flat(float* master, void* packed, const void* X, int n, float* out, cudaStream_t st) {
    launch_mlp_forward(flat_params(master, packed), X, n, out, st);
}
void launch_mlp_forward_tc(const void* W1T, const void* W2T, const void* W3T, const float* b1, const float* b2,
                           const float* b3, const void* X, int n, float* out, int* err, int max_ctas, cudaStream_t st);
void mlp_forward_tc_flat(float* master, void* packed, const void* X, int n, float* out, int* err, cudaStream_t st) {
    const MlpParams p = flat_params(master, packed);
    launch_mlp_forward_tc(p.W1T, p.W2T, p.W3T, p.b1, p.b2, p.b3, X, n, out, err, 2 * device_sms(), st);
}
int mlp_train_flat(float* master, void* packed, const void* X, const float* Y, int n, float* part, cudaStream_t st) {
    return launch_mlp_train(flat_params(master, packed), X, Y, n, part, st);
}
void mlp_adamw_flat(float* master, void* packed, const float* part, int nblocks, float lr, float b1, float b2,
                    float eps, float wd, int step, float* m, float* v, float* grad_out, float* loss_out,
                    cudaStream_t st) {
    launch_mlp_adamw(flat_params(master, packed), part, nblocks, lr, b1, b2, eps, wd, step, m, v, grad_out, loss_out,
                     st);
}

}  // namespace dphd

namespace dphd {

namespace {

// Per-node features (16): displacement (q - X)/dx, last step (q - q_prev)/dx, the last step's correction
// (q - q_tilde_prev)/dx (0 without a previous prediction), h^2/m f_ext/dx, height above the contact plane /dx,
// log10 of the node's mean PD stiffness / 7, Dirichlet flag, and the node's current contact multiplier (the
// previous frame's lambda) in the output's scale h^2/(m dx), clipped at 4 (0 off the contact set); also the inertial
// prediction q_tilde = q + h v + h^2/m (f_ext + m g) (the warm start is q_tilde + dx * MLP).
__global__ void k_mlp_features(FeatureArgs a, const double* __restrict__ q, const double* __restrict__ qp,
                               const double* __restrict__ v, const double* __restrict__ f,
                               const double* __restrict__ prev_base, const float* __restrict__ lam_node,
                               __nv_bfloat16* __restrict__ X, double* __restrict__ base) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    float feat[16];
    double qt[3];
    for (int d = 0; d < 3; ++d) {
        const int k = 3 * i + d;
        qt[d] = q[k] + a.h * v[k] + a.h2m * f[k] + a.h2m * a.gforce[d];
        base[k] = qt[d];
        feat[d] = (float)((q[k] - a.X[k]) * a.inv_dx);
        feat[3 + d] = (float)((q[k] - qp[k]) * a.inv_dx);
        feat[6 + d] = prev_base ? (float)((q[k] - prev_base[k]) * a.inv_dx) : 0.f;
        feat[9 + d] = (float)(a.h2m * f[k] * a.inv_dx);
    }
    // height above the contact plane in cells, clamped to [-2, 2]: only the layer next to the plane is told apart
    // (unclamped, the feature would grow with the body's size and leave the training range on larger meshes)
    feat[12] = a.plane ? fminf(2.f, fmaxf(-2.f, (float)((a.pn[0] * q[3 * i] + a.pn[1] * q[3 * i + 1] +
                                                         a.pn[2] * q[3 * i + 2] + a.poff) * a.inv_dx)))
                       : 0.f;
    feat[13] = a.wlog[i];
    feat[14] = a.fixed[i] ? 1.f : 0.f;
    feat[15] = lam_node ? lam_node[i] : 0.f;
    for (int c = 0; c < 16; ++c) X[(size_t)i * 16 + c] = __float2bfloat16_rn(feat[c]);
}

__global__ void k_mlp_apply(int n3, const double* __restrict__ base, const float* __restrict__ out, double dx,
                            const unsigned char* __restrict__ fixed_dof, const double* __restrict__ fval,
                            double* __restrict__ q_init) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n3) return;
    q_init[k] = fixed_dof[k] ? fval[k] : base[k] + dx * (double)out[(size_t)(k / 3) * 8 + k % 3];
}

// The scaled multipliers are clipped at kLamClip in the feature and the target: impact frames reach tens of the
// resting values, and a few such rows would dominate the squared loss of a warm start.
constexpr double kLamClip = 4.0;

// Training targets, 4 per node: (q_next - q_tilde)/dx and the frame's contact multiplier in the scale h^2/(m dx)
// (column 3: 0 here, the candidates' values are written by k_mlp_target_lambda after this kernel).
__global__ void k_mlp_target(int n3, const double* __restrict__ q_next, const double* __restrict__ base,
                             double inv_dx, float* __restrict__ Y) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n3) return;
    Y[(size_t)(k / 3) * 4 + k % 3] = (float)((q_next[k] - base[k]) * inv_dx);
    if (k % 3 == 0) Y[(size_t)(k / 3) * 4 + 3] = 0.f;
}

// Column 3: the change of the multiplier over the frame, (lambda_final - lambda_prev) * scale, clipped to
// [-kLamClip, kLamClip] (the network predicts a correction of the previous frame's multiplier).
__global__ void k_mlp_target_lambda(int K, const int* __restrict__ cand, const double* __restrict__ lam,
                                    const double* __restrict__ lam_prev, double scale, float* __restrict__ Y) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const double d = (lam[k] - (lam_prev ? lam_prev[k] : 0.0)) * scale;
    Y[(size_t)cand[k] * 4 + 3] = (float)fmax(-kLamClip, fmin(d, kLamClip));
}

// Node-indexed contact multipliers in the network's scale (the lambda feature): 0 off the candidate set.
__global__ void k_mlp_lambda_zero(int n, float* __restrict__ lam_node) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) lam_node[i] = 0.f;
}
__global__ void k_mlp_lambda_scatter(int K, const int* __restrict__ cand, const double* __restrict__ lam, double scale,
                                     float* __restrict__ lam_node) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) lam_node[cand[k]] = (float)fmin(lam[k] * scale, kLamClip);
}

// The predicted initial contact multipliers: lambda_k <- max(0, lambda_k + out[node_k][3] / scale), the previous
// frame's multiplier corrected by the network.
__global__ void k_mlp_lambda_apply(int K, const int* __restrict__ cand, const float* __restrict__ out, double inv_scale,
                                   double* __restrict__ lam) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const double v = lam[k] + (double)out[(size_t)cand[k] * 8 + 3] * inv_scale;
    lam[k] = v > 0.0 ? v : 0.0;
}

}  // namespace

void launch_mlp_features(const FeatureArgs& a, const double* q, const double* qp, const double* v, const double* f,
                         const double* prev_base, const float* lam_node, void* X, double* base, cudaStream_t st) {
    k_mlp_features<<<(a.n + 255) / 256, 256, 0, st>>>(a, q, qp, v, f, prev_base, lam_node,
                                                      reinterpret_cast<__nv_bfloat16*>(X), base);
}
void launch_mlp_lambda_nodes(int n, int K, const int* cand, const double* lam, double scale, float* lam_node,
                             cudaStream_t st) {
    k_mlp_lambda_zero<<<(n + 255) / 256, 256, 0, st>>>(n, lam_node);
    if (K > 0) k_mlp_lambda_scatter<<<(K + 255) / 256, 256, 0, st>>>(K, cand, lam, scale, lam_node);
}
void launch_mlp_target_lambda(int K, const int* cand, const double* lam, const double* lam_prev, double scale,
                              float* Y, cudaStream_t st) {
    if (K > 0) k_mlp_target_lambda<<<(K + 255) / 256, 256, 0, st>>>(K, cand, lam, lam_prev, scale, Y);
}
void launch_mlp_lambda_apply(int K, const int* cand, const float* out, double inv_scale, double* lam, cudaStream_t st) {
    if (K > 0) k_mlp_lambda_apply<<<(K + 255) / 256, 256, 0, st>>>(K, cand, out, inv_scale, lam);
}
void launch_mlp_apply(int n3, const double* base, const float* out, double dx, const unsigned char* fixed_dof,
                      const double* fval, double* q_init, cudaStream_t st) {
    k_mlp_apply<<<(n3 + 255) / 256, 256, 0, st>>>(n3, base, out, dx, fixed_dof, fval, q_init);
}
// The learned start at the contact candidates.  Mode 1: a candidate in contact in the previous frame (lambda > 0)
// keeps its previous gap (a resting contact stays at rest), the others are moved out of the half space if the
// prediction penetrates it; the tangential components stay as predicted.  Mode 2: a candidate in contact keeps
// its previous position altogether (the plain solver's start there), the others keep the prediction.
__global__ void k_ws_contact_start(int K, int mode, const int* __restrict__ cand, const double* __restrict__ lam,
                                   double n0, double n1, double n2, double off,
                                   const unsigned char* __restrict__ fixed_dof, const double* __restrict__ q_prev,
                                   double* __restrict__ q_init) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    const int i = cand[k];
    if (fixed_dof[3 * i] || fixed_dof[3 * i + 1] || fixed_dof[3 * i + 2]) return;
    double* x = q_init + 3 * (size_t)i;
    const double* xp = q_prev + 3 * (size_t)i;
    if (mode == 2) {
        if (lam[k] > 0.0) {
            x[0] = xp[0];
            x[1] = xp[1];
            x[2] = xp[2];
        }
        return;
    }
    const double d = n0 * x[0] + n1 * x[1] + n2 * x[2] + off;
    const double dp = n0 * xp[0] + n1 * xp[1] + n2 * xp[2] + off;
    const double target = lam[k] > 0.0 ? dp : (d < 0.0 ? 0.0 : d);
    const double s = target - d;
    x[0] += s * n0;
    x[1] += s * n1;
    x[2] += s * n2;
}

void launch_ws_contact_start(int K, int mode, const int* cand, const double* lam, const double* n, double off,
                             const unsigned char* fixed_dof, const double* q_prev, double* q_init, cudaStream_t st) {
    if (K > 0)
        k_ws_contact_start<<<(K + 255) / 256, 256, 0, st>>>(K, mode, cand, lam, n[0], n[1], n[2], off, fixed_dof,
                                                             q_prev, q_init);
}

void launch_mlp_target(int n3, const double* q_next, const double* base, double inv_dx, float* Y, cudaStream_t st) {
    k_mlp_target<<<(n3 + 255) / 256, 256, 0, st>>>(n3, q_next, base, inv_dx, Y);
}

}  // namespace dphd
