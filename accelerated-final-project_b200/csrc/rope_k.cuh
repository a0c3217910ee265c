// "Rotate once and keep it": writes RoPE(X) for a [B,H,L,D] tensor, the producer a KV-cache caller runs
// when keys are appended, so that attention can then take K as already rotated (the *_Q_ONLY encodings).
// Replaces rope_kernel, final/rope.cu:1240-1280, as used by attention_forward_separate_rope
// (final/rope.cu:1379-1416) - without that kernel's position taken modulo 64 (:1257): the position
// of row l of every (b,h) slice is pos0 + l.
//
// Memory-bound element-wise work: a thread owns one 16-byte vector position of one row (two vectors for
// the rotate-half pairing: columns d and d + rotary_dim/2) and takes a share of the (b,h) slices with it, so the
// angle arithmetic - theta = (float)pos * (1 / powf(base, 2i / rotary_dim)), sincosf, exactly the fp32
// arithmetic of the reference tables (final/rope.cu:20-40) - is done once per (row, pair) and share and not once per
// element.  The products are fp32; a 16-bit result is rounded once.  The slices of a thread are loaded four at a time
// and the shares are cut so that the grid fills the chip, and two tensors (Q and K of a call) go in one launch: with one
// thread walking over all slices, one load in flight, a position took slices x DRAM latency whatever the sizes (an fp16
// attention call of 8 x 12 heads, 1000 x 1000, head_d 64 with its two encoding launches: 166 us; now 72 us).
#pragma once

#include "tc_common.cuh"

namespace b200attn {

constexpr int RK_UNROLL = 4;   // slices a thread has in flight

struct RopeKParams {
    const void *X;
    void *Y;
    long long BH;
    int L, D, rd;
    const void *X2;           // optional second tensor [BH][L2][D], encoded by the same rule (blockIdx.z = 1)
    void *Y2;
    int L2;
    int half;                 // 0: pairs (2i, 2i+1); 1: pairs (i, i + rd/2)
    int pos0;
    float base;
    const float *cos_cache, *sin_cache;   // optional [>= pos0 + L][rd], value of pair i at columns 2i and 2i+1
    int sinus;                // 1: additive sinusoidal encoding instead of a rotation - x[2i] += sin, x[2i+1] += cos of
                              // pos / 10000^(2i/D) (final/sinusoidal.cu:143-161); then rd = D, half = 0, base = 10000
};

template <typename T> struct RopeVec;
template <> struct RopeVec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void open(const uint4 &v, float (&x)[4]) {
        x[0] = __uint_as_float(v.x); x[1] = __uint_as_float(v.y); x[2] = __uint_as_float(v.z); x[3] = __uint_as_float(v.w);
    }
    static __device__ __forceinline__ void store(float *p, const float (&x)[4]) {
        *reinterpret_cast<float4 *>(p) = make_float4(x[0], x[1], x[2], x[3]);
    }
};
template <> struct RopeVec<__half> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void open(const uint4 &v, float (&x)[8]) {
        const __half *h = reinterpret_cast<const __half *>(&v);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __half2float(h[e]);
    }
    static __device__ __forceinline__ void store(__half *p, const float (&x)[8]) {
        uint4 v;
        __half2 *h = reinterpret_cast<__half2 *>(&v);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2half2_rn(x[2 * e], x[2 * e + 1]);
        *reinterpret_cast<uint4 *>(p) = v;
    }
};
template <> struct RopeVec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void open(const uint4 &v, float (&x)[8]) {
        const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __bfloat162float(h[e]);
    }
    static __device__ __forceinline__ void store(__nv_bfloat16 *p, const float (&x)[8]) {
        uint4 v;
        __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
        *reinterpret_cast<uint4 *>(p) = v;
    }
};

__device__ __forceinline__ void rope_angle(const RopeKParams &p, int pos, int pair, float &c, float &s) {
    if (p.cos_cache != nullptr) {
        c = p.cos_cache[(long long)pos * p.rd + 2 * pair];
        s = p.sin_cache[(long long)pos * p.rd + 2 * pair];
    } else {
        const float freq = 1.0f / powf(p.base, (2.0f * (float)pair) / (float)p.rd);
        sincosf((float)pos * freq, &s, &c);
    }
}

// Vector path: D, rd (interleaved) or rd/2 (half) are multiples of the vector width and the pointers are
// 16-byte aligned.  Work items of a row: interleaved - D/N vectors; half - rd/(2N) vector pairs plus
// (D - rd)/N copy vectors.  gridDim.y shares the slices.
template <typename T>
__global__ void __launch_bounds__(256) rope_k_vec_kernel(const RopeKParams p) {
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int N = RopeVec<T>::N;
    const T *X = reinterpret_cast<const T *>(blockIdx.z ? p.X2 : p.X);
    T *Y = reinterpret_cast<T *>(blockIdx.z ? p.Y2 : p.Y);
    const int L = blockIdx.z ? p.L2 : p.L;
    const int nrot = p.half ? p.rd / (2 * N) : p.rd / N;   // items that rotate
    const int nitem = nrot + (p.D - p.rd) / N;
    const long long total = (long long)L * nitem;
    const long long slab = (long long)L * p.D;
    const long long step = (long long)gridDim.y;
    auto ld = [&](long long bh, long long off) { return bh < p.BH ? *reinterpret_cast<const uint4 *>(X + bh * slab + off) : make_uint4(0, 0, 0, 0); };
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(w / nitem), it = (int)(w - (long long)l * nitem);
        const int pos = p.pos0 + l;
        const long long row = (long long)l * p.D;
        if (it >= nrot) {   // beyond rotary_dim: copy
            const long long off = row + p.rd + (long long)(it - nrot) * N;
            for (long long bh = blockIdx.y; bh < p.BH; bh += RK_UNROLL * step) {
                uint4 v[RK_UNROLL];
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u) v[u] = ld(bh + u * step, off);
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u)
                    if (bh + u * step < p.BH) *reinterpret_cast<uint4 *>(Y + (bh + u * step) * slab + off) = v[u];
            }
        } else if (p.half) {
            const int d = it * N;   // columns d..d+N-1 pair with d + rd/2 ..
            float c[N], s[N];
#pragma unroll
            for (int e = 0; e < N; ++e) rope_angle(p, pos, d + e, c[e], s[e]);
            for (long long bh = blockIdx.y; bh < p.BH; bh += RK_UNROLL * step) {
                uint4 v0[RK_UNROLL], v1[RK_UNROLL];
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u) { v0[u] = ld(bh + u * step, row + d); v1[u] = ld(bh + u * step, row + d + p.rd / 2); }
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u) {
                    if (bh + u * step >= p.BH) break;
                    float lo[N], hi[N], ylo[N], yhi[N];
                    RopeVec<T>::open(v0[u], lo);
                    RopeVec<T>::open(v1[u], hi);
#pragma unroll
                    for (int e = 0; e < N; ++e) { ylo[e] = lo[e] * c[e] - hi[e] * s[e]; yhi[e] = lo[e] * s[e] + hi[e] * c[e]; }
                    RopeVec<T>::store(Y + (bh + u * step) * slab + row + d, ylo);
                    RopeVec<T>::store(Y + (bh + u * step) * slab + row + d + p.rd / 2, yhi);
                }
            }
        } else {
            const int d = it * N;   // pairs (d, d+1), (d+2, d+3), ...
            float c[N / 2], s[N / 2];
#pragma unroll
            for (int e = 0; e < N / 2; ++e) rope_angle(p, pos, d / 2 + e, c[e], s[e]);
            for (long long bh = blockIdx.y; bh < p.BH; bh += RK_UNROLL * step) {
                uint4 v[RK_UNROLL];
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u) v[u] = ld(bh + u * step, row + d);
#pragma unroll
                for (int u = 0; u < RK_UNROLL; ++u) {
                    if (bh + u * step >= p.BH) break;
                    float x[N], y[N];
                    RopeVec<T>::open(v[u], x);
#pragma unroll
                    for (int e = 0; e < N / 2; ++e) {
                        if (p.sinus) { y[2 * e] = x[2 * e] + s[e]; y[2 * e + 1] = x[2 * e + 1] + c[e]; }
                        else { y[2 * e] = x[2 * e] * c[e] - x[2 * e + 1] * s[e]; y[2 * e + 1] = x[2 * e] * s[e] + x[2 * e + 1] * c[e]; }
                    }
                    RopeVec<T>::store(Y + (bh + u * step) * slab + row + d, y);
                }
            }
        }
    }
}

// Any shape and alignment: a thread owns one pair (or one copied column) of one row.
template <typename T>
__global__ void __launch_bounds__(256) rope_k_scalar_kernel(const RopeKParams p) {
    grid_launch_dependents();
    grid_dependency_wait();
    const T *X = reinterpret_cast<const T *>(blockIdx.z ? p.X2 : p.X);
    T *Y = reinterpret_cast<T *>(blockIdx.z ? p.Y2 : p.Y);
    const int L = blockIdx.z ? p.L2 : p.L;
    const int npair = p.rd / 2, nitem = npair + (p.D - p.rd);
    const long long total = (long long)L * nitem;
    const long long slab = (long long)L * p.D;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(w / nitem), it = (int)(w - (long long)l * nitem);
        const long long row = (long long)l * p.D;
        if (it >= npair) {
            const long long off = row + p.rd + (it - npair);
            for (long long bh = blockIdx.y; bh < p.BH; bh += gridDim.y) Y[bh * slab + off] = X[bh * slab + off];
        } else {
            float c, s;
            rope_angle(p, p.pos0 + l, it, c, s);
            const int d0 = p.half ? it : 2 * it, d1 = p.half ? it + npair : 2 * it + 1;
            for (long long bh = blockIdx.y; bh < p.BH; bh += gridDim.y) {
                const float a = to_f32(X[bh * slab + row + d0]), b = to_f32(X[bh * slab + row + d1]);
                Y[bh * slab + row + d0] = OutCvt<T>::one(p.sinus ? a + s : a * c - b * s);
                Y[bh * slab + row + d1] = OutCvt<T>::one(p.sinus ? b + c : a * s + b * c);
            }
        }
    }
}

template <typename T>
inline cudaError_t launch_rope_k(const RopeKParams &p, int sm_count, cudaStream_t st) {
    constexpr int N = RopeVec<T>::N;
    const bool two = p.X2 != nullptr;
    const bool aligned = (((uintptr_t)p.X | (uintptr_t)p.Y | (uintptr_t)p.X2 | (uintptr_t)p.Y2) & 15) == 0;
    const bool vec = aligned && p.D % N == 0 && (p.half ? (p.rd % (2 * N) == 0) : (p.rd % N == 0));
    const long long per_row = vec ? (p.half ? p.rd / (2 * N) : p.rd / N) + (p.D - p.rd) / N : p.rd / 2 + (p.D - p.rd);
    const long long items = (long long)(two && p.L2 > p.L ? p.L2 : p.L) * per_row;
    long long blocks = (items + 255) / 256;
    const long long cap = (long long)sm_count * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    // shares of the slices: enough blocks for two waves of the chip, but no share below one round of RK_UNROLL slices
    // (a share repeats the angles)
    long long shares = cap / (blocks * (two ? 2 : 1));
    const long long most = (p.BH + RK_UNROLL - 1) / RK_UNROLL;
    if (shares > most) shares = most;
    if (shares > 65535) shares = 65535;
    if (shares < 1) shares = 1;
    const dim3 grid((unsigned)blocks, (unsigned)shares, two ? 2 : 1);
    return vec ? launch_dependent(rope_k_vec_kernel<T>, grid, 256, 0, 1, st, p) : launch_dependent(rope_k_scalar_kernel<T>, grid, 256, 0, 1, st, p);
}

}  // namespace b200attn
