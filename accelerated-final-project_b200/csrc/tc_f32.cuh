// Attention forward for sequences longer than 64 on the tensor cores, at fp32 accuracy: fp32 tensors, and 16-bit tensors of the
// head widths that the 16-bit kernels do not take (no multiple of 64; 192 with an encoding).
//
// An fp32 value is cut into three bf16 pieces x = x1 + x2 + x3 (8 significant bits each: the sum is exact), and a product
// a b is taken as a1 b1 + (a1 b2 + a2 b1) + (a1 b3 + a2 b2 + a3 b1): what is left out is below 2^-22 |a b| (2^-26 on average; the
// first piece is cut off, not rounded, so that a large value does not become an infinity: a2 reaches 2^-7 a).  Values below 2^-110
// lose low bits, to an absolute error of 2^-134 (of V 2^-103 and 2^-127).  Six bf16 MMAs cost what three tf32 MMAs on a hi / lo pair cost and keep two more bits.  The leading products
// have an accumulator of their own and are added to the small ones in fp32 by the thread that reads them, and P V starts a
// fresh accumulator per 64 keys, summed in registers: the chain of roundings at the full magnitude is as short as
// head_d / 16 and len_k / 64.  (Replaces, for these shapes, the FFMA kernels of splitd.cuh; same mathematics as the
// reference's fp32 kernel, final/attention.cu:84-191: softmax statistics, probabilities and sums are fp32.)
// A 16-bit tensor is fewer pieces (bf16 one, fp16 two, an encoded Q or K three) and its result is rounded once, at the end.  The 16-bit
// kernel of tc_fa.cuh at these widths (P and encoded operands rounded to 16 bits) was no replacement for the CUDA-core kernels, which
// hold both in fp32: 2 x 16 heads, 777 x 1000, head_d 96, bf16, its output lay 2.5e-3 from theirs; this one lies 5e-5 from it (a result
// in some thousands rounds the other way), in 126 us against 717 us on the CUDA cores and 22 us there.
//
//   f32_split_kernel    Q, K, V -> three bf16 planes each, columns padded to whole groups of 64 with zeros; a positional
//                       encoding is applied here, once per element, with the fp32 arithmetic of the reference tables;
//   f32_scores_kernel   score tile [128 queries x 128 keys] per CTA, planes streamed by TMA in chunks of 64 columns; the
//                       epilogue writes the raw scores (fp32, four keys of a row per 16 bytes, rows side by side) and, per
//                       row, raises the maximum kept in global memory;
//   f32_pv_kernel       unit = (head, 128 queries, 64 output columns), the keys cut over a cluster of up to 8 CTAs where the
//                       units alone would leave SMs idle.  A row's maximum is known when it starts, so partial outputs
//                       and sums of exponentials are plain sums (added through distributed shared memory in the order of
//                       the CTAs) and nothing is ever rescaled.
//
// Why two kernels: the three planes of P, Q, K and V of a one-kernel form fill shared memory at head_d 128 and exceed it
// beyond, while the fp32 scores of the sizes in use stay in the L2.
// Infinities and NaN: a non-finite value is its first piece, the others are zero, and the sum of the leading products is the result
// wherever it is not finite (f3_sum): as in FFMA but for an infinity times a subnormal.
// Every wait is bounded.
#pragma once

#include <type_traits>

#include "tc_bf16.cuh"

namespace b200attn {

constexpr int F3_T = 128;                    // queries and keys per tile
constexpr int F3_SLAB = F3_T * 128;          // [128 rows x 64 bf16]: one plane of a 64-column chunk
// score kernel, operands of `nq` pieces: a stage is the planes of Q, then those of K; fewer pieces, more stages
__host__ __device__ constexpr int f3_stage(int nq) { return 2 * nq * F3_SLAB; }
__host__ __device__ constexpr int f3_stages(int nq) { return nq == 3 ? 2 : nq == 2 ? 3 : 4; }
constexpr int F3_VSLAB = 64 * 128;           // [64 keys x 64 bf16]
constexpr int F3_VSTAGE = 3 * F3_VSLAB;      // P V kernel: the pieces of V of 64 keys x 64 columns
constexpr int F3_SSTEP = 64 * F3_T * 4;      // scores of 64 keys as the score kernel leaves them
constexpr int F3_PBUF = 3 * F3_SLAB;         // P1 P2 P3 [128 rows x 64 keys]
constexpr int F3_A_THREADS = 576;            // score kernel: warp 0 loads, warp 1 issues, warps 2-17 four threads per query row
constexpr int F3_B_THREADS = 608;            // P V kernel: the same, warp 0 loads the scores and warp 18 loads V
constexpr int F3_MAX_CLUSTER = 8;
constexpr int F3_OPITCH = 68;                // floats per row of the partial output in shared memory
constexpr float F3_VSCALE = 1.0f / 128;      // V goes through the MMAs this much smaller: 64 of its products add up without overflow

struct F32Params {
    int heads;                 // heads of this pass
    int Lq, Lk, D, Dp;         // Dp = head_d rounded up to 64
    int nq, nk, ndb;           // query tiles, key tiles, blocks of 64 output columns
    int upc;                   // P V kernel: steps of 64 keys per CTA of the cluster
    float c;                   // log2(e) / sqrt(head_d)
    float share, unshare;      // a power of two not above 1 / (steps of 64 keys): unnormalised sums of finite values stay finite; 1 / (share * F3_VSCALE)
    float *S;                  // [heads][nq][nk][32 groups of 4 keys][128 rows][4]
    int *rowmax;               // [heads][nq * 128] largest score of a row, as f3_key; the split kernel starts it at the lowest key
    void *O;                   // [heads * Lq][D]
    int vec_out;               // stores of four columns
    unsigned *err, *err_sys;
    unsigned spin_limit;
};

// two fp32 values as packed pairs of their bf16 pieces; the sum of the pieces is exact for finite values
__device__ __forceinline__ void f3_split2(float x0, float x1, uint32_t &a, uint32_t &b, uint32_t &c) {
    const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
    a = __byte_perm(u0, u1, 0x7632);   // truncation: the first piece of a large value must not round up to infinity
    const float r0 = x0 - __uint_as_float(u0 & 0xffff0000u), r1 = x1 - __uint_as_float(u1 & 0xffff0000u);
    b = pack_bf16x2(r0, r1);
    c = pack_bf16x2(r0 - __uint_as_float(b << 16), r1 - __uint_as_float(b & 0xffff0000u));
}
// fp32 values as integers of the same order (NaN aside), and back
__device__ __forceinline__ int f3_key(float x) { const int i = __float_as_int(x); return i >= 0 ? i : i ^ 0x7fffffff; }
__device__ __forceinline__ float f3_unkey(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
// two fp32 additions, multiply-adds
__device__ __forceinline__ float2 f3_add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 f3_fma2(float2 a, float b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tmov.b64 z, {%5, %6};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 f3_pair(const uint32_t *r) { return make_float2(__uint_as_float(r[0]), __uint_as_float(r[1])); }
// Sums of the leading products and the smaller ones (low: null or the third set).  A sum of leading products that is not finite is the
// result: of a non-finite operand only the first piece holds it (the others are zero, times which the smaller products are NaN),
// and of finite operands whose products overflow a lower piece may have the other sign.  One look for all N: looking at each sum cost the
// P V kernel 6 % (32 heads, 2048 x 2048, head_d 64, the call 311 -> 332 us).
template <int N> __device__ __forceinline__ void f3_sums(const uint32_t (&lead)[N], const uint32_t (&mid)[N], const uint32_t *low, float2 (&v)[N / 2]) {
    float2 look = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const float2 m = f3_pair(mid + 2 * i);
        v[i] = f3_add2(f3_pair(lead + 2 * i), low != nullptr ? f3_add2(m, f3_pair(low + 2 * i)) : m);
        look = f3_fma2(v[i], 0.0f, look);
    }
    if (!(look.x + look.y == 0.0f)) {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float2 a = f3_pair(lead + 2 * i);
            if (!(fabsf(a.x) < INFINITY)) v[i].x = a.x;
            if (!(fabsf(a.y) < INFINITY)) v[i].y = a.y;
        }
    }
}

// ---- split (and encode) ---------------------------------------------------------------------------
struct F32SplitTensor {
    const void *X;
    __nv_bfloat16 *Y;          // [pieces][heads][L][Dp]
    int L;
    int encode;                // the encoding applies to this tensor
    int pieces;
    float scale;               // 1, for V F3_VSCALE
};
struct F32SplitParams {
    F32SplitTensor t[3];       // blockIdx.z
    int heads, D, Dp;
    int pe, rd;
    float base;
    const float *cos_cache, *sin_cache;
    int *rowmax;               // nrows entries, set to the key of -inf
    long long nrows;
};

// A thread owns eight columns of one row position and takes a share (gridDim.y) of the heads with them, so that the angles
// are computed once per share; the loads of two heads are in flight together.
template <typename T>
__global__ void __launch_bounds__(256) f32_split_kernel(const F32SplitParams p) {
    grid_launch_dependents();
    grid_dependency_wait();
    const F32SplitTensor t = p.t[blockIdx.z];
    const T *X = reinterpret_cast<const T *>(t.X);
    const int ng = p.Dp >> 3, D = p.D;
    const long long total = (long long)t.L * ng, slab = (long long)t.L * D, yslab = (long long)t.L * p.Dp, plane = yslab * p.heads;
    const bool sinus = p.pe == PE_SINUSOIDAL, half = pe_pairs_halves(p.pe);
    const bool vec = D % (16 / (int)sizeof(T)) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const int step = gridDim.y;
    if (blockIdx.z == 0)
        for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < p.nrows; i += (long long)gridDim.x * gridDim.y * blockDim.x)
            p.rowmax[i] = f3_key(-INFINITY);
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(w / ng), d0 = (int)(w - (long long)l * ng) * 8;
        const int n = min(8, D - d0);            // real columns, <= 0 in the padding
        const bool enc = t.encode && n > 0 && (sinus || d0 < p.rd);
        float cs[8], sn[8];   // per column (interleaved pairs: the two columns of a pair share theirs)
        if (enc) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (!half && (e & 1)) { cs[e] = cs[e - 1]; sn[e] = sn[e - 1]; continue; }
                const int d = d0 + e, pair = half ? (d < (p.rd >> 1) ? d : d - (p.rd >> 1)) : d >> 1;
                cs[e] = 1.0f; sn[e] = 0.0f;
                if (d < (sinus ? D : p.rd)) {
                    if (p.cos_cache != nullptr && !sinus) {
                        cs[e] = p.cos_cache[(long long)l * p.rd + 2 * pair];
                        sn[e] = p.sin_cache[(long long)l * p.rd + 2 * pair];
                    } else {
                        // same arithmetic as the reference tables (final/rope.cu:20-40, final/sinusoidal.cu:848)
                        const float freq = 1.0f / powf(p.base, (2.0f * (float)pair) / (float)(sinus ? D : p.rd));
                        sincosf((float)l * freq, &sn[e], &cs[e]);
                    }
                }
            }
        }
        auto load = [&](int h, float (&x)[8]) {
            const T *xp = X + h * slab + (long long)l * D + d0;
            if (vec && n == 8) {
                uint4 raw[sizeof(T) / 2];
#pragma unroll
                for (int i = 0; i < (int)sizeof(T) / 2; ++i) raw[i] = reinterpret_cast<const uint4 *>(xp)[i];
                const T *e8 = reinterpret_cast<const T *>(raw);
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = to_f32(e8[e]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = e < n ? to_f32(xp[e]) : 0.0f;
            }
        };
        auto store = [&](int h, float (&x)[8]) {
            if (enc) {
                if (sinus) {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e < n) x[e] += (e & 1) ? cs[e] : sn[e];
                } else if (half) {
                    const T *xr = X + h * slab + (long long)l * D;
                    const int hr = p.rd >> 1;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int d = d0 + e;
                        if (d < hr) x[e] = x[e] * cs[e] - to_f32(xr[d + hr]) * sn[e];
                        else if (d < p.rd) x[e] = to_f32(xr[d - hr]) * sn[e] + x[e] * cs[e];
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 8; e += 2)
                        if (d0 + e + 1 < p.rd) {
                            const float a = x[e], b = x[e + 1];
                            x[e] = a * cs[e] - b * sn[e];
                            x[e + 1] = a * sn[e] + b * cs[e];
                        }
                }
            }
            uint32_t a[4], b[4], c[4];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] *= t.scale;
#pragma unroll
            for (int e = 0; e < 4; ++e) f3_split2(x[2 * e], x[2 * e + 1], a[e], b[e], c[e]);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if ((__float_as_uint(x[e]) & 0x7f800000u) == 0x7f800000u) {   // the value in the first piece (a NaN stays one), zero in the others
                    const uint32_t keep = (e & 1) ? 0x0000ffffu : 0xffff0000u;
                    b[e >> 1] &= keep; c[e >> 1] &= keep;
                    if (x[e] != x[e]) a[e >> 1] |= (e & 1) ? 0x00400000u : 0x00000040u;
                }
            __nv_bfloat16 *yp = t.Y + h * yslab + (long long)l * p.Dp + d0;
            *reinterpret_cast<uint4 *>(yp) = make_uint4(a[0], a[1], a[2], a[3]);
            if (t.pieces > 1) *reinterpret_cast<uint4 *>(yp + plane) = make_uint4(b[0], b[1], b[2], b[3]);
            if (t.pieces > 2) *reinterpret_cast<uint4 *>(yp + 2 * plane) = make_uint4(c[0], c[1], c[2], c[3]);
        };
        for (int h = blockIdx.y; h < p.heads; h += 2 * step) {
            float x0[8], x1[8];
            const bool two = h + step < p.heads;
            load(h, x0);
            if (two) load(h + step, x1);
            store(h, x0);
            if (two) store(h + step, x1);
        }
    }
}

// ---- scores ---------------------------------------------------------------------------------------
#define F3_FAIL_AT(site, cond)                                                                      \
    if (cond) {                                                                                     \
        report_kernel_error(p.err, p.err_sys, (unsigned)KERR_MBAR_TIMEOUT | (1u << (7 + (site))));  \
        failed = true;                                                                              \
        break;                                                                                      \
    }

// the same for a wait of a whole warp: either all of its lanes go on or none
#define F3_WARP_WAIT(site, bar, parity)                                                                          \
    if (!__all_sync(0xffffffffu, mbar_wait(&(bar), (uint32_t)(parity), lim))) {                                  \
        if (lane == 0) report_kernel_error(p.err, p.err_sys, (unsigned)KERR_MBAR_TIMEOUT | (1u << (7 + (site)))); \
        failed = true;                                                                                           \
        break;                                                                                                   \
    }

// Persistent score kernel: a CTA per SM takes tiles [128 queries x 128 keys] in turn.  Planes of 64-column chunks pass through two
// stages; a group of two chunks (128 columns) accumulates in one of two pairs of accumulators, the leading products and the
// small ones apart, and the epilogue warps add the groups of a tile up in registers while the next group is multiplied.  (The
// groups also keep the chain short in which the tensor core cuts sums off, always towards zero: with one accumulator over
// head_d 512 the output erred by 7.8e-7 against 64 bits on normal inputs, with groups of 128 by 2.1e-7; the FFMA kernels: 4.1e-7.)
template <int NQ>   // pieces of Q and K
__global__ void __launch_bounds__(F3_A_THREADS, 1)
f32_scores_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const F32Params p) {
    constexpr int STAGE = f3_stage(NQ), NST = f3_stages(NQ);
    extern __shared__ unsigned char f3_smem_raw[];
    __shared__ uint64_t full[NST], empty[NST], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    unsigned char *smem = f3_smem_raw + ((1024u - (smem_u32(f3_smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nch = p.Dp >> 6, per_head = p.nq * p.nk, tiles = per_head * p.heads;
    const uint32_t lim = p.spin_limit;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 16); }
        mbar_fence_init();
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;       // pair g & 1 at column 256 (g & 1): leading products, then (+ 128) the small ones
    grid_launch_dependents();
    grid_dependency_wait();
    bool failed = false;
    const bool skip = *reinterpret_cast<volatile unsigned *>(p.err) != 0;   // an earlier kernel of the call failed

    if (skip) {
        // fall through to the common exit
    } else if (warp == 0) {
        if (elect_one()) {
            int s = 0, ph = 0;
            for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
                const int h = tile / per_head, r = tile - h * per_head, qt = r / p.nk, kt = r - qt * p.nk;
                for (int ch = 0; ch < nch; ++ch) {
                    F3_FAIL_AT(0, !mbar_wait(&empty[s], (uint32_t)ph ^ 1u, lim));
                    unsigned char *st = smem + (size_t)s * STAGE;
                    mbar_expect_tx(&full[s], STAGE);
#pragma unroll
                    for (int i = 0; i < NQ; ++i) {
                        tma_load_4d(st + i * F3_SLAB, &tmQ, 0, qt * F3_T, ch, i * p.heads + h, &full[s]);
                        tma_load_4d(st + (NQ + i) * F3_SLAB, &tmK, 0, kt * F3_T, ch, i * p.heads + h, &full[s]);
                    }
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t id128 = umma_idesc_bf16(128, 128, 0, 0), id256 = umma_idesc_bf16(128, 256, 0, 0);
            int s = 0, ph = 0;
            uint32_t g = 0;   // groups so far
            for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
                for (int ch = 0; ch < nch; ++ch) {
                    const bool first = (ch & 1) == 0;
                    if (first) F3_FAIL_AT(1, !mbar_wait(&acc_empty[g & 1], ((g >> 1) & 1) ^ 1u, lim));
                    F3_FAIL_AT(1, !mbar_wait(&full[s], (uint32_t)ph, lim));
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + (size_t)s * STAGE), ta = tmem + 256u * (g & 1);
                    const uint64_t q1 = umma_desc_k_sw128(sa), k1 = umma_desc_k_sw128(sa + NQ * F3_SLAB);
                    constexpr uint64_t PL = F3_SLAB >> 4;   // from a plane to the next, in descriptor units
                    // (one accumulator after the other: an MMA waits for the one before it where their columns overlap in part)
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_bf16(ta, q1 + 2 * k, k1 + 2 * k, NQ > 1 ? id256 : id128, (!first || k != 0) ? 1u : 0u);   // Q1 [K1; K2]
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (NQ > 1) umma_bf16(ta + 128, q1 + PL + 2 * k, k1 + 2 * k, id128, 1u);      // Q2 K1
                        if (NQ > 2) umma_bf16(ta + 128, q1 + 2 * k, k1 + 2 * PL + 2 * k, id128, 1u);  // Q1 K3
                        if (NQ > 1) umma_bf16(ta + 128, q1 + PL + 2 * k, k1 + PL + 2 * k, id128, 1u); // Q2 K2
                        if (NQ > 2) umma_bf16(ta + 128, q1 + 2 * PL + 2 * k, k1 + 2 * k, id128, 1u);  // Q3 K1
                    }
                    umma_commit(&empty[s]);
                    if (!first || ch + 1 == nch) { umma_commit(&acc_full[g & 1]); ++g; }
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
            }
        }
    } else {
        // ---- thread = (query row, quarter): the scores of 32 keys and their maximum.  (Four threads per row: with two, the chain tensor
        // memory -> registers -> global of a tile took longer than its MMAs.) ----
        const int qr = (warp - 2) >> 2, q = warp & 3, row = 32 * q + lane;
        const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16) + 32u * qr;
        uint32_t g = 0;
        for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
            const int h = tile / per_head, r = tile - h * per_head, qt = r / p.nk, kt = r - qt * p.nk;
            const int qrow = qt * F3_T + row, valid = min(32, p.Lk - kt * F3_T - 32 * qr);   // real keys of this quarter (none: <= 0)
            float s[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) s[j] = 0.0f;
            for (int c = 0; c < nch; c += 2, ++g) {
                F3_WARP_WAIT(2, acc_full[g & 1], (g >> 1) & 1);
                tc_fence_after();
                const uint32_t ta = tl + 256u * (g & 1);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t a[16], b[16];
                    tmem_ld16(ta + 16 * i, a);
                    if (NQ > 1) tmem_ld16(ta + 128 + 16 * i, b);
                    tmem_ld_wait();
                    float2 v[8];
                    if (NQ > 1) f3_sums<16>(a, b, nullptr, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) s[16 * i + j] += NQ > 1 ? (j & 1 ? v[j >> 1].y : v[j >> 1].x) : __uint_as_float(a[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[g & 1]);
            }
            if (failed) break;
            if (valid < 32) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (j >= valid) s[j] = -INFINITY;   // keys that do not exist: exp2(-inf) = 0
            }
            // (the P V kernel reads steps of 64 keys: a quarter without keys is written where its neighbour has some)
            if (qrow < p.Lq && valid > ((qr & 1) ? -32 : 0)) {
                float4 *sp = reinterpret_cast<float4 *>(p.S) + ((long long)tile * 32 + 8 * qr) * F3_T + row;
                float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    sp[(j >> 2) * F3_T] = make_float4(s[j], s[j + 1], s[j + 2], s[j + 3]);
                    m0 = fmaxf(m0, s[j]); m1 = fmaxf(m1, s[j + 1]); m2 = fmaxf(m2, s[j + 2]); m3 = fmaxf(m3, s[j + 3]);
                }
                atomicMax(p.rowmax + ((long long)h * p.nq * F3_T + qrow), f3_key(fmaxf(fmaxf(m0, m1), fmaxf(m2, m3))));
            }
        }
    }
    if (failed) for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies and MMAs in flight drain
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---- P V ------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// The keys go in steps of 64, which two sets of eight warps take in turn, each with a score stage, a P buffer and accumulators of
// its own: one's softmax runs under the other's MMAs.  (Two threads of a set share a row, 32 keys and 32 output columns each: with
// one thread, two warps per scheduler spent their time on each other's latencies, 39 % of the issue slots used.)  Per 16 keys three MMAs: P1 [V1 | V2 | V3] (N = 192), P2 [V1 | V2], P3 V1, into columns
// that collect the products of one order of magnitude (1, 2^-8, 2^-16).  A set adds the accumulators of its step up and
// folds them into its running output (32 registers a thread) before it hands over the next P; the exponentials of that P
// are computed before it waits.  (Scores through shared memory: loaded into registers a step ahead they cost a step their latency.)
template <typename T, int NV>   // the result's type, pieces of V
__global__ void __launch_bounds__(F3_B_THREADS, 1)
f32_pv_kernel(const __grid_constant__ CUtensorMap tmV, const F32Params p) {
    extern __shared__ unsigned char f3_smem_raw[];
    __shared__ uint64_t v_full[2], v_empty[2], s_full[2], s_empty[2], p_full[2], pv_done[2];
    __shared__ float l_part[4][F3_T];
    __shared__ uint32_t tmem_slot;
    unsigned char *smem = f3_smem_raw + ((1024u - (smem_u32(f3_smem_raw) & 1023u)) & 1023u);
    unsigned char *p_smem = smem, *v_smem = smem + 2 * F3_PBUF, *s_smem = v_smem + 2 * F3_VSTAGE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x, ncl = gridDim.x;    // the cluster is the grid's x extent
    const int qt = blockIdx.y / p.ndb, db = blockIdx.y - qt * p.ndb, h = blockIdx.z;
    const int nu = (p.Lk + 63) >> 6;                 // steps of 64 keys
    const int u0 = min(nu, rank * p.upc), n = min(nu, u0 + p.upc) - u0;
    const uint32_t lim = p.spin_limit;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 8);
            mbar_init(&p_full[i], 8); mbar_init(&pv_done[i], 1);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmV);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;       // step u: columns [256 (u & 1), + 192)
    grid_launch_dependents();
    grid_dependency_wait();
    bool failed = false;
    const bool skip = *reinterpret_cast<volatile unsigned *>(p.err) != 0;
    // warps 2-17: thread = (query row, set of warps: every other step of keys, half of a step's keys and of the output columns)
    const int wg = warp >= 10 ? 1 : 0, hf = ((warp - 2) >> 2) & 1, q = warp & 3, row = 32 * q + lane;
    const float *S_unit = p.S + ((((long long)h * p.nq + qt) * p.nk) * 32 + 16ll * u0) * F3_T * 4;
    float o[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) o[j] = 0.0f;
    float l = 0.0f;

    if (skip) {
        // fall through to the common exit
    } else if (warp == 0) {
        if (elect_one()) {
            for (int u = 0; u < n; ++u) {
                const int b = u & 1;
                F3_FAIL_AT(0, !mbar_wait(&s_empty[b], (uint32_t)((u >> 1) & 1) ^ 1u, lim));
                mbar_expect_tx(&s_full[b], F3_SSTEP);
                bulk_g2s(s_smem + (size_t)b * F3_SSTEP, S_unit + (long long)u * (F3_SSTEP / 4), F3_SSTEP, &s_full[b]);
            }
        }
    } else if (warp == 18) {   // (a thread of its own: V waits for MMAs, and the scores of the next step must not wait behind it)
        if (elect_one()) {
            for (int u = 0; u < n; ++u) {
                const int b = u & 1;
                F3_FAIL_AT(0, !mbar_wait(&v_empty[b], (uint32_t)((u >> 1) & 1) ^ 1u, lim));
                unsigned char *st = v_smem + (size_t)b * F3_VSTAGE;
                mbar_expect_tx(&v_full[b], NV * F3_VSLAB);
#pragma unroll
                for (int i = 0; i < NV; ++i) tma_load_4d(st + i * F3_VSLAB, &tmV, 0, (u0 + u) * 64, db, i * p.heads + h, &v_full[b]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t id192 = umma_idesc_bf16(128, 192, 0, 1), id128 = umma_idesc_bf16(128, 128, 0, 1), id64 = umma_idesc_bf16(128, 64, 0, 1);
            for (int u = 0; u < n; ++u) {
                const int b = u & 1;
                const uint32_t par = (uint32_t)((u >> 1) & 1);
                F3_FAIL_AT(1, !mbar_wait(&v_full[b], par, lim));
                F3_FAIL_AT(2, !mbar_wait(&p_full[b], par, lim));
                tc_fence_after();
                const uint32_t va = smem_u32(v_smem + (size_t)b * F3_VSTAGE), to = tmem + 256u * (uint32_t)b;
                const uint64_t pa = umma_desc_k_sw128(smem_u32(p_smem + (size_t)b * F3_PBUF));
                // (one set of columns after the other: an MMA waits for the one before it where their columns overlap in part)
                const uint64_t vd = umma_desc_mn_sw128(va, F3_VSLAB);
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16(to, pa + 2 * k, vd + 128 * k, NV == 3 ? id192 : NV == 2 ? id128 : id64, k != 0);
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16(to + 64, pa + (F3_SLAB >> 4) + 2 * k, vd + 128 * k, NV == 3 ? id128 : id64, NV > 1 || k != 0);
                if (NV == 2) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_bf16(to + 128, pa + (F3_SLAB >> 4) + 2 * k, vd + (F3_VSLAB >> 4) + 128 * k, id64, k != 0);   // P2 V2
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16(to + 128, pa + 2 * (F3_SLAB >> 4) + 2 * k, vd + 128 * k, id64, NV > 1 || k != 0);
                umma_commit(&v_empty[b]);
                umma_commit(&pv_done[b]);
            }
        }
    } else {
        const int qrow = qt * F3_T + row;
        const bool above = p.c > 1.0f;   // head_d 1 and 2: a finite score times c need not be finite, its distance from the maximum comes first
        float m = 0.0f;   // (rows that do not exist: whatever they hold stays in them and is not stored)
        if (qrow < p.Lq) m = f3_unkey(__ldcg(p.rowmax + (long long)h * p.nq * F3_T + qrow)) * (above ? 1.0f : p.c);
        const uint32_t prow = smem_u32(p_smem + (size_t)wg * F3_PBUF) + (uint32_t)row * 128u, sw = (uint32_t)(row & 7);
        const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + 256u * (uint32_t)wg + 32u * (uint32_t)hf;
        const float4 *sp = reinterpret_cast<const float4 *>(s_smem + (size_t)wg * F3_SSTEP) + row;
        auto fold = [&]() {   // o += the three accumulators of this set
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t a[8], b[8], c[8];
                tmem_ld8(ta + 8 * g, a);
                tmem_ld8(ta + 64 + 8 * g, b);
                tmem_ld8(ta + 128 + 8 * g, c);
                tmem_ld_wait();
                float2 v[4];
                f3_sums<8>(a, b, c, v);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 x = f3_fma2(v[j], p.share, make_float2(o[8 * g + 2 * j], o[8 * g + 2 * j + 1]));
                    o[8 * g + 2 * j] = x.x; o[8 * g + 2 * j + 1] = x.y;
                }
            }
            tc_fence_before();
        };
        int i = 0;   // steps of this set so far
        for (int u = wg; u < n; u += 2, ++i) {
            F3_WARP_WAIT(3, s_full[wg], i & 1);
            float e[32];   // the step's scores of this thread: the stage is free for the next step's at once
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 v = sp[(8 * hf + c) * F3_T];
                e[4 * c] = v.x; e[4 * c + 1] = v.y; e[4 * c + 2] = v.z; e[4 * c + 3] = v.w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[wg]);
            float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f, l3 = 0.0f;
            if (above) {   // (the whole grid takes the same branch)
#pragma unroll
                for (int c = 0; c < 32; ++c) e[c] = (e[c] - m) * p.c;
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) e[c] = fmaf(e[c], p.c, -m);
            }
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
                e[c] = fast_exp2(e[c]); e[c + 1] = fast_exp2(e[c + 1]); e[c + 2] = fast_exp2(e[c + 2]); e[c + 3] = fast_exp2(e[c + 3]);
                l0 += e[c]; l1 += e[c + 1]; l2 += e[c + 2]; l3 += e[c + 3];
            }
            l += (l0 + l1) + (l2 + l3);
            if (i > 0) {
                F3_WARP_WAIT(3, pv_done[wg], (i - 1) & 1);   // P may be overwritten, the products are there
                fold();
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {   // eight keys, 16 bytes of a row of each piece of P
                uint32_t a[4], b[4], d[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) f3_split2(e[8 * c + 2 * k], e[8 * c + 2 * k + 1], a[k], b[k], d[k]);
                const uint32_t at = prow + (((uint32_t)(4 * hf + c) ^ sw) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + F3_SLAB), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 2 * F3_SLAB), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]) : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[wg]);
        }
        if (!failed && i > 0) {
            do {
                F3_WARP_WAIT(4, pv_done[wg], (i - 1) & 1);
                fold();
            } while (false);
        }
    }
    if (failed) for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();   // every product of this CTA is done: the partial outputs of the two sets go over P
    tc_fence_after();
    if (warp >= 2 && warp < 18) {
        float *os = reinterpret_cast<float *>(p_smem) + (wg * F3_T + row) * F3_OPITCH + 32 * hf;
#pragma unroll
        for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4 *>(os + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
        l_part[2 * wg + hf][row] = l;
    }
    __syncthreads();
    if (ncl > 1) { cluster_arrive(); cluster_wait(); }
    if (!skip) {
        // each CTA of the cluster adds up and stores its share of the rows
        const int per = F3_T / ncl, r0 = rank * per, w = min(64, p.D - db * 64);
        const uint32_t mine = smem_u32(p_smem), lmine = smem_u32(&l_part[0][0]);
        for (int i = threadIdx.x; i < per * 16; i += F3_B_THREADS) {
            const int orow = r0 + (i >> 4), c = (i & 15) * 4, qrow = qt * F3_T + orow;
            if (qrow >= p.Lq || c >= w) continue;
            const uint32_t at = mine + (uint32_t)(orow * F3_OPITCH + c) * 4u, lat = lmine + (uint32_t)orow * 4u;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            float sum = 0.0f;
            for (int r = 0; r < ncl; ++r) {
                const uint32_t peer = ncl > 1 ? map_to_rank(at, (uint32_t)r) : at, lpeer = ncl > 1 ? map_to_rank(lat, (uint32_t)r) : lat;
                const float4 x = ld_cluster_v4(peer), y = ld_cluster_v4(peer + F3_T * F3_OPITCH * 4);
                sum += (ld_cluster_f32(lpeer) + ld_cluster_f32(lpeer + F3_T * 4)) + (ld_cluster_f32(lpeer + 2 * F3_T * 4) + ld_cluster_f32(lpeer + 3 * F3_T * 4));
                v.x += x.x + y.x; v.y += x.y + y.y; v.z += x.z + y.z; v.w += x.w + y.w;
            }
            const float inv = p.unshare * (1.0f / sum);
            v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
            T *op = reinterpret_cast<T *>(p.O) + ((long long)h * p.Lq + qrow) * p.D + db * 64 + c;
            if (p.vec_out) {
                if constexpr (sizeof(T) == 4) *reinterpret_cast<float4 *>(op) = v;
                else {
                    constexpr bool H = std::is_same<T, __half>::value;
                    *reinterpret_cast<uint2 *>(op) = make_uint2(pack_16x2(v.x, v.y, H), pack_16x2(v.z, v.w, H));
                }
            } else {
                op[0] = OutCvt<T>::one(v.x);
                if (c + 1 < w) op[1] = OutCvt<T>::one(v.y);
                if (c + 2 < w) op[2] = OutCvt<T>::one(v.z);
                if (c + 3 < w) op[3] = OutCvt<T>::one(v.w);
            }
        }
    }
    if (ncl > 1) { cluster_arrive(); cluster_wait(); }   // a peer may still be reading this CTA's partial output
    if (warp == 1) tmem_dealloc(tmem, 512);
}

#undef F3_FAIL_AT
#undef F3_WARP_WAIT

// ---- host side ------------------------------------------------------------------------------------
struct F32Scratch {   // per device, grown on demand
    void *buf = nullptr;
    size_t bytes = 0;
    bool attr[3] = {};   // fp32, fp16, bf16
    void release() {
        if (buf) cudaFree(buf);
        buf = nullptr; bytes = 0;
    }
};

inline bool f32tc_supported(const b200attn_args &a) {
    if (a.len_q <= 64 && a.len_k <= 64) return false;
    // Few rows on one side are padded to whole tiles here, and with enough blocks for the chip the CUDA-core kernels are done before the
    // split is (us there / here, fp32: 148 heads, 1 x 65, head_d 512 55 / 94, 1000 heads, 16 x 100, head_d 128 141 / 184, 300 heads, 200 x 8,
    // head_d 64 46 / 55; bf16: 300 heads, 1 x 128, head_d 80 44 / 52).  Below the lines this is the faster one almost everywhere (64 heads, 1 x 1000,
    // head_d 128 110 / 74; 148 heads, 300 x 32, head_d 64 51 / 39; still the slower one by up to a quarter: 1000 heads of head_d 16).
    const long long blocks = (long long)a.batch_sz * a.num_heads * ((a.len_q + 63) / 64) * ((a.head_d + 63) / 64);
    const int few = a.len_q < a.len_k ? a.len_q : a.len_k, many = a.len_q < a.len_k ? a.len_k : a.len_q;
    if ((few <= 4 && blocks >= 200) || (few <= 16 && blocks >= 300) || (few <= 32 && many <= 512 && blocks >= 1000)) return false;
    if (a.dtype == B200ATTN_F32) return a.head_d <= 512;
    // 16 bit: the widths up to 256 whose 16-bit kernels would round what the CUDA-core kernels hold in fp32
    if (a.head_d % 8 != 0 || a.head_d > 256 || (a.head_d % 64 == 0 && (a.head_d != 192 || a.len_q <= 64))) return false;
    return (((uintptr_t)a.Q | (uintptr_t)a.K | (uintptr_t)a.V | (uintptr_t)a.out) & 15) == 0;
}

// Returns B200ATTN_OK, -1 when the shape should run on another path (also when the scratch could not be allocated: nothing
// has been launched then), or a status with tc_bf16_error() set.
template <typename T>
inline int f32tc_launch(const b200attn_args &a, int rd, float base, F32Scratch &sc, unsigned *err_dev, unsigned *err_sys, int sm_count, unsigned spin_limit,
                     size_t scratch_cap, cudaStream_t st, std::atomic<unsigned long long> *launches) {
    const long long BH = (long long)a.batch_sz * a.num_heads;
    const int Lq = a.len_q, Lk = a.len_k, D = a.head_d;
    // pieces that make up a value: of V, and of Q and K (fp32 values once encoded)
    constexpr int NV = sizeof(T) == 4 ? 3 : std::is_same<T, __half>::value ? 2 : 1;
    const int nqp = a.pe != B200ATTN_PE_NONE ? 3 : NV;
    auto smem_a = [](int n) { return f3_stages(n) * (size_t)f3_stage(n) + 1024; };
    const size_t smem_b = 2 * (size_t)(F3_PBUF + F3_VSTAGE + F3_SSTEP) + 1024;
    const int type = sizeof(T) == 4 ? 0 : std::is_same<T, __half>::value ? 1 : 2;
    if (!sc.attr[type]) {
        if (cudaFuncSetAttribute(f32_scores_kernel<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_a(NV)) != cudaSuccess ||
            cudaFuncSetAttribute(f32_scores_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_a(3)) != cudaSuccess ||
            cudaFuncSetAttribute(f32_pv_kernel<T, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_b) != cudaSuccess) {
            (void)cudaGetLastError();
            snprintf(t_tc_error, sizeof t_tc_error, "cudaFuncSetAttribute(max dynamic shared memory) failed");
            return B200ATTN_ERR_CUDA;
        }
        sc.attr[type] = true;
    }
    F32Params p{};
    p.Lq = Lq; p.Lk = Lk; p.D = D; p.Dp = (D + 63) & ~63;
    const long long nq = ((long long)Lq + F3_T - 1) / F3_T, nk = ((long long)Lk + F3_T - 1) / F3_T, ndb = p.Dp / 64;
    if (nq * nk >= (1ll << 30) || nq * ndb > 65535) return -1;
    p.nq = (int)nq; p.nk = (int)nk; p.ndb = (int)ndb;
    // a pass takes as many heads as the scratch cap has room for
    const size_t qb = (size_t)Lq * p.Dp * 2 * nqp, kb = (size_t)Lk * p.Dp * 2 * nqp, vb = (size_t)Lk * p.Dp * 2 * NV, sb = (size_t)nq * nk * F3_T * F3_T * 4, tb = (size_t)nq * F3_T * 4;
    const size_t per_head = qb + kb + vb + sb + tb;
    long long G = (long long)(scratch_cap / per_head);
    if (G < 1) G = 1;
    if (G > BH) G = BH;
    if (G > 20000) G = 20000;   // grid dimension, and three planes of heads in a tensor-map coordinate
    if (G * nq * nk >= (1ll << 30)) G = (1ll << 30) / (nq * nk);
    const size_t want = (size_t)G * per_head + 5 * 256;
    if (want > sc.bytes) {
        if (sc.buf) { cudaDeviceSynchronize(); cudaFree(sc.buf); }
        sc.buf = nullptr; sc.bytes = 0;
        if (cudaMalloc(&sc.buf, want) != cudaSuccess) { (void)cudaGetLastError(); sc.buf = nullptr; return -1; }
        sc.bytes = want;
    }
    p.c = 1.4426950408889634f / sqrtf((float)D);
    int steps_log2 = 0;
    while ((64ll << steps_log2) < Lk) ++steps_log2;
    p.share = ldexpf(1.0f, -steps_log2);
    p.unshare = 1.0f / (p.share * F3_VSCALE);
    p.vec_out = D % 4 == 0 && ((uintptr_t)a.out & (4 * sizeof(T) - 1)) == 0;
    p.err = err_dev; p.err_sys = err_sys; p.spin_limit = spin_limit;
    for (long long h0 = 0; h0 < BH; h0 += G) {
        const int n = (int)(BH - h0 < G ? BH - h0 : G);
        auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
        unsigned char *b = (unsigned char *)sc.buf;
        __nv_bfloat16 *qpl = (__nv_bfloat16 *)b; b += up(n * qb);
        __nv_bfloat16 *kpl = (__nv_bfloat16 *)b; b += up(n * kb);
        __nv_bfloat16 *vpl = (__nv_bfloat16 *)b; b += up(n * vb);
        p.S = (float *)b; b += up(n * sb);
        p.rowmax = (int *)b;
        p.heads = n;
        p.O = (T *)a.out + (size_t)h0 * Lq * D;
        F32SplitParams s{};
        s.heads = n; s.D = D; s.Dp = p.Dp; s.pe = a.pe;
        s.rd = rd; s.base = a.pe == B200ATTN_PE_SINUSOIDAL ? 10000.0f : base;
        s.cos_cache = a.cos_cache; s.sin_cache = a.sin_cache;
        s.rowmax = p.rowmax; s.nrows = (long long)n * nq * F3_T;
        s.t[0] = {(const T *)a.Q + (size_t)h0 * Lq * D, qpl, Lq, a.pe != B200ATTN_PE_NONE, nqp, 1.0f};
        s.t[1] = {(const T *)a.K + (size_t)h0 * Lk * D, kpl, Lk, pe_encodes_k(a.pe), nqp, 1.0f};
        s.t[2] = {(const T *)a.V + (size_t)h0 * Lk * D, vpl, Lk, 0, NV, F3_VSCALE};
        CUtensorMap tmQ, tmK, tmV;
        if (!make_tmap_grouped_heads(&tmQ, qpl, (long long)nqp * n, Lq, p.Dp, F3_T, 1) || !make_tmap_grouped_heads(&tmK, kpl, (long long)nqp * n, Lk, p.Dp, F3_T, 1) ||
            !make_tmap_grouped_heads(&tmV, vpl, (long long)NV * n, Lk, p.Dp, 64, 1)) {
            snprintf(t_tc_error, sizeof t_tc_error, "cuTensorMapEncodeTiled failed");
            return h0 == 0 ? -1 : B200ATTN_ERR_CUDA;
        }
        // split: about four blocks per SM; a share of the heads repeats the angles
        const long long items = (long long)(Lq > Lk ? Lq : Lk) * (p.Dp / 8);
        long long blocks = (items + 255) / 256, shares = 1;
        const long long cap = (long long)sm_count * 8 / 3;
        if (blocks > cap) blocks = cap;
        shares = cap / blocks;
        if (shares > (n + 1) / 2) shares = (n + 1) / 2;
        if (shares < 1) shares = 1;
        cudaError_t e = launch_dependent(f32_split_kernel<T>, dim3((unsigned)blocks, (unsigned)shares, 3), 256, 0, 1, st, s);
        // scores: a CTA per SM, a tile at a time
        const long long tiles = nq * nk * n;
        const unsigned grid = (unsigned)(tiles < sm_count ? tiles : sm_count);
        if (e == cudaSuccess) e = launch_dependent(nqp == 3 ? f32_scores_kernel<3> : f32_scores_kernel<NV>, dim3(grid), F3_A_THREADS, smem_a(nqp), 1, st, tmQ, tmK, p);
        // P V: the keys are cut while that still adds CTAs to idle SMs and leaves each a step for either set of warps
        const int nu = (Lk + 63) / 64;
        int ncl = 1;
        while (ncl < F3_MAX_CLUSTER && 4 * ncl <= nu && nq * ndb * n * ncl * 2 <= sm_count) ncl *= 2;
        p.upc = (nu + ncl - 1) / ncl;
        if (e == cudaSuccess) e = launch_dependent(f32_pv_kernel<T, NV>, dim3((unsigned)ncl, (unsigned)(nq * ndb), (unsigned)n), F3_B_THREADS, smem_b, ncl, st, tmV, p);
        if (e != cudaSuccess) { snprintf(t_tc_error, sizeof t_tc_error, "launch of the fp32 tensor-core kernels failed: %s", cudaGetErrorString(e)); return B200ATTN_ERR_CUDA; }
        launches->fetch_add(3);
    }
    return B200ATTN_OK;
}

inline int f32tc_run(const b200attn_args &a, int rd, float base, F32Scratch &sc, unsigned *err_dev, unsigned *err_sys, int sm_count, unsigned spin_limit,
                     size_t scratch_cap, cudaStream_t st, std::atomic<unsigned long long> *launches) {
    return a.dtype == B200ATTN_F32 ? f32tc_launch<float>(a, rd, base, sc, err_dev, err_sys, sm_count, spin_limit, scratch_cap, st, launches)
         : a.dtype == B200ATTN_F16 ? f32tc_launch<__half>(a, rd, base, sc, err_dev, err_sys, sm_count, spin_limit, scratch_cap, st, launches)
                                   : f32tc_launch<__nv_bfloat16>(a, rd, base, sc, err_dev, err_sys, sm_count, spin_limit, scratch_cap, st, launches);
}

}  // namespace b200attn
