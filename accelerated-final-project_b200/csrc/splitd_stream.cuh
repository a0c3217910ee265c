// Attention forward for short sequences (len_q, len_k <= 64) and wide heads with STREAMED column slices: the decomposition of
// splitd_tc.cuh (a CTA owns a column slice of Q, K and V of one head, error-compensated tf32 MMAs, partial scores summed in an
// L2-resident scratch) for slices of any width, for fp32 and 16-bit tensors, with the positional encodings whose pairs are
// neighbouring columns, and for several independent problems of one shape in one launch.
//
// splitd_tc.cuh keeps a whole slice of V in shared memory, so a slice is at most 256 columns and a call at most #SMs / (head_d /
// 256) heads; everything beyond, and everything with an encoding or 16-bit tensors, ran on the CUDA-core kernels of splitd.cuh.
// Here both contractions stream: atoms of 32 columns of Q and K pass through landing slots into operand stages, then V passes
// through a ring in blocks of four atoms while the block before it is multiplied and the one before that is stored.  The
// kernel is bound by its HBM traffic (every input byte is read once) once a CTA has a few blocks; below that by the chain
// load -> scores -> reduction over the slices -> softmax -> P V -> store that splitd_tc.cuh describes.
//
//   warp 0       TMA loads, the head's arrival counter
//   warp 1       MMAs
//   warps 2-7    landed atoms -> (encoding) -> hi | lo operand stage; landed V -> hi and lo (16-bit V: -> its fp32 operand layout)
//   warps 8-11   partial scores -> scratch, softmax, P, epilogue of each block of 128 output columns
//
// Precision: operands are cut into bf16 pieces whose sum is exact (fp32 and encoded values three, fp16 two, bf16 one; P three) and
// the products are collected by their order of magnitude in accumulators of their own (x1 y1 | x1 y2 + x2 y1 | x1 y3 + x2 y2 +
// x3 y1); what is left out is below 2^-22 of a product, on average 2^-26 (the first piece is cut off, not rounded: x2 reaches 2^-7 x).  A score accumulator takes 128 columns, the sums over
// these are added up in fp32 registers: the tensor core cuts a sum off where it does not fit, always towards zero.  Against 64
// bits (uniform inputs, head_d 2048 to 8192) a hi / lo tf32 form of this kernel erred by 6e-7 to 8e-7, the CUDA-core kernels
// by 1.1e-7 to 1.8e-7, this form by 0.8e-7 to 1.0e-7.  The encoding and the softmax are fp32 as in splitd.cuh.
// Infinities and NaN go through the MMAs like other values: a sum of leading products that is not finite is the result, whatever
// the smaller products are (a lower piece of such a value is NaN).  The epilogue looks for such sums only in blocks of V that
// hold such a value.
// The score scratch is one buffer, cleared by its user: a call starts after the one before it in the stream is complete.  (The ring
// of splitd_tc.cuh, whose generations the host counts, is for calls that overlap; a call captured into a graph is counted there
// but runs when the graph is launched, never or often, and later calls then waited for a generation that did not come.)
// The slices of a head wait for each other's scores, and the launch does not promise that they run together: while another stream's
// kernel holds some of the SMs, some slices wait for room.  A slice says that it runs (cnt_cur, upper half) when it starts; until all
// of them have said so the others' patience is some thousands of times the limit of the waits on work that is running, so such a call
// takes until there is room, as a cooperative launch would.  (Launched as one: 14.3 -> 16.4 us for 4 heads, 64 x 64, head_d 2048, RoPE.)
#pragma once

#include <type_traits>

#include "splitd_tc.cuh"

namespace b200attn {

constexpr int SW_THREADS = 384;
constexpr int SW_SPLIT = 192;             // threads of warps 2-7
constexpr int SW_NR = 4;                  // landing slots of 16 KB
constexpr int SW_NST = 4;                 // operand stages of one atom; two share the 128-byte rows of their planes
constexpr int SW_PL = 64 * 128;           // a plane [64 rows x 64 bf16]
constexpr int SW_STAGE = 6 * SW_PL;       // two atoms: Q1 Q2 Q3 K1 K2 K3
constexpr int SW_VBLK = 4 * ST_SLAB;      // a block of V as it lands: four atoms [64 keys x 32 columns] fp32
constexpr int SW_VOP = 6 * SW_PL;         // its operand: V1 V2 V3, each [2 groups of 64 columns][64 keys][128 B]
constexpr int SW_NV = 3;                  // V ring: slots 0 and 1 have room of their own, 2 lies over landing slots
constexpr int SW_GROUP = 4;               // atoms per score accumulator
constexpr int SW_MAXP = 16;               // problems per launch

// Shared memory: V slots 0, 1 | while the scores are computed: operand stages, landing slots
//                             | afterwards: two V operands (stages), P1 P2 P3 (landing slots 0, 1), V slot 2 (landing slots 2, 3)
constexpr size_t SW_SMEM = 2 * (size_t)SW_VBLK + 2 * (size_t)SW_STAGE + SW_NR * (size_t)ST_CHUNK + 1024;
static_assert(SW_NR == 4 && SW_VOP == SW_STAGE && 3 * SW_PL <= 2 * ST_CHUNK && SW_VBLK == 2 * ST_CHUNK, "the second use of the shared memory relies on these");

template <int NP> struct SwProblems {
    CUtensorMap q[NP], k[NP], v[NP];
    void *O[NP];
};

struct SwParams {
    int BH;                  // heads of one problem
    int Lq, Lk, D;
    int natoms, nsplit;      // atoms of 32 columns; slices per head
    int pe, rd;
    const float2 *tab;       // [64 positions][16 natoms] (cos, sin) of a pair of columns; what leaves a pair alone where it is not encoded
    float scale;
    float *S;                // [heads of the launch][64][64]
    unsigned *counters;      // [heads][2]: warps that have added their scores + 65536 x slices that run, warps that have read the sums
    unsigned *err, *err_sys;
    unsigned spin_limit, wait_extra;
};

struct SwBars {
    uint64_t full[SW_NR], raw_free[SW_NR];
    uint64_t ready[SW_NST], st_free[SW_NST];
    uint64_t acc_full[2], acc_empty[2];     // a group of atoms has been multiplied / read
    uint64_t s_full, head_ok, p_ready;
    uint64_t v_full[SW_NV], v_free[SW_NV];
    uint64_t v_ready[2], vop_free[2];
    uint64_t o_full[2], o_empty[2];
};

// What depends on the other slices of the head: longer waits, cut short when the thread that waits for those has given up.
constexpr uint32_t SW_ROOM = 4096;   // times the poll limit
__device__ __forceinline__ bool sw_wait_head(uint64_t *bar, uint32_t parity, uint32_t lim, unsigned *fail) {
    if (mbar_test_wait(bar, parity)) return true;
    for (unsigned long long it = 0; it < (unsigned long long)lim * SW_ROOM; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (it > 64) {
            __nanosleep(32);
            if ((it & 63) == 0 && *reinterpret_cast<volatile unsigned *>(fail) != 0u) return false;
        }
    }
    return false;
}

#define SW_FAIL_AT(site, cond)                                                                       \
    if (cond) {                                                                                      \
        report_kernel_error(p.err, p.err_sys, (unsigned)KERR_MBAR_TIMEOUT | (1u << (7 + (site))));   \
        *reinterpret_cast<volatile unsigned *>(&s_fail) = 1u;                                        \
        failed = true;                                                                               \
        break;                                                                                       \
    }

// the same for a wait of a whole warp: either all of its lanes go on or none
#define SW_WARP_WAIT(site, bar, parity)                                                                          \
    SW_WARP_ALL(site, mbar_wait(&(bar), (uint32_t)(parity), lim))
#define SW_WARP_WAIT_HEAD(site, bar, parity)                                                                     \
    SW_WARP_ALL(site, sw_wait_head(&(bar), (uint32_t)(parity), lim, &s_fail))
#define SW_WARP_ALL(site, waited)                                                                                \
    if (!__all_sync(0xffffffffu, waited)) {                                                                      \
        if (lane == 0) report_kernel_error(p.err, p.err_sys, (unsigned)KERR_MBAR_TIMEOUT | (1u << (7 + (site)))); \
        *reinterpret_cast<volatile unsigned *>(&s_fail) = 1u;                                                    \
        failed = true;                                                                                           \
        break;                                                                                                   \
    }


// ---- (cos, sin) of the encodings whose pairs are columns (2i, 2i + 1), positions 0 to 63: the arithmetic of the reference tables
// (final/rope.cu:20-40, final/sinusoidal.cu:143-161) ----
__global__ void __launch_bounds__(256) sw_table_kernel(float2 *tab, int npairs, int D, int rd, float base, int sinus) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 64 * npairs; i += gridDim.x * blockDim.x) {
        const int pos = i / npairs, pair = i - pos * npairs;
        float c = sinus ? 0.0f : 1.0f, s = 0.0f;
        if (sinus ? 2 * pair < D : 2 * pair + 1 < rd) {
            const float freq = 1.0f / powf(base, (2.0f * (float)pair) / (float)rd);
            sincosf((float)pos * freq, &s, &c);
        }
        tab[i] = make_float2(c, s);
    }
}

// encodes the pair (a, b) of columns (fp32, the products and sums of splitd.cuh's load_slice)
__device__ __forceinline__ void sw_encode(float &a, float &b, bool sinus, float c, float s) {
    if (sinus) { a += s; b += c; }
    else { const float x = a, y = b; a = x * c - y * s; b = x * s + y * c; }
}

// eight fp32 values as N bf16 pieces each, packed; returns a number that is NaN when one of the values is not finite
template <int N> __device__ __forceinline__ float sw_pieces(const float (&x)[8], uint4 (&out)[N]) {
    uint32_t w[3][4];
    float odd = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t u0 = __float_as_uint(x[2 * i]), u1 = __float_as_uint(x[2 * i + 1]);
        w[0][i] = __byte_perm(u0, u1, 0x7632);   // truncation: the first piece of a large value must not round up to infinity
        const float r0 = x[2 * i] - __uint_as_float(u0 & 0xffff0000u), r1 = x[2 * i + 1] - __uint_as_float(u1 & 0xffff0000u);
        odd += r0 + r1;                          // inf - inf, NaN - NaN
        if (N > 1) w[1][i] = pack_bf16x2(r0, r1);
        if (N > 2) w[2][i] = pack_bf16x2(r0 - __uint_as_float(w[1][i] << 16), r1 - __uint_as_float(w[1][i] & 0xffff0000u));
    }
#pragma unroll
    for (int n = 0; n < N; ++n) out[n] = make_uint4(w[n][0], w[n][1], w[n][2], w[n][3]);
    return odd;
}

// eight elements of a row of an atom as it lands (fp32: 128-byte swizzled rows of 128 bytes; 16 bit: plain rows of 64 bytes)
template <typename T> __device__ __forceinline__ void sw_open8(const unsigned char *slab, int row, int pc, float (&x)[8]) {
    if constexpr (sizeof(T) == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(slab + st_swz(row, 8 * pc)), b = *reinterpret_cast<const float4 *>(slab + st_swz(row, 8 * pc + 4));
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
        const uint4 v = *reinterpret_cast<const uint4 *>(slab + row * 64 + pc * 16);
        const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = to_f32(e[i]);
    }
}

// The first pieces of eight fp32 values as they landed, some of them not finite: one of a NaN stays a NaN when its low bits are cut off.
__device__ __noinline__ void sw_keep_nan(const unsigned char *slab, int row, int pc, unsigned char *first) {
    for (int i = 0; i < 8; ++i)
        if ((*reinterpret_cast<const uint32_t *>(slab + st_swz(row, 8 * pc + i)) & 0x7fffffffu) > 0x7f800000u) *reinterpret_cast<uint16_t *>(first + 2 * i) |= 0x0040;
}

// Reports that the head's other slices did not arrive.  (A call that takes the address of the parameters: with one the compiler keeps a copy
// of them at hand, without it reads them from the constant bank, beside up to 6 KB of tensor maps: 16 problems of 4 heads, 64 x 64,
// head_d 2048 take 43.1 us with it and 47.6 us without.)
__device__ __noinline__ void sw_report(const SwParams &p, unsigned bits) { report_kernel_error(p.err, p.err_sys, bits); }

template <typename T, bool PE, int NP>
__global__ void __launch_bounds__(SW_THREADS, 1)
sw_kernel(const __grid_constant__ SwProblems<NP> pr, const SwParams p) {
    constexpr bool W = sizeof(T) == 4;              // fp32 tensors
    constexpr int NVP = W ? 3 : std::is_same<T, __half>::value ? 2 : 1;   // pieces of V
    constexpr int NQP = PE ? 3 : NVP;               // pieces of Q and K
    constexpr uint32_t RB = 32 * sizeof(T);         // bytes of a row of an atom as it lands
    constexpr uint32_t ASLAB = 64 * RB;             // an atom of one operand as it lands
    extern __shared__ __align__(256) unsigned char sw_smem_raw[];
    __shared__ SwBars bars;
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned s_fail, s_odd_v[2];   // a non-finite value in block n of V: n + 1
    unsigned char *smem = sw_smem_raw + ((1024u - (smem_u32(sw_smem_raw) & 1023u)) & 1023u);
    unsigned char *stages = smem + 2 * SW_VBLK, *raw = stages + 2 * SW_STAGE;
    unsigned char *v_op = stages, *p_buf = raw;
    auto v_slot = [&](int s) { return s < 2 ? smem + (size_t)s * SW_VBLK : raw + 2 * ST_CHUNK; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slice = blockIdx.x, head = blockIdx.y;
    const int prob = NP == 1 ? 0 : head / p.BH, bh = NP == 1 ? head : head - prob * p.BH;
    const int Lq = p.Lq, Lk = p.Lk, kpad = (Lk + 15) & ~15;
    const int nat = (p.natoms - slice + p.nsplit - 1) / p.nsplit;   // atoms slice, slice + nsplit, ...
    const int nblk = (nat + 3) >> 2;
    auto atom_col = [&](int c) { return (slice + c * p.nsplit) * ST_ATOM; };
    const uint32_t lim = p.spin_limit;
    float *S_cur = p.S + (size_t)head * 4096;
    unsigned *cnt_cur = p.counters + (size_t)head * 2;
    const CUtensorMap *tmQ = &pr.q[prob], *tmK = &pr.k[prob], *tmV = &pr.v[prob];

    auto load_atom = [&](int c, int r) {
        unsigned char *st = raw + (size_t)r * ST_CHUNK;
        mbar_expect_tx(&bars.full[r], (uint32_t)(Lq + Lk) * RB);
        tma_load_2d(st, tmQ, atom_col(c), bh * Lq, &bars.full[r]);
        tma_load_2d(st + ST_SLAB, tmK, atom_col(c), bh * Lk, &bars.full[r]);
    };
    auto load_v = [&](int b, int s) {
        const int na = min(4, nat - 4 * b);
        mbar_expect_tx(&bars.v_full[s], (uint32_t)(na * Lk) * RB);
        for (int i = 0; i < na; ++i) tma_load_2d(v_slot(s) + (size_t)i * ASLAB, tmV, atom_col(4 * b + i), bh * Lk, &bars.v_full[s]);
    };

    if (threadIdx.x == 0) {
        tma_prefetch_desc(tmQ); tma_prefetch_desc(tmK); tma_prefetch_desc(tmV);
        for (int i = 0; i < SW_NR; ++i) { mbar_init(&bars.full[i], 1); mbar_init(&bars.raw_free[i], 6); }
        for (int i = 0; i < SW_NST; ++i) { mbar_init(&bars.ready[i], 6); mbar_init(&bars.st_free[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars.acc_full[i], 1); mbar_init(&bars.acc_empty[i], 4);
            mbar_init(&bars.v_ready[i], 6); mbar_init(&bars.vop_free[i], 1);
            mbar_init(&bars.o_full[i], 1); mbar_init(&bars.o_empty[i], 4);
        }
        for (int i = 0; i < SW_NV; ++i) { mbar_init(&bars.v_full[i], 1); mbar_init(&bars.v_free[i], 6); }
        mbar_init(&bars.s_full, 1); mbar_init(&bars.head_ok, 1); mbar_init(&bars.p_ready, 4);
        s_fail = 0u; s_odd_v[0] = s_odd_v[1] = 0u;
        mbar_fence_init();
        grid_dependency_wait();   // (a no-op unless launched as a programmatic dependent)
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 65536;" ::"l"(cnt_cur) : "memory");   // this slice runs
        for (int c = 0; c < nat && c < SW_NR; ++c) load_atom(c, c);
        for (int b = 0; b < nblk && b < 2; ++b) load_v(b, b);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // scores of group g of atoms, and later output block b: columns [256 (g & 1), + 192), 64 per order of magnitude of the products
    const uint32_t tmem = tmem_slot;
    bool failed = false;
    grid_launch_dependents();
    grid_dependency_wait();

    if (warp == 0) {
        if (elect_one()) {
            do {
                for (int c = SW_NR, r = 0, par = 0; c < nat; ++c) {
                    SW_FAIL_AT(0, !mbar_wait(&bars.raw_free[r], (uint32_t)par, lim));
                    load_atom(c, r);
                    if (++r == SW_NR) { r = 0; par ^= 1; }
                }
                if (failed) break;
                if (nblk > 2) {   // V over the landing slots, once everything in them has been multiplied
                    SW_FAIL_AT(1, !mbar_wait(&bars.s_full, 0, lim));
                    load_v(2, 2);
                }
                // the head's scores are complete when every read-out warp of every slice has arrived
                const unsigned want = 4u * (unsigned)p.nsplit + p.wait_extra;
                unsigned seen = 0, polls = 0;
                for (unsigned it = 0; polls < lim; ++it) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(cnt_cur) : "memory");
                    if ((seen & 0xffffu) >= want) break;
                    const bool all = (seen >> 16) == (unsigned)p.nsplit;
                    __nanosleep(all ? 20 : 500);
                    if (all || (it & (SW_ROOM / 16 - 1)) == 0) ++polls;   // (some twenty times as long a poll)
                }
                if ((seen & 0xffffu) < want) {
                    sw_report(p, (unsigned)KERR_HEAD_BARRIER_TIMEOUT);
                    *reinterpret_cast<volatile unsigned *>(&s_fail) = 1u;
                }
                mbar_arrive(&bars.head_ok);
                if ((seen & 0xffffu) < want) break;
                for (int b = SW_NV, s = 0, par = 0; b < nblk; ++b) {
                    SW_FAIL_AT(2, !sw_wait_head(&bars.v_free[s], (uint32_t)par, lim, &s_fail));
                    load_v(b, s);
                    if (++s == SW_NV) { s = 0; par ^= 1; }
                }
            } while (false);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            do {
                // scores, M = 64: per 16 columns Q1 [K1; K2; K3], Q2 [K1; K2], Q3 K1
                const uint32_t id64 = umma_idesc_bf16(64, 64, 0, 0), id128 = umma_idesc_bf16(64, 128, 0, 0), id192 = umma_idesc_bf16(64, 192, 0, 0);
                for (int c = 0; c < nat; ++c) {
                    const int j = c & (SW_NST - 1), g = c / SW_GROUP;
                    const bool first = c % SW_GROUP == 0;
                    SW_FAIL_AT(3, !mbar_wait(&bars.ready[j], (uint32_t)((c / SW_NST) & 1), lim));
                    if (first) SW_FAIL_AT(3, !mbar_wait(&bars.acc_empty[g & 1], (uint32_t)((g >> 1) & 1) ^ 1u, lim));
                    tc_fence_after();
                    const uint32_t ts = tmem + 256u * (uint32_t)(g & 1);
                    const uint32_t sa = smem_u32(stages + (size_t)(j >> 1) * SW_STAGE) + 64u * (uint32_t)(j & 1);
                    constexpr uint64_t PL = SW_PL >> 4;   // from a plane to the next, in descriptor units
                    const uint64_t q1 = umma_desc_k_sw128(sa), k1 = umma_desc_k_sw128(sa + 3 * SW_PL);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const uint32_t acc = (!first || k != 0) ? 1u : 0u;
                        if (NQP == 3) {
                            umma_bf16(ts, q1 + 2 * k, k1 + 2 * k, id192, acc);
                            umma_bf16(ts + 64, q1 + PL + 2 * k, k1 + 2 * k, id128, 1u);
                            umma_bf16(ts + 128, q1 + 2 * PL + 2 * k, k1 + 2 * k, id64, 1u);
                        } else if (NQP == 2) {
                            umma_bf16(ts, q1 + 2 * k, k1 + 2 * k, id128, acc);
                            umma_bf16(ts + 64, q1 + PL + 2 * k, k1 + 2 * k, id64, 1u);
                            umma_bf16(ts + 128, q1 + PL + 2 * k, k1 + PL + 2 * k, id64, acc);
                        } else {
                            umma_bf16(ts, q1 + 2 * k, k1 + 2 * k, id64, acc);
                        }
                    }
                    umma_commit(&bars.st_free[j]);
                    if (c + 1 == nat || (c + 1) % SW_GROUP == 0) umma_commit(&bars.acc_full[g & 1]);
                }
                if (failed) break;
                umma_commit(&bars.s_full);
                // O[:, block]^T = V^T P^T: V the M-major A operand, P1 P2 P3 one K-major B operand; per 16 keys V1 [P1 | P2 | P3], V2 [P1 | P2], V3 P1
                SW_FAIL_AT(4, !sw_wait_head(&bars.p_ready, 0, lim, &s_fail));
                const uint32_t iv64 = umma_idesc_bf16(128, 64, 1, 0), iv128 = umma_idesc_bf16(128, 128, 1, 0), iv192 = umma_idesc_bf16(128, 192, 1, 0);
                const uint64_t dp = umma_desc_k_sw128(smem_u32(p_buf));
                for (int b = 0; b < nblk; ++b) {
                    const int e = b & 1;
                    SW_FAIL_AT(5, !sw_wait_head(&bars.v_ready[e], (uint32_t)((b >> 1) & 1), lim, &s_fail));
                    SW_FAIL_AT(6, !sw_wait_head(&bars.o_empty[e], (uint32_t)((b >> 1) & 1) ^ 1u, lim, &s_fail));
                    tc_fence_after();
                    const uint32_t va = smem_u32(v_op + (size_t)e * SW_VOP), to = tmem + 256u * (uint32_t)e;
                    for (int k = 0; k < (kpad >> 4); ++k) {
                        const uint64_t v1 = umma_desc_mn_sw128(va + (uint32_t)k * 2048u, SW_PL);
                        umma_bf16(to, v1, dp + 2 * k, iv192, k != 0);
                        if (NVP > 1) umma_bf16(to + 64, v1 + (2 * SW_PL >> 4), dp + 2 * k, iv128, 1u);
                        if (NVP > 2) umma_bf16(to + 128, v1 + (4 * SW_PL >> 4), dp + 2 * k, iv64, 1u);
                    }
                    umma_commit(&bars.vop_free[e]);
                    umma_commit(&bars.o_full[e]);
                }
            } while (false);
        }
    } else if (warp < 8) {
        const int t = threadIdx.x - 64;   // 0..191
        const bool sinus = p.pe == PE_SINUSOIDAL;
        const bool enc_k = pe_encodes_k(p.pe);
        for (int c = 0; c < nat; ++c) {
            // pieces of eight columns: piece idx = (operand, row, place in the row), three rounds
            float4 ang[3][2];
            if (PE) {   // requested before the wait, so that they travel while the atom does
#pragma unroll
                for (int n = 0; n < 3; ++n) {
                    const int idx = t + n * SW_SPLIT, row = (idx >> 2) & 63, pc = idx & 3;
                    if (idx < (enc_k ? 512 : 256)) {
                        // (four pairs, 32 bytes: (cos, sin) of the pairs, two pairs per 16 bytes)
                        const float4 *tp = reinterpret_cast<const float4 *>(p.tab + (size_t)row * 16 * p.natoms + (atom_col(c) >> 1) + 4 * pc);
                        ang[n][0] = __ldg(tp); ang[n][1] = __ldg(tp + 1);
                    }
                }
            }
            const int r = c & (SW_NR - 1), j = c & (SW_NST - 1);
            SW_WARP_WAIT(7, bars.full[r], (c / SW_NR) & 1);
            SW_WARP_WAIT(8, bars.st_free[j], ((c / SW_NST) & 1) ^ 1);
            const unsigned char *src = raw + (size_t)r * ST_CHUNK;
            unsigned char *dst = stages + (size_t)(j >> 1) * SW_STAGE;
            float odd = 0.0f;
            auto first = [&](int op, int row, int pc) { return dst + op * 3 * SW_PL + row * 128 + (((4 * (j & 1) + pc) ^ (row & 7)) << 4); };
            const bool part = !sinus && atom_col(c) + ST_ATOM > p.rd;   // pairs from rotary_dim on are left alone, infinities too
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const int idx = t + n * SW_SPLIT, op = idx >> 8, row = (idx >> 2) & 63, pc = idx & 3;
                if (idx < 512 && row < (op ? Lk : Lq)) {
                    float x[8];
                    sw_open8<T>(src + op * ST_SLAB, row, pc, x);
                    if (PE && (!op || enc_k)) {
                        const int left = part ? p.rd - (atom_col(c) + 8 * pc) : 8;
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (4 * e < left) sw_encode(x[4 * e], x[4 * e + 1], sinus, ang[n][e].x, ang[n][e].y);
                            if (4 * e + 2 < left) sw_encode(x[4 * e + 2], x[4 * e + 3], sinus, ang[n][e].z, ang[n][e].w);
                        }
                    }
                    uint4 w[NQP];
                    odd += sw_pieces<NQP>(x, w);
                    unsigned char *d = first(op, row, pc);
#pragma unroll
                    for (int i = 0; i < NQP; ++i) *reinterpret_cast<uint4 *>(d + i * SW_PL) = w[i];
                }
            }
            if (W && odd != odd)
                for (int idx = t; idx < 512; idx += SW_SPLIT) {
                    const int op = idx >> 8, row = (idx >> 2) & 63, pc = idx & 3;
                    if (row < (op ? Lk : Lq)) sw_keep_nan(src + op * ST_SLAB, row, pc, first(op, row, pc));
                }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&bars.ready[j]); mbar_arrive(&bars.raw_free[r]); }
        }
        // ---- V: its pieces in the M-major layout; key rows [Lk, kpad) are zero ----
        if (!failed) {
            do {
                SW_WARP_WAIT(9, bars.s_full, 0);   // the stages may be overwritten
                for (int b = 0, s = 0, par = 0; b < nblk; ++b) {
                    const int e = b & 1, na = min(4, nat - 4 * b);
                    SW_WARP_WAIT_HEAD(10, bars.v_full[s], par);
                    SW_WARP_WAIT_HEAD(11, bars.vop_free[e], ((b >> 1) & 1) ^ 1);
                    const unsigned char *in = v_slot(s);
                    unsigned char *out = v_op + (size_t)e * SW_VOP;
                    float odd = 0.0f;
                    auto first = [&](int a, int row, int pc) { return out + (a >> 1) * SW_PL + row * 128 + (((4 * (a & 1) + pc) ^ (row & 7)) << 4); };
                    for (int idx = t; idx < (na << 8); idx += SW_SPLIT) {
                        const int a = idx >> 8, row = (idx >> 2) & 63, pc = idx & 3;
                        if (row < kpad) {
                            float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                            if (row < Lk) sw_open8<T>(in + a * ASLAB, row, pc, x);
                            uint4 w[NVP];
                            odd += sw_pieces<NVP>(x, w);
                            unsigned char *d = first(a, row, pc);
#pragma unroll
                            for (int i = 0; i < NVP; ++i) *reinterpret_cast<uint4 *>(d + i * 2 * SW_PL) = w[i];
                        }
                    }
                    if (__any_sync(0xffffffffu, odd != odd)) {
                        if (W)
                            for (int idx = t; idx < (na << 8); idx += SW_SPLIT) {
                                const int a = idx >> 8, row = (idx >> 2) & 63, pc = idx & 3;
                                if (row < Lk) sw_keep_nan(in + a * ASLAB, row, pc, first(a, row, pc));
                            }
                        // the word still belongs to block b - 2 until its epilogue has read it
                        SW_WARP_WAIT_HEAD(11, bars.o_empty[e], ((b >> 1) & 1) ^ 1);
                        if (lane == 0) *reinterpret_cast<volatile unsigned *>(&s_odd_v[e]) = (unsigned)b + 1u;
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(&bars.v_ready[e]); mbar_arrive(&bars.v_free[s]); }
                    if (++s == SW_NV) { s = 0; par ^= 1; }
                }
            } while (false);
        }
    } else {
        // ---- warps 8-11, one quadrant of tensor-memory lanes each ----
        const int q = warp & 3, w4 = warp - 8;
        const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16);
        do {
            // partial scores (M = 64: row r is in lane 32 (r / 16) + r % 16): summed over the groups of atoms, then added to the head's in the scratch
            float acc[64];
#pragma unroll
            for (int j = 0; j < 64; ++j) acc[j] = 0.0f;
            const int ngrp = (nat + SW_GROUP - 1) / SW_GROUP;
            for (int g = 0; g < ngrp; ++g) {
                SW_WARP_WAIT(12, bars.acc_full[g & 1], (g >> 1) & 1);
                tc_fence_after();
                const uint32_t ts = tq + 256u * (uint32_t)(g & 1);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t r0[16], r1[16], r2[16];
                    tmem_ld16(ts + 16 * k, r0);
                    if (NQP > 1) { tmem_ld16(ts + 64 + 16 * k, r1); tmem_ld16(ts + 128 + 16 * k, r2); }
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        // (products that overflow: the smaller ones may be infinities of the other sign, a third piece need not have its value's)
                        const float lead = __uint_as_float(r0[j]);
                        acc[16 * k + j] += NQP > 1 && fabsf(lead) < INFINITY ? lead + (__uint_as_float(r1[j]) + __uint_as_float(r2[j])) : lead;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.acc_empty[g & 1]);
            }
            if (failed) break;
            if (__any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned *>(&s_fail) != 0u)) { failed = true; break; }
            const int row = 16 * q + lane;
            if (lane < 16 && row < Lq) {
                float *srow = S_cur + (size_t)row * 64;
#pragma unroll
                for (int j = 0; j < 64; j += 4) red_add_v4(srow + j, acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
            }
            __syncwarp();
            if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt_cur) : "memory");
            SW_WARP_WAIT(14, bars.s_full, 0);    // P goes where atoms landed
            SW_WARP_WAIT_HEAD(14, bars.head_ok, 0);
            if (__any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned *>(&s_fail) != 0u)) { failed = true; break; }
            // softmax: half a warp per row, four keys per lane; warp w4 owns rows [16 w4, 16 w4 + 16)
            constexpr int RPW = 8;
            const int cg = lane & 15, r2 = lane >> 4;
            float4 sv[RPW];
#pragma unroll
            for (int k = 0; k < RPW; ++k) {
                const int i = 16 * w4 + 2 * k + r2;
                sv[k] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
                if (i < Lq && 4 * cg < Lk) sv[k] = __ldcg(reinterpret_cast<const float4 *>(S_cur + (size_t)i * 64) + cg);
            }
            float mx[RPW], tot[RPW];
#pragma unroll
            for (int k = 0; k < RPW; ++k) {
                sv[k].x = (4 * cg + 0 < Lk) ? sv[k].x * p.scale : -INFINITY;
                sv[k].y = (4 * cg + 1 < Lk) ? sv[k].y * p.scale : -INFINITY;
                sv[k].z = (4 * cg + 2 < Lk) ? sv[k].z * p.scale : -INFINITY;
                sv[k].w = (4 * cg + 3 < Lk) ? sv[k].w * p.scale : -INFINITY;
                mx[k] = fmaxf(fmaxf(sv[k].x, sv[k].y), fmaxf(sv[k].z, sv[k].w));
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < RPW; ++k) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
#pragma unroll
            for (int k = 0; k < RPW; ++k) {
                sv[k].x = __expf(sv[k].x - mx[k]); sv[k].y = __expf(sv[k].y - mx[k]);   // arguments are <= 0 (2 ulp)
                sv[k].z = __expf(sv[k].z - mx[k]); sv[k].w = __expf(sv[k].w - mx[k]);
                tot[k] = (sv[k].x + sv[k].y) + (sv[k].z + sv[k].w);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < RPW; ++k) tot[k] += __shfl_xor_sync(0xffffffffu, tot[k], o);
#pragma unroll
            for (int k = 0; k < RPW; ++k) {
                const int i = 16 * w4 + 2 * k + r2;
                const float inv = __frcp_rn(tot[k]);
                if (i < Lq && 4 * cg < kpad) {
                    const float x[8] = {sv[k].x * inv, sv[k].y * inv, sv[k].z * inv, sv[k].w * inv, 0.f, 0.f, 0.f, 0.f};
                    uint4 w[3];
                    sw_pieces<3>(x, w);
                    unsigned char *d = p_buf + i * 128 + (((cg >> 1) ^ (i & 7)) << 4) + (cg & 1) * 8;
#pragma unroll
                    for (int n = 0; n < 3; ++n) *reinterpret_cast<uint2 *>(d + n * SW_PL) = make_uint2(w[n].x, w[n].y);
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.p_ready);
            // this warp has read the head's scores; the last of all slices' warps to say so clears them for the next call
            unsigned old = 0;
            if (lane == 0) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(cnt_cur + 1) : "memory");
            old = __shfl_sync(0xffffffffu, old, 0);
            if (old == 4u * (unsigned)p.nsplit - 1u) {
                float4 *z = reinterpret_cast<float4 *>(S_cur);
#pragma unroll 4
                for (int i = lane; i < 1024; i += 32) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < 2) cnt_cur[lane] = 0u;
            }
            // ---- epilogue: the thread of tensor-memory lane 32 q + l holds output column l of atom 4 b + q; the four lanes of a quad
            // transpose 4 rows x 4 columns, so that a store instruction writes whole lines ----
            for (int b = 0; b < nblk; ++b) {
                const int e = b & 1, a = 4 * b + q;
                SW_WARP_WAIT_HEAD(15, bars.o_full[e], (b >> 1) & 1);
                tc_fence_after();
                const bool odd = __any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned *>(&s_odd_v[e]) == (unsigned)b + 1u);   // a non-finite value in the block
                if (a < nat) {
                    const uint32_t ta = tq + 256u * (uint32_t)e;
                    const int col0 = atom_col(a) + (lane & ~3);   // head_d is a multiple of 4: the four columns are inside or outside together
                    T *obase = reinterpret_cast<T *>(pr.O[prob]) + (long long)bh * Lq * p.D + col0;
                    for (int n0 = 0; n0 < Lq; n0 += 16) {
                        uint32_t x0[16], x1[16], x2[16];
                        tmem_ld16(ta + n0, x0);
                        tmem_ld16(ta + 64 + n0, x1);
                        tmem_ld16(ta + 128 + n0, x2);
                        tmem_ld_wait();
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(x0[j]) + (__uint_as_float(x1[j]) + __uint_as_float(x2[j]));
                        if (odd) {   // (the leading products once more: held on to, they cost every block)
                            tmem_ld16(ta + n0, x0);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (!(fabsf(__uint_as_float(x0[j])) < INFINITY)) v[j] = __uint_as_float(x0[j]);
                        }
#pragma unroll
                        for (int t4 = 0; t4 < 4; ++t4) {
                            st_quad_transpose(v[4 * t4], v[4 * t4 + 1], v[4 * t4 + 2], v[4 * t4 + 3], lane);
                            const int orow = n0 + 4 * t4 + (lane & 3);
                            if (orow < Lq && col0 < p.D) {
                                T *op = obase + (long long)orow * p.D;
                                if constexpr (W) {
                                    *reinterpret_cast<float4 *>(op) = make_float4(v[4 * t4], v[4 * t4 + 1], v[4 * t4 + 2], v[4 * t4 + 3]);
                                } else {
                                    constexpr bool H = std::is_same<T, __half>::value;
                                    *reinterpret_cast<uint2 *>(op) = make_uint2(pack_16x2(v[4 * t4], v[4 * t4 + 1], H), pack_16x2(v[4 * t4 + 2], v[4 * t4 + 3], H));
                                }
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.o_empty[e]);
            }
        } while (false);
    }
    __syncthreads();
    if (*reinterpret_cast<volatile unsigned *>(&s_fail) != 0u) for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies and MMAs in flight drain
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

#undef SW_FAIL_AT
#undef SW_WARP_WAIT
#undef SW_WARP_WAIT_HEAD
#undef SW_WARP_ALL

// The angle tables of the encodings in use, kept between calls (64 positions: 4 KB per 16 columns).  None is given up for another
// - a captured call keeps a pointer to its own - so there is an end to them: an encoding beyond it, or one first met while the
// stream is being captured (its table would be filled when the graph is launched only), has none.
struct SwTables {
    struct Entry { float2 *tab; int D, rd, sinus; float base; };
    static constexpr int kEntries = 1024;
    static constexpr size_t kBytes = (size_t)128 << 20;
    Entry e[kEntries] = {};
    int count = 0;
    size_t bytes = 0;
    const float2 *get(int D, int rd, float base, int sinus, cudaStream_t st, std::atomic<unsigned long long> *launches) {
        for (int i = count; i-- > 0;)
            if (e[i].D == D && e[i].rd == rd && e[i].base == base && e[i].sinus == sinus) return e[i].tab;
        const int npairs = 16 * ((D + ST_ATOM - 1) / ST_ATOM);
        const size_t n = (size_t)64 * npairs * sizeof(float2);
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        if (count >= kEntries || bytes + n > kBytes || cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) {
            (void)cudaGetLastError();
            return nullptr;
        }
        float2 *tab = nullptr;
        if (cudaMalloc((void **)&tab, n) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
        sw_table_kernel<<<296, 256, 0, st>>>(tab, npairs, D, rd, base, sinus);
        if (cudaGetLastError() != cudaSuccess) { cudaFree(tab); return nullptr; }
        launches->fetch_add(1);
        e[count++] = {tab, D, rd, sinus, base};
        bytes += n;
        return tab;
    }
    void release() {
        while (count > 0) cudaFree(e[--count].tab);
        bytes = 0;
    }
};

}  // namespace b200attn
