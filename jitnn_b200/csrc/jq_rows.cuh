// The rows kernel: y[m, n] = x[m, k] . W[n, k]^T (+ bias) in FP32 for up to 16 rows of x on the 5th-generation tensor cores, every weight read once.
//
// What bounds it. At 6.5 TB/s an SM gets a unit of 128 rows x 256 k of Q4_K (18 KB) in 770 clocks. The tensor core needs 270 of them: an MMA of 128
// weights' rows x 32 columns x 16 k whose weights lie in tensor memory takes 16 clocks, one of 16 columns 9. What is scarce is instructions: a unit is 64 KB of halves to
// be made by the warps, and with 1050 instructions per scheduler and unit, a fifth of the time without the next instruction at hand (long unrolled
// code of five roles), the same product as an instance of the matrix kernel (jq_matmul.cuh) took 1800 clocks a unit. So the weights are made with as few
// instructions as there are:
// * A quant in the low bits of a half IS the subnormal half q 2^-24: 1.1 logic operations a pair and one fused multiply-add that
//   multiplies by the scale and takes off the middle of the quants' range, exactly (Q4_K, Q5_K: (q - 8) scale <= 1008 is a half). Bits 4 .. 7
//   stay in place, as 16 q. The pairs are values 0 and 2, 1 and 3 of four; x's image has the same order.
// * d and dmin go to the sums: the mins, times the sums of x over 32 values, have columns of their own in tensor memory.
// * Where quant x scale does not fit a half (Q6_K 13 bits, 32-element formats 15 to 18) the operand is the quants alone, and every scale has an accumulator of
//   its own: its 16 or 32 k times hi and lo of x, which the warps that add up multiply by the scale, for 16 (8) multiply-adds a row and 8 columns. (As two halves,
//   hi = scale q rounded and lo = the rest, a weight takes two instructions a pair and twice the stores to tensor memory more. 32000 x 4096, 8 and 16 rows, so and as quants,
//   us: Q6_K 41.4, 42.0 and 32.2, 38.2; Q8_0 41.9, 42.4 and 26.0, 30.3; Q4_0 37.6, 38.4 and 23.9, 28.9; Q4_1 43.6, 44.6 and 27.9, 35.0; the error against 64 bits
//   2.0e-7 of the norm and 1.1e-7, as a sum of 16 or 32 terms is all that the tensor core cuts off.) Q6_K is still bound by its
//   instructions (1180 per scheduler and unit with 8 rows, 0.55 of the issue slots; four groups of warps that make weights in place of two: 33.2).
//
// x is split into halves hi + lo, 22 bits a value, times a power of two per row and 256 values (image_kernel in jq_rows.cu): NT + NT columns of one B
// operand, NT = 8 or 16 rows of x; a unit's part of the image is one contiguous copy, 8.5 or 17 KB. An accumulator of both hi and lo holds 256 (Q5_K: 128)
// terms before its sums are added up in registers, rounded to nearest: the tensor core cuts sums off towards zero.
//
// Roles: warp 0 brings in raw units, warp 2 the image, one bulk copy each; warp 1 issues the MMAs; warps 4 .. 3 + FOLD add up, eight columns each (a warp may only
// read its quarter of tensor memory's lanes): four with NT = 8, eight with 16; the eight behind them are two groups that turn raw units into operands in
// tensor memory, thread = row of W. Q4_K, Q5_K: an operand is a unit, the groups take units in turn. The others: an operand is half a unit's k, and each group
// makes its half of every unit. (The fold's loop over halves and the makers' loops are unrolled: as loops they were 3 to 6 % slower.)
//
// k is cut into eight ranges whatever the grid is; a range's units are added up in order, then the ranges. So a row shard gives bitwise what the whole
// weight gives, and a cluster of 2, 4 or 8 thread blocks may share the ranges (their sums meet through distributed shared memory) where there
// are too few tiles of rows to fill the chip.
//
// Every wait is bounded: one that runs out records a code (as jq_matmul.cuh's), raises the thread block's abort flag, and all roles leave their loops.
#pragma once

#include "jq_matmul.cuh"
#include "jq_rows_image.cuh"

namespace jq {
namespace rows {

using mm::add2;
using mm::elect_one;
using mm::f2;
using mm::fma2;
using mm::hadd2;
using mm::hfma2;
using mm::hmul2;
using mm::lds16;
using mm::mul2;
using mm::pack2;
using mm::unpack2;

constexpr int RANGES = 8;
constexpr int MAX_WEIGHTS = 3;
constexpr int MAX_RAW = 6, MAX_IMG = 6, MAX_OPERANDS = 4, MAX_ACC = 4, MAX_FACTORS = 8;

struct Args {
    const uint8_t* q[MAX_WEIGHTS];
    const uint8_t* aux[MAX_WEIGHTS];
    float* y[MAX_WEIGHTS];
    int64_t n[MAX_WEIGHTS];
    int ft_end[MAX_WEIGHTS];  // tiles of 128 rows up to and including each weight
    const uint8_t* image;     // [units][image_bytes]
    const float* scales;      // [units][NT]
    const float* bias;        // of the first weight, or null
    int units, m;
    int first_ft, ftiles;     // this launch's tiles: the first, and the one behind the last
    int followed;             // another launch of the same product is behind
    int ksplit;               // thread blocks that share a tile's ranges
    int raw, img;             // ring depths
    int* status;
    long long wait_clocks;
};

__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t lds4(uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}
// A scale of x or a bias, behind the wait for the kernel that writes it: not a read-only load, which might be moved in front of that wait. L2: from L2, past L1.
template <bool L2>
__device__ __forceinline__ float load_scale(const float* p) {
    float v;
    if constexpr (L2) {
        asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    } else {
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    }
    return v;
}
__device__ __forceinline__ void sts_pair(uint32_t at, float a, float b) { asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(a), "f"(b) : "memory"); }
__device__ __forceinline__ void st_tmem16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
// D (tensor memory) = or += A (tensor memory) . B (shared memory, K-major core matrices without swizzle)
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "r"((128u >> 4) | (1u << 14))  // 128 bytes between groups of 8 columns
        : "memory");
}
__device__ __forceinline__ uint32_t desc(uint32_t addr, int n) { return ((addr & 0x3FFFFu) >> 4) | ((uint32_t)(n * 16) >> 4 << 16); }  // between the two halves of a step
constexpr uint32_t idesc(int n) { return (1u << 4) | ((uint32_t)(128 >> 4) << 24) | ((uint32_t)(n >> 3) << 17); }

constexpr uint32_t dup(uint32_t half_bits) { return half_bits * 0x10001u; }

// Several barriers at once for a whole warp. A poll that finds its phase complete takes a warp among four busy ones 200 clocks and more, one after the
// other; the answers to several polls come back together. What is not complete is waited for in turn, by a wait that suspends the warp: a loop
// of polls takes issue slots from the very warps it waits for.
struct Phase {
    uint32_t bar, parity;
    int code;
};
template <typename... P>
__device__ __forceinline__ bool wait_all(volatile int* abort_flag, const Args& p, const P&... phases) {
    constexpr int COUNT = sizeof...(P);
    bool ready[COUNT];
    int i = 0;
    ((ready[i++] = tc::mbar_test(phases.bar, phases.parity)), ...);
    i = 0;
    return ((__all_sync(0xffffffffu, ready[i++]) || mm::wait_warp(phases.bar, phases.parity, abort_flag, p, phases.code)) && ...);
}

__device__ __forceinline__ void ld(float (&r)[8], uint32_t addr) { mm::ld_tmem8(r, addr); }

// ---- the formats -------------------------------------------------------------------------------------------------------------------
// HALVES: operands per unit, each of 128 columns / HALVES; GROUP: consecutive k with one scale that the fold multiplies by, 0 where the scales are in the
// operand; MINS: the sums of x have a part (what is the same for 32 weights, the middle of the quants and the min: 8 more columns of an operand, the eight
// values' hi parts and lo parts, whose products have an accumulator of their own); ACCS: accumulators per unit, without GROUP.
// make(): operand `half` of the row's unit into this lane's columns from `to` on, and what the fold multiplies the sums by into `fac`.
template <int TYPE>
struct Rw;

// Eight values of at most `bound` as columns of halves, hi then lo, times a power of two; the fold multiplies by its inverse.
__device__ __forceinline__ float sums_part(const float (&e)[8], float bound, uint32_t to) {
    const uint32_t ex = min(max(__float_as_uint(bound) >> 23, 40u), 250u);
    const float by = __uint_as_float((267u - ex) << 23);  // below 2^14
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        mm::split_pair(e[2 * i] * by, e[2 * i + 1] * by, v[i], v[4 + i]);
    }
    mm::st_tmem8(to, v);
    return __uint_as_float((ex - 13u) << 23);
}

// Q4_K and Q5_K: values scale (q - mid) 2^-14.
template <bool FIVE>
struct RwK45 {
    static constexpr int ROW = FIVE ? 176 : 144, AUX = 0, HALVES = 1, GROUP = 0, ACCS = FIVE ? 2 : 1;
    static constexpr bool MINS = true;
    __device__ static __forceinline__ void make(uint32_t uq, uint32_t, int row, int, uint32_t to, uint32_t fac) {
        const uint32_t at = uq + (uint32_t)(row * ROW);
        const uint4 h = lds16(at);
        uint4 q0 = lds16(at + (FIVE ? 48 : 16)), q1 = lds16(at + (FIVE ? 64 : 32));
        uint4 b0 = make_uint4(0, 0, 0, 0), b1 = b0;
        if constexpr (FIVE) {
            b0 = lds16(at + 16);
            b1 = lds16(at + 32);
        }
        const uint32_t sc0 = h.y & 0x3f3f3f3fu, sc1 = and_or(h.y >> 2, 0x30303030u, h.w & 0x0f0f0f0fu);
        const uint32_t mn0 = h.z & 0x3f3f3f3fu, mn1 = and_or(h.z >> 2, 0x30303030u, (h.w >> 4) & 0x0f0f0f0fu);
        {
            const float d = half_bits_to_float(h.x), dmin = half_bits_to_float(h.x >> 16), mid = d * (FIVE ? 16.0f : 8.0f);
            float e[8];  // mid d scale - dmin min; a byte in the mantissa of 2^23
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float sc = __uint_as_float(__byte_perm(i < 4 ? sc0 : sc1, 0x4B000000u, 0x7540u + (uint32_t)(i & 3))) - 8388608.0f;
                const float mn = __uint_as_float(__byte_perm(i < 4 ? mn0 : mn1, 0x4B000000u, 0x7540u + (uint32_t)(i & 3))) - 8388608.0f;
                e[i] = fmaf(-dmin, mn, mid * sc);
            }
            const float f1 = sums_part(e, fmaxf(63.0f * fabsf(mid), 63.0f * fabsf(dmin)) * 2.0f, to + 128);
            sts_pair(fac, d * 16384.0f, f1);
        }
#pragma unroll 1
        for (int j = 0; j < 4; j++) {
            const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            const uint32_t g[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            if (j < 3) {
                q0 = lds16(at + (FIVE ? 80 : 48) + 32 * (uint32_t)j);
                q1 = lds16(at + (FIVE ? 96 : 64) + 32 * (uint32_t)j);
            }
            const uint32_t sc = j < 2 ? sc0 : sc1, pick = 0x4040u + 0x0202u * (uint32_t)(j & 1);
            const uint32_t a = hadd2(__byte_perm(sc, 0x64646464u, pick), 0xE400E400u), b = hadd2(__byte_perm(sc, 0x64646464u, pick + 0x0101u), 0xE400E400u);
            // q 2^-24 x scale 2^10 and 16 q 2^-24 x scale 2^6, minus mid scale 2^-14
            const uint32_t sa = hmul2(a, dup(0x6400)), sb = hmul2(b, dup(0x5400)), ca = hmul2(a, FIVE ? dup(0x9400) : dup(0x9000)),
                           cb = hmul2(b, FIVE ? dup(0x9400) : dup(0x9000));
            uint32_t lo[16], hi[16];
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const uint32_t v = w[x], u = v >> 8;
                uint32_t l0 = v & 0x000F000Fu, l1 = u & 0x000F000Fu, h0 = v & 0x00F000F0u, h1 = u & 0x00F000F0u;
                if constexpr (FIVE) {
                    const uint32_t t = g[x] >> (2 * j);  // bits 2 j and 2 j + 1 of every byte, to bit 4 and bit 8
                    l0 = and_or(t << 4, 0x00100010u, l0);
                    l1 = and_or(t >> 4, 0x00100010u, l1);
                    h0 = and_or(t << 7, 0x01000100u, h0);
                    h1 = and_or(t >> 1, 0x01000100u, h1);
                }
                lo[2 * x] = hfma2(l0, sa, ca);
                lo[2 * x + 1] = hfma2(l1, sa, ca);
                hi[2 * x] = hfma2(h0, sb, cb);
                hi[2 * x + 1] = hfma2(h1, sb, cb);
            }
            st_tmem16(to + 32 * (uint32_t)j, lo);
            st_tmem16(to + 32 * (uint32_t)j + 16, hi);
        }
    }
};
template <>
struct Rw<JQ_TYPE_Q4_K> : RwK45<false> {};
template <>
struct Rw<JQ_TYPE_Q5_K> : RwK45<true> {};

// The other formats' products of quant and scale do not fit a half: the operand is the quants alone, and the sums over the k of one scale come out of the
// tensor core one by one. fac: the scales of the half's groups (bytes or halves in .x and .y), .z what else the fold multiplies by.
template <>
struct Rw<JQ_TYPE_Q6_K> {
    static constexpr int ROW = 208, AUX = 2, HALVES = 2, GROUP = 16, ACCS = 2;
    static constexpr bool MINS = false;
    __device__ static __forceinline__ void make(uint32_t uq, uint32_t ua, int row, int half, uint32_t to, uint32_t fac) {
        const uint32_t at = uq + (uint32_t)(row * ROW), l = at + 64u * (uint32_t)half, h = at + 128u + 32u * (uint32_t)half;
        const uint32_t s0 = lds4(at + 192u + 8u * (uint32_t)half) ^ 0x80808080u, s1 = lds4(at + 196u + 8u * (uint32_t)half) ^ 0x80808080u;
        const uint32_t dw = lds4(ua + 4u * (uint32_t)(row >> 1));
        mm::sts16(fac, s0, s1, __float_as_uint(half_bits_to_float((row & 1) != 0 ? dw >> 16 : dw)), 0u);
#pragma unroll
        for (int p = 0; p < 2; p++) {  // bytes 16 p .. 16 p + 15 of the half's runs of 32
            const uint4 qa = lds16(l + 16u * (uint32_t)p), qb = lds16(l + 32u + 16u * (uint32_t)p), qh = lds16(h + 16u * (uint32_t)p);
            const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w}, wh[4] = {qh.x, qh.y, qh.z, qh.w};
            uint32_t q[4][8];  // runs 0 .. 3: low nibbles of a and b, high nibbles of a and b
#pragma unroll
            for (int x = 0; x < 4; x++) {
#pragma unroll
                for (int odd = 0; odd < 2; odd++) {
                    const uint32_t a = wa[x] >> (8 * odd), b = wb[x] >> (8 * odd), t = wh[x] >> (8 * odd), t2 = t << 2, t4 = t << 4;
                    const int i = 2 * x + odd;  // 1024 + q, and 1024 + 16 q; minus 32
                    q[0][i] = hadd2(and_or(a, 0x000F000Fu, and_or(t4, 0x00300030u, 0x64006400u)), 0xE420E420u);
                    q[1][i] = hadd2(and_or(b, 0x000F000Fu, and_or(t2, 0x00300030u, 0x64006400u)), 0xE420E420u);
                    q[2][i] = hfma2(and_or(a, 0x00F000F0u, and_or(t4, 0x03000300u, 0x64006400u)), 0x2C002C00u, 0xD600D600u);
                    q[3][i] = hfma2(and_or(b, 0x00F000F0u, and_or(t2, 0x03000300u, 0x64006400u)), 0x2C002C00u, 0xD600D600u);
                }
            }
#pragma unroll
            for (int run = 0; run < 4; run++) {
                mm::st_tmem8(to + (uint32_t)(16 * run) + 8u * (uint32_t)p, q[run]);
            }
        }
    }
};

template <int TYPE>
struct Rw32 {
    static constexpr bool Q8 = TYPE == JQ_TYPE_Q8_0, MINS = TYPE == JQ_TYPE_Q4_1;
    static constexpr int ROW = Q8 ? 256 : 128, AUX = MINS ? 32 : 16, HALVES = 2, GROUP = 32, ACCS = 2;
    __device__ static __forceinline__ void make(uint32_t uq, uint32_t ua, int row, int half, uint32_t to, uint32_t fac) {
        const uint32_t at = uq + (uint32_t)(row * ROW), au = ua + (uint32_t)(row * AUX);
        if constexpr (MINS) {
            const uint4 d0 = lds16(au), d1 = lds16(au + 16);
            uint32_t f1 = 0;
            if (half == 1) {
                const uint32_t a[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
                float c[8], bound = 0.0f;  // 8 d + m
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    c[i] = fmaf(8.0f, half_bits_to_float(a[i]), half_bits_to_float(a[i] >> 16));
                    bound = fmaxf(bound, fabsf(c[i]));
                }
                f1 = __float_as_uint(sums_part(c, bound, to + 64));
            }
            const uint4 d = half ? d1 : d0;
            mm::sts16(fac, __byte_perm(d.x, d.y, 0x5410), __byte_perm(d.z, d.w, 0x5410), f1, 0u);
        } else {
            const uint4 d = lds16(au);
            mm::sts16(fac, half ? d.z : d.x, half ? d.w : d.y, 0u, 0u);
        }
#pragma unroll
        for (int b = 0; b < 4; b++) {  // blocks of 32 of the half
            uint32_t v[16];
            if constexpr (Q8) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const uint4 q = lds16(at + 16u * (uint32_t)swizzle_piece(8 * half + 2 * b + c, row));
                    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        const uint32_t u = w[x] ^ 0x80808080u;  // q + 128 under 0x64: 1024 + that
                        v[8 * c + 2 * x] = hadd2(__byte_perm(u, 0x64646464u, 0x4240), 0xE480E480u);
                        v[8 * c + 2 * x + 1] = hadd2(__byte_perm(u, 0x64646464u, 0x4341), 0xE480E480u);
                    }
                }
            } else {
                const uint4 q = lds16(at + 16u * (uint32_t)swizzle_piece(4 * half + b, row));
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int x = 0; x < 4; x++) {  // low nibbles, high nibbles: 1024 + q, 1024 + 16 q; minus 8
                    const uint32_t u = w[x] >> 8;
                    v[2 * x] = hadd2(and_or(w[x], 0x000F000Fu, 0x64006400u), 0xE408E408u);
                    v[2 * x + 1] = hadd2(and_or(u, 0x000F000Fu, 0x64006400u), 0xE408E408u);
                    v[8 + 2 * x] = hfma2(and_or(w[x], 0x00F000F0u, 0x64006400u), 0x2C002C00u, 0xD480D480u);
                    v[8 + 2 * x + 1] = hfma2(and_or(u, 0x00F000F0u, 0x64006400u), 0x2C002C00u, 0xD480D480u);
                }
            }
            st_tmem16(to + 16u * (uint32_t)b, v);
        }
    }
};
template <>
struct Rw<JQ_TYPE_Q8_0> : Rw32<JQ_TYPE_Q8_0> {};
template <>
struct Rw<JQ_TYPE_Q4_0> : Rw32<JQ_TYPE_Q4_0> {};
template <>
struct Rw<JQ_TYPE_Q4_1> : Rw32<JQ_TYPE_Q4_1> {};

// Tensor memory: slots of accumulators, then those of the mins' sums (16 columns each), behind them the operands. Without GROUP a slot is one
// accumulator of N columns, hi and lo; with it, the accumulators of an operand's groups, 16 columns each: an MMA with the hi columns and one with the lo
// columns of x add to the same. (An MMA of 128 rows has at least 16 columns: with NT = 8 the upper eight are whatever lies behind in the image, and not read.)
template <int TYPE, int NT>
struct Shape {
    using F = Rw<TYPE>;
    static constexpr int UNIT_Q = 128 * F::ROW, UNIT_A = 128 * F::AUX, UNIT = UNIT_Q + UNIT_A;
    static constexpr int N = 2 * NT, STEP = step_bytes(NT), IMAGE = image_bytes(NT);
    static constexpr bool GROUPED = F::GROUP > 0;
    static constexpr int A_COLS = 128 / F::HALVES + (F::MINS ? 8 : 0), OPERANDS = GROUPED ? 4 : 3;
    static constexpr int PER_HALF = GROUPED ? 128 / F::GROUP : 0;  // groups of an operand
    static constexpr int SLOT = GROUPED ? 16 * PER_HALF : N, ACC = !GROUPED || F::GROUP == 16 ? 2 : (F::MINS ? 3 : 4), MIN_ACC = F::MINS ? 2 : 0;
    static constexpr int ACC_COLS = ACC * SLOT + MIN_ACC * 16;
    static_assert(ACC_COLS + OPERANDS * A_COLS <= 512 && OPERANDS <= MAX_OPERANDS && ACC <= MAX_ACC, "tensor memory");
    static constexpr int FACTORS = GROUPED ? 4 : 8, FAC_HALF = GROUPED ? 2048 : 1024, FAC = GROUPED ? 2 * FAC_HALF : FAC_HALF;  // units whose factors are kept, bytes
    static constexpr int GROUPS = 2, FOLD = NT / 2, THREADS = (4 + FOLD + 4 * GROUPS) * 32;  // warps that make weights (groups of four), that add up
    static constexpr int C = 8;  // columns (rows of x) of a fold warp
    static constexpr int SCALES = FOLD * 16 * C * 4;  // bytes of the fold warps' scales of x
    static constexpr int TAIL = FACTORS * FAC + SCALES + 1024;  // and barriers
};
constexpr int part_bytes(int ksplit, int nt) { return ksplit > 1 ? RANGES / ksplit * nt * 512 : 0; }

// AFTER: another launch of the same product is in front. A product may be cut by tiles into several launches, which read and write nothing of each
// other's: the one behind starts as SMs become free, without waiting for the one in front, once that one knows that x's image is complete. It ends
// after it, though, so whoever waits for the last waits for all. What it reads of the image kernel's work is in L2 by then (that kernel had ended before the
// launch in front let this one start), and it reads it there: the image by bulk copies, the scales past L1. (Past L1 in every launch: Q4_K 32000 x 4096, 16
// rows 24.6 -> 25.2 us, as eight warps of every SM read the same lines.)
template <int TYPE, int NT, bool AFTER>
__global__ void __launch_bounds__((Shape<TYPE, NT>::THREADS), 1) rows_kernel(const __grid_constant__ Args p) {
    using F = Rw<TYPE>;
    using S = Shape<TYPE, NT>;
    constexpr int GROUPS = S::GROUPS, FOLD = S::FOLD, THREADS = S::THREADS, C = S::C, N = S::N, STEP = S::STEP, IMAGE = S::IMAGE;
    constexpr int OPERANDS = S::OPERANDS, FACTORS = S::FACTORS;
    constexpr bool GROUPED = S::GROUPED;
    extern __shared__ uint8_t smem_unaligned[];
    const uint32_t base = (tc::smem_u32(smem_unaligned) + 127u) & ~127u;  // sums of this thread block's ranges (ksplit > 1), then the rings
    const uint32_t img0 = base + (uint32_t)(p.ksplit > 1 ? RANGES / p.ksplit * NT * 512 : 0), raw0 = img0 + (uint32_t)(p.img * IMAGE), fac0 = raw0 + (uint32_t)(p.raw * S::UNIT);
    const uint32_t scl0 = fac0 + FACTORS * S::FAC, bars = scl0 + S::SCALES;
    const uint32_t img_full = bars, img_free = img_full + 8 * MAX_IMG, raw_full = img_free + 8 * MAX_IMG, raw_free = raw_full + 8 * MAX_RAW;
    const uint32_t full_a = raw_free + 8 * MAX_RAW, free_a = full_a + 8 * MAX_OPERANDS, acc_full = free_a + 8 * MAX_OPERANDS, acc_free = acc_full + 8 * MAX_ACC;
    const uint32_t fac_full = acc_free + 8 * MAX_ACC, slot_s = fac_full + 8 * MAX_FACTORS;
    uint8_t* const generic = smem_unaligned + (slot_s - tc::smem_u32(smem_unaligned));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(generic);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(generic + 4);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int range = p.ksplit == 1 ? 0 : (int)mm::cluster_rank();
    const int cluster_id = (int)blockIdx.x / p.ksplit, clusters = (int)gridDim.x / p.ksplit;
    const int u0 = (int)((int64_t)range * p.units / p.ksplit), u1 = (int)((int64_t)(range + 1) * p.units / p.ksplit);

    if (threadIdx.x == 0) {
        for (int i = 0; i < MAX_IMG; i++) {
            tc::mbar_init(img_full + 8 * i, 1);
            tc::mbar_init(img_free + 8 * i, 1);
        }
        for (int i = 0; i < MAX_RAW; i++) {
            tc::mbar_init(raw_full + 8 * i, 1);
            tc::mbar_init(raw_free + 8 * i, 4 * F::HALVES);
        }
        for (int i = 0; i < OPERANDS; i++) {
            tc::mbar_init(full_a + 8 * i, 4);
            tc::mbar_init(free_a + 8 * i, 1);
        }
        for (int i = 0; i < MAX_ACC; i++) {
            tc::mbar_init(acc_full + 8 * i, 1);
            tc::mbar_init(acc_free + 8 * i, FOLD);
        }
        for (int i = 0; i < MAX_FACTORS; i++) {
            tc::mbar_init(fac_full + 8 * i, 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot_s) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    if (p.ksplit > 1) {
        mm::cluster_sync();
    }
    tc::fence_after_sync();
    if (AFTER || !p.followed) {
        asm volatile("griddepcontrol.launch_dependents;");
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t tmem_m = tmem + S::ACC * S::SLOT, tmem_a = tmem + S::ACC_COLS;

    auto weight_of = [&](int ft, int& ft0) {
        const int w = ft < p.ft_end[0] ? 0 : (ft < p.ft_end[1] ? 1 : 2);
        ft0 = w == 0 ? 0 : (w == 1 ? p.ft_end[0] : p.ft_end[1]);
        return w;
    };
    bool ok = true;
    if (warp == 0) {
        // ---- raw units -------------------------------------------------------------------------------------------------------------
        if (lane == 0) {
            int r = 0;
            uint32_t ph = 1;
            for (int ft = p.first_ft + cluster_id; ft < p.ftiles && ok; ft += clusters) {
                int ft0;
                const int w = weight_of(ft, ft0);
                const int64_t first = (int64_t)(ft - ft0) * p.units;
                const uint8_t* const q = mm::pick(p.q, w) + first * S::UNIT_Q;
                const uint8_t* const a = mm::pick(p.aux, w) + first * S::UNIT_A;
                for (int u = u0; u < u1; u++) {
                    if (!(ok = mm::wait(raw_free + 8 * r, ph, abort_flag, p, 8))) {
                        break;
                    }
                    const uint32_t to = raw0 + (uint32_t)(r * S::UNIT), bar = raw_full + 8 * r;
                    tc::mbar_expect_tx(bar, S::UNIT);
                    tc::bulk_load(to, q + (int64_t)u * S::UNIT_Q, S::UNIT_Q, bar);
                    if constexpr (F::AUX > 0) {
                        tc::bulk_load(to + S::UNIT_Q, a + (int64_t)u * S::UNIT_A, S::UNIT_A, bar);
                    }
                    if (++r == p.raw) {
                        r = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 2) {
        // ---- the image ---------------------------------------------------------------------------------------------------------------
        if (lane == 0) {
            if constexpr (!AFTER) {
                asm volatile("griddepcontrol.wait;" ::: "memory");  // the kernel in front writes it
                asm volatile("griddepcontrol.launch_dependents;");
            }
            int s = 0;
            uint32_t ph = 1;
            for (int ft = p.first_ft + cluster_id; ft < p.ftiles && ok; ft += clusters) {
                for (int u = u0; u < u1; u++) {
                    if (!(ok = mm::wait<true>(img_free + 8 * s, ph, abort_flag, p, 3))) {
                        break;
                    }
                    tc::mbar_expect_tx(img_full + 8 * s, IMAGE);
                    tc::bulk_load(img0 + (uint32_t)(s * IMAGE), p.image + (int64_t)u * IMAGE, IMAGE, img_full + 8 * s);
                    if (++s == p.img) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMAs: an operand's in one go (an election between them costs as much as several). What the next operand needs is asked for before they are
        // issued: an answer takes 200 clocks, with those of all polls together, and by then it is mostly yes.
        constexpr int BUFS = F::ACCS / F::HALVES, STEPS = 16 / F::HALVES;  // slots of accumulators and steps of 16 k of an operand
        const int turns = (p.ftiles - p.first_ft - cluster_id + clusters - 1) / clusters * (u1 - u0) * F::HALVES;
        int a = 0, s = 0, buf = 0, half = 0;
        uint32_t pa = 0, ps = 0, pb = 1;
        bool ready = false;
        for (int t = 0; t < turns; t++) {
            uint32_t d[BUFS], d_bar[BUFS], dm = 0;
            Phase free[BUFS];
#pragma unroll
            for (int i = 0; i < BUFS; i++) {
                d[i] = tmem + (uint32_t)(buf * S::SLOT);
                dm = tmem_m + 16u * (uint32_t)(GROUPED ? (t >> 1) & 1 : buf);
                d_bar[i] = acc_full + 8 * buf;
                free[i] = Phase{acc_free + 8 * buf, pb, 5};
                if (++buf == S::ACC) {
                    buf = 0;
                    pb ^= 1;
                }
            }
            if (!__all_sync(0xffffffffu, ready) &&
                !(ok = wait_all(abort_flag, p, Phase{full_a + 8 * a, pa, 2}, Phase{img_full + 8 * s, ps, 3}, free[0], free[BUFS - 1]))) {
                break;
            }
            tc::fence_after_sync();
            const uint32_t img = desc(img0 + (uint32_t)(s * IMAGE), N), ta = tmem_a + (uint32_t)(a * S::A_COLS), bd = img + (uint32_t)(half * STEPS * (STEP >> 4));
            const uint32_t a_bar = free_a + 8 * a, s_bar = img_free + 8 * s;
            const bool last = F::HALVES == 1 || half == 1;
            if (++a == OPERANDS) {
                a = 0;
                pa ^= 1;
            }
            if (last && ++s == p.img) {
                s = 0;
                ps ^= 1;
            }
            half = last ? 0 : 1;
            ready = tc::mbar_test(full_a + 8 * a, pa);
            ready = tc::mbar_test(img_full + 8 * s, ps) && ready;
            ready = tc::mbar_test(acc_free + 8 * buf, pb) && ready;
            if constexpr (BUFS == 2) {  // (all of them)
                ready = tc::mbar_test(acc_free + 8 * (buf + 1), pb) && ready;
            }
            if (elect_one()) {
                auto sums_of_x = [&]() {  // times the lo columns, then the hi columns
                    mma(dm, ta + 128 / F::HALVES, img + 16 * (STEP >> 4) + NT, idesc(16), 0u);
                    mma(dm, ta + 128 / F::HALVES, img + 16 * (STEP >> 4), idesc(16), 1u);
                };
                if constexpr (GROUPED) {
                    constexpr int KS = F::GROUP / 16;  // steps of a group
#pragma unroll
                    for (int g = 0; g < S::PER_HALF; g++) {
#pragma unroll
                        for (int i = 0; i < 2 * KS; i++) {  // lo first, while the accumulator is small
                            const int step = g * KS + i % KS;
                            mma(d[0] + 16 * g, ta + 8 * step, bd + step * (STEP >> 4) + (i < KS ? NT : 0), idesc(16), i == 0 ? 0u : 1u);
                        }
                    }
                    if (F::MINS && last) {
                        sums_of_x();
                    }
                    tc::umma_commit(d_bar[0]);
                } else {
#pragma unroll
                    for (int i = 0; i < STEPS; i++) {
                        const int b = i / (STEPS / BUFS);
                        mma(d[b], ta + 8 * i, bd + i * (STEP >> 4), idesc(N), i % (STEPS / BUFS) == 0 ? 0u : 1u);  // (hi | lo)
                        if (F::MINS && i == STEPS - 1) {
                            sums_of_x();
                        }
                        if ((i + 1) % (STEPS / BUFS) == 0) {
                            tc::umma_commit(d_bar[b]);
                        }
                    }
                }
                tc::umma_commit(a_bar);
                if (last) {
                    tc::umma_commit(s_bar);
                }
            }
            __syncwarp();
        }
    } else if (warp >= 4 + FOLD) {
        // ---- weights -------------------------------------------------------------------------------------------------------------------
        const int group = (warp - 4 - FOLD) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t to0 = tmem_a + ((uint32_t)((warp & 3) * 32) << 16);
        const int units = (p.ftiles - p.first_ft - cluster_id + clusters - 1) / clusters * (u1 - u0);
        // A group makes one operand (half) of every TAKE-th unit. Without halves the places in the ring of raw units go in turn too (its depth is even), so no
        // group tests a barrier that is a turn of the ring behind.
        constexpr int TAKE = GROUPS / F::HALVES;
        const int half = group % F::HALVES;
        int r = group / F::HALVES, o = group;
        uint32_t pr = 0, po = 1;
        for (int unit = r; unit < units; unit += TAKE) {
            if (!(ok = wait_all(abort_flag, p, Phase{raw_full + 8 * r, pr, 6}, Phase{free_a + 8 * o, po, 1}))) {
                break;
            }
            tc::fence_after_sync();
            const int slot = unit & (FACTORS - 1);
            const uint32_t uq = raw0 + (uint32_t)(r * S::UNIT), fac = fac0 + (uint32_t)(slot * S::FAC + half * S::FAC_HALF + row * (GROUPED ? 16 : 8));
            F::make(uq, uq + S::UNIT_Q, row, half, to0 + (uint32_t)(o * S::A_COLS), fac);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                tc::mbar_arrive(full_a + 8 * o);
                tc::mbar_arrive(fac_full + 8 * (slot * F::HALVES + half));
                tc::mbar_arrive(raw_free + 8 * r);  // (all that was read of the unit has been used)
            }
            if ((r += TAKE) >= p.raw) {
                r -= p.raw;
                pr ^= 1;
            }
            if ((o += GROUPS) >= OPERANDS) {
                o -= OPERANDS;
                po ^= 1;
            }
        }
    } else if (warp >= 4) {
        // ---- sums ----------------------------------------------------------------------------------------------------------------------
        if constexpr (!AFTER) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // x's scales; and y may be read by the kernel in front
        }
        const int lane_row = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int c0 = (warp - 4) / 4 * C;  // this warp's columns
        const uint32_t scl = scl0 + (uint32_t)(warp - 4) * (16 * C * 4);
        int chunk = 0, buf = 0;
        uint32_t pb = 0;
        // The scales of x of 16 units at a time: a load takes up to 2000 clocks while the weights stream, so it is asked for a whole block ahead.
        constexpr int NEXT = 16 * C / 32;
        float next[NEXT];
        auto fetch = [&](int u) {
#pragma unroll
            for (int i = 0; i < NEXT; i++) {
                const int at = lane + 32 * i, on = at / C;
                next[i] = u + on < u1 ? load_scale<AFTER>(p.scales + (int64_t)(u + on) * NT + c0 + at % C) : 0.0f;
            }
        };
        const bool keep = u1 - u0 <= 16;  // (a short contraction's stay for the next tile)
        fetch(u0);
        for (int ft = p.first_ft + cluster_id; ft < p.ftiles && ok; ft += clusters) {
            int ft0;
            const int w = weight_of(ft, ft0);
            const int64_t row = (int64_t)(ft - ft0) * 128 + lane_row, n = mm::pick(p.n, w);
            const float bias = w == 0 && p.bias != nullptr && row < n ? load_scale<AFTER>(p.bias + row) : 0.0f;  // (on its way while the tile is multiplied)
            f2 sum[C / 2], total[C / 2];
#pragma unroll
            for (int i = 0; i < C / 2; i++) {
                sum[i] = total[i] = 0;
            }
            int v = 0;  // the range that the unit belongs to
            while (v < RANGES - 1 && (int)((int64_t)(v + 1) * p.units / RANGES) <= u0) {
                v++;
            }
            int v_end = (int)((int64_t)(v + 1) * p.units / RANGES);
            for (int u = u0; u < u1; u++, chunk++) {
                if (((u - u0) & 15) == 0 && (!keep || ft == p.first_ft + cluster_id)) {
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < NEXT; i++) {
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(scl + (uint32_t)(lane + 32 * i) * 4u), "f"(next[i]) : "memory");
                    }
                    __syncwarp();
                    if (!keep) {
                        fetch(u + 16 < u1 ? u + 16 : u0);
                    }
                }
                const uint32_t xs = scl + (uint32_t)((u - u0) & 15) * (C * 4);
                uint4 x4[C / 4];
#pragma unroll
                for (int j = 0; j < C / 4; j++) {
                    x4[j] = lds16(xs + 16u * (uint32_t)j);
                }
                const int slot = chunk & (FACTORS - 1);
                const uint32_t fac_phase = (uint32_t)(chunk / FACTORS) & 1u;
                f2 t[C / 2];  // the unit's sums
                auto took = [&]() {  // a slot's sums are in registers
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        tc::mbar_arrive(acc_free + 8 * buf);
                    }
                    if (++buf == S::ACC) {
                        buf = 0;
                        pb ^= 1;
                    }
                };
                if constexpr (GROUPED) {
                    uint4 fc;
#pragma unroll
                    for (int i = 0; i < C / 2; i++) {
                        t[i] = 0;
                    }
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        if (!(ok = wait_all(abort_flag, p, Phase{fac_full + 8 * (slot * 2 + half), fac_phase, 6}, Phase{acc_full + 8 * buf, pb, 4}))) {
                            break;
                        }
                        tc::fence_after_sync();
                        fc = lds16(fac0 + (uint32_t)(slot * S::FAC + half * S::FAC_HALF + lane_row * 16));
                        float mn[C];
#pragma unroll
                        for (int part = 0; part < S::PER_HALF / 4; part++) {
                            float v[4][C];
#pragma unroll
                            for (int g = 0; g < 4; g++) {
                                ld(v[g], tmem + lanes + (uint32_t)(buf * S::SLOT + 16 * (4 * part + g) + c0));
                            }
                            if (F::MINS && half == 1) {
                                ld(mn, tmem_m + lanes + (uint32_t)((chunk & 1) * 16 + c0));
                            }
                            mm::ld_tmem_done();
                            if (part == S::PER_HALF / 4 - 1) {
                                took();
                            }
                            const uint32_t w = part == 0 ? fc.x : fc.y;
#pragma unroll
                            for (int g = 0; g < 4; g++) {
                                float sc;
                                if constexpr (F::GROUP == 16) {  // a byte + 128 in the mantissa of 2^23
                                    sc = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + (uint32_t)g)) - 8388736.0f;
                                } else {
                                    const uint32_t bits = g < 2 ? fc.x : fc.y;
                                    sc = half_bits_to_float(g % 2 != 0 ? bits >> 16 : bits);
                                }
                                const f2 s2 = pack2(sc, sc);
#pragma unroll
                                for (int i = 0; i < C / 2; i++) {
                                    const f2 e = pack2(v[g][2 * i], v[g][2 * i + 1]);
                                    t[i] = fma2(e, s2, t[i]);
                                }
                            }
                        }
                        if (F::MINS && half == 1) {
                            const f2 f = pack2(__uint_as_float(fc.z), __uint_as_float(fc.z));
#pragma unroll
                            for (int i = 0; i < C / 2; i++) {
                                t[i] = fma2(pack2(mn[2 * i], mn[2 * i + 1]), f, t[i]);
                            }
                        }
                    }
                    if constexpr (F::GROUP == 16) {
                        const f2 f = pack2(__uint_as_float(fc.z), __uint_as_float(fc.z));
#pragma unroll
                        for (int i = 0; i < C / 2; i++) {
                            t[i] = mul2(t[i], f);
                        }
                    }
                } else {
                    if (!(ok = wait_all(abort_flag, p, Phase{fac_full + 8 * slot, fac_phase, 6}, Phase{acc_full + 8 * buf, pb, 4}))) {
                        break;
                    }
                    float f0, f1;
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(f0), "=f"(f1) : "r"(fac0 + (uint32_t)(slot * S::FAC + lane_row * 8)));
                    const f2 ff0 = pack2(f0, f0), ff1 = pack2(f1, f1);
#pragma unroll
                    for (int acc = 0; acc < F::ACCS; acc++) {
                        if (acc > 0 && !(ok = mm::wait_warp<true>(acc_full + 8 * buf, pb, abort_flag, p, 4))) {
                            break;
                        }
                        tc::fence_after_sync();
                        float hi[C], lo[C], mn[C];
                        ld(hi, tmem + lanes + (uint32_t)(buf * N + c0));
                        ld(lo, tmem + lanes + (uint32_t)(buf * N + NT + c0));
                        const bool mins = acc == F::ACCS - 1;
                        if (mins) {
                            ld(mn, tmem_m + lanes + (uint32_t)(buf * 16 + c0));
                        }
                        mm::ld_tmem_done();
                        took();
#pragma unroll
                        for (int i = 0; i < C / 2; i++) {
                            const f2 e = add2(pack2(hi[2 * i], hi[2 * i + 1]), pack2(lo[2 * i], lo[2 * i + 1]));
                            t[i] = acc == 0 ? mul2(e, ff0) : fma2(e, ff0, t[i]);
                            if (mins) {
                                t[i] = fma2(pack2(mn[2 * i], mn[2 * i + 1]), ff1, t[i]);
                            }
                        }
                    }
                }
                if (!ok) {
                    break;
                }
#pragma unroll
                for (int j = 0; j < C / 4; j++) {
                    sum[2 * j] = fma2(t[2 * j], pack2(__uint_as_float(x4[j].x), __uint_as_float(x4[j].y)), sum[2 * j]);
                    sum[2 * j + 1] = fma2(t[2 * j + 1], pack2(__uint_as_float(x4[j].z), __uint_as_float(x4[j].w)), sum[2 * j + 1]);
                }
                if (u + 1 == v_end) {  // the end of a range
                    const int slot = v - range * (RANGES / p.ksplit);
#pragma unroll
                    for (int i = 0; i < C / 2; i++) {
                        if (p.ksplit > 1) {
                            float a, b;
                            unpack2(sum[i], a, b);
                            const uint32_t at = base + (uint32_t)(((slot * NT + c0 + 2 * i) * 128 + lane_row) * 4);
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(a) : "memory");
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 512u), "f"(b) : "memory");
                        } else {
                            total[i] = add2(total[i], sum[i]);
                        }
                        sum[i] = 0;
                    }
                    do {
                        v++;
                        v_end = (int)((int64_t)(v + 1) * p.units / RANGES);
                    } while (v < RANGES - 1 && v_end <= u + 1);
                }
            }
            if (!ok || p.ksplit > 1) {
                break;  // (one tile per cluster)
            }
            if (row < n) {
                float* at = mm::pick(p.y, w) + (int64_t)c0 * n + row;
#pragma unroll
                for (int i = 0; i < C; i++, at += n) {
                    float v[2];
                    unpack2(total[i / 2], v[0], v[1]);
                    if (c0 + i < p.m) {
                        *at = v[i % 2] + bias;
                    }
                }
            }
        }
    }

    // ---- exit -----------------------------------------------------------------------------------------------------------------------
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        for (int i = 0; i < 1000; i++) {
            __nanosleep(1000);  // copies that may still be in flight land long before this millisecond is over
        }
    }
    __syncthreads();
    if (p.ksplit > 1) {
        mm::cluster_sync();  // the sums of all ranges are there
        if (*abort_flag == 0) {
            int ft0;
            const int ft = p.first_ft + cluster_id, w = weight_of(ft, ft0);
            const int64_t f0 = (int64_t)(ft - ft0) * 128, n = mm::pick(p.n, w);
            float* const y = mm::pick(p.y, w);
            const int per = RANGES / p.ksplit;
            static_assert(THREADS % 128 == 0, "a thread's columns are of the same row");
            const int row = threadIdx.x & 127;
            const float bias = w == 0 && p.bias != nullptr && f0 + row < n ? load_scale<AFTER>(p.bias + f0 + row) : 0.0f;
            // columns range, range + ksplit, ... of the tile; a thread adds up one row's eight ranges
            for (int i = threadIdx.x; i < NT / p.ksplit * 128; i += THREADS) {
                const int col = range + (i >> 7) * p.ksplit;
                float e[RANGES];
#pragma unroll
                for (int g = 0; g < RANGES; g++) {
                    const bool there = (int64_t)g * p.units / RANGES < (int64_t)(g + 1) * p.units / RANGES;  // (a range without units has no sums)
                    const uint32_t from = mm::map_rank(base + (uint32_t)(((g % per * NT + col) * 128 + row) * 4), (uint32_t)(g / per));
                    e[g] = 0.0f;
                    if (there) {
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(e[g]) : "r"(from));
                    }
                }
                float t = 0.0f;
#pragma unroll
                for (int g = 0; g < RANGES; g++) {
                    t += e[g];
                }
                if (f0 + row < n && col < p.m) {
                    y[(int64_t)col * n + f0 + row] = t + bias;
                }
            }
        }
        __syncthreads();
        mm::cluster_sync();  // no thread block ends while others read its sums
    }
    if (AFTER && threadIdx.x == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    if (warp == 1) {
        tc::fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

}  // namespace rows
}  // namespace jq
