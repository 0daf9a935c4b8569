// How a dequantiser thread of the matrix kernel (jq_matmul.cuh) turns raw blocks in shared memory into weights.
//
// A unit is 128 rows x 256 k of a tiled weight as it lies in device memory. Dq<TYPE>::head reads what a row's 256 values share, load()
// the quants of 64 consecutive k (chunk c of the row), values() turns half of them (`part`) into two runs of 16 values; run r starts at
// 16-byte piece piece(part, r) of the chunk when values take two bytes.
//
// The quant goes under the exponent of a power of two with one byte permute (no integer-to-float conversion, which runs at a
// quarter of the rate), and one packed FMA applies scale and offset to two weights: a (P + q) + (c - P a) with P = 16, 32, 64 or
// 32768. For Q8_0, Q4_0 and Q6_K every operand and result is exact, so the value is the reference's; for Q4_K, Q5_K and Q4_1 the
// constant is rounded once, at most 2^-24 of the largest weight that the block can hold, which is what FP32 keeps anyway.
// f0 and f1 are powers of two that the values of the chunk's first and second 32 are multiplied by (exactly). bounds(): the sizes that no
// weight of blocks 4 h .. 4 h + 3 of 32 values exceeds (the backward product's powers of two).
#pragma once

#include "jq_formats.cuh"

namespace jq {
namespace mm {

// two floats in a 64-bit register pair and the packed operations on them
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint4 lds16(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// Byte i of `bytes` as the third byte of a float whose top byte is that of `top`.
__device__ __forceinline__ float under3(uint32_t bytes, uint32_t top, int i) { return __uint_as_float(__byte_perm(bytes, top, 0x7044u | ((uint32_t)i << 8))); }
// ... and as the second byte.
__device__ __forceinline__ float under2(uint32_t bytes, uint32_t top, int i) { return __uint_as_float(__byte_perm(bytes, top, 0x7404u | ((uint32_t)i << 4))); }

// The largest of eight halves' magnitudes (as bits).
__device__ __forceinline__ uint32_t max_half8(const uint4& v) {
    uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
    return max(m & 0xffffu, m >> 16);
}

// Words of the scales and mins of sub-blocks 4 (c >> 1) .. + 3 (GgufKernels.java:74-83), one byte each.
__device__ __forceinline__ void scale_min_words(const uint4& h, int c, uint32_t& sc, uint32_t& mn) {
    const uint32_t high_sc = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u), high_mn = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u);
    sc = c < 2 ? h.y & 0x3f3f3f3fu : high_sc;
    mn = c < 2 ? h.z & 0x3f3f3f3fu : high_mn;
}

template <int TYPE>
struct Dq;

// ---- Q4_K, Q5_K ---------------------------------------------------------------------------------------------------------------
template <int TYPE>
struct DqK45 {
    static constexpr bool Q5 = TYPE == JQ_TYPE_Q5_K;
    static constexpr int ROW = Q5 ? 176 : 144, UNIT_Q = TILE_ROWS * ROW, UNIT_A = 0;
    struct Head {
        uint4 h;      // d, dmin, scales
        uint4 hi[2];  // Q5_K: fifth bits
    };
    struct Raw {
        uint4 q[2];
    };
    __device__ static __forceinline__ int piece(int part, int run) { return 4 * run + 2 * part; }
    __device__ static __forceinline__ Head head(uint32_t uq, uint32_t, int row) {
        Head r;
        r.h = lds16(uq + (uint32_t)row * ROW);
        if constexpr (Q5) {
            r.hi[0] = lds16(uq + (uint32_t)row * ROW + 16);
            r.hi[1] = lds16(uq + (uint32_t)row * ROW + 32);
        }
        return r;
    }
    __device__ static __forceinline__ Raw load(uint32_t uq, int row, int c) {
        const uint32_t at = uq + (uint32_t)row * ROW + (Q5 ? 48 : 16) + 32 * c;
        return Raw{{lds16(at), lds16(at + 16)}};
    }
    __device__ static __forceinline__ void bounds(const Head& r, int h, float (&b)[4]) {
        const float d = fabsf(half_bits_to_float(r.h.x)) * (Q5 ? 31.0f : 15.0f), dmin = fabsf(half_bits_to_float(r.h.x >> 16));
        uint32_t sc, mn;  // sub-blocks 4 h .. 4 h + 3
        scale_min_words(r.h, 2 * h, sc, mn);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            b[i] = fmaf(d, (float)byte_of(sc, i), dmin * (float)byte_of(mn, i));
        }
    }
    __device__ static __forceinline__ void values(const Head& r, const Raw& raw, int c, int part, float f0, float f1, f2 (&w0)[8], f2 (&w1)[8]) {
        const uint4 q = raw.q[part];
        const float d = half_bits_to_float(r.h.x), dmin = half_bits_to_float(r.h.x >> 16);
        uint32_t sc, mn;  // sub-blocks 2c and 2c + 1
        scale_min_words(r.h, c, sc, mn);
        sc >>= 16 * (c & 1);
        mn >>= 16 * (c & 1);
        // exact: 11 + 6 bits
        const float a0 = d * f0 * (under2(sc, 0x47000000u, 0) - 32768.0f), a1 = d * f1 * (under2(sc, 0x47000000u, 1) - 32768.0f);
        const float m0 = under2(mn, 0x47000000u, 0) - 32768.0f, m1 = under2(mn, 0x47000000u, 1) - 32768.0f;
        constexpr float P = Q5 ? 32.0f : 16.0f;
        const float k0 = -fmaf(P, a0, dmin * f0 * m0), k1 = -fmaf(P, a1, dmin * f1 * m1);
        const f2 A0 = pack2(a0, a0), A1 = pack2(a1, a1), K0 = pack2(k0, k0), K1 = pack2(k1, k1);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        const uint32_t g[4] = {r.hi[part].x, r.hi[part].y, r.hi[part].z, r.hi[part].w};
#pragma unroll
        for (int x = 0; x < 4; x++) {
            uint32_t lo, hi, top;
            if constexpr (Q5) {
                const uint32_t s = g[x] >> (2 * c);
                lo = ((w[x] << 2) & 0x3c3c3c3cu) | ((s << 6) & 0x40404040u);
                hi = ((w[x] >> 2) & 0x3c3c3c3cu) | ((s << 5) & 0x40404040u);
                top = 0x42000000u;  // 32 + q: q in mantissa bits 18..22
            } else {
                lo = ((w[x] << 3) & 0x78787878u) | 0x80808080u;
                hi = ((w[x] >> 1) & 0x78787878u) | 0x80808080u;
                top = 0x41000000u;  // 16 + q: q in mantissa bits 19..22
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                w0[2 * x + i] = fma2(A0, pack2(under3(lo, top, 2 * i), under3(lo, top, 2 * i + 1)), K0);
                w1[2 * x + i] = fma2(A1, pack2(under3(hi, top, 2 * i), under3(hi, top, 2 * i + 1)), K1);
            }
        }
    }
};
template <>
struct Dq<JQ_TYPE_Q4_K> : DqK45<JQ_TYPE_Q4_K> {};
template <>
struct Dq<JQ_TYPE_Q5_K> : DqK45<JQ_TYPE_Q5_K> {};

// ---- Q6_K ---------------------------------------------------------------------------------------------------------------------
template <>
struct Dq<JQ_TYPE_Q6_K> {
    static constexpr int ROW = 208, UNIT_Q = TILE_ROWS * ROW, UNIT_A = TILE_ROWS * 2;
    struct Head {
        uint4 sv;
        float d;
    };
    struct Raw {
        uint4 la[2], lb[2], hq[2];
    };
    __device__ static __forceinline__ int piece(int part, int run) { return 4 * run + 2 * part; }
    __device__ static __forceinline__ Head head(uint32_t uq, uint32_t ua, int row) {
        Head r;
        r.sv = lds16(uq + (uint32_t)row * ROW + 192);
        unsigned short d;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(d) : "r"(ua + 2u * (uint32_t)row));
        r.d = __half2float(__ushort_as_half(d));
        return r;
    }
    __device__ static __forceinline__ Raw load(uint32_t uq, int row, int c) {
        const uint32_t l = uq + (uint32_t)row * ROW + 64 * (c >> 1), h = uq + (uint32_t)row * ROW + 128 + 32 * (c >> 1);
        return Raw{{lds16(l), lds16(l + 16)}, {lds16(l + 32), lds16(l + 48)}, {lds16(h), lds16(h + 16)}};
    }
    __device__ static __forceinline__ void bounds(const Head& r, int h, float (&b)[4]) {
        const float d = 32.0f * fabsf(r.d);
#pragma unroll
        for (int i = 0; i < 4; i++) {  // the scales of 32 values are two bytes
            const uint32_t s = (h == 0 ? (i < 2 ? r.sv.x : r.sv.y) : (i < 2 ? r.sv.z : r.sv.w)) >> (16 * (i & 1));
            b[i] = d * (float)max(abs((int)(int8_t)(s & 0xff)), abs((int)(int8_t)((s >> 8) & 0xff)));
        }
    }
    __device__ static __forceinline__ void values(const Head& r, const Raw& raw, int c, int part, float f0, float f1, f2 (&w0)[8], f2 (&w1)[8]) {
        // 64 values: pair p of half n of the super-block (jq_formats.cuh)
        const int n = c >> 1, p = c & 1;
        const uint4 la = raw.la[part], lb = raw.lb[part], hq = raw.hq[part];
        const uint32_t sw = n == 0 ? (p == 0 ? r.sv.x : r.sv.y) : (p == 0 ? r.sv.z : r.sv.w);
        const float a0 = r.d * f0 * (float)(int)(int8_t)byte_of(sw, part), a1 = r.d * f1 * (float)(int)(int8_t)byte_of(sw, part + 2);
        const f2 A0 = pack2(a0, a0), A1 = pack2(a1, a1), K0 = pack2(-96.0f * a0, -96.0f * a0), K1 = pack2(-96.0f * a1, -96.0f * a1);
        const uint32_t wa[4] = {la.x, la.y, la.z, la.w}, wb[4] = {lb.x, lb.y, lb.z, lb.w}, wh[4] = {hq.x, hq.y, hq.z, hq.w};
#pragma unroll
        for (int x = 0; x < 4; x++) {
            // 64 + q under 0x42: bit 7 set, q in bits 1..6
            const uint32_t a = wa[x] >> (4 * p), b = wb[x] >> (4 * p), h = wh[x] >> (4 * p);
            const uint32_t qa = ((a << 1) & 0x1e1e1e1eu) | ((h << 5) & 0x60606060u) | 0x80808080u;
            const uint32_t qb = ((b << 1) & 0x1e1e1e1eu) | ((h << 3) & 0x60606060u) | 0x80808080u;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                w0[2 * x + i] = fma2(A0, pack2(under3(qa, 0x42000000u, 2 * i), under3(qa, 0x42000000u, 2 * i + 1)), K0);
                w1[2 * x + i] = fma2(A1, pack2(under3(qb, 0x42000000u, 2 * i), under3(qb, 0x42000000u, 2 * i + 1)), K1);
            }
        }
    }
};

// ---- Q8_0, Q4_0, Q4_1: half `part` of a chunk is one of its two 32-element blocks ------------------------------------------------
template <>
struct Dq<JQ_TYPE_Q8_0> {
    static constexpr int ROW = 256, UNIT_Q = TILE_ROWS * ROW, UNIT_A = TILE_ROWS * 16;
    struct Head {
        uint4 d;
    };
    struct Raw {
        uint4 q[4];
    };
    __device__ static __forceinline__ int piece(int part, int run) { return 4 * part + 2 * run; }
    __device__ static __forceinline__ Head head(uint32_t, uint32_t ua, int row) { return Head{lds16(ua + 16u * (uint32_t)row)}; }
    __device__ static __forceinline__ Raw load(uint32_t uq, int row, int c) {
        const uint32_t base = uq + (uint32_t)row * ROW;
        return Raw{{lds16(base + 16 * swizzle_piece(4 * c, row)), lds16(base + 16 * swizzle_piece(4 * c + 1, row)), lds16(base + 16 * swizzle_piece(4 * c + 2, row)),
                    lds16(base + 16 * swizzle_piece(4 * c + 3, row))}};
    }
    __device__ static __forceinline__ void bounds(const Head& r, int h, float (&b)[4]) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            b[i] = 128.0f * fabsf(half_bits_to_float((h == 0 ? (i < 2 ? r.d.x : r.d.y) : (i < 2 ? r.d.z : r.d.w)) >> (16 * (i & 1))));
        }
    }
    __device__ static __forceinline__ void values(const Head& r, const Raw& raw, int c, int part, float f0, float f1, f2 (&w0)[8], f2 (&w1)[8]) {
        const uint4 qa = raw.q[2 * part], qb = raw.q[2 * part + 1];
        const uint32_t dw = c == 0 ? r.d.x : (c == 1 ? r.d.y : (c == 2 ? r.d.z : r.d.w));
        const float d = half_bits_to_float(dw >> (16 * part)) * (part == 0 ? f0 : f1);
        const f2 D = pack2(d, d), K = pack2(-32896.0f * d, -32896.0f * d);  // 32768 + 128
        const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
        for (int x = 0; x < 8; x++) {
            const uint32_t u = w[x] ^ 0x80808080u;  // q + 128
            const f2 v0 = fma2(D, pack2(under2(u, 0x47000000u, 0), under2(u, 0x47000000u, 1)), K);
            const f2 v1 = fma2(D, pack2(under2(u, 0x47000000u, 2), under2(u, 0x47000000u, 3)), K);
            if (x < 4) {
                w0[2 * x] = v0; w0[2 * x + 1] = v1;
            } else {
                w1[2 * (x - 4)] = v0; w1[2 * (x - 4) + 1] = v1;
            }
        }
    }
};

template <int TYPE>
struct DqN {
    static constexpr bool HAS_MIN = TYPE == JQ_TYPE_Q4_1;
    static constexpr int ROW = 128, UNIT_Q = TILE_ROWS * ROW, UNIT_A = TILE_ROWS * (HAS_MIN ? 32 : 16);
    struct Head {
        uint4 d;   // Q4_0: eight d; Q4_1: d, m of blocks 0..3
        uint4 d2;  // Q4_1: d, m of blocks 4..7
    };
    struct Raw {
        uint4 q[2];
    };
    __device__ static __forceinline__ int piece(int part, int run) { return 4 * part + 2 * run; }
    __device__ static __forceinline__ Head head(uint32_t, uint32_t ua, int row) {
        Head r;
        r.d = lds16(ua + (HAS_MIN ? 32u : 16u) * (uint32_t)row);
        if constexpr (HAS_MIN) {
            r.d2 = lds16(ua + 32u * (uint32_t)row + 16);
        }
        return r;
    }
    __device__ static __forceinline__ Raw load(uint32_t uq, int row, int c) {
        const uint32_t base = uq + (uint32_t)row * ROW;
        return Raw{{lds16(base + 16 * swizzle_piece(2 * c, row)), lds16(base + 16 * swizzle_piece(2 * c + 1, row))}};
    }
    __device__ static __forceinline__ void bounds(const Head& r, int h, float (&b)[4]) {
        if constexpr (HAS_MIN) {
            const uint4 four = h == 0 ? r.d : r.d2;
            const uint32_t dm[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                b[i] = fmaf(15.0f, fabsf(half_bits_to_float(dm[i])), fabsf(half_bits_to_float(dm[i] >> 16)));
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                b[i] = 8.0f * fabsf(half_bits_to_float((h == 0 ? (i < 2 ? r.d.x : r.d.y) : (i < 2 ? r.d.z : r.d.w)) >> (16 * (i & 1))));
            }
        }
    }
    __device__ static __forceinline__ void values(const Head& r, const Raw& raw, int c, int part, float f0, float f1, f2 (&w0)[8], f2 (&w1)[8]) {
        const uint4 q = raw.q[part];
        const float fac = part == 0 ? f0 : f1;
        float d, k;
        if constexpr (HAS_MIN) {
            const uint4 four = c < 2 ? r.d : r.d2;
            const uint32_t dm = (c & 1) == 0 ? (part == 0 ? four.x : four.y) : (part == 0 ? four.z : four.w);
            d = half_bits_to_float(dm) * fac;
            k = fmaf(-16.0f, d, half_bits_to_float(dm >> 16) * fac);
        } else {
            const uint32_t dw = c == 0 ? r.d.x : (c == 1 ? r.d.y : (c == 2 ? r.d.z : r.d.w));
            d = half_bits_to_float(dw >> (16 * part)) * fac;
            k = -24.0f * d;
        }
        const f2 D = pack2(d, d), K = pack2(k, k);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const uint32_t lo = ((w[x] << 3) & 0x78787878u) | 0x80808080u, hi = ((w[x] >> 1) & 0x78787878u) | 0x80808080u;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                w0[2 * x + i] = fma2(D, pack2(under3(lo, 0x41000000u, 2 * i), under3(lo, 0x41000000u, 2 * i + 1)), K);
                w1[2 * x + i] = fma2(D, pack2(under3(hi, 0x41000000u, 2 * i), under3(hi, 0x41000000u, 2 * i + 1)), K);
            }
        }
    }
};
template <>
struct Dq<JQ_TYPE_Q4_0> : DqN<JQ_TYPE_Q4_0> {};
template <>
struct Dq<JQ_TYPE_Q4_1> : DqN<JQ_TYPE_Q4_1> {};

// ---- the forward FP32 product's weights: half arithmetic ------------------------------------------------------------------------------
// A row's 256 weights of a unit are a factor (applied in FP32 when the unit's sums are folded) times values that halves hold exactly, in one
// part or two:
//   Q4_K, Q5_K  d x (scale (q - mid) + scale mid - r min), r = dmin / d, mid = 8 or 16: scale (q - mid) <= 1008 is a half (see factor for a dmin far
//               above d). The rest is the same for 32 values, so it is not added to each value but multiplied with the sum of x over the 32 (EXT:
//               16 more columns of the contraction per unit, scale_j mid - r min_j as hi and lo halves, against the sums that split_kernel
//               wrote there). With q - mid in the place of q the accumulators hold smaller sums, of which less is cut off.
//   Q6_K        d x scale (q - 32): 13 bits, hi = the product rounded to a half, lo = fma(scale, q - 32, -hi), which is exact
//   Q8_0, Q4_0  2^e x d' q with d' = 2^-e d exact: hi and lo in the same way; Q4_1 likewise with q - 8, its m' + 8 d' through the 16 more columns
// The quants become halves with one byte permute per pair (1024 + q under the exponent 0x64). About 1.3 (K-quants) to 2.3 instructions per
// weight; going through FP32 and splitting the result takes 5 and was issue bound at twice the time.

__device__ __forceinline__ uint32_t h2_dup(float v) {
    const __half2 h = __float2half2_rn(v);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Bytes 2i and 2i + 1 as halves 1024 + byte.
__device__ __forceinline__ uint32_t bytes_to_halves(uint32_t w, int i) { return __byte_perm(w, 0x64646464u, i == 0 ? 0x4140u : 0x4342u); }
// hi and lo of two products s q.
__device__ __forceinline__ void product_hi_lo(uint32_t q, uint32_t s, uint32_t& hi, uint32_t& lo) {
    hi = hmul2(q, s);
    lo = hfma2(q, s, hi ^ 0x80008000u);
}
// A pair (a, b) of floats as halves hi, and what is left as halves lo.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const float2 back = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - back.x, b - back.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// TILES: parts per weight; EXT: the 16 more columns. factor(): the row's factor. values(): run `run` (0, 1) of half `part` of chunk c.
template <int TYPE>
struct Half;

template <int TYPE>
struct HalfK45 {
    using D = Dq<TYPE>;
    static constexpr bool Q5 = TYPE == JQ_TYPE_Q5_K;
    static constexpr int TILES = 1;
    static constexpr bool EXT = true;
    // d; where a min's weight -r min might not fit a half (dmin above 952 d), d 2^p with the smallest p that brings the block's mins below 2^15. The
    // scales are then divided by 2^p, which is exact: sub-blocks whose min is 0 or 1 keep their values beside others whose min is 63.
    __device__ static __forceinline__ float factor(const typename D::Head& h) {
        const float d = half_bits_to_float(h.h.x), dmin = half_bits_to_float(h.h.x >> 16);
        if (!(63.0f * fabsf(dmin) > 60000.0f * fabsf(d))) {
            return d;
        }
        if (d == 0.0f) {
            return dmin;  // the mins alone
        }
        uint32_t sc, m0, m1;
        scale_min_words(h.h, 0, sc, m0);
        scale_min_words(h.h, 2, sc, m1);
        m0 = __vmaxu4(m0, m1);
        m0 = max(max(m0 & 0xffu, (m0 >> 8) & 0xffu), max((m0 >> 16) & 0xffu, m0 >> 24));
        const int p = (int)(__float_as_uint(fabsf(dmin) / fabsf(d) * (float)m0) >> 23) - (127 + 14);
        return p <= 0 ? d : d * __uint_as_float((uint32_t)(127 + p) << 23);
    }
    static constexpr float MID = Q5 ? 16.0f : 8.0f;
    // 1 / 2^p, see factor. Beyond 2^20 the scales' part of a weight is below 2^-25 of the block's largest, and halves would round it
    __device__ static __forceinline__ float scale_by(float d, float f) {
        const float by = f == d ? 1.0f : d / f;
        return fabsf(by) < 9.5367431640625e-7f ? 0.0f : by;
    }
    struct Scales {
        uint32_t s0, c0, s1, c1;  // as pairs of halves, for sub-blocks 2c and 2c + 1: what 1024 + 16 q (Q5_K: 8 q) is multiplied by, and what is added
    };
    __device__ static __forceinline__ Scales scales(const typename D::Head& h, int c) {
        uint32_t sc, mn;
        scale_min_words(h.h, c, sc, mn);
        // byte under 0x64: 1024 + scale
        uint32_t a = hadd2(__byte_perm(sc, 0x64646464u, (c & 1) ? 0x4242u : 0x4040u), 0xe400e400u);
        uint32_t b = hadd2(__byte_perm(sc, 0x64646464u, (c & 1) ? 0x4343u : 0x4141u), 0xe400e400u);
        const float d = half_bits_to_float(h.h.x), f = factor(h);
        if (f != d) {  // rare
            const uint32_t ratio = h2_dup(scale_by(d, f));
            a = hmul2(a, ratio);
            b = hmul2(b, ratio);
        }
        // / 16 and x -(1024 / 16 + 8); / 8 and x -(1024 / 8 + 16): all exact
        constexpr uint32_t BY = Q5 ? 0x30003000u : 0x2c002c00u, OFF = Q5 ? 0xd880d880u : 0xd480d480u;
        return Scales{hmul2(a, BY), hmul2(a, OFF), hmul2(b, BY), hmul2(b, OFF)};
    }
    __device__ static __forceinline__ void values(const typename D::Head& h, const typename D::Raw& raw, const Scales& s, int c, int part, int run, uint32_t (&hi)[8],
                                                  uint32_t (&)[8]) {
        const uint4 q = raw.q[part];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        const uint4 five = Q5 ? h.hi[part] : make_uint4(0, 0, 0, 0);
        const uint32_t g[4] = {five.x, five.y, five.z, five.w};
#pragma unroll
        for (int x = 0; x < 4; x++) {
            uint32_t v;
            if constexpr (Q5) {
                const uint32_t bit = g[x] >> (2 * c + run);
                v = ((run == 0 ? w[x] << 3 : w[x] >> 1) & 0x78787878u) | ((bit << 7) & 0x80808080u);
            } else {
                v = (run == 0 ? w[x] << 4 : w[x]) & 0xf0f0f0f0u;
            }
            hi[2 * x] = hfma2(bytes_to_halves(v, 0), run == 0 ? s.s0 : s.s1, run == 0 ? s.c0 : s.c1);
            hi[2 * x + 1] = hfma2(bytes_to_halves(v, 1), run == 0 ? s.s0 : s.s1, run == 0 ? s.c0 : s.c1);
        }
    }
    // The 16 more columns: scale mid - r min of the eight sub-blocks, hi then lo.
    __device__ static __forceinline__ void ext(const typename D::Head& h, uint32_t (&v)[8]) {
        const float d = half_bits_to_float(h.h.x), f = factor(h), r = f != 0.0f ? half_bits_to_float(h.h.x >> 16) / f : 0.0f, mid = MID * scale_by(d, f);
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            uint32_t sc, mn;
            scale_min_words(h.h, c, sc, mn);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float a = under2(mn, 0x47000000u, 2 * i) - 32768.0f, b = under2(mn, 0x47000000u, 2 * i + 1) - 32768.0f;
                const float sa = under2(sc, 0x47000000u, 2 * i) - 32768.0f, sb = under2(sc, 0x47000000u, 2 * i + 1) - 32768.0f;
                split_pair(fmaf(-r, a, mid * sa), fmaf(-r, b, mid * sb), v[c + i], v[4 + c + i]);
            }
        }
    }
};
template <>
struct Half<JQ_TYPE_Q4_K> : HalfK45<JQ_TYPE_Q4_K> {};
template <>
struct Half<JQ_TYPE_Q5_K> : HalfK45<JQ_TYPE_Q5_K> {};

template <>
struct Half<JQ_TYPE_Q6_K> {
    using D = Dq<JQ_TYPE_Q6_K>;
    static constexpr int TILES = 2;
    static constexpr bool EXT = false;
    struct Scales {
        uint32_t word;  // the int8 scales of the chunk's four runs
    };
    __device__ static __forceinline__ float factor(const D::Head& h) { return h.d; }
    __device__ static __forceinline__ Scales scales(const D::Head& h, int c) {
        return Scales{c == 0 ? h.sv.x : (c == 1 ? h.sv.y : (c == 2 ? h.sv.z : h.sv.w))};
    }
    __device__ static __forceinline__ void values(const D::Head&, const D::Raw& raw, const Scales& sc, int c, int part, int run, uint32_t (&hi)[8], uint32_t (&lo)[8]) {
        const int p = c & 1;
        const uint4 l = run == 0 ? raw.la[part] : raw.lb[part], hq = raw.hq[part];
        const uint32_t wl[4] = {l.x, l.y, l.z, l.w}, wh[4] = {hq.x, hq.y, hq.z, hq.w};
        // scale + 128 under 0x64, minus 1152
        const uint32_t s = hadd2(__byte_perm(sc.word ^ 0x80808080u, 0x64646464u, 0x4040u + 0x0101u * (uint32_t)(part + 2 * run)), 0xe480e480u);
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const uint32_t a = wl[x] >> (4 * p), b = wh[x] >> (4 * p);
            const uint32_t v = (a & 0x0f0f0f0fu) | ((run == 0 ? b << 4 : b << 2) & 0x30303030u);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                product_hi_lo(hadd2(bytes_to_halves(v, i), 0xe420e420u), s, hi[2 * x + i], lo[2 * x + i]);  // - 1056
            }
        }
    }
    __device__ static __forceinline__ void ext(const D::Head&, uint32_t (&)[8]) {}
};

// The exponent field of the largest of a row's eight block scales (as bits of a half): 2^(exponent - 131) brings it to [2^4, 2^5).
__device__ __forceinline__ uint32_t scale_exponent(uint32_t half_bits) {
    const uint32_t e = __float_as_uint(half_bits_to_float(half_bits)) >> 23;
    return e < 40u ? 40u : (e > 200u ? 200u : e);
}

template <int TYPE>
struct Half32 {
    using D = Dq<TYPE>;
    static constexpr int TILES = 2;
    static constexpr bool EXT = TYPE == JQ_TYPE_Q4_1;
    static constexpr bool Q8 = TYPE == JQ_TYPE_Q8_0;
    struct Scales {
        uint32_t s[2];  // d' of the chunk's two blocks as pairs of halves
    };
    __device__ static __forceinline__ uint32_t exponent(const typename D::Head& h) {
        if constexpr (EXT) {  // d, m interleaved: m counts an eighth
            const uint32_t a[8] = {h.d.x, h.d.y, h.d.z, h.d.w, h.d2.x, h.d2.y, h.d2.z, h.d2.w};
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t mag = a[i] & 0x7fff7fffu;
                const uint32_t min8 = mag >> 16;
                m = max(m, max(mag & 0xffffu, min8 > 0x0c00u ? min8 - 0x0c00u : 0u));  // exponent field less 3
            }
            return scale_exponent(m);
        } else {
            return scale_exponent(max_half8(h.d));
        }
    }
    __device__ static __forceinline__ float factor(const typename D::Head& h) { return __uint_as_float((exponent(h) - 4u) << 23); }
    __device__ static __forceinline__ uint32_t d_bits(const typename D::Head& h, int c, int part) {
        if constexpr (EXT) {
            const uint4 four = c < 2 ? h.d : h.d2;
            return (c & 1) == 0 ? (part == 0 ? four.x : four.y) : (part == 0 ? four.z : four.w);
        } else {
            return (c == 0 ? h.d.x : (c == 1 ? h.d.y : (c == 2 ? h.d.z : h.d.w))) >> (16 * part);
        }
    }
    __device__ static __forceinline__ Scales scales(const typename D::Head& h, int c) {
        const float inv = __uint_as_float((258u - exponent(h)) << 23);  // 2^(4 + 127 - e)
        return Scales{{h2_dup(half_bits_to_float(d_bits(h, c, 0)) * inv), h2_dup(half_bits_to_float(d_bits(h, c, 1)) * inv)}};
    }
    __device__ static __forceinline__ void values(const typename D::Head&, const typename D::Raw& raw, const Scales& sc, int, int part, int run, uint32_t (&hi)[8],
                                                  uint32_t (&lo)[8]) {
        const uint4 q = Q8 ? raw.q[(2 * part + run) % (Q8 ? 4 : 2)] : raw.q[part];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        const uint32_t offset = Q8 ? 0xe480e480u : 0xe408e408u;  // -(1024 + 128), -(1024 + 8)
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const uint32_t v = Q8 ? w[x] ^ 0x80808080u : ((run == 0 ? w[x] : w[x] >> 4) & 0x0f0f0f0fu);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                product_hi_lo(hadd2(bytes_to_halves(v, i), offset), sc.s[part], hi[2 * x + i], lo[2 * x + i]);
            }
        }
    }
    __device__ static __forceinline__ void ext(const typename D::Head& h, uint32_t (&v)[8]) {
        if constexpr (EXT) {
            const float inv = __uint_as_float((258u - exponent(h)) << 23);
            const uint32_t a[8] = {h.d.x, h.d.y, h.d.z, h.d.w, h.d2.x, h.d2.y, h.d2.z, h.d2.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                split_pair(fmaf(8.0f, half_bits_to_float(a[2 * i]), half_bits_to_float(a[2 * i] >> 16)) * inv,
                           fmaf(8.0f, half_bits_to_float(a[2 * i + 1]), half_bits_to_float(a[2 * i + 1] >> 16)) * inv, v[i], v[4 + i]);
            }
        }
    }
};
template <>
struct Half<JQ_TYPE_Q8_0> : Half32<JQ_TYPE_Q8_0> {};
template <>
struct Half<JQ_TYPE_Q4_0> : Half32<JQ_TYPE_Q4_0> {};
template <>
struct Half<JQ_TYPE_Q4_1> : Half32<JQ_TYPE_Q4_1> {};

}  // namespace mm
}  // namespace jq
