// What the activation images of the integer GEMVs have in common: eight values a lane of a warp's 256 become 22-bit fixed point relative to the largest
// magnitude, as three signed base-256 digits.
#pragma once

#include "jq_common.cuh"

namespace jq {

// The exponent field of s = 2^floor(log2(largest magnitude of the warp's 256 values)), at least `least` (so that 2^21 / s and the smallest weight of
// a digit stay normal), at most that of the largest finite values: |x| / s < 2, on which the digits depend; bad: a NaN or an Inf is among them. Magnitudes are compared as integers: NaN > Inf > every finite value.
__device__ __forceinline__ uint32_t image_exponent(const float (&xv)[8], uint32_t least, bool& bad) {
    uint32_t amb = 0u;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        amb = max(amb, __float_as_uint(xv[i]) & 0x7fffffffu);
    }
    amb = __reduce_max_sync(0xffffffffu, amb);
    bad = amb >= 0x7f800000u;
    const uint32_t e = amb & 0x7f800000u;
    return e < least ? least : (e > 0x7f000000u ? 0x7f000000u : e);
}

// dw[d][h]: digit d of values 4 h .. 4 h + 3, a signed byte each.
// X = rint(x 2^21 / s) lands in the mantissa of x 2^21 / s + 1.5 * 2^23 (the product is exact: s is a power of two). With 128 added at every byte position
// the three low bytes of Y = X + 0x808080 are the digits plus 128 each (X = d0 + 256 d1 + 65536 d2 with -128 <= d < 128 has exactly one such form,
// and |X| <= 2^22 keeps the top digit within a signed byte after the carries), so digit = byte ^ 0x80.
__device__ __forceinline__ void image_digits(const float (&xv)[8], uint32_t e, uint32_t (&dw)[3][2]) {
    const float inv = __uint_as_float(0x7f000000u - e + (21u << 23));
    uint32_t Y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        Y[i] = __float_as_uint(fmaf(xv[i], inv, 12582912.0f)) - 0x4b400000u + 0x00808080u;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t t01 = __byte_perm(Y[4 * h], Y[4 * h + 1], 0x5140), t23 = __byte_perm(Y[4 * h + 2], Y[4 * h + 3], 0x5140);
        const uint32_t h01 = __byte_perm(Y[4 * h], Y[4 * h + 1], 0x0062), h23 = __byte_perm(Y[4 * h + 2], Y[4 * h + 3], 0x0062);
        dw[0][h] = __byte_perm(t01, t23, 0x5410) ^ 0x80808080u;
        dw[1][h] = __byte_perm(t01, t23, 0x7632) ^ 0x80808080u;
        dw[2][h] = __byte_perm(h01, h23, 0x5410) ^ 0x80808080u;
    }
}

__device__ __forceinline__ int digit_sum(const uint32_t (&w)[2]) { return __dp4a((int)w[0], 0x01010101, __dp4a((int)w[1], 0x01010101, 0)); }

}  // namespace jq
