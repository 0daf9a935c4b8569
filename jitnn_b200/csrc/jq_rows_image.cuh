// The image of x that the rows kernel (jq_rows.cuh) reads: its layout and the warp-level routine that makes one step of one row. Kernels that produce
// activations include this to write the image in the place of a float vector.
#pragma once

#include "jq_matmul_dequant.cuh"

namespace jq {
namespace rows {

constexpr int MAX_NT = 16;  // NT: rows of x that an instance takes, 8 or 16; 2 NT columns
inline int nt_of(int m) { return m <= 8 ? 8 : 16; }
__host__ __device__ constexpr int step_bytes(int nt) { return 2 * nt * 32; }           // 16 k of the image: [8 k][8 columns][8 rows of 16 bytes]
__host__ __device__ constexpr int image_bytes(int nt) { return 17 * step_bytes(nt); }  // a unit: 256 k, then the sums of x over its runs of 32, twice, as 16 more k

// One warp: lane L holds the values 8 L .. 8 L + 7 of step u of a row. The row's 256 values times a power of two that brings the largest to [2^9, 2^10),
// hi = that rounded to half precision, lo = the rest rounded to half precision: 22 significant bits for everything down to 2^-13 of the largest.
// 256 values that hold a NaN or an Inf get the scale NaN, which reaches every output of that row.
template <int NT>
__device__ __forceinline__ void store_image(const float (&v)[8], int64_t u, int row, uint8_t* image, float* scales, int lane) {
    constexpr int N = 2 * NT, STEP = step_bytes(NT);
    uint32_t am = 0;  // the largest magnitude as bits: an Inf or a NaN is larger than any number
#pragma unroll
    for (int i = 0; i < 8; i++) {
        am = max(am, __float_as_uint(v[i]) & 0x7fffffffu);
    }
    am = __reduce_max_sync(0xffffffffu, am);
    const bool bad = am >= 0x7f800000u;
    uint32_t e = am >> 23;
    e = e < 14u ? 14u : (e > 254u ? 254u : e);
    const float f = __uint_as_float((263u - e) << 23);
    uint32_t hi[4], lo[4];  // of four values 0 and 2, 1 and 3
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = v[(i >> 1) * 4 + (i & 1)] * f, c = v[(i >> 1) * 4 + (i & 1) + 2] * f;
        mm::split_pair(a, c, hi[i], lo[i]);
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i])), l = __half22float2(*reinterpret_cast<const __half2*>(&lo[i]));
        sum += (h.x + l.x) + (h.y + l.y);
    }
    // lane = step of 16 and half of it; columns row (hi) and NT + row (lo), 128 bytes per eight columns
    uint8_t* const unit = image + u * image_bytes(NT);
    const int col = (row >> 3) * 128 + (row & 7) * 16;
    uint8_t* const to = unit + (lane >> 1) * STEP + (lane & 1) * (N * 16) + col;
    *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(to + NT * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    // the sums over runs of 32 (four lanes), up to 2^15, twice
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const __half sh = __float2half_rn(sum), sl = __float2half_rn(sum - __half2float(sh));
    if ((lane & 3) == 0) {
        __half* const run = reinterpret_cast<__half*>(unit + 16 * STEP + col) + (lane >> 2);
        run[0] = run[N * 8] = sh;
        run[NT * 8] = run[(N + NT) * 8] = sl;
    }
    if (lane == 0) {
        scales[u * NT + row] = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((e - 9u) << 23);
    }
}

}  // namespace rows
}  // namespace jq
