// Bit-exact dequantisation of an uploaded weight to float32 (Gguf.dequantize / Quant.dequantize of
// the reference: ops/Gguf.java:68-73,127-133, ops/Quant.java:52-60,137-144).
#include "jq_formats.cuh"

namespace jq {

// Four consecutive weights of a block of 256 (of eight 32-element blocks), starting at e (a multiple of 4), with the arithmetic of
// jq_formats.cuh (one rounded operation per step, the reference's order). Integers become floats exactly through 2^15 + q.
__device__ __forceinline__ float byte_float(uint32_t w, int i) { return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7404u | ((uint32_t)i << 4))) - 32768.0f; }

__device__ __forceinline__ uint32_t ld4(const uint8_t* p) { return __ldg(reinterpret_cast<const uint32_t*>(p)); }

template <int TYPE>
struct Four;

template <int TYPE>
struct FourK45 {
    static constexpr bool Q5 = TYPE == JQ_TYPE_Q5_K;
    uint4 h;
    uint32_t q, hi;
    __device__ __forceinline__ void load(const View& v, int64_t row, int64_t b, int e) {
        const uint8_t* p = v.q + tiled_offset(row, b, v.k >> 8, Q5 ? 176 : 144);
        h = ld16(p);
        q = ld4(p + (Q5 ? 48 : 16) + 32 * (e >> 6) + (e & 31));
        hi = Q5 ? ld4(p + 16 + (e & 31)) : 0;
    }
    __device__ __forceinline__ float4 values(int e) const {
        const int sub = e >> 5;
        int sc, mn;
        k_scale_min(h.y, h.z, h.w, sub, sc, mn);
        const float a = __fmul_rn(half_bits_to_float(h.x), (float)sc), m = __fmul_rn(half_bits_to_float(h.x >> 16), (float)mn);
        uint32_t w = (q >> (4 * (sub & 1))) & 0x0f0f0f0fu;
        if (Q5) {
            w |= ((hi >> sub) & 0x01010101u) << 4;
        }
        return make_float4(__fsub_rn(__fmul_rn(a, byte_float(w, 0)), m), __fsub_rn(__fmul_rn(a, byte_float(w, 1)), m), __fsub_rn(__fmul_rn(a, byte_float(w, 2)), m),
                           __fsub_rn(__fmul_rn(a, byte_float(w, 3)), m));
    }
};
template <>
struct Four<JQ_TYPE_Q4_K> : FourK45<JQ_TYPE_Q4_K> {};
template <>
struct Four<JQ_TYPE_Q5_K> : FourK45<JQ_TYPE_Q5_K> {};

template <>
struct Four<JQ_TYPE_Q6_K> {
    uint32_t l, h, sd;
    __device__ __forceinline__ void load(const View& v, int64_t row, int64_t b, int e) {
        const int64_t at = tiled_index(row, b, v.k >> 8);
        const uint8_t* p = v.q + at * 208;
        const int n = e >> 7, kk = (e >> 5) & 3, i = e & 31;
        l = ld4(p + 64 * n + 32 * (kk & 1) + i);
        h = ld4(p + 128 + 32 * n + i);
        sd = __ldg(p + 192 + 8 * n + 2 * kk + (i >> 4)) | ((uint32_t)__ldg(reinterpret_cast<const unsigned short*>(v.aux) + at) << 16);
    }
    __device__ __forceinline__ float4 values(int e) const {
        const int kk = (e >> 5) & 3;
        const uint32_t w = ((l >> (4 * (kk >> 1))) & 0x0f0f0f0fu) | (((h >> (2 * kk)) & 0x03030303u) << 4);
        const float a = __fmul_rn(half_bits_to_float(sd >> 16), (float)(int)(int8_t)(sd & 0xff));
        return make_float4(__fmul_rn(a, byte_float(w, 0) - 32.0f), __fmul_rn(a, byte_float(w, 1) - 32.0f), __fmul_rn(a, byte_float(w, 2) - 32.0f),
                           __fmul_rn(a, byte_float(w, 3) - 32.0f));
    }
};

template <>
struct Four<JQ_TYPE_Q8_0> {
    uint32_t q, d;
    __device__ __forceinline__ void load(const View& v, int64_t row, int64_t b, int e) {
        const int64_t at = tiled_index(row, b, tiled_steps(v.k));
        q = ld4(v.q + at * 256 + 16 * swizzle_piece(e >> 4, row) + (e & 15));
        d = __ldg(reinterpret_cast<const unsigned short*>(v.aux) + at * 8 + (e >> 5));
    }
    __device__ __forceinline__ float4 values(int) const {
        const uint32_t w = q ^ 0x80808080u;
        const float f = half_bits_to_float(d);
        return make_float4(__fmul_rn(f, byte_float(w, 0) - 128.0f), __fmul_rn(f, byte_float(w, 1) - 128.0f), __fmul_rn(f, byte_float(w, 2) - 128.0f),
                           __fmul_rn(f, byte_float(w, 3) - 128.0f));
    }
};

template <int TYPE>
struct FourN {
    static constexpr bool HAS_MIN = TYPE == JQ_TYPE_Q4_1;
    uint32_t q, d;
    __device__ __forceinline__ void load(const View& v, int64_t row, int64_t b, int e) {
        const int64_t at = tiled_index(row, b, tiled_steps(v.k));
        q = ld4(v.q + at * 128 + 16 * swizzle_piece(e >> 5, row) + (e & 15));
        d = HAS_MIN ? ld4(v.aux + (at * 8 + (e >> 5)) * 4) : (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(v.aux) + at * 8 + (e >> 5));
    }
    __device__ __forceinline__ float one(uint32_t w, int i) const {
        const float f = half_bits_to_float(d);
        return HAS_MIN ? __fadd_rn(__fmul_rn(byte_float(w, i), f), half_bits_to_float(d >> 16)) : __fmul_rn(byte_float(w, i) - 8.0f, f);
    }
    __device__ __forceinline__ float4 values(int e) const {
        const uint32_t w = (q >> (4 * ((e >> 4) & 1))) & 0x0f0f0f0fu;
        return make_float4(one(w, 0), one(w, 1), one(w, 2), one(w, 3));
    }
};
template <>
struct Four<JQ_TYPE_Q4_0> : FourN<JQ_TYPE_Q4_0> {};
template <>
struct Four<JQ_TYPE_Q4_1> : FourN<JQ_TYPE_Q4_1> {};

// A warp takes 256 values of ROWS rows: lane i the values 4 i .. and 128 + 4 i .. of each, so that every store of the warp is 512 contiguous
// bytes; eight warps take neighbouring steps of k. Memory bound: the 4 output bytes per weight are 80 % and more of the traffic. (One
// thread per 16 or 64 consecutive weights left stores of 16 bytes at strides of 64 to 256.)
constexpr int ROWS = 4;
template <int TYPE>
__global__ void __launch_bounds__(256) dequantize_kernel(View v, float* __restrict__ dst) {
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), r0 = (int64_t)blockIdx.y * ROWS;
    if (b >= tiled_steps(v.k)) {
        return;
    }
    Four<TYPE> f[ROWS][2];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        const int64_t row = r0 + r < v.n ? r0 + r : v.n - 1;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            f[r][j].load(v, row, b, 128 * j + 4 * lane);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int e = 128 * j + 4 * lane;
            if (r0 + r < v.n && b * 256 + e < v.k) {
                *reinterpret_cast<float4*>(dst + (r0 + r) * v.k + b * 256 + e) = f[r][j].values(e);
            }
        }
    }
}

// ---- formats that are dequantised only (no linear kernel): verbatim bytes ----
__device__ __forceinline__ int u8(const uint8_t* w, int64_t at) { return w[at]; }
__device__ __forceinline__ float f16(const uint8_t* w, int64_t at) {
    return __half2float(__ushort_as_half((unsigned short)(w[at] | (w[at + 1] << 8))));
}
__device__ __forceinline__ int bit32(const uint8_t* w, int64_t at, int bit) { return (u8(w, at + bit / 8) >> (bit % 8)) & 1; }

// kernels/GgufKernels.java:147-198 of the reference (Q5_0, Q5_1, Q2_K, Q3_K), one rounded float
// operation per arithmetic step.
__device__ __forceinline__ float extra_value(int type, const uint8_t* w, int64_t i) {
    if (type == JQ_TYPE_Q5_0) {
        int64_t base = (i / 32) * 22;
        int e = (int)(i % 32);
        int b = u8(w, base + 6 + e % 16);
        int q = (e < 16 ? b & 15 : b >> 4) + 16 * bit32(w, base + 2, e);
        return __fmul_rn((float)(q - 16), f16(w, base));
    }
    if (type == JQ_TYPE_Q5_1) {
        int64_t base = (i / 32) * 24;
        int e = (int)(i % 32);
        int b = u8(w, base + 8 + e % 16);
        int q = (e < 16 ? b & 15 : b >> 4) + 16 * bit32(w, base + 4, e);
        return __fadd_rn(__fmul_rn((float)q, f16(w, base)), f16(w, base + 2));
    }
    if (type == JQ_TYPE_Q2_K) {
        int64_t base = (i / 256) * 84;
        int e = (int)(i % 256);
        int n = e / 128, j = (e % 128) / 32, l = e % 32;
        int sc = u8(w, base + n * 8 + j * 2 + l / 16);
        int q = (u8(w, base + 16 + n * 32 + l) >> (2 * j)) & 3;
        float a = __fmul_rn(__fmul_rn(f16(w, base + 80), (float)(sc & 15)), (float)q);
        return __fsub_rn(a, __fmul_rn(f16(w, base + 82), (float)(sc >> 4)));
    }
    // Q3_K
    int64_t base = (i / 256) * 110;
    int e = (int)(i % 256);
    int n = e / 128, j = (e % 128) / 32, l = e % 32;
    int is = n * 8 + j * 2 + l / 16;
    int q = (u8(w, base + 32 + n * 32 + l) >> (2 * j)) & 3;
    int high = (u8(w, base + l) >> (4 * n + j)) & 1;
    int64_t s = base + 96;
    int low = is < 8 ? u8(w, s + is) & 15 : u8(w, s + is - 8) >> 4;
    int hi2 = (u8(w, s + 8 + is % 4) >> (2 * (is / 4))) & 3;
    int scale = low + 16 * hi2 - 32;
    return __fmul_rn(__fmul_rn(f16(w, base + 108), (float)scale), (float)(q - (high == 1 ? 0 : 4)));
}

// Four consecutive values per thread (they share a block), so that stores are 16 bytes each.
template <int TYPE>
__global__ void __launch_bounds__(256) dequantize_extra_kernel(const uint8_t* __restrict__ w, float* __restrict__ dst, int64_t count) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i < count) {
        *reinterpret_cast<float4*>(dst + i) = make_float4(extra_value(TYPE, w, i), extra_value(TYPE, w, i + 1), extra_value(TYPE, w, i + 2), extra_value(TYPE, w, i + 3));
    }
}

template <int TYPE>
static int run_extra(const View& v, float* dst, cudaStream_t s) {
    const int64_t count = v.n * v.k;
    if (count == 0) {
        return JQ_OK;
    }
    dequantize_extra_kernel<TYPE><<<(unsigned)((count / 4 + 255) / 256), 256, 0, s>>>(v.q, dst, count);
    count_launch();
    return check_launch("dequantize_extra_kernel");
}

template <int TYPE>
static int run(const View& v, float* dst, cudaStream_t s) {
    if (v.n == 0 || v.k == 0) {
        return JQ_OK;
    }
    constexpr int64_t GROUP = 128 * 1024;  // rows per launch: a grid has at most 65535 rows of CTAs; a multiple of 128, so the tiles go on
    const int64_t steps = tiled_steps(v.k);
    for (int64_t r0 = 0; r0 < v.n; r0 += GROUP) {
        View part = v;
        part.n = v.n - r0 < GROUP ? v.n - r0 : GROUP;
        part.q = v.q + tiled_index(r0, 0, steps) * (256 / Fmt<TYPE>::QK) * plane_q_bytes(TYPE);
        part.aux = v.aux == nullptr ? nullptr : v.aux + tiled_index(r0, 0, steps) * (256 / Fmt<TYPE>::QK) * plane_aux_bytes(TYPE);
        const dim3 grid((unsigned)((steps + 7) / 8), (unsigned)((part.n + ROWS - 1) / ROWS));
        dequantize_kernel<TYPE><<<grid, 256, 0, s>>>(part, dst + r0 * v.k);
        count_launch();
    }
    return check_launch("dequantize_kernel");
}

int launch_dequantize(const View& v, float* dst, cudaStream_t s) {
    switch (v.type) {
        case JQ_TYPE_Q8_0: return run<JQ_TYPE_Q8_0>(v, dst, s);
        case JQ_TYPE_Q4_0: return run<JQ_TYPE_Q4_0>(v, dst, s);
        case JQ_TYPE_Q4_1: return run<JQ_TYPE_Q4_1>(v, dst, s);
        case JQ_TYPE_Q4_K: return run<JQ_TYPE_Q4_K>(v, dst, s);
        case JQ_TYPE_Q5_K: return run<JQ_TYPE_Q5_K>(v, dst, s);
        case JQ_TYPE_Q6_K: return run<JQ_TYPE_Q6_K>(v, dst, s);
        case JQ_TYPE_Q5_0: return run_extra<JQ_TYPE_Q5_0>(v, dst, s);
        case JQ_TYPE_Q5_1: return run_extra<JQ_TYPE_Q5_1>(v, dst, s);
        case JQ_TYPE_Q2_K: return run_extra<JQ_TYPE_Q2_K>(v, dst, s);
        case JQ_TYPE_Q3_K: return run_extra<JQ_TYPE_Q3_K>(v, dst, s);
        default: return fail(JQ_ERR_UNSUPPORTED, "dequantize: unknown type %d", v.type);
    }
}

}  // namespace jq
