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
// bytes; neighbouring warps take neighbouring steps of k. The weights are on their way before the kernel in front has ended (nothing writes them): Q6_K 4096 x 11008
// 39.4 -> 36.5 us, 4096 x 4096 17.9 -> 15.3, 1024 x 1024 4.6 -> 2.8. Memory bound: the 4 output bytes per weight are 80 % and more of the traffic. (One
// thread per 16 or 64 consecutive weights left stores of 16 bytes at strides of 64 to 256.)
constexpr int ROWS = 4;
constexpr int THREADS = 256;
template <int TYPE>
__global__ void __launch_bounds__(THREADS) dequantize_kernel(View v, float* __restrict__ dst, int steps) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int lane = threadIdx.x & 31;
    const uint32_t task = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);  // (warps that the last step of a row leaves idle would be every tenth at k = 11008)
    const int64_t b = task % (uint32_t)steps, r0 = (int64_t)(task / (uint32_t)steps) * ROWS;
    if (r0 >= v.n) {
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
    asm volatile("griddepcontrol.wait;" ::: "memory");  // dst may be in use by the kernel in front
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
__device__ __forceinline__ uint32_t ld2(const uint8_t* p) { return __ldg(reinterpret_cast<const unsigned short*>(p)); }
__device__ __forceinline__ uint32_t ld2x2(const uint8_t* p) { return ld2(p) | ld2(p + 2) << 16; }  // (where a block starts on an even address only)
// Bits 0 .. 3 to bit 4 of four bytes.
__device__ __forceinline__ uint32_t bits_to_bytes(uint32_t h) { return ((h & 15u) * 0x00204081u & 0x01010101u) << 4; }

// Four consecutive values, which share a scale: kernels/GgufKernels.java:147-198 of the reference (Q5_0, Q5_1, Q2_K, Q3_K), one rounded float operation
// per arithmetic step.
template <int TYPE>
__device__ __forceinline__ float4 extra_values(const uint8_t* w, int64_t i) {
    if constexpr (TYPE == JQ_TYPE_Q5_0) {
        const uint8_t* p = w + (i >> 5) * 22;
        const int e = (int)(i & 31);
        const uint32_t q = ((ld2x2(p + 6 + (e & 15)) >> (e & 16 ? 4 : 0)) & 0x0f0f0f0fu) | bits_to_bytes(ld2x2(p + 2) >> e);
        const float d = half_bits_to_float(ld2(p));
        return make_float4(__fmul_rn(byte_float(q, 0) - 16.0f, d), __fmul_rn(byte_float(q, 1) - 16.0f, d), __fmul_rn(byte_float(q, 2) - 16.0f, d), __fmul_rn(byte_float(q, 3) - 16.0f, d));
    } else if constexpr (TYPE == JQ_TYPE_Q5_1) {
        const uint8_t* p = w + (i >> 5) * 24;
        const int e = (int)(i & 31);
        const uint32_t q = ((ld4(p + 8 + (e & 15)) >> (e & 16 ? 4 : 0)) & 0x0f0f0f0fu) | bits_to_bytes(ld4(p + 4) >> e), dm = ld4(p);
        const float d = half_bits_to_float(dm), m = half_bits_to_float(dm >> 16);
        return make_float4(__fadd_rn(__fmul_rn(byte_float(q, 0), d), m), __fadd_rn(__fmul_rn(byte_float(q, 1), d), m), __fadd_rn(__fmul_rn(byte_float(q, 2), d), m),
                           __fadd_rn(__fmul_rn(byte_float(q, 3), d), m));
    } else if constexpr (TYPE == JQ_TYPE_Q2_K) {
        const uint8_t* p = w + (i >> 8) * 84;
        const int n = (int)(i >> 7) & 1, j = (int)(i >> 5) & 3, l = (int)(i & 31);
        const uint32_t sc = __ldg(p + n * 8 + j * 2 + (l >> 4)), q = (ld4(p + 16 + n * 32 + l) >> (2 * j)) & 0x03030303u, dm = ld4(p + 80);
        const float d = __fmul_rn(half_bits_to_float(dm), (float)(sc & 15)), m = __fmul_rn(half_bits_to_float(dm >> 16), (float)(sc >> 4));
        return make_float4(__fsub_rn(__fmul_rn(d, byte_float(q, 0)), m), __fsub_rn(__fmul_rn(d, byte_float(q, 1)), m), __fsub_rn(__fmul_rn(d, byte_float(q, 2)), m),
                           __fsub_rn(__fmul_rn(d, byte_float(q, 3)), m));
    } else {
        const uint8_t* p = w + (i >> 8) * 110;
        const int n = (int)(i >> 7) & 1, j = (int)(i >> 5) & 3, l = (int)(i & 31), is = n * 8 + j * 2 + (l >> 4);
        // (quant) + 4 (its bit in the mask), minus 4
        const uint32_t q = ((ld2x2(p + 32 + n * 32 + l) >> (2 * j)) & 0x03030303u) | ((ld2x2(p + l) >> (4 * n + j)) & 0x01010101u) << 2;
        const int low = __ldg(p + 96 + (is & 7)), high = __ldg(p + 104 + (is & 3));
        const int scale = (is < 8 ? low & 15 : low >> 4) + 16 * (high >> (2 * (is >> 2)) & 3) - 32;
        const float d = __fmul_rn(half_bits_to_float(ld2(p + 108)), (float)scale);
        return make_float4(__fmul_rn(d, byte_float(q, 0) - 4.0f), __fmul_rn(d, byte_float(q, 1) - 4.0f), __fmul_rn(d, byte_float(q, 2) - 4.0f), __fmul_rn(d, byte_float(q, 3) - 4.0f));
    }
}

// A warp's stores are 512 contiguous bytes; a thread has the loads of PIECES of them in flight. (With every value of its own, made from loads of single bytes,
// instructions bound it: 4096 x 11008 Q5_0 71.7 us, Q5_1 74.0, Q2_K 86.4, Q3_K 112.8; now 42.9, 34.2, 34.6, 43.7, and 47 with one piece in flight; floor 30 to 33. Q5_0's and
// Q3_K's blocks start on even addresses, so that four quants are two loads.)
constexpr int PIECES = 2;
template <int TYPE>
__global__ void __launch_bounds__(THREADS) dequantize_extra_kernel(const uint8_t* __restrict__ w, float* __restrict__ dst, int64_t count) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int64_t i0 = ((int64_t)blockIdx.x * (PIECES * THREADS) + threadIdx.x) * 4;
    float4 v[PIECES];
#pragma unroll
    for (int j = 0; j < PIECES; j++) {
        const int64_t i = i0 + j * (THREADS * 4);
        v[j] = extra_values<TYPE>(w, i < count ? i : 0);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // dst may be in use by the kernel in front
#pragma unroll
    for (int j = 0; j < PIECES; j++) {
        const int64_t i = i0 + j * (THREADS * 4);
        if (i < count) {
            *reinterpret_cast<float4*>(dst + i) = v[j];
        }
    }
}

// `ctas` thread blocks, launched programmatically.
struct Config {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
};
static Config& launch_config(int64_t ctas, cudaStream_t s) {
    static thread_local Config c;
    c.attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    c.attr[0].val.programmaticStreamSerializationAllowed = 1;
    c.cfg.attrs = c.attr;
    c.cfg.numAttrs = 1;
    c.cfg.gridDim = dim3((unsigned)ctas);
    c.cfg.blockDim = dim3(THREADS);
    c.cfg.stream = s;
    return c;
}

template <int TYPE>
static int run_extra(const View& v, float* dst, cudaStream_t s) {
    const int64_t count = v.n * v.k;
    if (count == 0) {
        return JQ_OK;
    }
    JQ_CUDA(cudaLaunchKernelEx(&launch_config((count / 4 + PIECES * THREADS - 1) / (PIECES * THREADS), s).cfg, dequantize_extra_kernel<TYPE>, (const uint8_t*)v.q, dst, count));
    count_launch();
    return JQ_OK;
}

template <int TYPE>
static int run(const View& v, float* dst, cudaStream_t s) {
    if (v.n == 0 || v.k == 0) {
        return JQ_OK;
    }
    constexpr int64_t GROUP = 128 * 1024;  // rows per launch, a multiple of 128, so the tiles go on: (at most 2^31 values) / 256 / ROWS tasks fit 32 bits
    const int64_t steps = tiled_steps(v.k);
    for (int64_t r0 = 0; r0 < v.n; r0 += GROUP) {
        View part = v;
        part.n = v.n - r0 < GROUP ? v.n - r0 : GROUP;
        part.q = v.q + tiled_index(r0, 0, steps) * (256 / Fmt<TYPE>::QK) * plane_q_bytes(TYPE);
        part.aux = v.aux == nullptr ? nullptr : v.aux + tiled_index(r0, 0, steps) * (256 / Fmt<TYPE>::QK) * plane_aux_bytes(TYPE);
        const int64_t tasks = steps * ((part.n + ROWS - 1) / ROWS);
        JQ_CUDA(cudaLaunchKernelEx(&launch_config((tasks + THREADS / 32 - 1) / (THREADS / 32), s).cfg, dequantize_kernel<TYPE>, part, dst + r0 * v.k, (int)steps));
        count_launch();
    }
    return JQ_OK;
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
