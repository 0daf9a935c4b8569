// FP32 -> Q8_0 quantiser (F.quantizeQ8 of the reference), following the host form
// ops/Quant.java:102-118, which computes the scale and the quotients in double: the blocks equal the reference's bit for bit.
#include <cuda_fp16.h>

#include "jq_common.cuh"

namespace jq {

namespace {

// 4096 x 11008 (4096 x 4096): 35.2 us (15.4) with 64 threads, 35.7 (15.7) with 128, 37.1 (16.3) with 256; floor 35 (13). Warps that stay for the whole call, with
// asynchronous copies of the next chunks on their way, 41 (17.4).
constexpr int THREADS = 64;
constexpr int PER_THREAD = 8;                         // float4 in flight per thread
constexpr int CTA_BLOCKS = THREADS * PER_THREAD / 8;  // 64 blocks: 8 KB read, 2176 bytes written

// q = v / d rounded half away from zero, clamped, in the reference's double arithmetic.
__device__ __noinline__ int quantise_exactly(float v, float d) {
    const double s = (double)v / (double)d;
    long long q = s >= 0 ? (long long)(s + 0.5) : -(long long)(-s + 0.5);
    q = q > 127 ? 127 : q;
    q = q < -127 ? -127 : q;
    return (int)q;
}

// The same from v times 1 / d in single precision, which is off by at most 2^-22.9 of itself, that is 2^-15 below 128: it settles the result
// unless it lies within 2^-14 of a half (or beyond 127.4, or is a NaN); `sure` says whether it does. A double division for every value
// bound the kernel (4096 x 4096: 70 us), then a float one and conversions to integer (29 us). The integer stands in the low bits of
// s + 1.5 2^23.
__device__ __forceinline__ uint32_t quantise(float v, float inv, bool& sure) {
    const float s = v * inv, m = s + 12582912.0f;
    sure = sure && fabsf(s - (m - 12582912.0f)) < 0.49993896f && fabsf(s) < 127.4f;
    return __float_as_uint(m);
}

// The largest of eight values' magnitudes over eight lanes each: lane `part` of the eight gets that of value `part`, in seven shuffles.
__device__ __forceinline__ float share_max(const float (&am)[8], int part) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        a[i] = fmaxf((part & 4) ? am[i + 4] : am[i], __shfl_xor_sync(0xffffffffu, (part & 4) ? am[i] : am[i + 4], 4));
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        b[i] = fmaxf((part & 2) ? a[i + 2] : a[i], __shfl_xor_sync(0xffffffffu, (part & 2) ? a[i] : a[i + 2], 2));
    }
    return fmaxf((part & 1) ? b[1] : b[0], __shfl_xor_sync(0xffffffffu, (part & 1) ? b[0] : b[1], 1));
}

// Eight threads per block of 32, four values each; the CTA's blocks are put together in shared memory and leave as 16-byte stores (a block
// is 34 bytes, so nothing wider than two bytes is aligned by itself). Memory bound: 4 + 34/32 bytes per value. Each of the eight threads makes the scale of one
// of their eight blocks: where each makes all eight, a division and a reciprocal for every four values, those bound the kernel (4096 x 4096 20.6 us against 15.4;
// 4096 x 11008 45.1 against 35.2).
__global__ void __launch_bounds__(THREADS) quantize_q8_0_kernel(const float* x, uint8_t* out, int64_t blocks, bool wide) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // x is written, and out may be read, by the kernel in front
    __shared__ __align__(16) uint8_t stage[CTA_BLOCKS * 34];
    const int64_t b0 = (int64_t)blockIdx.x * CTA_BLOCKS;
    const int tid = threadIdx.x, part = tid & 7;
    float4 v[PER_THREAD];
#pragma unroll
    for (int i = 0; i < PER_THREAD; i++) {
        const int64_t b = b0 + i * (THREADS / 8) + (tid >> 3);
        v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (b < blocks) {
            const float* p = x + b * 32 + part * 4;
            if (wide) {
                v[i] = *reinterpret_cast<const float4*>(p);
            } else {
                v[i] = make_float4(p[0], p[1], p[2], p[3]);
            }
        }
    }
    float am[PER_THREAD];
#pragma unroll
    for (int i = 0; i < PER_THREAD; i++) {
        am[i] = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
    }
    // (float)((double)amax / 127.0): a number of 25 bits in the middle between two floats, times 127, has more than 24 bits, so the quotient
    // is never such a middle nor within 2^-31 of one, and rounding it to double first cannot matter
    const float my_d = __fdiv_rn(share_max(am, part), 127.0f), my_inv = __frcp_rn(my_d);
    const int lane = tid & 31;
    *reinterpret_cast<unsigned short*>(stage + (part * (THREADS / 8) + (tid >> 3)) * 34) = __half_as_ushort(__float2half_rn(my_d));
#pragma unroll
    for (int i = 0; i < PER_THREAD; i++) {
        const float inv = __shfl_sync(0xffffffffu, my_inv, (lane & 24) | i);
        uint8_t* blk = stage + (i * (THREADS / 8) + (tid >> 3)) * 34;
        bool sure = true;
        uint32_t q0 = quantise(v[i].x, inv, sure), q1 = quantise(v[i].y, inv, sure), q2 = quantise(v[i].z, inv, sure), q3 = quantise(v[i].w, inv, sure);
        if (__any_sync(0xffffffffu, !sure)) {  // (a block of zeros has d = 0 and comes here too)
            const float d = __shfl_sync(0xffffffffu, my_d, (lane & 24) | i);
            if (!sure) {
                q0 = d > 0.0f ? (uint32_t)quantise_exactly(v[i].x, d) : 0u;
                q1 = d > 0.0f ? (uint32_t)quantise_exactly(v[i].y, d) : 0u;
                q2 = d > 0.0f ? (uint32_t)quantise_exactly(v[i].z, d) : 0u;
                q3 = d > 0.0f ? (uint32_t)quantise_exactly(v[i].w, d) : 0u;
            }
        }
        unsigned short* to = reinterpret_cast<unsigned short*>(blk + 2 + part * 4);
        to[0] = (unsigned short)__byte_perm(q0, q1, 0x0040);
        to[1] = (unsigned short)__byte_perm(q2, q3, 0x0040);
    }
    __syncthreads();
    const int64_t left = blocks - b0;
    const int bytes = (int)(left < CTA_BLOCKS ? left : CTA_BLOCKS) * 34;
    uint8_t* dst = out + b0 * 34;  // a multiple of 2176, which 16 divides
    const int whole = wide ? bytes / 16 : 0;
    for (int i = tid; i < whole; i += THREADS) {
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(stage)[i];
    }
    for (int i = whole * 16 + tid; i < bytes; i += THREADS) {
        dst[i] = stage[i];
    }
}

}  // namespace

int launch_quantize_q8_0(const float* x, int64_t blocks, uint8_t* out, cudaStream_t s) {
    if (blocks == 0) {
        return JQ_OK;
    }
    const bool wide = (((uintptr_t)x | (uintptr_t)out) & 15) == 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((blocks + CTA_BLOCKS - 1) / CTA_BLOCKS));
    cfg.blockDim = dim3(THREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    JQ_CUDA(cudaLaunchKernelEx(&cfg, quantize_q8_0_kernel, x, out, blocks, wide));
    count_launch();
    return JQ_OK;
}

}  // namespace jq
