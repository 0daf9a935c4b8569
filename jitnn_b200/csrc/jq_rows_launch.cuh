// Instances of the rows kernel for one weight format and their launch. Each format is a translation unit of its own (jq_rows_<format>.cu), so that they
// compile side by side.
#pragma once

#include "jq_rows.cuh"

namespace jq {
namespace rows {

// Ring depths for a.ksplit; returns the bytes of shared memory.
template <int TYPE, int NT>
size_t configure(Args& a) {
    using S = Shape<TYPE, NT>;
    constexpr int IMAGE = S::IMAGE;
    const int room = 227 * 1024 - 128 - S::TAIL - part_bytes(a.ksplit, NT), step = Rw<TYPE>::HALVES == 1 ? S::GROUPS : 1;
    a.raw = step == 1 ? 2 : step;
    a.img = 2;
    while (a.raw + step <= MAX_RAW && (a.raw + step) * S::UNIT + 3 * IMAGE <= room) {
        a.raw += step;
    }
    while (a.img < MAX_IMG && a.raw * S::UNIT + (a.img + 1) * IMAGE <= room) {
        a.img++;
    }
    return (size_t)(128 + S::TAIL + part_bytes(a.ksplit, NT) + a.raw * S::UNIT + a.img * IMAGE);
}

template <int TYPE, int NT, bool AFTER>
int launch_instance(Args& a, int ctas, cudaStream_t s) {
    auto kernel = rows_kernel<TYPE, NT, AFTER>;
    static std::atomic<uint64_t> configured{0};  // the opt-in for large dynamic shared memory is per device
    int dev = 0;
    JQ_CUDA(cudaGetDevice(&dev));
    if ((configured.load(std::memory_order_relaxed) >> (dev & 63) & 1) == 0) {
        JQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured.fetch_or((uint64_t)1 << (dev & 63));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(Shape<TYPE, NT>::THREADS);
    cfg.dynamicSmemBytes = configure<TYPE, NT>(a);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // barriers, tensor memory and the first raw units before the kernel in front ends
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)a.ksplit;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.ksplit > 1 ? 2 : 1;
    JQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    count_launch();
    return JQ_OK;
}

template <int TYPE>
int launch_format(Args& a, int ctas, bool after, cudaStream_t s) {
    if (a.m <= 8) {  // 32000 x 4096, 8 rows by either, us: Q4_K 21.8 and 24.9, Q6_K 32.2 and 38.2, Q8_0 26.0 and 30.3
        return after ? launch_instance<TYPE, 8, true>(a, ctas, s) : launch_instance<TYPE, 8, false>(a, ctas, s);
    }
    return after ? launch_instance<TYPE, 16, true>(a, ctas, s) : launch_instance<TYPE, 16, false>(a, ctas, s);
}

int launch_q4_k(Args& a, int ctas, bool after, cudaStream_t s);
int launch_q5_k(Args& a, int ctas, bool after, cudaStream_t s);
int launch_q6_k(Args& a, int ctas, bool after, cudaStream_t s);
int launch_q8_0(Args& a, int ctas, bool after, cudaStream_t s);
int launch_q4_0(Args& a, int ctas, bool after, cudaStream_t s);
int launch_q4_1(Args& a, int ctas, bool after, cudaStream_t s);

}  // namespace rows
}  // namespace jq
