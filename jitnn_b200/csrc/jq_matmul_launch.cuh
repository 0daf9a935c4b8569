// Instances of the matrix kernel for one weight format and their launch. Each format is a translation unit of its own
// (jq_matmul_<format>.cu), so that they compile side by side.
#pragma once

#include "jq_matmul.cuh"

namespace jq {
namespace mm {

struct Plan {
    bool fp32, bwd;
    int nmax;  // the instance, by the widest tile of rows of x it takes
    int ctas;  // grid
    size_t smem;
};

// What the host has to know of an instance's Shape.
struct Facts {
    int groups, turn, turns, a_cols, b_tiles, columns;  // columns: accumulator columns per row of x
    int operands, scales;
    bool owned, ext, paired;
};
template <int TYPE, bool FP32, bool BWD, int NMAX>
constexpr Facts facts_of() {
    using W = Shape<TYPE, FP32, BWD, NMAX>;
    return Facts{W::GROUPS, W::TURN, W::TURNS, W::A_COLS, W::B_TILES, W::JOINED ? 2 : 1, W::OPERANDS, W::SCALES, W::OWNED, W::EXT, W::PAIRED};
}
template <int TYPE>
Facts facts_format(bool fp32, bool bwd, int nmax) {
    if (!fp32) {
        return nmax <= 128 ? facts_of<TYPE, false, false, 128>() : facts_of<TYPE, false, false, 256>();
    }
    if (bwd) {
        return nmax <= 32 ? facts_of<TYPE, true, true, 32>() : facts_of<TYPE, true, true, 128>();
    }
    return nmax <= 32 ? facts_of<TYPE, true, false, 32>() : facts_of<TYPE, true, false, 128>();
}

template <int TYPE, bool FP32, bool BWD, int NMAX>
int launch_instance(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) {
    auto kernel = matmul_kernel<TYPE, FP32, BWD, NMAX>;
    static std::atomic<uint64_t> configured{0};  // the opt-in for large dynamic shared memory is per device
    int dev = 0;
    JQ_CUDA(cudaGetDevice(&dev));
    if ((configured.load(std::memory_order_relaxed) >> (dev & 63) & 1) == 0) {
        JQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured.fetch_or((uint64_t)1 << (dev & 63));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.ctas);
    cfg.blockDim = dim3((Shape<TYPE, FP32, BWD, NMAX>::THREADS));
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // barriers, tensor memory and the first raw blocks before the kernel in front ends
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)args.ksplit;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = args.ksplit > 1 ? 2 : 1;
    JQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, args, map));
    count_launch();
    return JQ_OK;
}

template <int TYPE>
int launch_format(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) {
    if (!plan.fp32) {
        return plan.nmax <= 128 ? launch_instance<TYPE, false, false, 128>(plan, args, map, s) : launch_instance<TYPE, false, false, 256>(plan, args, map, s);
    }
    if (plan.bwd) {
        return plan.nmax <= 32 ? launch_instance<TYPE, true, true, 32>(plan, args, map, s) : launch_instance<TYPE, true, true, 128>(plan, args, map, s);
    }
    return plan.nmax <= 32 ? launch_instance<TYPE, true, false, 32>(plan, args, map, s) : launch_instance<TYPE, true, false, 128>(plan, args, map, s);
}

int launch_q4_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);
int launch_q5_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);
int launch_q6_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);
int launch_q8_0(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);
int launch_q4_0(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);
int launch_q4_1(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s);

}  // namespace mm
}  // namespace jq
