// Device-side helpers for kernels built on the Blackwell copy engine and tensor memory: mbarriers with bounded waits,
// bulk and tensor-map copies into shared memory (no multicast anywhere), tcgen05 fences, tensor-memory allocation.
#pragma once

#include <cuda.h>

#include "jq_common.cuh"

namespace jq {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// The same without ever suspending the thread: true if the phase with the given parity is complete.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// A wait gave up: `status` is a status word (page-locked host memory); of several codes written at a time any one will do.
__device__ __forceinline__ void record_status(int* status, int code) {
    *reinterpret_cast<volatile int*>(status) = code;
    __threadfence_system();
}

// Waits for the phase with the given parity, for at most `limit` clocks of the SM (a poll may suspend the thread for a time the
// hardware chooses, so the bound counts time, not polls). Gives up earlier when another role of the CTA has given up (abort
// flag in shared memory); a wait that runs out records `code` in the status word.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code, long long limit) {
    if (mbar_try(bar, parity)) {
        return true;
    }
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try(bar, parity)) {
            return true;
        }
        if (*abort_flag != 0) {
            return false;
        }
        if (clock64() - t0 > limit) {
            record_status(status, code);
            *abort_flag = 1;
            return false;
        }
    }
}

// Between a warp's reads of shared memory and the arrival that lets the copy engine fill it again. A barrier among the lanes orders their loads
// against each other's, not against the copy engine, and a load whose value is used later may be made behind the arrival; the fence between
// the proxies orders them.
__device__ __forceinline__ void reads_before_refill() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
}

// One contiguous run of bytes (a multiple of 16, both addresses 16-byte aligned) from global into shared memory.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// A box of a rank-2 tensor map; c0 is the innermost coordinate (c0 times the element size must be a multiple of 16 bytes).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
                 "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Arrives on the mbarrier once every tcgen05 operation this thread has issued so far has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

}  // namespace tc

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (the library does not link libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled();

}  // namespace jq
