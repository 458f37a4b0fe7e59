// tma_pipe.cuh -- what the kernels that stage tiles by the Tensor Memory Accelerator share:
// mbarriers with bounded waits, the tile copy, and the host's tensor-map encoder.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace tomo {

constexpr unsigned long long PIPE_WAIT_NS = 1000000000ull;  // bound of every wait: one second

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for the phase of parity `parity` to complete, as a whole warp; false once a second has
// passed (the clock is read every 256 polls; a poll may itself suspend the thread for a short
// while). One answer for the 32 lanes, which may see the phase or the second pass at different
// polls: they vote at every poll, so all control flow and __syncwarp() after a wait that gave up
// stay uniform over the warp. (A phase that one lane has seen stays visible to the others: the
// next one needs this warp's arrival.)
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long* b, unsigned parity) {
    unsigned long long t0 = 0;
    for (unsigned i = 0;; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(b)), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, done)) return true;
        if ((i & 255u) == 0) {
            const unsigned long long t = global_ns();
            if (i == 0) t0 = t;
            else if (__any_sync(0xffffffffu, t - t0 > PIPE_WAIT_NS)) return false;
        }
    }
}
__device__ __forceinline__ void tma_load_3d(float* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_addr(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
        : "memory");
}

// The FP32 word at byte address a + OFF of shared memory.
template <int OFF>
__device__ __forceinline__ float lds_f32(unsigned a) {
    float r;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(r) : "r"(a), "n"(OFF));
    return r;
}

// The driver's cuTensorMapEncodeTiled (null where the driver does not have it).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn tma_encode_fn();

}  // namespace tomo
