// Asynchronous copies into shared memory for sm_100a: bulk copies (the
// non-tensor form of TMA) that complete on an mbarrier, bounded waits, and the
// two instructions of programmatic dependent launch.
//
// Every wait has an iteration limit.  A wait that runs out returns false; the
// caller then records it in a status word, skips the data it waited for and
// leaves in order, so a fault in the protocol never hangs the GPU.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nnis {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// The first 1,024-byte boundary at or after `smem` in shared memory, by an offset: a pointer that came out of an integer has no
// space that the compiler knows, and is read and written by generic accesses with addresses of twice the registers.
__device__ __forceinline__ unsigned char* shared_1024(unsigned char* smem) { return smem + (-smem_addr(smem) & 1023u); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals));
}

// Makes barrier initialisation visible to the async proxy before copies use it.
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// Waits for the phase with the given parity; false after `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = 1u << 22) {
    for (uint32_t i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// global -> shared, `bytes` a multiple of 16, both addresses 16-byte aligned;
// completion is counted in bytes on `bar`.
__device__ __forceinline__ void bulk_load(void* dst_smem, const void* src_gmem, uint32_t bytes,
                                          uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_addr(dst_smem)), "l"(src_gmem), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// Programmatic dependent launch.  `pdl_wait`: everything the preceding kernel
// wrote is visible after it (a no-op without the launch attribute).
// `pdl_launch_dependents`: the next kernel may begin its own preamble.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace nnis
