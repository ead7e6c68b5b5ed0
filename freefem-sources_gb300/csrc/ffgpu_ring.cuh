// ffgpu_ring.cuh -- matrix entries staged through shared memory: each warp keeps a few stages filled
// ahead of its lanes by bulk copies, one mbarrier per stage.  Lane 0 expects a stage's bytes and issues
// its copies (16-byte aligned, whole slots of 32 entries); the warp waits for the stage, reads it, and
// after a __syncwarp() lane 0 fills it again.  Every wait is bounded in time.
#pragma once
#include <stdint.h>

namespace ffgpu {

constexpr unsigned long long kRingWaitNs = 1000000000ull;

__device__ __forceinline__ uint32_t ring_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ring_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar), "l"(pol)
        : "memory");
}
__device__ __forceinline__ uint32_t ring_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done;
}
// whole warp; false when the second allowed runs out
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok = ring_try(bar, parity);
    if (!__all_sync(0xffffffffu, ok)) {
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        do {
            ok = ring_try(bar, parity);
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        } while (!__all_sync(0xffffffffu, ok) && __any_sync(0xffffffffu, t - t0 <= kRingWaitNs));
    }
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void ring_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// matrix streams leave the L2 to the vectors
__device__ __forceinline__ uint64_t ring_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
// one thread; the threads that wait come after a barrier of their own
__device__ __forceinline__ void ring_init(uint32_t bar, int stages) {
    for (int k = 0; k < stages; ++k)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8 * k), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

}  // namespace ffgpu
