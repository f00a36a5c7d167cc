// mbarriers, bulk copies and shared-memory loads of the forward projectors that stage voxel
// columns (proj_staged.cu, proj_sums.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ctsim {

constexpr unsigned kFull = 0xffffffffu;  // all lanes of a warp

// Error flag bit of a stage wait that ran out (ctsim_plan_check reports the flag).
constexpr int kErrStageWait = 4;

// Every wait is bounded by a number of polls (a copy normally lands in microseconds).
constexpr int kMbarPolls = 1 << 22;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
// Makes the initialised barriers visible to the copy engine (async proxy).
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// One arrival that also announces `bytes` of copies to complete on this phase.
__device__ __forceinline__ void mbar_arrive_expect(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// One plain arrival (release: the arriving thread's earlier shared-memory reads are done).
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Global -> shared bulk copy (16-byte aligned addresses, size a multiple of 16), its
// bytes counted on `bar`.  No multicast: the destination is this block's own memory.
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Waits for the phase of the given parity to complete; false after kMbarPolls polls.
// SLEEP: ns between polls (a warp with time to spare leaves its issue slots to the others).
template <int SLEEP = 0>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    const uint32_t a = smem_addr(bar);
    for (int i = 0; i < kMbarPolls; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (SLEEP) __nanosleep(SLEEP);
    }
    return false;
}

__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
}  // namespace ctsim
