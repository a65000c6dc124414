// mbarrier, bulk-copy (TMA unit) and asynchronous-copy helpers for kernels that stage global memory through a
// ring of shared-memory stages.  Every wait is bounded: when the limit runs out the waiter raises the CTA's
// abort flag (so the CTA's other waits give up at once) and ORs `who` into a status word in device
// memory that the host reads through cera_cuda_kernel_status.  Copies go to this CTA's shared memory; of a pair they may
// count their bytes on the other CTA's barrier.
#pragma once

#include "common.cuh"

namespace cera {
namespace tma {

constexpr uint32_t SPIN_LIMIT = 1u << 22;  // polls of ~50-100 ns: a fraction of a second at most

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Returns false when the limit ran out or another warp of the CTA already gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag, unsigned int *status,
                                          unsigned int who) {
    for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
        if (mbar_test(bar, parity)) return true;
        if (*abort_flag) return false;
        if (i > 64) __nanosleep(40);
    }
    *abort_flag = 1;
    atomicOr(status, who);
    return false;
}
// The same with mbarrier.try_wait, which suspends the thread in hardware for a bounded time instead of spinning on
// test_wait: far fewer issued instructions while a copy is in flight.  Bounded like mbar_wait.
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_blocking(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag, unsigned int *status,
                                                   unsigned int who) {
    for (uint32_t i = 0; i < (SPIN_LIMIT >> 4); ++i) {  // each try may block for microseconds: keep the total bound comparable
        if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicOr(status, who);
    return false;
}
// For a whole warp that goes on to warp-wide instructions: one answer for all of its lanes.  Of a wait that is given up each lane by itself may see the phase
// complete or the abort flag, and those that went on would run the instructions without the rest.  (A vote on what the lanes' own waits returned cost
// an attention over 16384 positions 1.3 us of 77, a product with 49 stages a CTA 1.4 of 69; in the place of each lane's branch 0.3 and nothing.)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag, unsigned int *status, unsigned int who) {
    for (uint32_t i = 0; i < (SPIN_LIMIT >> 4); ++i) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    atomicOr(status, who);
    return false;
}
// One contiguous global range (16-byte aligned, a multiple of 16 bytes) -> this CTA's shared memory; the bytes are
// counted on `bar`.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// A box of a tensor map (the map lives in constant / parameter space) -> this CTA's shared memory; x * element size must be
// a multiple of 16 bytes.
__device__ __forceinline__ void tensor_g2s_2d(void *dst, const void *map, int32_t x, int32_t y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
                 : "memory");
}

// ---- barriers of another CTA of the cluster ----
__device__ __forceinline__ uint32_t smem_of_rank(const void *p, uint32_t rank) {  // the same object in that CTA's shared memory
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// Its scope is this CTA: what it may hand over is TMEM that has been read (tcgen05.wait::ld, and tc_fence_before ahead of it), never memory.  Operands that
// the other CTA's products read are handed over by their own tensor copies, which count their bytes on that CTA's barrier (tensor_g2s_2d_pair_if).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// ---- for a warp that runs a loop of requests together, issued by the lane for which `me` is true (see elect_one) ----
__device__ __forceinline__ void mbar_expect_tx_if(uint64_t *bar, uint32_t bytes, uint32_t me) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes), "r"(me)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s_if(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint32_t me) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "r"(me)
        : "memory");
}
__device__ __forceinline__ void tensor_g2s_2d_if(void *dst, const void *map, int32_t x, int32_t y, uint64_t *bar, uint32_t me) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(me)
        : "memory");
}
// Its bytes counted on a barrier (cluster address) of this CTA or its cta_group::2 peer.
__device__ __forceinline__ void tensor_g2s_2d_pair_if(void *dst, const void *map, int32_t x, int32_t y, uint32_t bar, uint32_t me) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(smem_u32(dst)),
        "l"(map), "r"(bar), "r"(x), "r"(y), "r"(me)
        : "memory");
}

// 16 bytes global -> shared through the LSU's asynchronous copy path (L1-bypassing).
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// Arrive on `bar` once every cp.async this thread has issued so far has landed (the arrival is one of the
// barrier's expected count).
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace tma
}  // namespace cera
