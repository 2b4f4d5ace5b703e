// PTX wrappers for kernels on CTA pairs (tcgen05 with cta_group::2: two CTAs of a cluster, one MMA over both tensor memories).
// No load is multicast: a TMA copy lands in the shared memory of the CTA that issues it.
#pragma once

#include "tc_common.cuh"

namespace rwkvq {
namespace tc {

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// address of `local` in the shared memory of CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled load into THIS CTA's shared memory whose bytes are counted on the barrier of the pair's leader CTA
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, int x, int y, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {      // the same warp in both CTAs
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// all MMAs issued so far by this thread have completed -> arrive on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
    const unsigned short mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
// mbar_arrive_cluster by lane 0 of a whole warp, predicated instead of branched around, and without ordering ordinary memory: for a
// warp whose only work behind the barrier is tensor-memory loads and stores, completed (tcgen05.wait) and fenced
// (tc_fence_before_sync).  A release at cluster scope waits for everything the thread has in flight, about 0.4 us, which a
// barrier of every step cannot afford.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t}"
                 ::"r"(cluster_addr), "r"(lane) : "memory");
}
// The end of a pair's producer warp: waits until every stage of its ring has been released.  A multicast commit arrives in both CTAs
// on its own time, and the last ones on a stage's barrier release nothing that a later step would wait for: without this a CTA could
// leave while the peer's commit is still on its way into what is then another CTA's shared memory.  `rp` is the step after the last
// one; a stage that was never used passes at once (its barrier is in phase 0).  The result is the warp's.
__device__ __forceinline__ bool pair_drain_ring(uint64_t* empty, RingPos rp, int stages, const volatile int* abort_flag, unsigned long long limit_ns) {
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < stages && ok; ++i, rp.next(stages)) ok = mbar_wait(&empty[rp.i], rp.phase ^ 1, abort_flag, limit_ns);
    return __all_sync(0xffffffffu, ok);
}

}  // namespace tc
}  // namespace rwkvq
