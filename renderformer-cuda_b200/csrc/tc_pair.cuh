// Inline-PTX helpers for kernels on CTA pairs (clusters of two, tcgen05 cta_group::2): cluster barrier and addresses, copies whose
// bytes count on the pair's first CTA, products over both CTAs' operands, tile stores from shared memory. sm_100a only.
#pragma once
#include "attention_tc.cuh"

namespace rfk {
namespace pair_ptx {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the location `smem_addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// its two halves, for work between them; every thread of both CTAs makes each once, whole warps together
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// An arrival on a barrier of the pair's other CTA, and the waiting side's poll for such arrivals. Both name the cluster: the default scope is
// the CTA, which orders nothing between the accumulator reads of one CTA's threads and the products that the other issues into it next.
__device__ __forceinline__ void remote_arrive(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool poll_remote(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(tc::smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Waits of one thread and of a whole warp for a phase that other CTAs' threads arrive for and that no other can follow yet: nearly always
// over, so that one poll is all; behind a wait of the CTA's scope a last poll acquires for the cluster.
__device__ __forceinline__ bool wait_remote(uint64_t* bar, uint32_t parity, volatile int* abort) {
    if (poll_remote(bar, parity)) return true;
    return tc::mbar_wait_slow(bar, parity, abort) && poll_remote(bar, parity);
}
__device__ __forceinline__ bool wait_remote_warp(uint64_t* bar, uint32_t parity, volatile int* abort) {
    if (__all_sync(0xffffffffu, poll_remote(bar, parity))) return true;
    return tc::mbar_wait_warp(bar, parity, abort) && __all_sync(0xffffffffu, poll_remote(bar, parity));
}

// ---- shared <-> global tile copies
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until at most N of this thread's committed store groups still READ their shared-memory source
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
// per-CTA tiled copy whose bytes are counted on a barrier that may live in the pair's other CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst_smem, const void* tmap, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}

// ---- tensor memory of both CTAs: one whole warp in each of the two issues these together (every tcgen05 instruction of a kernel names
// the same cta_group); each CTA gets its address in its own shared memory
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_addr(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- products and their completion
__device__ __forceinline__ void umma_pair_f16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(tc::kDescHiSw128) : "memory");
}
// one arrival on the barrier at this shared-memory offset in BOTH CTAs of the pair when every product issued so far is complete
__device__ __forceinline__ void umma_pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(tc::smem_addr(bar)), "h"((uint16_t)3) : "memory");
}
// bounded pause on the abort path: lets copies that were started a moment ago land
__device__ __forceinline__ void drain_pause() {
    const uint64_t t0 = tc::global_timer_ns();
    for (int i = 0; i < 4096 && tc::global_timer_ns() - t0 < 50000; ++i) __nanosleep(256);
}

// Byte offset of 16-byte chunk j (0..7) of row r (0..31) inside a staging buffer of 32 rows x 128 bytes (SWIZZLE_128B box layout).
__device__ __forceinline__ uint32_t staged(int r, int j) { return (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)); }

}  // namespace pair_ptx
}  // namespace rfk
