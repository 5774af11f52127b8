// tcgen05 / tensor-memory PTX wrappers and descriptors shared by the tensor-core kernels
// (gemm_tcgen05.cu: bf16 and tf32 contractions; bool_tcgen05.cu: 8-bit integer counts).
#pragma once
#include "common.cuh"
#include "pair_exit.cuh"

namespace tpw {
namespace {

constexpr uint32_t kSpinLimit = 1u << 26;

// ---- PTX wrappers (tcgen05) ---------------------------------------------------------------------
// CTA pairs (cta_group::2): two CTAs of a cluster, on neighbouring SMs, work on one tile of twice the rows: each holds its own
// rows of A, half of the rows of B and the accumulator of its own rows, so B crosses L2 -> SM once per pair.  Rank 0 issues the
// MMAs for both; the copies of both complete on rank 0's barriers, and a commit arrives at the same barrier of both CTAs.
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of rank `rank`'s copy of a shared variable
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar) {   // arrives at this barrier in both CTAs
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}
// the same for a CTA by itself
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    if (PAIR)
        tc_commit_pair(bar);
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                     : "memory");
}
// copy into this CTA's shared memory that completes on a barrier of the pair (shared::cluster address)
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, uint32_t cluster_bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(cluster_bar)
        : "memory");
}
// Shared memory written by threads and then read by the copy engine; 3-D tiled store shared -> global as a bulk async-group (the tensor
// map clips what lies outside the tensor; c0 must keep c0 * element size a multiple of 16 bytes and no coordinate may be negative),
// its commit, and the wait until every committed store has read its shared-memory source.
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// try_wait on a barrier at which threads of the other CTA arrive
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives lane (base + t)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes, 128-byte swizzle:
// start address >> 4 in bits [0,14), stride between 8-row groups (1024 B) >> 4 in bits [32,46),
// descriptor version 1 in bits [46,48), swizzle mode 2 (128 B) in bits [61,64).  The leading
// byte offset is not used by swizzled K-major layouts (set to 1).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Raises the abort flag of both CTAs of a pair (the flag lies at the same offset in both), or of the one CTA.
__device__ __forceinline__ void raise_abort(int *abort_flag, uint32_t ctas) {
    for (uint32_t r = 0; r < ctas; ++r)
        asm volatile("st.volatile.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(abort_flag, r)), "r"(1) : "memory");
}
// Bounded mbarrier wait that also gives up when another role raised the abort flag.  PAIR: threads of the other CTA arrive too.
template <bool PAIR = false>
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    auto done = [&]() { return PAIR ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
    if (done()) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        if (done()) return true;
        if ((it & 63u) == 63u && (*abort_flag || globaltimer_ns() - t0 > kWaitBudgetNs)) return false;
    }
    return false;
}

// How far the roles of a pair came, at the same offset of both CTAs' shared memory: operand uses issued by either producer, uses
// read (their slots' empty barriers committed), accumulators handed to the epilogue.  Written once by each role when it stops.
struct PairCounts {
    uint32_t issued[2], used, filled;
};
__device__ __forceinline__ void publish(uint32_t *word, uint32_t value, uint32_t ctas) {
    for (uint32_t r = 0; r < ctas; ++r)
        asm volatile("st.volatile.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(word, r)), "r"(value) : "memory");
}
// bytes of a copy that was never issued, counted as arrived
__device__ __forceinline__ void mbar_complete_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(cluster_addr(bar, 0)), "r"(bytes) : "memory");
}
// The producer's last step in a run without errors: the commits that release the slots have arrived in this CTA (pair_exit.cuh).
__device__ __forceinline__ bool wait_for_releases(uint64_t *empty, uint32_t issued, uint32_t slots, volatile int *abort_flag) {
    for (uint32_t u = first_of_last_uses(issued, slots); u < issued; ++u)
        if (!wait_or_abort(&empty[u % slots], parity_of_use(u, slots), abort_flag)) return false;
    return true;
}
// The same after a wait that gave up, by one thread of each CTA when all roles of both have stopped: copies and commits that are still
// under way arrive, each waited for with the usual bound.  bytes(u): what one CTA copies for use u.
template <typename F>
__device__ __noinline__ void drain_pair(uint64_t *full, uint64_t *empty, uint64_t *tmem_full, uint32_t slots, volatile PairCounts *c,
                                        uint32_t rank, F bytes) {
    const uint32_t i0 = c->issued[0], i1 = c->issued[1], used = c->used, filled = c->filled;
    if (rank == 0) {
        for (uint32_t u = used; u < (i0 > i1 ? i0 : i1); ++u) {
            const PairDebt debt = debt_of_use(u, i0, i1);
            if (debt == PairDebt::arm_other) mbar_expect_tx(&full[u % slots], bytes(u));
            if (debt == PairDebt::forgive) mbar_complete_tx(&full[u % slots], bytes(u));
        }
        for (uint32_t u = used; u < (i0 > i1 ? i0 : i1); ++u) mbar_wait_bounded(&full[u % slots], parity_of_use(u, slots));
    }
    for (uint32_t u = first_of_last_uses(used, slots); u < used; ++u) mbar_wait_bounded(&empty[u % slots], parity_of_use(u, slots));
    for (uint32_t u = first_of_last_uses(filled, 2); u < filled; ++u) mbar_wait_bounded(&tmem_full[u % 2], parity_of_use(u, 2));
}

} // namespace
} // namespace tpw
