// What kernels on pairs of CTAs (clusters of two, tcgen05 cta_group::2) share: barriers and stores of the other CTA,
// bounded waits that give up in both, per-CTA loads signalled on the first CTA, the MMA over both SMs and
// its commit.  CTAS = 1 gives the same code on single CTAs.
#pragma once
#include "omni_ptx.cuh"

namespace {

// ------------------------------------------------------------------ cluster-scope helpers
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the same offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrive on a barrier that may live in the peer CTA (shared::cluster address)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same with the default ordering (release at CTA scope): for arrivals that only say "done"
// -- a stage was consumed, copies into this CTA's own shared memory have landed -- and publish no
// data written through the generic proxy into another CTA.  A cluster-scope release costs
// hundreds of nanoseconds and these arrivals sit on the per-stage critical path.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t cluster_addr, int a, int b, int c, int d) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}

// What a CTA needs to give up cleanly: its own flag, its peer's, the status word.
struct Abort {
    volatile int *flag;
    uint32_t peer_flag;          // shared::cluster address of the peer's flag; 0 without a peer
    uint32_t *status;
    __device__ __forceinline__ void raise(uint32_t bits) const {
        *flag = 1;
        if (peer_flag) st_cluster_u32(peer_flag, 1u);
        atomicOr(status, bits);
    }
};

// Bounded wait on a barrier of this CTA by a whole warp.  False: the limit ran out or someone in the pair gave up.
// CLUSTER: acquire at cluster scope, for the one hand-over whose data another CTA wrote with
// ordinary stores (the item ring); everything else is signalled by the asynchronous units.
// The lanes stay together: the vote makes the outcome, and with it every stage counter and address of the loop around it, uniform for
// the compiler, and nothing is called.  us, waits lane by lane with a function behind the first polls, in the epilogue, gather and softmax
// warps -> these, in turn, each alone under its own clock, on two GPUs: attention half of 37 tokens 29.1 -> 28.7 and 28.9 -> 28.7, 300 48.5 -> 47.4
// and 48.3 -> 47.6, 1030 in 6 records 64.9 -> 64.3 and 65.2 -> 64.6, 16384 in 16 839 -> 827 and 860 -> 849; MoE block the same within 0.7 %.
// (Spills are not the reason: the expert kernels have none either way, and attention_kernel reloads 120 bytes where it reloaded 52.)
template <bool CLUSTER>
__device__ __forceinline__ bool xwait_warp(uint32_t bar, uint32_t parity, const Abort &ab) {
    uint64_t t0 = 0;
    for (int i = 0;; i++) {
        if (__all_sync(0xffffffffu, CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity))) return true;
        if ((i & 63) == 63) {
            if (__any_sync(0xffffffffu, *ab.flag)) return false;
            const uint64_t t = globaltimer_ns();
            if (!t0) t0 = t;
            if (__any_sync(0xffffffffu, t - t0 > WAIT_LIMIT_NS)) {
                if (elect_one()) ab.raise(OMNI_ST_TIMEOUT);
                return false;
            }
        }
    }
}
__device__ __forceinline__ int uniform_i32(int v) { return __reduce_min_sync(0xffffffffu, v); }

// The same for a wait that is long as a rule and in no hurry: sleeps between polls, so that the
// warp does not take issue slots from the epilogue warps of its scheduler.
__device__ __forceinline__ bool xwait_lazy(uint32_t bar, uint32_t parity, const Abort &ab) {
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        __nanosleep(100);
        if (*ab.flag) return false;
        if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) { ab.raise(OMNI_ST_TIMEOUT); return false; }
    }
    return true;
}

// TMA loads whose completion is signalled on a barrier of the pair's first CTA.  Each CTA
// issues its own loads into its own shared memory: nothing here is a multicast.
template <int CTAS>
__device__ __forceinline__ void xtma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar, uint64_t policy) {
    if (CTAS == 2)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "l"(policy) : "memory");
    else
        tma_load_2d_hint(dst, map, x, y, bar, policy);
}
template <int CTAS>
__device__ __forceinline__ void xtma_4d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, int w, uint32_t bar, uint64_t policy) {
    if (CTAS == 2)
        asm volatile(
            "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w), "l"(policy) : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w), "l"(policy) : "memory");
}

template <int CTAS>
__device__ __forceinline__ void xtmem_alloc(uint32_t dst_smem, uint32_t cols) {
    if (CTAS == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        tmem_alloc(dst_smem, cols);
        tmem_relinquish();
    }
}
template <int CTAS>
__device__ __forceinline__ void xtmem_dealloc(uint32_t addr, uint32_t cols) {
    if (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
    else tmem_dealloc(addr, cols);
}
// D[tmem] (+)= A[smem] . B[smem]^T.  With CTAS = 2 the instruction spans both SMs of the pair:
// A = 128 rows per CTA, B = N/2 rows per CTA, at the same shared-memory offsets in both.
template <int CTAS>
__device__ __forceinline__ void xmma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if (CTAS == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    else
        umma_bf16(d_tmem, a_desc, b_desc, idesc, accumulate);
}
// One arrival on the barrier at this offset in EVERY CTA of the pair once all MMAs issued so far
// by this thread have completed (a barrier signal to both CTAs, not a data transfer).
template <int CTAS>
__device__ __forceinline__ void xcommit(uint32_t bar) {
    if (CTAS == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        umma_commit(bar);
}

}  // namespace
