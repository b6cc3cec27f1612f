// device_util.cuh -- small sm_100a building blocks shared by the kernels:
// streaming loads, relaxed GPU-scope flag traffic, bounded waits and the
// warp-wide decoupled look-back.
#pragma once

#include <cstdint>

#include "hgap_internal.h"

namespace hgap {

constexpr unsigned kFull = 0xffffffffu;
// A wait gives up after this long (ns of %globaltimer) and flags kDevTimeout.
constexpr uint64_t kWaitLimitNs = 500ull * 1000 * 1000;
// The same for a warp that waits for another one's look-back: that has kWaitLimitNs for
// every record that is late, so it may rightly take longer than one of them.
constexpr uint64_t kCtaWaitLimitNs = 20 * kWaitLimitNs;

__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t ld_stream_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint64_t ld_relaxed_u64(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_u64(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ------------------------------------------- bulk copies into shared memory --
// One-dimensional bulk copy (the TMA engine, no tensor map) from global to
// this CTA's shared memory, completing on an mbarrier with a byte count.
// Both addresses 16-byte aligned, size a multiple of 16; the copy lands in this
// CTA alone.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Per-thread asynchronous 16-byte copies from global to this CTA's shared
// memory (no registers held): a thread waits for its own copies with
// cp_async_wait_all, and a CTA barrier after that shows them to the others.
// Both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst_smem)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// makes initialised mbarriers visible to the async proxy (bulk copies)
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// orders this thread's earlier generic-proxy shared accesses (made visible to
// it by a CTA barrier) before a following bulk copy into the same bytes
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// A barrier of `threads` of the CTA's threads (whole warps), the others not taking part.
__device__ __forceinline__ void named_barrier(uint32_t id, uint32_t threads) {
    asm volatile("barrier.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Counts towards that barrier without waiting for it.
__device__ __forceinline__ void named_barrier_arrive(uint32_t id, uint32_t threads) {
    asm volatile("barrier.arrive.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void bulk_load(void* dst_smem, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(dst_smem)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}

// The wait suspends the warp for about this long instead of spinning.
constexpr uint32_t kTryWaitNs = 20000;

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(kTryWaitNs)
        : "memory");
    return ok != 0;
}

// Waits for the phase of `bar` with the given parity to complete.  Bounded:
// after limit_ns it flags kDevTimeout and returns false; with `bail`, a wait
// of more than kBailNs also gives up as soon as a timeout is already flagged
// (the kernel's output is void then, and it only has to finish).  The lanes of
// a warp give up each on its own clock.
constexpr uint64_t kBailNs = 200000;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* status, bool bail,
                                          uint64_t limit_ns = kWaitLimitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        const uint64_t waited = global_timer_ns() - t0;
        if (waited > limit_ns || (bail && waited > kBailNs && (ld_relaxed_u32(status) & kDevTimeout))) {
            atomicOr(status, kDevTimeout);
            return false;
        }
    }
}

// The wait limit of a launch's look-back waits (the test hook may shorten it).
__device__ __forceinline__ uint64_t wait_limit(const LookbackHook& h) {
    return h.wait_ns ? h.wait_ns : kWaitLimitNs;
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
    return v;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, d);
        if (lane >= (uint32_t)d) v += t;
    }
    return v;
}

// Single-pass decoupled look-back (the reference's scheme,
// encoder/src/encoder.cu:222-263, decoder/src/decoder.cu:601-638) run by one
// full warp, with a window of 32 predecessors per round trip, one a lane, the
// nearest in lane 0.  One load a lane: all look-backs read the same few lines,
// and a wider window costs each of them more than the round trips it saves
// (decoder, 32 / 64 / 128 records: Zipf(1.2) 256 MiB 443 / 453 / 479 us, BF16
// mantissa 371 / 378 / 392).
// Only the records between the tile and the nearest inclusive prefix matter.
// The window is loaded without blocking; records in front of the nearest
// unpublished one are summed at once and left behind, and the next window
// starts at that one, so a wait costs one round trip after its record appears
// (waiting for one record at a time and then loading the window again
// took one of these cycles per late predecessor).
// Publishing the aggregate and resolving the prefix are separate steps, so a
// CTA can publish a tile's aggregate, decode its next tile, and resolve the
// first tile afterwards, when its predecessors have long been published.
// `first`: the tile starts its own scan (tile 0, or a batched job's first
// tile); it publishes its inclusive prefix at once and resolves to 0, so no
// look-back ever crosses into another job's tiles.
__device__ __forceinline__ void lookback_publish(uint64_t* rec, uint64_t tile, uint64_t agg, bool first) {
    st_relaxed_u64(rec + tile, (first ? kFlagP : kFlagA) | (agg & kValueMask));
}

// `limit_ns` bounds the wait for each record; `publish` = false keeps the
// inclusive prefix unpublished (the bounded-wait test hook only: LookbackHook).
__device__ __forceinline__ uint64_t lookback_resolve(uint64_t* rec, uint64_t tile, uint64_t agg, bool first,
                                                     uint32_t* status, uint32_t lane, uint64_t limit_ns,
                                                     bool publish = true) {
    if (first) return 0;
    uint64_t excl = 0, t0 = 0;
    int64_t top = (int64_t)tile - 1;
    for (;;) {
        const int64_t i = top - (int64_t)lane;
        const uint64_t v = i >= 0 ? ld_relaxed_u64(rec + i) : kFlagP;
        // the window's nearest inclusive prefix / unpublished record
        const uint32_t pmask = __ballot_sync(kFull, (v & kFlagP) != 0), zmask = __ballot_sync(kFull, v == 0);
        const int gp = pmask ? __ffs(pmask) - 1 : 32, gz = zmask ? __ffs(zmask) - 1 : 32;
        const int take = gz < gp ? gz : gp < 32 ? gp + 1 : 32;  // records to sum
        excl += warp_sum_u64((int)lane < take ? v & kValueMask : 0);
        if (gp < gz) break;
        top -= take;
        if (take) {
            t0 = 0;
        } else {  // the nearest record is unpublished: bounded
            const uint64_t now = global_timer_ns();
            bool give_up = false;
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) give_up = true;
            if (__any_sync(kFull, give_up)) {
                if (lane == 0) atomicOr(status, kDevTimeout);
                return excl;
            }
            if (ld_relaxed_u32(status) & kDevTimeout) return excl;  // given up elsewhere: the status says so
        }
    }
    if (lane == 0 && publish) st_relaxed_u64(rec + tile, kFlagP | ((excl + agg) & kValueMask));
    return excl;
}

}  // namespace hgap
