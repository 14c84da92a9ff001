// mbarrier and bulk-copy (TMA, non-tensor form) primitives for sm_100a, as inline PTX.
// Only the plain global -> shared::cta bulk copy is used: no cluster multicast anywhere.
// Every wait is bounded: after the limit the caller records a status and leaves.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace lg {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: each try_wait itself blocks for a hardware-defined slice, so ~2^20 rounds is far
// beyond any legitimate delay (tens of milliseconds at least) and still ends by itself.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 20); it++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (it > 64) __nanosleep(64);
    }
    return false;
}

// Plain bulk copy global -> this CTA's shared memory; completion is counted on an mbarrier.
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Tiled TMA load of a 3-D box (global -> this CTA's shared memory), no multicast; completion is
// counted on an mbarrier.  dst 128-byte aligned; coordinate x times the element size a multiple of 16 B.
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_prefetch_descriptor(const void* tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// `size` bytes (all or none: then src is not read) and zeros behind them
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t size) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, uint32_t size) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}

// Arrival of a CTA at a counter in global memory, by one thread behind a barrier: orders what the whole CTA wrote before that
// barrier against what the last arriver's CTA reads behind the barrier that follows.  With this
// instead of a fence by every thread, and one more by every thread of the last CTA, calls back to back on one weight: 4096 x 4096, q = 3, one row 5.53 -> 4.92 us, 12288
// x 12288 17.56 -> 16.95, two rows of 8192 x 8192, q = 2 11.6 -> 10.3, 16 rows (gemm_tc) 22.4 -> 21.8, 128 rows (gemm_hl) 33.0 -> 31.8.
__device__ __forceinline__ unsigned arrive_acq_rel(unsigned* counter) {
    unsigned prev;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
    return prev;
}

}  // namespace lg
