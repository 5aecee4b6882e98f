// Thin wrappers over the sm_100a bulk-copy (TMA) and mbarrier PTX used by the streaming kernels.
// Every wait is bounded: after kSpinLimit failed polls the caller records an error and moves on,
// so a missed completion can never hang the GPU.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace runit {

constexpr uint32_t kSpinLimit = 1u << 16;   // polls of mbarrier.try_wait (each may suspend for a while)

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint32_t bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Returns false if the phase did not complete within the spin limit.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSpinLimit; i++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// For the thread that starts copies (or MMAs) 0 .. issued - 1, in order, on a ring of `ring` barriers: waits (bounded) for those that can
// still be in flight, so that nothing arrives after a block that gave up has handed back its shared and tensor memory.
__device__ __forceinline__ void mbar_drain(uint32_t bars, uint32_t ring, uint32_t issued) {
    for (uint32_t i = issued < ring ? 0 : issued - ring; i < issued; i++) mbar_wait(bars + 8 * (i % ring), (i / ring) & 1);
}
// The same for copies that are counted on no barrier that the thread could wait on (a peer CTA's): some two milliseconds, a thousand times what a
// copy takes.
__device__ __forceinline__ void copies_settle() {
    const long long t0 = clock64();
    while (clock64() - t0 < (1ll << 22)) __nanosleep(1000);
}
// 2-D tiled load: box (c0 = innermost coordinate in elements, c1 = row) -> dense shared tile.
// c0 * element size must be a multiple of 16 bytes; dst must be 128-byte aligned.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
// 2-D tiled store of a dense shared tile, in the executing thread's bulk group; the same rule for c0.  Rows and columns outside the tensor are not
// written.  Generic writes to the tile need fence_proxy_async before.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int32_t c0, int32_t c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(src)
                 : "memory");
}
// 1-D bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Thread-block clusters: rank of this CTA in its cluster, cluster-wide barrier, and a float read from the
// shared memory of another CTA of the cluster (distributed shared memory).
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(const float* local_smem_ptr, uint32_t cta_rank) {
    uint32_t laddr = (uint32_t)__cvta_generic_to_shared(local_smem_ptr), raddr;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(laddr), "r"(cta_rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(raddr) : "memory");
    return v;
}

// Programmatic dependent launch (griddepcontrol): no-ops when the kernel was launched without the attribute.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace runit
