// Tensor Memory Accelerator (TMA) helpers for sm_100a: tensor-map encoding
// on the host and the inline-PTX bulk tensor copies / mbarrier operations the
// column passes use.  No multicast form is used anywhere.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace dk {

constexpr unsigned kWaitLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
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

// Bounded wait: gives up after `limit` polls (kWaitLimit in the kernels) and
// raises *flag, the device's flag that decon_device_status reads (conv.cu);
// the CTA then skips its compute and store.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* flag,
                                                  unsigned limit = kWaitLimit) {
    for (unsigned i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(flag, 1);
    return false;
}

// For a CTA that leaves because a wait gave up: copies of its own may still be on
// their way into shared memory that another CTA gets next.  Waits for them, bounded
// too; by one thread, after the CTA's last barrier.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    for (unsigned i = 0; i < kWaitLimit; ++i)
        if (mbar_try_wait(bar, parity)) return;
}

// 3-D tiled bulk tensor load global -> shared, completion on an mbarrier.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

// Host: rank-3 tensor map over a spectrum buffer [d2][d1][pitch] of elements
// of esize bytes (8: complex64 as two floats, 4: half2) with boxes of T
// elements x b1 x b2, no swizzle.  False if the driver entry point is
// unavailable or the encode fails.
bool encode_tile_map(CUtensorMap* map, const void* base, int esize, int64_t pitch, int64_t d1, int64_t d2,
                     int T, int b1, int b2);

}  // namespace dk
