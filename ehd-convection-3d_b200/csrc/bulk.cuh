// bulk.cuh -- bulk copies global -> shared on mbarriers, and the e_y, e_z of a
// run-time direction, for the row kernels.
#pragma once

#include "common.cuh"

namespace ehd {

namespace {

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned phase) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}
// one contiguous global -> shared copy completing on the barrier; both
// addresses 16-byte aligned and the size a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes,
                                         unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

constexpr unsigned kWaitLimit = 1u << 24;  // try_wait polls before giving up

// e_y + 1 and e_z + 1 of all directions, 2 bits per direction, for lookups
// with a run-time d (a constexpr table indexed at run time lands in local
// memory)
constexpr unsigned long long pack_e(int comp) {
    unsigned long long v = 0;
    for (int d = 0; d < Q; ++d)
        v |= (unsigned long long)((comp == 1 ? ey_of(d) : ez_of(d)) + 1) << (2 * d);
    return v;
}
constexpr unsigned long long kEyPack = pack_e(1), kEzPack = pack_e(2);
__device__ __forceinline__ int ey_rt(int d) { return (int)((kEyPack >> (2 * d)) & 3u) - 1; }
__device__ __forceinline__ int ez_rt(int d) { return (int)((kEzPack >> (2 * d)) & 3u) - 1; }

}  // namespace

}  // namespace ehd
