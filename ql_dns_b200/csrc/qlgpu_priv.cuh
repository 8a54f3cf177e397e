// qlgpu_priv.cuh -- allocation of Blackwell tensor memory (TMEM) as per-thread
// scratch.  Warp w owns TMEM lanes 32*(w%4)..+31 (the 32x32b access shape); a
// thread's values are consecutive 32-bit columns of its own lane.  tcgen05.ld /
// tcgen05.st are warp-wide (.sync.aligned), so every call is warp-convergent.
#pragma once
#include <cstdint>

namespace qlgpu {

__device__ __forceinline__ void tmem_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// One full warp allocates ncols (power of two, 32..512) and writes the base to *dst.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(d), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(ncols) : "memory");
}

}  // namespace qlgpu
