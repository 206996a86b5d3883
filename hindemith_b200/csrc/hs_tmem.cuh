// hs_tmem.cuh -- tensor memory as per-warp storage.
//
// The sweeps keep data that a warp alone writes and reads back (coefficients) in tensor memory:
// 32 lanes x 32-bit columns, 64 KB per SM sub-partition, read at about 900 B per clock and SM
// where shared memory, which the shuffles also use, delivers 128.
#pragma once

#include "hs_common.cuh"

namespace hs {

// ---- tensor memory as per-warp storage (32 lanes x 32-bit columns; warp w of a CTA reaches
// lanes 32 (w % 4) .. + 31)

__device__ __forceinline__ void tmem_st16(unsigned addr, const float (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(r[0]), "f"(r[1]), "f"(r[2]),
        "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]), "f"(r[10]),
        "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), "r"(addr));
}
__device__ __forceinline__ void tmem_ld16(float (&r)[16], unsigned addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
          "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(addr));
}
// The loaded registers hold their values after this wait; they pass through it as operands so
// that no use of them can be scheduled before it.
__device__ __forceinline__ void tmem_wait_ld(float (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]),
                   "+f"(r[7]), "+f"(r[8]), "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]),
                   "+f"(r[14]), "+f"(r[15]));
}
__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Tensor memory of a CTA: one warp allocates `cols` columns (a power of two from 32) for all.
__device__ __forceinline__ void tmem_alloc(unsigned *base, int cols) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(base);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
// After the allocating warp: every warp sees the base.
__device__ __forceinline__ unsigned tmem_base_of(const unsigned *base) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return *(volatile const unsigned *)base;
}
__device__ __forceinline__ void tmem_dealloc(unsigned base, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}

}  // namespace hs
