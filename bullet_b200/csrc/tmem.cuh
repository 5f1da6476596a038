// Tensor memory as storage: each warp of a CTA reads and writes the 32 lanes (warp % 4) of its columns, one 32-bit word per lane
// and column.  256 KB per SM beside shared memory, with a data path of its own.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// One whole warp: all 512 columns, which start at column 0 (`word`: where the instruction writes that).  Waits while another CTA
// of the SM holds any.  Other warps may use them behind a barrier.
__device__ __forceinline__ void tmem_alloc_all(uint32_t* word) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"((uint32_t)__cvta_generic_to_shared(word)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_all() { asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(0)); }
// `columns` columns of the lanes of warp `warp` that no other warp of the CTA is given
__device__ __forceinline__ uint32_t tmem_own(int warp, int columns) { return (uint32_t)(warp & 3) << 21 | (uint32_t)(columns * (warp >> 2)); }

// Whole warps, converged.  What was put may be got by the same warp after tmem_stored().
__device__ __forceinline__ void tmem_put8(uint32_t at, const float4& a, const float4& b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(at), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ void tmem_stored() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Two neighbouring fours.  (The wait is part of the statement: nothing reads the words before they have arrived.)
__device__ __forceinline__ void tmem_get8(uint32_t at, float4& a, float4& b) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\ntcgen05.wait::ld.sync.aligned;"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "r"(at)
                 : "memory");
}

}  // namespace b200
