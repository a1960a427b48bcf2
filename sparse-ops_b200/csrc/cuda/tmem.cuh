// tmem.cuh -- tensor memory as a store of gathered operands.
//
// An SM's tensor memory is 128 lanes x 512 columns of 4 bytes; a warp reaches the 32 lanes of its quadrant (warp
// index % 4), lane l of the warp the tensor-memory lane l.  A load names a column, the same for the whole warp:
// consecutive columns from it arrive in consecutive registers of each lane.  So an operand whose place is the same for
// all lanes of a warp -- the input under a tap of a sparse convolution -- can come from there: 16 columns take 11.6
// clocks per quadrant, 704 bytes per clock and SM, where shared memory delivers 128 (measured).
#pragma once

#include "common.cuh"

namespace spx {

constexpr uint32_t kTmemColumns = 512;

// By one whole warp; the address of the first column is left in shared memory.  Waits in hardware while another
// kernel's CTA on the SM holds columns: not to be called before pdl_wait(), or each could wait for the other.
__device__ __forceinline__ void tmem_alloc_all(uint32_t* at) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(at)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_all(uint32_t tmem) {       // by the warp that allocated
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}
// Loads and stores are asynchronous: a value is there after the wait, and other threads see what was stored after
// wait, fence_before, a barrier, fence_after.
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(float (&v)[8], uint32_t at) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(at));
}
__device__ __forceinline__ void tmem_st8(uint32_t at, const float (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(at), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// Waits for this thread's loads; the values pass through it, so that nothing uses them before.
template <int G>
__device__ __forceinline__ void tmem_wait_ld(float (&v)[G][8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < G; ++g)
        asm volatile("" : "+f"(v[g][0]), "+f"(v[g][1]), "+f"(v[g][2]), "+f"(v[g][3]), "+f"(v[g][4]), "+f"(v[g][5]), "+f"(v[g][6]), "+f"(v[g][7]));
}

}  // namespace spx
