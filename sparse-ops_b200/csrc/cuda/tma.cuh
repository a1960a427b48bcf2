// tma.cuh -- bulk tensor copies (TMA) into shared memory with bounded waits, shared by the kernels
// that stage a dense operand (conv.cu, spmm_tile.cu).
#pragma once

#include "common.cuh"

#include <cuda.h>            // CUtensorMap and its enums only; the encoder is looked up at run time
#include <cudaTypedefs.h>

namespace spx {

// One thread asks the copy unit for a whole box; the unit writes it into shared memory (zeros where
// the box leaves the tensor) and signals an mbarrier with the byte count.  No multicast, the tensor
// maps cover this GPU's own operands only.
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
                   "r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(map), "r"(c0), "r"(c1),
                   "r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
// Arrives, and returns how many arrivals of the phase were pending before this one.
__device__ __forceinline__ uint32_t mbar_arrive_pending(uint64_t* bar) {
    uint32_t pending;
    asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.shared::cta.b64 s, [%1];\n\tmbarrier.pending_count.b64 %0, s;\n\t}"
                 : "=r"(pending) : "r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
    return pending;
}
// Acquires the arrivals of a phase that is known to be complete.
__device__ __forceinline__ void mbar_acquire(uint64_t* bar, uint32_t parity) {
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%0], %1;\n\t}"
                 ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(parity) : "memory");
}
// Waits for the phase with the given parity; gives up one second (of the GPU's wall clock) after
// its 256th unsuccessful poll and returns false, so a copy that never completes cannot hang the GPU.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
    uint64_t t0 = 0;
    for (uint32_t i = 1;; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(a), "r"(parity) : "memory");
        if (done) return true;
        if ((i & 255u) == 0) {
            uint64_t now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > 1000000000ull) return false;
        }
    }
}

// The two words of a handle through which a kernel reports a bounded wait that ran out: one in device
// memory, which CTAs that start later read and leave on, and one in pinned host memory (only ever
// written by the kernels: a read of host memory costs an SM about a microsecond), which the next call
// that would use bulk copies on the handle reports.  Absent (null) when they cannot be allocated.
void ensure_tma_words(spx_ell* e);
// SPX_ERR_CUDA once after a wait on the handle ran out (bulk copies are then off for the handle).
int check_tma_words(spx_ell* e, const char* what);
// cuTensorMapEncodeTiled, looked up through the runtime (the library does not link libcuda); null when absent.
PFN_cuTensorMapEncodeTiled tensor_map_encoder();

}  // namespace spx
