// peer_out.cuh -- where the SpMM kernels' epilogue stores its finished vectors.
#pragma once

#include "common.cuh"

namespace spx {

constexpr int kMaxPeers = 8;

// Destinations of the epilogue.  Plain SpMM: one pointer (this GPU's Y).  Row-sharded SpMM with
// the all-gather fused in: the full Y buffer of every rank (this GPU's own and its peers' buffers
// mapped over NVLink); each finished output vector is stored to all of them with ordinary 16-byte
// stores, so the exchange overlaps the multiply instead of following it.
struct PeerOut {
    float* p[kMaxPeers];
    int n;
    int mcast;          // p[0] is an NVLink multicast address: one multimem.st reaches every rank's buffer
    uint64_t row0;      // first row of this rank's slab inside the full buffers
};

// One finished vector to every destination.  Peer list: one ordinary 16-byte store per buffer (the
// GPU sends the vector once per peer).  Multicast address: a single multimem.st, replicated to all
// bound GPUs (this one included) by the NVSwitch, so the vector leaves this GPU once.
__device__ __forceinline__ void store_out(const PeerOut& out, size_t at, const float4& o) {
    if (out.mcast) {
        asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};"
                     ::"l"(out.p[0] + at), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
        return;
    }
#pragma unroll
    for (int g = 0; g < kMaxPeers; ++g)
        if (g < out.n) *reinterpret_cast<float4*>(out.p[g] + at) = o;
}
__device__ __forceinline__ void store_out(const PeerOut& out, size_t at, float o) {
    if (out.mcast) {
        asm volatile("multimem.st.relaxed.sys.global.f32 [%0], %1;" ::"l"(out.p[0] + at), "f"(o) : "memory");
        return;
    }
#pragma unroll
    for (int g = 0; g < kMaxPeers; ++g)
        if (g < out.n) out.p[g][at] = o;
}

}  // namespace spx
