// spmm.cu -- ELLPACK SpMM  Y = act(bias + E * X)  for sm_100a.
//
// Replaces ellpack_matmul_fused<USE_MASK,FUSE_RELU> of the reference
// (src/ellpack_matmul.cpp:11-92).  Arithmetic contract kept from the reference: every output
// element starts from bias[i] (or 0) and receives ONE fused multiply-add per stored nonzero
// of row i, in storage order (:56-66); the activation follows (:68-70).  A thread owns whole
// output elements, so the result is bit-identical to the reference for every C, and no
// padding slot is ever multiplied.
//
// Kernels (launch_spmm_bcast chooses):
//   spmm_chain, spmm_direct   X fits in shared memory: staged whole, chains fed from there
//   spmm_tile_kernel          (spmm_tile.cu) columns are used often enough by the rows of a CTA to stage X
//                             block by block
//   spmm_rows                 everything else: rows of X gathered through L1 / L2
//   spmm_gather_half          44 <= C <= 128 and many short rows
//   spmm_gather_staged        a few long rows decide the duration (row shard of a skewed matrix)
// Column panels are the slow grid dimension so that all CTAs in flight work on the same X panel.
// Rows are taken from the handle's sorted row schedule (longest first), so the warps of a CTA
// and the CTAs of a wave carry equal work.
#include "common.cuh"
#include "peer_out.cuh"
#include "tma.cuh"

#include <algorithm>
#include <cstdlib>

namespace {

using spx::PeerOut;
using spx::kMaxPeers;
using spx::store_out;

constexpr int kGatherWarps = 8;

// Linear block id -> (row block, column panel).  Normally panel-major: all row blocks of panel 0,
// then panel 1, ... so that the CTAs in flight share one panel of X in L2.  The first `head` row
// blocks (the longest rows of the sorted schedule) can instead be issued first, for all panels:
// a long row is one dependent chain of gathers, and when the whole kernel is only a few such chains
// long, a chain that starts with the last panel would end well after everything else.
struct BlockMap {
    uint32_t blocks;      // grid size
    uint32_t row_blocks;  // CTAs per panel
    uint32_t panels;
    uint32_t head;        // row blocks issued first, panel-minor
};

__device__ __forceinline__ void decode_block(const BlockMap& bm, uint32_t b, uint32_t& rb, uint32_t& panel) {
    const uint32_t head_blocks = bm.head * bm.panels;
    if (b < head_blocks) {
        rb = b / bm.panels;
        panel = b % bm.panels;
    } else {
        const uint32_t t = b - head_blocks, rest = bm.row_blocks - bm.head;
        panel = t / rest;
        rb = bm.head + t % rest;
    }
}

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

__device__ __forceinline__ void fma4(float4& a, float w, const float4& x) {
    a.x = fmaf(w, x.x, a.x);
    a.y = fmaf(w, x.y, a.y);
    a.z = fmaf(w, x.z, a.z);
    a.w = fmaf(w, x.w, a.w);
}

// ---------------------------------------------------------------------------------------
// spmm_gather_staged: the kernel for matrices whose longest rows decide the duration (few rows
// per GPU, skewed lengths: a row shard of a power-law matrix).  Same chain per output element
// as the other kernels.  Differences: (1) the first `head` row blocks of the schedule -- the rows
// with 512 and more stored entries -- are issued first, for all their panels, and run on
// 128-column panels with eight rows of X in flight per round trip; all other row blocks follow
// panel-major on 256-column panels with four.  (2) A row's (w, idx) slab travels 32 entries at a
// time, one batch ahead, through a double-buffered 256-byte staging area of the warp in shared
// memory (cp.async) and is handed to the lanes with 16-byte broadcast loads, one per four
// entries, instead of two shuffles per entry: the chain of a long row no longer waits for slab
// reads.  (3) Loads and FMAs carry the predicate "entry exists"; nothing is zero-filled.
// ---------------------------------------------------------------------------------------
struct StagedMap {
    uint32_t blocks;        // grid size
    uint32_t row_blocks;    // row blocks (one row per warp)
    uint32_t head;          // row blocks on the narrow path, issued first, panel-minor
    uint32_t head_panels;   // 128-column panels
    uint32_t panels;        // panels of the other row blocks: 256 columns, or 128 when all_narrow
    uint32_t all_narrow;    // every row on 128-column panels (panel-major, so one 128-column panel of X is in use at a time)
    uint32_t rest_ascending;    // the rows behind the head run shortest first (see launch_spmm_bcast)
};

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// One row on one panel of 128 * NV columns, G rows of X per round trip; the lane owns columns
// c0 + 128 * v + 0..3.
template <int NV, int G>
__device__ __forceinline__ void staged_row(const float* __restrict__ w, const uint32_t* __restrict__ k, uint32_t nn,
                                           const float* __restrict__ X, uint32_t c0, uint32_t C, uint32_t ldxb, float b, int act,
                                           const PeerOut& out, size_t out_at, float* sw, uint32_t* sk, int lane)
{
    static_assert(G % 4 == 0 && 32 % G == 0, "groups are made of 16-byte quads");
    bool on[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) on[v] = (c0 + 128u * v) < C;   // C % 4 == 0 on this path
    float4 acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = make_float4(b, b, b, b);
    const char* xbase = reinterpret_cast<const char*>(X + c0);

    if ((uint32_t)lane < nn) {
        cp_async4(sw + lane, w + lane);
        cp_async4(sk + lane, k + lane);
    }
    cp_async_commit();
    const uint32_t batches = (nn + 31) >> 5;
    for (uint32_t bt = 0; bt < batches; ++bt) {
        const float* bw = sw + (bt & 1) * 32;
        const uint32_t* bk = sk + (bt & 1) * 32;
        cp_async_wait_all();
        __syncwarp();       // batch bt has landed for all lanes; the other buffer is no longer read
        const uint32_t jn = (bt + 1) * 32 + lane;
        if (jn < nn) {      // next batch in flight while this one is multiplied
            cp_async4(sw + ((bt + 1) & 1) * 32 + lane, w + jn);
            cp_async4(sk + ((bt + 1) & 1) * 32 + lane, k + jn);
        }
        cp_async_commit();
        const uint32_t cnt = min(32u, nn - bt * 32);
        for (uint32_t t = 0; t < cnt; t += G) {
            float wt[G];
            uint32_t kt[G];
#pragma unroll
            for (int q = 0; q < G / 4; ++q) {
                const float4 w4 = *reinterpret_cast<const float4*>(bw + t + 4 * q);
                const uint4 k4 = *reinterpret_cast<const uint4*>(bk + t + 4 * q);
                wt[4 * q] = w4.x; wt[4 * q + 1] = w4.y; wt[4 * q + 2] = w4.z; wt[4 * q + 3] = w4.w;
                kt[4 * q] = k4.x; kt[4 * q + 1] = k4.y; kt[4 * q + 2] = k4.z; kt[4 * q + 3] = k4.w;
            }
            const uint32_t left = cnt - t;
            float4 xv[G][NV];
#pragma unroll
            for (int u = 0; u < G; ++u) {       // issue all gathers of the group first
                if ((uint32_t)u < left) {
                    const char* xr = xbase + (size_t)kt[u] * ldxb;
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (on[v]) xv[u][v] = __ldg(reinterpret_cast<const float4*>(xr + 512 * v));
                }
            }
#pragma unroll
            for (int u = 0; u < G; ++u) {       // then the FMA chain, strictly in storage order
                if ((uint32_t)u < left) {
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (on[v]) fma4(acc[v], wt[u], xv[u][v]);
                }
            }
        }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (on[v]) {
            float4 o = acc[v];
            if (act != SPX_ACT_NONE) {
                o.x = spx::apply_act(o.x, act); o.y = spx::apply_act(o.y, act);
                o.z = spx::apply_act(o.z, act); o.w = spx::apply_act(o.w, act);
            }
            const size_t at = out_at + 128 * v;
            store_out(out, at, o);
        }
    }
}

__global__ void __launch_bounds__(kGatherWarps * 32, 4)
spmm_gather_staged(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                   const uint2* __restrict__ rows,
                   uint32_t m, uint32_t pitch,
                   const float* __restrict__ X, uint32_t C, uint32_t ldxb,
                   const float* __restrict__ bias, int act, PeerOut out, uint64_t ldy, StagedMap sm)
{
    extern __shared__ __align__(16) float s_stage[];           // per warp: 64 weights, then 64 column ids
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* s_w = s_stage + warp * 128;
    uint32_t* s_k = reinterpret_cast<uint32_t*>(s_w + 64);
    const uint32_t head_blocks = sm.head * sm.head_panels;
    const bool narrow = blockIdx.x < head_blocks;
    uint32_t rb, panel;
    if (narrow) {
        rb = blockIdx.x / sm.head_panels;
        panel = blockIdx.x % sm.head_panels;
    } else {
        const uint32_t t = blockIdx.x - head_blocks, rest = sm.row_blocks - sm.head;
        panel = t / rest;
        rb = sm.head + t % rest;
    }
    uint32_t slot = rb * (blockDim.x >> 5) + warp;
    if (slot >= m) return;                      // whole warp leaves together
    if (!narrow && sm.rest_ascending) {
        const uint32_t first = sm.head * (blockDim.x >> 5);      // schedule slots [first, m) in reverse
        slot = first + (m - 1 - slot);
    }
    const uint2 ri = __ldg(rows + slot);
    const uint32_t row = ri.x;
    const float b = bias ? __ldg(bias + row) : 0.0f;
    const uint32_t nn = ri.y;
    const float* __restrict__ w = Wd + (size_t)row * pitch;
    const uint32_t* __restrict__ k = idx + (size_t)row * pitch;
    const size_t out_row = (size_t)(out.row0 + row) * ldy;
    if (narrow || sm.all_narrow) {
        const uint32_t c0 = panel * 128u + 4u * lane;
        staged_row<1, 8>(w, k, nn, X, c0, C, ldxb, b, act, out, out_row + c0, s_w, s_k, lane);
    } else {
        const uint32_t c0 = panel * 256u + 4u * lane;
        staged_row<2, 4>(w, k, nn, X, c0, C, ldxb, b, act, out, out_row + c0, s_w, s_k, lane);
    }
}

// ---------------------------------------------------------------------------------------
// spmm_gather_half: short rows, 32 < C <= 128.  With a full warp per row a lane would own at most one float4 and the
// per-entry work that does not scale with the width (two shuffles, the row address, the loop)
// would be spread over 4 FMAs; here 16 lanes share a row and own NV float4 each, a warp carries
// two neighbouring rows of the sorted schedule, and every shuffle / address / load instruction
// serves both rows.  Same chain per output element.
// ---------------------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(kGatherWarps * 32, 4)
spmm_gather_half(const float* __restrict__ Wd, const uint32_t* __restrict__ idx, const uint2* __restrict__ rows,
                 uint32_t m, uint32_t pitch,
                 const float* __restrict__ X, uint32_t C, uint64_t ldx,
                 const float* __restrict__ bias, int act, PeerOut out, uint64_t ldy, bool early)
{
    constexpr int G = 4;                        // gathers in flight per vector
    const int lane = threadIdx.x & 31;
    const int sl = lane & 15;
    const uint32_t slot = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 2 + (lane >> 4);
    const bool live = slot < m;
    const uint2 ri = live ? __ldg(rows + slot) : make_uint2(0u, 0u);
    const uint32_t row = ri.x;
    const uint32_t c0 = 4u * sl;
    bool on[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) on[v] = live && (c0 + 64u * v) < C;

    const uint32_t nn = ri.y;
    const uint32_t nmax = __reduce_max_sync(0xffffffffu, nn);       // the warp runs to its longer row
    const float* __restrict__ w = Wd + (size_t)row * pitch;
    const uint32_t* __restrict__ k = idx + (size_t)row * pitch;
    spx::pdl_wait();
    if (early) spx::pdl_launch();
    const float b = (live && bias) ? __ldg(bias + row) : 0.0f;
    float4 acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = make_float4(b, b, b, b);

    for (uint32_t j0 = 0; j0 < nmax; j0 += 16) {
        float wl = 0.0f;
        uint32_t kl = 0;
        if (j0 + sl < nn) {                     // 64-byte slab reads per half warp
            wl = __ldg(w + j0 + sl);
            kl = __ldg(k + j0 + sl);
        }
        const uint32_t cnt = j0 < nn ? min(16u, nn - j0) : 0u;      // entries of this lane's row in the batch
        const uint32_t cmax = min(16u, nmax - j0);
        for (uint32_t t0 = 0; t0 < cmax; t0 += G) {
            float wt[G];
            float4 xv[G][NV];
#pragma unroll
            for (int u = 0; u < G; ++u) {
                wt[u] = __shfl_sync(0xffffffffu, wl, (t0 + u) & 15, 16);
                const uint32_t kt = __shfl_sync(0xffffffffu, kl, (t0 + u) & 15, 16);
                const float* xr = X + (size_t)kt * ldx + c0;
                const bool have = (t0 + u) < cnt;
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    xv[u][v] = (have && on[v]) ? ldg4(xr + 64 * v) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < G; ++u) {
                if ((t0 + u) < cnt) {
#pragma unroll
                    for (int v = 0; v < NV; ++v) fma4(acc[v], wt[u], xv[u][v]);
                }
            }
        }
    }
    spx::pdl_launch();
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (on[v]) {
            float4 o = acc[v];
            if (act != SPX_ACT_NONE) {
                o.x = spx::apply_act(o.x, act); o.y = spx::apply_act(o.y, act);
                o.z = spx::apply_act(o.z, act); o.w = spx::apply_act(o.w, act);
            }
            const size_t at = (size_t)(out.row0 + row) * ldy + c0 + 64 * v;
            store_out(out, at, o);
        }
    }
}

// ---------------------------------------------------------------------------------------
// spmm_rows: rows of X gathered through L1 / L2, any width and alignment.  A warp owns RW rows of the sorted schedule (neighbours there have near-equal lengths), G lanes each; a lane
// owns NV vectors of V floats of its row's output, vector v at columns (v * G + g) * V.  V is the
// widest vector the operands' alignment allows; G and NV are chosen by the host so that few lanes
// stay idle (C = 77: 26 lanes x 3 single columns; C = 100: 3 rows x 9 lanes x 3 vectors).
//
// The rows' slabs travel 32 entries at a time, two batches ahead, through a ring in shared memory
// (cp.async) and reach the lanes by 16-byte broadcast loads, one per four entries; per entry and warp
// that is half a shared-memory wavefront instead of the two of a shuffle hand-off.  U entries' gathers are in
// flight per round trip.  Same chain per output element as in all kernels here.
// What bounds it: bytes of gathered operands over the L2 -> SM path (4096 x 4096, 10 %, C = 256: 72 us,
// 23.8 TB/s of gathers, L1 hits among them; 84.5 us with a shuffle hand-off and predicated loads), or with few
// rows the round trips of the longest one.
// ---------------------------------------------------------------------------------------
struct RowsArgs {
    const float* Wd;
    const uint32_t* idx;
    const uint2* rows;
    uint32_t m, pitch;
    const float* X;
    uint32_t C;
    uint64_t ldx;
    const float* bias;
    int act;
    uint64_t ldy;
    uint32_t G, RW;
    BlockMap bm;
    bool early;                         // spmm_rows: let the successor in before the end
    uint32_t n, Cp, batch;              // staged X: its rows, their pitch in shared memory, entries per batch
    PeerOut out;
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// The rows of a warp and their slabs on the way into its ring in shared memory: batches of BATCH
// entries per row, RING - 1 of them ahead of the one in use.  Ring rows are BATCH + 4 floats apart, so
// that the 16-byte reads of neighbouring rows hit different banks.
struct WarpRows {
    uint2 info;                 // lane i < RW: (row, length) of the warp's row i
    uint32_t nmax, nmin;        // over the warp's rows
    __device__ __forceinline__ WarpRows(const RowsArgs& a, uint32_t slot0) {
        const uint32_t lane = threadIdx.x & 31;
        const bool have = lane < a.RW && slot0 + lane < a.m;
        info = have ? __ldg(a.rows + slot0 + lane) : make_uint2(0u, 0u);
        nmax = __reduce_max_sync(0xffffffffu, info.y);
        nmin = __reduce_min_sync(0xffffffffu, have ? info.y : 0xffffffffu);
    }
    // Asks for batch b of every row (ring slot b % RING) and closes the group, empty or not.
    template <int BATCH, int RING>
    __device__ __forceinline__ void fill(const RowsArgs& a, float* s_w, uint32_t* s_k, uint32_t b) const {
        const uint32_t lane = threadIdx.x & 31, st = b % RING, RW = a.RW;
        if (b * BATCH < nmax) {
            for (uint32_t id = lane; id - lane < RW * (BATCH / 4); id += 32) {
                const uint32_t i = id / (BATCH / 4), part = id % (BATCH / 4);
                const uint32_t row = __shfl_sync(0xffffffffu, info.x, i & 31), nn = __shfl_sync(0xffffffffu, info.y, i & 31);
                const uint32_t j = b * BATCH + part * 4;
                if (i < RW && j < nn) {         // the pitch is a multiple of 32 entries: whole quads exist
                    const size_t at = (size_t)row * a.pitch + j;
                    cp_async16(s_w + (st * RW + i) * (BATCH + 4) + part * 4, a.Wd + at);
                    cp_async16(s_k + (st * RW + i) * (BATCH + 4) + part * 4, a.idx + at);
                }
            }
        }
        cp_async_commit();
    }
    template <int BATCH, int RING>
    __device__ __forceinline__ void start(const RowsArgs& a, float* s_w, uint32_t* s_k) const {
#pragma unroll 1
        for (uint32_t b = 0; b + 1 < RING; ++b) fill<BATCH, RING>(a, s_w, s_k, b);
    }
};
constexpr int kRowsWarps = 4;       // per CTA at most
constexpr int kRowsBatch = 32, kRowsRing = 3, kRowsStride = kRowsBatch + 4;

template <int V> struct VecT;
template <> struct VecT<1> { using T = float; };
template <> struct VecT<2> { using T = float2; };
template <> struct VecT<4> { using T = float4; };
template <int V>
__device__ __forceinline__ void load_vec(float (&d)[V], const float* p) {
    const typename VecT<V>::T t = __ldg(reinterpret_cast<const typename VecT<V>::T*>(p));
    memcpy(d, &t, sizeof(t));
}


// A lane's columns of X: rows of `stride` bytes from one base address per vector (an address is one
// widening multiply-add).
template <int V, int NV>
struct Gather {
    const char* g[NV];
    uint32_t stride;
    __device__ __forceinline__ void load(float (&d)[V], uint32_t k, int v) const {
        load_vec<V>(d, reinterpret_cast<const float*>(g[v] + (uint64_t)k * stride));
    }
};

// U entries of a row on their way: issue() asks for all their operands, multiply() runs the FMA chain in
// storage order.  FULL: all U exist; otherwise the first `have` do, and the others load row 0 of X (an
// unconditional load: under a predicate the compiler waits for each load before it issues the next)
// without their FMA.
template <int V, int NV, int U>
struct RowsGroup {
    float w[U];
    float x[U][NV][V];
    template <bool FULL>
    __device__ __forceinline__ void issue(const float* bw, const uint32_t* bk, uint32_t have, const Gather<V, NV>& from) {
#pragma unroll
        for (int q = 0; q < U / 4; ++q) {
            const uint4 k4 = *reinterpret_cast<const uint4*>(bk + 4 * q);
            const float4 w4 = *reinterpret_cast<const float4*>(bw + 4 * q);
            w[4 * q] = w4.x; w[4 * q + 1] = w4.y; w[4 * q + 2] = w4.z; w[4 * q + 3] = w4.w;
            const uint32_t k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < NV; ++v) from.load(x[4 * q + u][v], FULL || 4 * q + u < have ? k[u] : 0u, v);
        }
    }
    template <bool FULL>
    __device__ __forceinline__ void multiply(float (&acc)[NV][V], uint32_t have) const {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (FULL || u < have) {
#pragma unroll
                for (int v = 0; v < NV; ++v)
#pragma unroll
                    for (int i = 0; i < V; ++i) acc[v][i] = fmaf(w[u], x[u][v][i], acc[v][i]);
            }
    }
};

template <int V, int NV, int U, int MINB, bool PIPE>
__global__ void __launch_bounds__(kRowsWarps * 32, MINB)     // MINB x 4 warps: 64, 128 or 255 registers
spmm_rows(const __grid_constant__ RowsArgs a)
{
    constexpr int kBatch = kRowsBatch, kRing = kRowsRing, kRowStride = kRowsStride;
    static_assert(U % 4 == 0 && kBatch % U == 0, "groups are made of 16-byte quads");
    extern __shared__ __align__(16) float s_ring[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t G = a.G, RW = a.RW;
    float* s_w = s_ring + (size_t)warp * (kRing * RW * kRowStride * 2);
    uint32_t* s_k = reinterpret_cast<uint32_t*>(s_w + kRing * RW * kRowStride);
    uint32_t rb = blockIdx.x, panel = 0;
    if (a.bm.panels > 1) decode_block(a.bm, blockIdx.x, rb, panel);
    const uint32_t slot0 = (rb * warps + warp) * RW;

    WarpRows wr(a, slot0);
    wr.template start<kBatch, kRing>(a, s_w, s_k);
    const uint2 info = wr.info;
    const uint32_t nmax = wr.nmax, nmin = wr.nmin, nb = (nmax + kBatch - 1) / kBatch;

    const uint32_t rl = lane / G, g = lane - rl * G;
    const bool mine = rl < RW && slot0 + rl < a.m;
    const uint32_t row = __shfl_sync(0xffffffffu, info.x, rl & 31);
    const uint32_t nn_all = __shfl_sync(0xffffffffu, info.y, rl & 31);
    const uint32_t nn = mine ? nn_all : 0u;
    const uint32_t c0 = panel * (G * NV * V) + g * V;
    bool on[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) on[v] = mine && c0 + v * G * V < a.C;
    const uint32_t lrow = mine ? rl : 0u;

    spx::pdl_wait();
    if (a.early) spx::pdl_launch();
    const float b = (mine && a.bias) ? __ldg(a.bias + row) : 0.0f;
    float acc[NV][V];
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[v][i] = b;
    Gather<V, NV> x;                            // this lane's columns; an idle vector repeats the first one
    x.stride = (uint32_t)a.ldx * 4u;
#pragma unroll
    for (int v = 0; v < NV; ++v) x.g[v] = reinterpret_cast<const char*>(a.X + (on[v] ? c0 + v * G * V : 0u));

    if constexpr (PIPE) {
        // Few warps per SM: nothing hides a warp's round trips but its own work, so there are always one or two
        // groups of U on their way.  A group's ids and weights leave the ring when its gathers are issued.
        RowsGroup<V, NV, U> ga, gb;
        const uint32_t ng = (nmax + U - 1) / U;
        auto have_of = [&](uint32_t gi) { return nn > gi * U ? nn - gi * U : 0u; };
        auto issue = [&](RowsGroup<V, NV, U>& gr, uint32_t gi) {
            const uint32_t bt = gi / (kBatch / U), t = gi % (kBatch / U) * U;
            if (t == 0) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
                __syncwarp();                   // batch bt has landed; the slot of batch bt - 1 is no longer read
                wr.template fill<kBatch, kRing>(a, s_w, s_k, bt + kRing - 1);
            }
            const uint32_t at = ((bt % kRing) * RW + lrow) * kRowStride + t;
            if ((gi + 1) * U <= nmin) gr.template issue<true>(s_w + at, s_k + at, U, x);
            else gr.template issue<false>(s_w + at, s_k + at, have_of(gi), x);
        };
        auto multiply = [&](const RowsGroup<V, NV, U>& gr, uint32_t gi) {
            if ((gi + 1) * U <= nmin) gr.template multiply<true>(acc, U);
            else gr.template multiply<false>(acc, have_of(gi));
        };
        if (ng > 0) issue(ga, 0);
        if (ng > 1) issue(gb, 1);
        for (uint32_t gi = 0; gi < ng; gi += 2) {
            multiply(ga, gi);
            if (gi + 2 < ng) issue(ga, gi + 2);
            if (gi + 1 < ng) multiply(gb, gi + 1);
            if (gi + 3 < ng) issue(gb, gi + 3);
        }
    } else {
        for (uint32_t bt = 0; bt < nb; ++bt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
            __syncwarp();                           // batch bt has landed; the slot of batch bt - 1 is no longer read
            wr.template fill<kBatch, kRing>(a, s_w, s_k, bt + kRing - 1);
            const float* bw = s_w + ((bt % kRing) * RW + lrow) * kRowStride;
            const uint32_t* bk = s_k + ((bt % kRing) * RW + lrow) * kRowStride;
            const uint32_t cnt = nn > bt * kBatch ? min((uint32_t)kBatch, nn - bt * kBatch) : 0u;
            const uint32_t cmax = min((uint32_t)kBatch, nmax - bt * kBatch);
            const uint32_t cmin = nmin > bt * kBatch ? min((uint32_t)kBatch, nmin - bt * kBatch) : 0u;
            constexpr int T = U >= 16 ? 8 : 4;
            // groups that every row of the warp fills, then smaller ones.  Groups of 4 take the predicated path alone:
            // a second copy of the loop does not fit 64 registers (262144 power-law rows, C = 1024: 4.39 -> 4.20 ms).
            uint32_t t = 0;
            if constexpr (U > T) {
                for (; t + U <= cmin; t += U) {
                    RowsGroup<V, NV, U> g;
                    g.template issue<true>(bw + t, bk + t, U, x);
                    g.template multiply<true>(acc, U);
                }
            }
            for (; t < cmax; t += T) {
                const uint32_t have = cnt > t ? cnt - t : 0u;
                RowsGroup<V, NV, T> g;
                g.template issue<false>(bw + t, bk + t, have, x);
                g.template multiply<false>(acc, have);
            }
        }
    }
    spx::pdl_launch();
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (!on[v]) continue;
        if (a.act != SPX_ACT_NONE) {
#pragma unroll
            for (int i = 0; i < V; ++i) acc[v][i] = spx::apply_act(acc[v][i], a.act);
        }
        const size_t at = (size_t)(a.out.row0 + row) * a.ldy + c0 + v * G * V;
        if constexpr (V == 4) store_out(a.out, at, make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]));
        else
#pragma unroll
            for (int i = 0; i < V; ++i) store_out(a.out, at + i, acc[v][i]);
    }
}

// ---------------------------------------------------------------------------------------
// spmm_direct: X fits in shared memory, C is a multiple of 4 from 8 to 64 and the operands are aligned.  Such
// products are bound by latency: a row's FMA chain is serial, and there are not enough rows to hide
// a gather per entry.  So a CTA over R rows stages X whole, and splits its warps: the last two are producers that keep
// the rows' slabs coming (cp.async, batches of E entries, kChainRing - 1 ahead), the others are
// consumers: C / 4 lanes per row, which read (w, k) four entries at a time, gather one group of 8
// entries ahead of the group being multiplied and do nothing else.
// ---------------------------------------------------------------------------------------
constexpr int kChainRing = 4, kChainProducers = 64, kChainConsumers = 256;
constexpr uint64_t kChainX = 128 * 1024;        // bytes of X up to which it is staged

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// All of X into shared memory, rows Cp floats apart, by all threads of the CTA: asynchronous copies,
// so that no thread waits for one load before it asks for the next; ends with the copies landed and the CTA in step.
// Columns beyond C are not written: what is computed from them is never stored.
__device__ __forceinline__ void stage_x(float* s_x, const RowsArgs& a, uint32_t Cp)
{
    if (Cp == a.C && a.ldx == a.C && (reinterpret_cast<uintptr_t>(a.X) & 15) == 0) {
        const uint32_t total = a.n * Cp;
        for (uint32_t i = threadIdx.x * 4; i + 4 <= total; i += blockDim.x * 4) cp_async16(s_x + i, a.X + i);
        for (uint32_t i = (total & ~3u) + threadIdx.x; i < total; i += blockDim.x) cp_async4(s_x + i, a.X + i);
    } else {
        const uint32_t dk = blockDim.x / a.C, dc = blockDim.x - dk * a.C;
        uint32_t k = threadIdx.x / a.C, c = threadIdx.x - k * a.C;
        while (k < a.n) {
            cp_async4(s_x + k * Cp + c, a.X + (size_t)k * a.ldx + c);
            k += dk; c += dc;
            if (c >= a.C) { c -= a.C; ++k; }
        }
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
}

template <int V>
__device__ __forceinline__ void lds_vec(float (&d)[V], uint32_t at) {
    if constexpr (V == 1) asm("ld.shared.f32 %0, [%1];" : "=f"(d[0]) : "r"(at));
    if constexpr (V == 2) asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(d[0]), "=f"(d[1]) : "r"(at));
    if constexpr (V == 4)
        asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(at));
}

__global__ void __launch_bounds__(kChainConsumers + kChainProducers)
spmm_direct(const __grid_constant__ RowsArgs a)
{
    // named barriers: batch in ring slot s has landed (kFull + s), slot s is free again (kFree + s)
    constexpr int kFull = 1, kFree = 1 + kChainRing;
    constexpr int U = 8, V = 4;                 // entries per group, columns per lane
    extern __shared__ __align__(16) float s_mem[];
    const uint32_t R = a.RW, E = a.batch, stride = E + 4;           // E: 32, 64, 128 or 256 entries per row and batch
    const uint32_t Cp = a.Cp, L = Cp / V;
    float* s_w = s_mem + ((a.n * Cp + 3) & ~3u);
    uint32_t* s_k = reinterpret_cast<uint32_t*>(s_w + kChainRing * R * stride);
    uint2* s_info = reinterpret_cast<uint2*>(s_k + kChainRing * R * stride);
    const uint32_t slot0 = blockIdx.x * R;
    const uint32_t consumers = blockDim.x - kChainProducers;
    for (uint32_t i = threadIdx.x; i < R; i += blockDim.x) s_info[i] = slot0 + i < a.m ? __ldg(a.rows + slot0 + i) : make_uint2(0u, 0u);
    __syncthreads();
    const uint32_t nb = (s_info[0].y + E - 1) / E;                  // rows descend in length
    const bool producer = threadIdx.x >= consumers;
    auto fill = [&](uint32_t b) {               // producers: batch b into slot b % kChainRing, one group, empty or not
        const uint32_t shift = 29 - __clz(E);
        if (b < nb)
            for (uint32_t id = threadIdx.x - consumers; id < R << shift; id += kChainProducers) {
                const uint32_t i = id >> shift, at = (id & ((1u << shift) - 1u)) * 4, j = b * E + at;
                const uint2 ri = s_info[i];
                if (j < ri.y) {                 // the pitch is a multiple of 32 entries: whole quads exist
                    const size_t src = (size_t)ri.x * a.pitch + j;
                    const uint32_t dst = ((b % kChainRing) * R + i) * stride + at;
                    cp_async16(s_w + dst, a.Wd + src);
                    cp_async16(s_k + dst, a.idx + src);
                }
            }
        cp_async_commit();
    };
    if (producer)
        for (uint32_t b = 0; b + 1 < kChainRing; ++b) fill(b);
    spx::pdl_wait();
    spx::pdl_launch();
    stage_x(s_mem, a, Cp);

    if (producer) {
        for (uint32_t b = 0; b < nb; ++b) {
            // slot of batch b + ring - 1 is that of batch b - 1
            if (b >= 1 && b + kChainRing - 1 < nb) bar_sync(kFree + (b - 1) % kChainRing, blockDim.x);
            fill(b + kChainRing - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(kChainRing - 1) : "memory");
            bar_arrive(kFull + b % kChainRing, blockDim.x);
        }
        return;
    }

    const uint32_t i = threadIdx.x / L, g = threadIdx.x - i * L;
    const bool mine = i < R && slot0 + i < a.m;
    const uint2 ri = mine ? s_info[i] : make_uint2(0u, 0u);
    const uint32_t li = mine ? i : 0u;
    const float bias = (mine && a.bias) ? __ldg(a.bias + ri.x) : 0.0f;
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = bias;
    const uint32_t xs = (uint32_t)__cvta_generic_to_shared(s_mem) + g * V * 4u, xstride = Cp * 4u;
    const uint32_t warp_max = __reduce_max_sync(0xffffffffu, ri.y);
    for (uint32_t b = 0; b < nb; ++b) {
        bar_sync(kFull + b % kChainRing, blockDim.x);
        const float4* bw = reinterpret_cast<const float4*>(s_w + ((b % kChainRing) * R + li) * stride);
        const uint4* bk = reinterpret_cast<const uint4*>(s_k + ((b % kChainRing) * R + li) * stride);
        const uint32_t cnt = ri.y > b * E ? min(E, ri.y - b * E) : 0u;
        const uint32_t cmax = warp_max > b * E ? min(E, warp_max - b * E) : 0u;
        // A slot beyond the row's end reads row 0 of X and its FMA is skipped.
        float w[U], x[U][V];
        auto gather = [&](uint32_t t) {
#pragma unroll
            for (int q = 0; q < U / 4; ++q) {
                const float4 w4 = bw[t / 4 + q];
                const uint4 k4 = bk[t / 4 + q];
                w[4 * q] = w4.x; w[4 * q + 1] = w4.y; w[4 * q + 2] = w4.z; w[4 * q + 3] = w4.w;
                const uint32_t k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) lds_vec<V>(x[4 * q + u], xs + (t + 4 * q + u < cnt ? k[u] : 0u) * xstride);
            }
        };
        gather(0);
        for (uint32_t t = 0; t < cmax; t += U) {
            float wc[U], xc[U][V];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                wc[u] = w[u];
#pragma unroll
                for (int v = 0; v < V; ++v) xc[u][v] = x[u][v];
            }
            gather(min(t + U, E - U));          // the next group travels while this one is multiplied
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + u < cnt) {
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[v] = fmaf(wc[u], xc[u][v], acc[v]);
                }
        }
        if (b + kChainRing < nb) bar_arrive(kFree + b % kChainRing, blockDim.x);
    }
    if (!mine) return;
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = spx::apply_act(acc[v], a.act);
    const size_t at = (size_t)(a.out.row0 + ri.x) * a.ldy + g * V;
    store_out(a.out, at, make_float4(acc[0], acc[1], acc[2], acc[3]));
}

// ---------------------------------------------------------------------------------------
// spmm_chain<C>: X in shared memory and C <= 8 columns, any leading dimension.  With so few columns the
// serial FMA chain of a row (4 cycles an entry) and the instructions around it are what is left, so the
// gathering is taken off the chain: producer warps keep the slabs coming (cp.async), replace a batch of E
// column ids by the operands these select, 32 entries per instruction, transposed to one run per (row, column);
// one consumer lane per (row, column) walks its run with 16-byte reads of weights and operands, 1.5
// instructions per entry, while the producers prepare the next batch.  4096 x 4096, 10 %, C = 1: 39.6 us with
// a gather per entry, 10.3 us with the direct kernel above, 6.1 us here; C = 2 / 4: 8.0 / 13.3 us.
// ---------------------------------------------------------------------------------------
constexpr int kPreThreads = 256, kPreRing = 4;
template <int C>
__global__ void __launch_bounds__(kPreThreads)
spmm_chain(const __grid_constant__ RowsArgs a)
{
    // named barriers: operands of buffer 0 / 1 ready, buffer 0 / 1 free again, producers among themselves
    constexpr int kFull = 1, kFree = 3, kProducers = 5;
    constexpr uint32_t Cp = C == 3 ? 4 : C == 1 ? 1 : C == 2 ? 2 : (C + 3) / 4 * 4;
    extern __shared__ __align__(16) float s_mem[];
    const uint32_t R = a.RW, E = a.batch, stride = E + 4;           // E: 64, 128 or 256 entries per row and batch
    float* s_w = s_mem + ((a.n * Cp + 3) & ~3u);
    uint32_t* s_k = reinterpret_cast<uint32_t*>(s_w + kPreRing * R * stride);
    float* s_x = s_w + 2 * kPreRing * R * stride;                 // [2][row][column][entry]
    uint2* s_info = reinterpret_cast<uint2*>(s_x + 2 * R * C * stride);
    const uint32_t slot0 = blockIdx.x * R;
    for (uint32_t i = threadIdx.x; i < R; i += kPreThreads) s_info[i] = slot0 + i < a.m ? __ldg(a.rows + slot0 + i) : make_uint2(0u, 0u);
    __syncthreads();
    const uint32_t nb = (s_info[0].y + E - 1) / E;                  // rows descend in length
    const uint32_t consumers = (R * C + 31) / 32 * 32;              // threads
    const uint32_t t = threadIdx.x - consumers, P = kPreThreads - consumers;
    const uint32_t shift = 29 - __clz(E);
    auto fill = [&](uint32_t b) {
        if (b < nb)
            for (uint32_t id = t; id < R << shift; id += P) {
                const uint32_t i = id >> shift, at = (id & ((1u << shift) - 1u)) * 4, j = b * E + at;
                const uint2 ri = s_info[i];
                if (j < ri.y) {             // the pitch is a multiple of 32 entries: whole quads exist
                    const size_t src = (size_t)ri.x * a.pitch + j;
                    const uint32_t dst = ((b % kPreRing) * R + i) * stride + at;
                    cp_async16(s_w + dst, a.Wd + src);
                    cp_async16(s_k + dst, a.idx + src);
                }
            }
        cp_async_commit();
    };
    const bool producer = threadIdx.x >= consumers;
    if (producer)
        for (uint32_t b = 0; b < kPreRing - 2; ++b) fill(b);
    spx::pdl_wait();
    spx::pdl_launch();
    stage_x(s_mem, a, Cp);

    if (producer) {
        for (uint32_t b = 0; b < nb; ++b) {
            if (b >= 2) bar_sync(kFree + (b & 1), kPreThreads);     // batch b - 2 is done with: its operands and its slot
            asm volatile("cp.async.wait_group %0;" ::"n"(kPreRing - 3) : "memory");
            bar_sync(kProducers, P);
            const uint32_t* bk = s_k + (b % kPreRing) * R * stride;
            float* bx = s_x + (b & 1) * R * C * stride;
            // a warp takes 32 entries of a row at a time, four such units in flight
            constexpr int kUnits = 4;
            const uint32_t per = shift - 3, units = R << per, lane = t & 31;        // units per row: 2^per
            for (uint32_t u0 = t >> 5; u0 < units; u0 += kUnits * (P / 32)) {
                uint32_t k[kUnits], at[kUnits];
                bool live[kUnits];
#pragma unroll
                for (int q = 0; q < kUnits; ++q) {
                    const uint32_t u = u0 + q * (P / 32), i = u >> per, j = ((u & ((1u << per) - 1u)) << 5) + lane;
                    const uint32_t ui = u < units ? i : 0u, kq = bk[ui * stride + j];
                    live[q] = u < units && b * E + j < s_info[ui].y;
                    k[q] = live[q] ? kq : 0u;
                    at[q] = i * C * stride + j;
                }
                float x[kUnits][Cp];
#pragma unroll
                for (int q = 0; q < kUnits; ++q) {
                    const uint32_t from = (uint32_t)__cvta_generic_to_shared(s_mem) + k[q] * (Cp * 4u);
                    constexpr int V = Cp % 4 == 0 ? 4 : Cp;
#pragma unroll
                    for (int c = 0; c < Cp; c += V) {
                        float d[V];
                        lds_vec<V>(d, from + c * 4u);
#pragma unroll
                        for (int v = 0; v < V; ++v) x[q][c + v] = d[v];
                    }
                }
#pragma unroll
                for (int q = 0; q < kUnits; ++q)
                    if (live[q]) {
#pragma unroll
                        for (int c = 0; c < C; ++c) bx[at[q] + c * stride] = x[q][c];
                    }
            }
            bar_arrive(kFull + (b & 1), kPreThreads);
            fill(b + kPreRing - 2);
        }
        return;
    }

    const uint32_t i = threadIdx.x / C, c = threadIdx.x - i * C;
    const bool mine = i < R && slot0 + i < a.m;
    const uint2 ri = mine ? s_info[i] : make_uint2(0u, 0u);
    const uint32_t li = mine ? i : 0u;
    float acc = (mine && a.bias) ? __ldg(a.bias + ri.x) : 0.0f;
    for (uint32_t b = 0; b < nb; ++b) {
        bar_sync(kFull + (b & 1), kPreThreads);
        const float4* bw = reinterpret_cast<const float4*>(s_w + ((b % kPreRing) * R + li) * stride);
        const float4* bx = reinterpret_cast<const float4*>(s_x + (((b & 1) * R + li) * C + c) * stride);
        const uint32_t cnt = ri.y > b * E ? min(E, ri.y - b * E) : 0u;
        // two register sets of 16 entries: one is read while the other is multiplied
        float4 w0[4], x0[4], w1[4], x1[4];
        auto read = [&](float4 (&w)[4], float4 (&x)[4], uint32_t t) {
            const uint32_t at = min(t, E - 16) / 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) { w[q] = bw[at + q]; x[q] = bx[at + q]; }
        };
        auto multiply = [&](const float4 (&w)[4], const float4 (&x)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                acc = fmaf(w[q].x, x[q].x, acc);
                acc = fmaf(w[q].y, x[q].y, acc);
                acc = fmaf(w[q].z, x[q].z, acc);
                acc = fmaf(w[q].w, x[q].w, acc);
            }
        };
        auto multiply_some = [&](const float4 (&w)[4], const float4 (&x)[4], uint32_t left) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (4u * q < left) acc = fmaf(w[q].x, x[q].x, acc);
                if (4u * q + 1 < left) acc = fmaf(w[q].y, x[q].y, acc);
                if (4u * q + 2 < left) acc = fmaf(w[q].z, x[q].z, acc);
                if (4u * q + 3 < left) acc = fmaf(w[q].w, x[q].w, acc);
            }
        };
        uint32_t t = 0;
        read(w0, x0, 0);
        for (; t + 32 <= cnt; t += 32) {
            read(w1, x1, t + 16);
            multiply(w0, x0);
            read(w0, x0, t + 32);
            multiply(w1, x1);
        }
        if (t < cnt) {
            read(w1, x1, t + 16);
            multiply_some(w0, x0, cnt - t);
            multiply_some(w1, x1, cnt > t + 16 ? cnt - t - 16 : 0u);
        }
        if (b + 2 < nb) bar_arrive(kFree + (b & 1), kPreThreads);
    }
    if (mine) store_out(a.out, (size_t)(a.out.row0 + ri.x) * a.ldy + c, spx::apply_act(acc, a.act));
}

// Any shape at all, a thread per output element: leading dimensions beyond what the other kernels'
// 32-bit strides hold.
__global__ void __launch_bounds__(256)
spmm_simple(const __grid_constant__ RowsArgs a)
{
    spx::pdl_wait();
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)a.m * a.C) return;
    const uint32_t c = (uint32_t)(t % a.C);
    const uint2 ri = a.rows[t / a.C];
    float acc = a.bias ? a.bias[ri.x] : 0.0f;
    for (uint32_t j = 0; j < ri.y; ++j) {
        const size_t at = (size_t)ri.x * a.pitch + j;
        acc = fmaf(a.Wd[at], a.X[(size_t)a.idx[at] * a.ldx + c], acc);
    }
    store_out(a.out, (size_t)(a.out.row0 + ri.x) * a.ldy + c, spx::apply_act(acc, a.act));
}

}  // namespace

namespace spx {

// Warps (= rows) per CTA.  Large problems use 8; small ones use fewer so that the grid still has
// several CTAs per SM and the last wave is not mostly empty (a 4096-row matrix with 8 rows per CTA
// left the SMs idle 40 % of the kernel's duration).
static uint32_t gather_wpb(const spx_ell* e, uint32_t panels)
{
    const uint64_t want = (uint64_t)sm_count(e->device) * 8;
    for (uint32_t wpb : {8u, 4u, 2u})
        if ((uint64_t)((e->m + wpb - 1) / wpb) * panels >= want) return wpb;
    return 2;
}

// Whether the longest row's chain of gathers decides the kernel's duration (see
// spmm_gather_staged).  Estimates: the kernel moves 4*C bytes of X per stored entry at about
// 17 TB/s; the longest row's chain takes max_nnz / 4 round trips of about 1.2 us on the wide path.
// Measured on B200 (power-law rows, mean 64, max 2048, n = 65536, C = 1024), staged kernel against
// one panel-major launch of equal warps: 32768 rows 0.556 against 0.610 ms, 65536 rows 1.00 against 1.00 ms,
// 262144 rows 4.21 against 4.09 ms.  SPX_SPMM_STAGED=0|1 overrides.
static int staged_mode()
{
    static const int forced = [] { const char* v = getenv("SPX_SPMM_STAGED"); return v ? atoi(v) : -1; }();
    return forced;
}

static bool chain_bound(const spx_ell* e, uint32_t C)
{
    const int forced = staged_mode();
    if (C <= 128) return false;
    if (forced == 2) return true;                   // experiment: every row on 128-column panels
    if (e->long_rows == 0) return false;
    if (forced >= 0) return forced != 0;
    if (e->max_nnz * (uint64_t)e->m < 4 * e->nnz_total) return false;      // rows of near-equal length: nothing sticks out
    const double kernel_us = (double)e->nnz_total * C * 4.0 / 17e6 * (148.0 / sm_count(e->device));
    const double chain_us = e->max_nnz / 4.0 * 1.2;
    return chain_us > 0.4 * kernel_us;
}

static int finish_launch(cudaError_t err, const char* name)
{
    if (err != cudaSuccess) return fail(SPX_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(err));
    count_launch();
    return SPX_OK;
}

template <int V, int NV, int U, int MINB, bool PIPE = false>
static int launch_rows_one(const spx_ell* e, RowsArgs a, uint32_t panels, uint32_t wpb, cudaStream_t s)
{
    const size_t smem = (size_t)wpb * kRowsRing * a.RW * kRowsStride * 8;
    // Panels are the slow dimension; rows with 512 and more entries go first, for all panels (see BlockMap).
    const uint64_t rows_per_block = (uint64_t)a.RW * wpb, row_blocks = (e->m + rows_per_block - 1) / rows_per_block;
    if (row_blocks * panels > 0x7fffffffull) return fail(SPX_ERR_LIMIT, "spmm: grid too large");
    a.bm.row_blocks = (uint32_t)row_blocks;
    a.bm.panels = panels;
    a.bm.head = panels > 1 ? std::min<uint32_t>(a.bm.row_blocks, (uint32_t)((e->long_rows + rows_per_block - 1) / rows_per_block)) : 0u;
    a.bm.blocks = a.bm.row_blocks * panels;
    // The successor may come in while this grid runs if both fit the GPU whole; otherwise its first CTAs crowd the SMs
    // that are done early, and it runs out of balance (690 x 4077, 21 %, C = 128 28.4 us against 24.2; 645 x 5312,
    // 12 %, C = 32, which fits, 15.7 against 17.6).
    a.early = (uint64_t)a.bm.blocks * wpb * 2 <= (uint64_t)sm_count(e->device) * MINB * kRowsWarps;
    if (int rc = allow_smem<spmm_rows<V, NV, U, MINB, PIPE>>(e->device)) return rc;
    return finish_launch(launch_pdl(spmm_rows<V, NV, U, MINB, PIPE>, dim3(a.bm.blocks), dim3(wpb * 32), smem, s, a), "spmm_rows");
}

static uint32_t chain_pitch(uint32_t C) { return C <= 2 ? C : round_up(C, 4u); }

// X staged whole.  R rows per CTA: one CTA per SM while kChainConsumers threads carry them; the batch
// grows as R shrinks so that the barriers of a batch are spread over as many entries.
static int launch_direct(const spx_ell* e, RowsArgs a, cudaStream_t s)
{
    const uint32_t sms = sm_count(e->device);
    a.Cp = a.C;
    const uint32_t L = a.C / 4;
    a.RW = std::min<uint32_t>(kChainConsumers / L, std::max<uint32_t>(1u, (e->m + sms - 1) / sms));
    a.batch = a.RW > 32 ? 32 : a.RW > 16 ? 64 : a.RW > 8 ? 128 : 256;
    const auto bytes = [&] { return (size_t)a.RW * (a.batch + 4) * 2 * kChainRing * 4 + a.RW * sizeof(uint2) + (size_t)round_up(e->n * a.Cp, 4u) * 4; };
    while (a.RW > 1 && bytes() > 200 * 1024) a.RW = (a.RW + 1) / 2;
    const uint32_t threads = round_up(a.RW * L, 32u) + kChainProducers;
    const size_t smem = bytes();
    if (int rc = allow_smem<spmm_direct>(e->device)) return rc;
    return finish_launch(launch_pdl(spmm_direct, dim3((e->m + a.RW - 1) / a.RW), dim3(threads), smem, s, a), "spmm_direct");
}

template <int C>
static int launch_chain_one(const spx_ell* e, const RowsArgs& a, size_t smem, cudaStream_t s)
{
    if (int rc = allow_smem<spmm_chain<C>>(e->device)) return rc;
    return finish_launch(launch_pdl(spmm_chain<C>, dim3((e->m + a.RW - 1) / a.RW), dim3(kPreThreads), smem, s, a), "spmm_chain");
}
// R rows per CTA and batches of E entries.  The kernel takes as many batches as the longest row needs, each
// about 0.35 us of barriers and latency plus 5 ns per entry of the serial chains, or the time the SM's
// producers need for the operands of its resident CTAs: the combination with the least estimate of a few.
static int launch_chain(const spx_ell* e, RowsArgs a, cudaStream_t s)
{
    const uint32_t sms = sm_count(e->device), C = a.C;
    a.Cp = chain_pitch(C);
    const size_t x_bytes = (size_t)round_up(e->n * a.Cp, 4u) * 4;
    const auto bytes = [&](uint32_t R, uint32_t E) { return (size_t)R * (E + 4) * (2 * kPreRing + 2 * C) * 4 + R * sizeof(uint2) + x_bytes; };
    double best = 1e30;
    size_t smem = 0;
    const uint32_t most = std::min<uint32_t>(128 / C, std::max<uint32_t>(1u, (e->m + sms - 1) / sms));
    for (uint32_t split = 1; split <= 8; split *= 2)
        for (uint32_t E = 32; E <= 256; E *= 2) {
            const uint32_t R = (most + split - 1) / split;
            const size_t need = bytes(R, E);
            if (need > 220 * 1024) continue;
            const uint32_t ctas = (e->m + R - 1) / R, fit = std::min<uint32_t>(8u, (uint32_t)(227 * 1024 / (need + 1024)));
            const uint32_t on_sm = std::min(fit, (ctas + sms - 1) / sms), waves = (ctas + sms * fit - 1) / (sms * fit);
            const uint32_t batches = (e->max_nnz + E - 1) / E, len = std::min(E, e->max_nnz);
            const double us = waves * batches * std::max(0.35 + 0.005 * len, on_sm * R * len * (0.2 + 0.15 * C) * 1e-3);
            if (us < best) { best = us; a.RW = R; a.batch = E; smem = need; }
        }
#define SPX_CHAIN_CASE(N) case N: return launch_chain_one<N>(e, a, smem, s);
    switch (C) {
        SPX_CHAIN_CASE(1) SPX_CHAIN_CASE(2) SPX_CHAIN_CASE(3) SPX_CHAIN_CASE(4)
        SPX_CHAIN_CASE(5) SPX_CHAIN_CASE(6) SPX_CHAIN_CASE(7) SPX_CHAIN_CASE(8)
    }
#undef SPX_CHAIN_CASE
    return fail(SPX_ERR_LIMIT, "spmm: no kernel");
}

// Lanes, vectors per lane and gathers in flight of spmm_rows with V floats per vector.  NV vectors per
// lane: as few as cover the row, two (16-byte vectors) or three at most; wider X goes in panels.  U
// entries in flight per row: few warps per SM are bound by the latency of a round trip, many by its
// throughput, where the registers of a deep group only cost residency.  Measured at 4096 x 4096, 10 %:
// C = 256 72 us at U = 8 against 84 at 4 and 82 at 16; C = 128 43 us at 16 against 58 / 45 at 8 / 4; 1000
// rows, 2 %, C = 256: 7.5 / 9.9 / 12.8 us at 16 / 8 / 4; 28256 power-law rows, C = 576: 252 us at 4, 283 at 8.
template <int V>
static int launch_rows(const spx_ell* e, RowsArgs a, cudaStream_t s)
{
    const uint32_t q = (a.C + V - 1) / V;           // vectors per row
    const uint64_t sms = sm_count(e->device);
    const uint32_t nv_max = V == 4 ? 2 : 3;
    const uint32_t NV = std::min(nv_max, (q + 31) / 32);
    const uint32_t panels = (q + 32 * NV - 1) / (32 * NV);
    // One vector per lane: as few lanes as cover the row.  More: whole warps, the rest in the last vector; equal parts
    // would start off the 128-byte lines (2690 x 3809, 3.4 %, C = 704: 77 -> 52 us; 4096 x 4096, 10 %, C = 320: 157 -> 144).
    a.G = NV > 1 ? 32u : q;
    a.RW = std::min(32u / a.G, 16u);
    const uint64_t warps = (uint64_t)((e->m + a.RW - 1) / a.RW) * panels;
    uint32_t wpb = 4;                               // small CTAs: a finished one frees its warps at once
    while (wpb > 1 && (warps + wpb - 1) / wpb < sms * 4) wpb >>= 1;
    const double per_sm = (double)warps / sms;
    const bool brief = e->nnz_total < 100ull * e->m;    // rows too short for a deep group to pay for its registers
    int U;
    if (NV == 1) U = per_sm <= 8 ? 32 : per_sm < 48 || !brief ? 16 : 4;
    else         U = per_sm < (V == 4 ? 12 : 24) ? 16 : per_sm < 48 || !brief ? 8 : 4;
    // Single columns per lane are cheap enough in registers to keep a second group in flight (1312 x 2080, 27 %,
    // C = 37: 34 -> 23 us); 16-byte vectors are not (4096 x 4096, 10 %, C = 128: 42 -> 46 us).
    if constexpr (V == 1) {
        if (per_sm < 12 && NV == 1) return launch_rows_one<1, 1, 32, 2, true>(e, a, panels, wpb, s);
        if (per_sm < 12 && NV == 2) return launch_rows_one<1, 2, 16, 2, true>(e, a, panels, wpb, s);
        if (per_sm < 12) return launch_rows_one<1, 3, 16, 2, true>(e, a, panels, wpb, s);
    }
    if (NV == 1)
        return U == 32   ? launch_rows_one<V, 1, 32, 2>(e, a, panels, wpb, s)
               : U == 16 ? launch_rows_one<V, 1, 16, 2>(e, a, panels, wpb, s)
                         : launch_rows_one<V, 1, 4, 8>(e, a, panels, wpb, s);
    if (NV == 2 || V == 4)
        return U == 16  ? launch_rows_one<V, 2, 16, 2>(e, a, panels, wpb, s)
               : U == 8 ? launch_rows_one<V, 2, 8, 4>(e, a, panels, wpb, s)
                        : launch_rows_one<V, 2, 4, 8>(e, a, panels, wpb, s);
    if constexpr (V != 4)
        return U == 16  ? launch_rows_one<V, 3, 16, 2>(e, a, panels, wpb, s)
               : U == 8 ? launch_rows_one<V, 3, 8, 4>(e, a, panels, wpb, s)
                        : launch_rows_one<V, 3, 4, 8>(e, a, panels, wpb, s);
    return fail(SPX_ERR_LIMIT, "spmm: no kernel");
}

int launch_spmm_tile(spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias, int act, const PeerOut& out,
                     uint64_t ldy, bool vec_x, bool vec_out, uint32_t V, bool half, bool again, cudaStream_t s);

// Short rows: the ring of spmm_rows costs more than it hides, and half warps leave fewer lanes idle than its 11 to 31
// lanes a row do.  Measured, half against rows, back to back / alone: 20000 rows of 16 to 64 entries, C = 96 0.75 / 0.80,
// C = 48 0.85 / 0.90, C = 64 0.99 - 1.14 / 0.95 - 1.05, C = 40 0.96 - 1.17; 5000 rows, C = 68 to 128 0.72 - 0.86 / 0.82 - 0.91,
// C = 48 0.83 - 0.96 / 0.87 - 0.97; 3500 rows, C = 68 to 128 0.84 - 1.02 / 0.87 - 0.94, C = 48 0.94 - 1.4.
static bool takes_half(const spx_ell* e, uint32_t C)
{
    const uint64_t sms = sm_count(e->device);
    if (e->nnz_total >= 128ull * e->m) return false;
    return C > 64 && C <= 128 ? e->m >= 16 * sms : C >= 44 && C <= 60 && e->m >= 32 * sms;
}

static int launch_half(const spx_ell* e, const RowsArgs& a, cudaStream_t s)
{
    const uint32_t warps = (e->m + 1) / 2;
    uint32_t wpb = 8;
    while (wpb > 1 && (uint64_t)((warps + wpb - 1) / wpb) < (uint64_t)sm_count(e->device) * 8) wpb >>= 1;
    const dim3 grid((warps + wpb - 1) / wpb), block(wpb * 32);
    const bool early = (uint64_t)warps * 2 <= (uint64_t)sm_count(e->device) * 32;       // as in launch_rows_one: 64 registers
    return finish_launch(launch_pdl(a.C > 64 ? spmm_gather_half<2> : spmm_gather_half<1>, grid, block, 0, s, a.Wd, a.idx, a.rows, a.m, a.pitch,
                                    a.X, a.C, a.ldx, a.bias, a.act, a.out, a.ldy, early), "spmm_gather_half");
}

int launch_spmm(const spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias,
                int act, float* Y, uint64_t ldy, cudaStream_t s, bool again)
{
    float* one[1] = { Y };
    return launch_spmm_bcast(e, X, C, ldx, bias, act, one, 1, 0, ldy, s, false, again);
}

int launch_spmm_bcast(const spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias, int act,
                      float* const* Ys, uint32_t npeers, uint64_t row0, uint64_t ldy, cudaStream_t s, bool mcast, bool again)
{
    if (e->m == 0 || C == 0) return SPX_OK;
    if (npeers == 0 || npeers > (uint32_t)kMaxPeers) return fail(SPX_ERR_LIMIT, "spmm: 1..%d destination buffers supported", kMaxPeers);
    if (mcast && npeers != 1) return fail(SPX_ERR_ARG, "spmm: a multicast destination is one address");
    if (int rc = check_tma_words(const_cast<spx_ell*>(e), "spmm")) return rc;
    PeerOut out{};
    out.n = (int)npeers;
    out.mcast = mcast ? 1 : 0;
    out.row0 = row0;
    bool aligned = true;
    for (uint32_t g = 0; g < npeers; ++g) {
        if (!Ys[g]) return fail(SPX_ERR_ARG, "spmm: destination %u is null", g);
        out.p[g] = Ys[g];
        aligned = aligned && (reinterpret_cast<uintptr_t>(Ys[g]) & 15) == 0;
    }
    const bool vec_ok = (C % 4 == 0) && (ldx % 4 == 0) && (ldy % 4 == 0) &&
                        ((reinterpret_cast<uintptr_t>(X) & 15) == 0) && aligned;
    RowsArgs a{};
    a.Wd = e->Wd; a.idx = e->idx; a.rows = e->rows; a.m = e->m; a.pitch = e->pitch; a.n = e->n;
    a.X = X; a.C = C; a.ldx = ldx; a.bias = bias; a.act = act; a.ldy = ldy; a.out = out;
    // Few columns and X small enough for shared memory: spmm_rows pays a trip to L2 per group of entries, the staged
    // kernels pay for bringing X in, for their barriers, and in CTAs that share an SM.  They win where rows
    // are long and few.  Measured, rows against staged: 1024 rows of 300 entries C = 1 / 4 / 8 8.5 / 10.4 / 10.6 us
    // against 4.0 / 4.8 / 5.1; of 30 entries, C = 3 2.1 against 3.2; 8192 rows of 300, C = 3 13.9 against 18.5; 8192 of
    // 30, C = 7 4.5 against 20.  Odd widths above 4 serialise most; 4 and 8 columns are whole vectors.
    const uint64_t x_bytes = (uint64_t)e->n * chain_pitch(C) * 4;
    const bool staged = x_bytes <= kChainX && e->max_nnz > 0;      // without entries X is not read and may be null
    const uint64_t len = e->max_nnz, m = e->m;
    const bool chain = C == 1 ? len >= 80 && m <= 6000
                     : C == 3 ? (len >= 200 || (len >= 80 && x_bytes <= 32 * 1024)) && m <= (len >= 1000 ? 4500u : 2000u)
                     : C <= 4 ? len >= 60 && m <= 4500
                     : C < 8  ? len >= 250 && m <= len
                              : C == 8 && len >= 80 && m <= 2048;
    if (staged && chain) return launch_chain(e, a, s);
    if (staged && vec_ok && C >= 8 && C <= 64 && len >= 80 && m <= (uint64_t)sm_count(e->device) * (kChainConsumers / (C / 4)))
        return launch_direct(e, a, s);
    // what gathers X if X is not staged: vectors of V floats
    const uint32_t V = vec_ok ? 4 : C % 2 == 0 && ldx % 2 == 0 && (reinterpret_cast<uintptr_t>(X) & 7) == 0 ? 2 : 1;
    const bool half = vec_ok && takes_half(e, C);
    {
        const bool vec_x = C % 4 == 0 && ldx % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
        const int rc = launch_spmm_tile(const_cast<spx_ell*>(e), X, C, ldx, bias, act, out, ldy, vec_x, C % 4 == 0 && ldy % 4 == 0 && aligned, V, half, again, s);
        if (rc != -1) return rc;
    }
    if (ldx >= (1ull << 30)) {
        const uint64_t blocks = ((uint64_t)e->m * C + 255) / 256;
        if (blocks > 0x7fffffffull) return fail(SPX_ERR_LIMIT, "spmm: grid too large");
        return finish_launch(launch_pdl(spmm_simple, dim3((unsigned)blocks), dim3(256), 0, s, a), "spmm_simple");
    } else if (half) {
        return launch_half(e, a, s);
    } else if (vec_ok && C > 128) {
        // A row is one dependent chain of gathers, G rows of X per round trip to L2 (about a
        // microsecond under load).  When the longest row's chain is a large part of the whole
        // kernel (few rows per GPU, skewed lengths) it becomes the tail: spmm_gather_staged then
        // gives the rows with 512 and more entries 128-column panels with eight rows of X in
        // flight per round trip (half the round trips), issued first.
        if (chain_bound(e, C)) {
            const bool all_narrow = staged_mode() == 2;
            const uint32_t wpb = gather_wpb(e, (C + 255) / 256);
            StagedMap sm{};
            sm.all_narrow = all_narrow ? 1u : 0u;
            // With the exchange fused in, every finished row is 4*C bytes to each peer, whatever its
            // length.  In descending order the many short rows all finish at the end and the links
            // idle until then; shortest first behind the head keeps them busy from the start, while
            // the long rows (the head) still start at once.  SPX_SPMM_BCAST_ORDER=0 keeps descending.
            static const int order_env = [] { const char* v = getenv("SPX_SPMM_BCAST_ORDER"); return v ? atoi(v) : 1; }();
            sm.rest_ascending = ((npeers > 1 || mcast) && order_env) ? 1u : 0u;
            sm.row_blocks = (e->m + wpb - 1) / wpb;
            sm.panels = all_narrow ? (C + 127) / 128 : (C + 255) / 256;
            sm.head_panels = (C + 127) / 128;
            sm.head = all_narrow ? 0u : std::min<uint32_t>(sm.row_blocks, (e->long_rows + wpb - 1) / wpb);
            sm.blocks = sm.head * sm.head_panels + (sm.row_blocks - sm.head) * sm.panels;
            spmm_gather_staged<<<sm.blocks, wpb * 32, (size_t)wpb * 512, s>>>(e->Wd, e->idx, e->rows, e->m, e->pitch,
                                                                          X, C, (uint32_t)(ldx * 4), bias, act, out, ldy, sm);
            SPX_LAUNCH_CHECK("spmm_gather_staged");
            return SPX_OK;
        }
    }
    return V == 4 ? launch_rows<4>(e, a, s) : V == 2 ? launch_rows<2>(e, a, s) : launch_rows<1>(e, a, s);
}

}  // namespace spx
