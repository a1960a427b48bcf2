// spmm_tile.cu -- SpMM with the dense operand staged in shared memory block by block, for matrices whose
// columns are used several times by the rows of one CTA (iid-sparse weights of a few thousand columns).
//
// The gather kernels of spmm.cu fetch 4*C bytes of X per stored entry through L1 / L2, and L2 -> SM
// bandwidth (64 B/clk/SM) and L1 wavefronts bound them.  Here a CTA owns a slice of 32 * NV columns of X
// and up to 28 groups of 4 rows, walks the columns of E in chunks of 256, and brings a chunk's
// 256 x (32 * NV) block of X into one of three stages of shared memory with a bulk tensor copy: X crosses
// L2 -> SM once per CTA instead of once per entry, and every gather is a conflict-free 16-byte
// shared-memory read (8 lanes cover 128 contiguous bytes).  A warp owns one group: 8 lanes per row, NV
// float4 accumulators per lane for the whole kernel.  Per output element the entries still come in
// storage order, one FMA each: bit-identical to the other kernels.
//
// The entries come in a form of their own, built once per handle: per group a run of 128-byte steps, each
// 4 entries of each of the 4 rows, which a warp streams through a private ring in shared memory with
// cp.async.  So the hand-off of 16 entries costs 2 broadcast reads, and no search, no shuffle.  An entry's id
// is its row of X among the three staged chunks, so a step may mix entries of two neighbouring chunks: the rows
// of a group need not finish a chunk together, which would leave 19 (10 % dense) to 56 % (2 %) of the slots empty.
//
// Bound by shared-memory wavefronts (16 NV + 4 per step and warp) with many warps per SM, by the latency
// of a warp's steps (0.04 us each, 0.05 with slices of 64) and the phases with few; chunks of 128 columns, six of them staged, lose 1 to 60 % to
// the phases' fixed cost, 192 x 4 up to 4 %.  Measured against gathering: 4096 x 4096, 10 %, C = 64 / 128 / 256 / 512
// 18.9 / 32.7 / 60.8 / 121 us against 25.3 / 43.5 / 72.6 / 142; 8192 x 8192, 10 %, C = 64 62.9 against 103;
// 3512 x 3227, 19 %, C = 160 59.5 against 106; 4927 x 3082, 21 %, C = 160 86.8 against 159.
#include "common.cuh"
#include "tma.cuh"
#include "peer_out.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <optional>

namespace {

using spx::PeerOut;
using spx::store_out;

constexpr uint32_t kChunk = 256;        // columns of E per chunk (the largest extent of a box)
constexpr uint32_t kStages = 3;         // chunks of X in shared memory
constexpr uint32_t kWindow = 2;         // chunks that the entries of a phase may be in; the others are on their way
constexpr uint32_t kGroupRows = 4;
constexpr uint32_t kStepWords = 32;     // 128 bytes: 16 weights, 16 local column ids ([row][4 entries] each)
// A slot without an entry holds the weight -0.0f and the id of a row of zeros behind the stages: -0 * 0
// is -0, and adding -0 leaves every accumulator as it is, -0 and NaN included.
constexpr uint32_t kNone = kStages * kChunk;
constexpr uint32_t kNoWeight = 0x80000000u;
constexpr uint32_t kMaxWarps = 28;      // per CTA: leaves 72 registers a thread

// First entry of a row whose column is at least c.
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* __restrict__ k, uint32_t n, uint32_t c)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(k + mid) < c) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Warp per group.  Phase c of a group is what it multiplies between the arrival of chunk c and that of the
// next: as many whole blocks of four steps as the chunks up to c fill for all four rows, and at least the entries
// of chunk c - 1, whose stage is given back after the phase.  So slots stay empty at the rows' ends, and in rows
// with fewer than a few entries per chunk.
// cnt[group][chunk] = steps of the phase; pos[group][chunk] = the rows' first entries in it; total[group].
__global__ void __launch_bounds__(256)
tile_count_kernel(const uint32_t* __restrict__ idx, const uint2* __restrict__ rows, uint32_t m, uint32_t pitch, uint32_t groups,
                  uint32_t chunks, uint32_t* __restrict__ cnt, uint4* __restrict__ pos, uint32_t* __restrict__ total)
{
    const uint32_t lane = threadIdx.x & 31, g = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (g >= groups) return;
    uint2 ri[kGroupRows];
#pragma unroll
    for (uint32_t r = 0; r < kGroupRows; ++r) ri[r] = g * kGroupRows + r < m ? __ldg(rows + g * kGroupRows + r) : make_uint2(0u, 0u);
    uint4* __restrict__ p4 = pos + (size_t)g * chunks;
    for (uint32_t c = lane; c < chunks; c += 32) {          // first: where each row's entries up to chunk c end
        uint32_t end[kGroupRows];
#pragma unroll
        for (uint32_t r = 0; r < kGroupRows; ++r) end[r] = lower_bound(idx + (size_t)ri[r].x * pitch, ri[r].y, (c + 1) * kChunk);
        p4[c] = make_uint4(end[0], end[1], end[2], end[3]);
    }
    __syncwarp();
    // then, lane r for row r: the steps of each phase
    const uint32_t r = lane % kGroupRows, len = r == 0 ? ri[0].y : r == 1 ? ri[1].y : r == 2 ? ri[2].y : ri[3].y;
    uint32_t at = 0, sum = 0, past[kWindow] = {};           // past[i]: the end of the entries up to chunk c - i
    for (uint32_t c = 0; c < chunks; ++c) {
#pragma unroll
        for (int i = kWindow - 1; i > 0; --i) past[i] = past[i - 1];
        const uint4 e4 = p4[c];
        past[0] = r == 0 ? e4.x : r == 1 ? e4.y : r == 2 ? e4.z : e4.w;
        const uint32_t there = past[0] - at;                // entries that could be taken now
        const uint32_t due = c + 1 == chunks ? len : past[kWindow - 1];     // entries before this leave the stages
        const uint32_t must = due > at ? (due - at + 3) / 4 : 0u;
        const uint32_t can = past[0] == len ? 0xffffffffu : there / 4;      // a row without more to come holds nobody up
        const uint32_t all = __reduce_min_sync(0xffffffffu, can);
        uint32_t fit = all == 0xffffffffu ? 0u : all;       // ending with a block of the ring: no block is cut in two
        fit = fit >= 4 - (sum & 3) ? fit - ((sum + fit) & 3) : 0u;
        const uint32_t n = max(fit, __reduce_max_sync(0xffffffffu, must));
        __syncwarp();                                       // p4[c] has been read
        const uint32_t a0 = __shfl_sync(0xffffffffu, at, 0), a1 = __shfl_sync(0xffffffffu, at, 1);
        const uint32_t a2 = __shfl_sync(0xffffffffu, at, 2), a3 = __shfl_sync(0xffffffffu, at, 3);
        if (lane == 0) {
            p4[c] = make_uint4(a0, a1, a2, a3);
            cnt[(size_t)g * chunks + c] = n;
        }
        at += min(4 * n, there);
        sum += n;
    }
    if (lane == 0) total[g] = sum;
}

// Warp per group: its steps, phase after phase.
__global__ void __launch_bounds__(256)
tile_fill_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx, const uint2* __restrict__ rows, uint32_t m, uint32_t pitch,
                 uint32_t groups, uint32_t chunks, const uint32_t* __restrict__ cnt, const uint4* __restrict__ pos,
                 const uint32_t* __restrict__ off, uint32_t* __restrict__ steps)
{
    const uint32_t lane = threadIdx.x & 31, g = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (g >= groups) return;
    const uint32_t r = (lane / 4) % kGroupRows, e = lane % 4;       // this lane's slot; lanes 16.. write the ids
    const uint2 ri = g * kGroupRows + r < m ? __ldg(rows + g * kGroupRows + r) : make_uint2(0u, 0u);
    const size_t base = (size_t)ri.x * pitch;
    const uint4* __restrict__ p4 = pos + (size_t)g * chunks;
    auto mine = [&](const uint4& v) { return r == 0 ? v.x : r == 1 ? v.y : r == 2 ? v.z : v.w; };
    size_t at = (size_t)off[g] * kStepWords;
    for (uint32_t c = 0; c < chunks; ++c) {
        const uint32_t lo = mine(p4[c]), hi = c + 1 < chunks ? mine(p4[c + 1]) : ri.y;
        const uint32_t n_steps = cnt[(size_t)g * chunks + c];
        for (uint32_t s = 0; s < n_steps; ++s, at += kStepWords) {
            const uint32_t j = lo + 4 * s + e;
            const bool have = j < hi;
            if (lane < 16) steps[at + lane] = have ? __float_as_uint(__ldg(Wd + base + j)) : kNoWeight;
            else steps[at + lane] = have ? __ldg(idx + base + j) % (kStages * kChunk) : kNone;
        }
    }
}

struct TileArgs {
    const uint32_t* steps;
    const uint32_t* off;
    const uint32_t* cnt;
    const uint2* rows;
    uint32_t m, groups, chunks, row_blocks, C;
    int vec_out;                // 16-byte stores: C % 4 == 0 and aligned destinations
    const float* bias;
    int act;
    uint64_t ldy;
    int* failed;
    int* failed_host;
    uint32_t missing;           // tests: bytes waited for that no copy brings
    PeerOut out;
};

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ float4 lds128(uint32_t at) {
    float4 d;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w) : "r"(at) : "memory");
    return d;
}
__device__ __forceinline__ void fma_vec(float4& a, float w, const float4& x) {
    spx::fma_pair(a.x, a.y, w, x.x, x.y);
    spx::fma_pair(a.z, a.w, w, x.z, x.w);
}

// N consecutive steps: entry u of a step of this lane's row is at `at` (weights) and `at` + 64 (ids).
template <int NV, int N>
__device__ __forceinline__ void tile_steps(float4 (&acc)[NV], uint32_t at, uint32_t xs)
{
    constexpr int kAhead = NV == 1 ? 2 : 1;     // steps of gathered operands held in registers
    float4 w[N], k[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        w[i] = lds128(at + i * 128);
        k[i] = lds128(at + i * 128 + 64);
    }
    float4 x[kAhead][4][NV];
    auto gather = [&](int i) {
        const uint32_t id[4] = {__float_as_uint(k[i].x), __float_as_uint(k[i].y), __float_as_uint(k[i].z), __float_as_uint(k[i].w)};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) x[i % kAhead][u][v] = lds128(xs + id[u] * (NV * 128u) + v * 128u);
    };
    if (kAhead == 2) gather(0);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (kAhead == 1) gather(i);
        else if (i + 1 < N) gather(i + 1);
        const float wv[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) fma_vec(acc[v], wv[u], x[i % kAhead][u][v]);
    }
}

// X with rows of C floats at any alignment into rows of Cp floats (a multiple of 8, at least 32), zeros behind.
__global__ void __launch_bounds__(256)
align_rows_kernel(const float* __restrict__ X, uint64_t ldx, uint32_t n, uint32_t C, uint32_t Cp, float* __restrict__ dst)
{
    spx::pdl_wait();
    spx::pdl_launch();
    const uint32_t quads = Cp / 4;
    const uint64_t total = (uint64_t)n * quads;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = (uint32_t)(i / quads), c = (uint32_t)(i - (uint64_t)k * quads) * 4;
        const float* __restrict__ p = X + (size_t)k * ldx + c;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < C) v.x = __ldg(p);
        if (c + 1 < C) v.y = __ldg(p + 1);
        if (c + 2 < C) v.z = __ldg(p + 2);
        if (c + 3 < C) v.w = __ldg(p + 3);
        reinterpret_cast<float4*>(dst)[i] = v;
    }
}

template <int WARPS> constexpr uint32_t kRingBlocks = WARPS < (int)kMaxWarps ? 4 : 2;       // of four steps, per warp

// For CTAs of up to WARPS warps.  kMaxWarps of them pass their gathers at the rate of shared memory with one step's operands
// in registers; fewer wait for their own latencies, and have registers for two steps (kDeep below).  2048 x 2048, 30 %,
// C = 32 16.6 -> 11.1 us, 640 x 1955, 35 %, C = 35 18.9 -> 14.0; 4096 x 4096, 10 %, C = 64 24.7 -> 18.9; 3001 x 4999, 6 %,
// C = 64 19.0 -> 15.4.  The steps' places in their blocks are known to the compiler: with one loop of steps, whose next block
// and register set are found at run time, these were 16.1, -, 21.6 and 16.6.
template <int NV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
spmm_tile_kernel(const __grid_constant__ TileArgs a, const __grid_constant__ CUtensorMap tmap)
{
    constexpr bool kDeep = WARPS < (int)kMaxWarps;
    constexpr uint32_t kRing = kRingBlocks<WARPS>;
    constexpr uint32_t kPitch = NV * 128u;                  // bytes of a staged row of X
    constexpr uint32_t kBox = kChunk * kPitch;              // bytes of a staged chunk
    extern __shared__ __align__(128) unsigned char s_mem[]; // [kStages] chunks of X, a row of zeros, a ring per warp
    __shared__ __align__(8) uint64_t s_bar[kStages];
    __shared__ __align__(8) uint64_t s_free[kStages];       // arrivals of the warps that no longer read the chunk in stage s
    __shared__ uint32_t s_asked;                            // copies asked for
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t slice = blockIdx.x / a.row_blocks, rb = blockIdx.x % a.row_blocks;
    // Groups come in descending length: dealt round, every CTA gets its share of the long ones (4096 x 4096, 10 %: the
    // first CTA in order had 12 % more to read from shared memory than the average: C = 256 65.7 us against 61.3).
    const uint32_t group = warp * a.row_blocks + rb;
    const bool active = group < a.groups;
    const uint32_t nactive = (a.groups - rb + a.row_blocks - 1) / a.row_blocks;    // at least warp 0: row_blocks <= groups

    // the warp's steps and counts do not depend on the predecessor kernel
    // Known to the compiler it goes into the addresses, and CTAs of up to 20 warps take 0.7 % longer (51 shapes).
    uint32_t ring_blocks = kRing;
    if (kDeep) asm volatile("" : "+r"(ring_blocks));
    const uint32_t ring_mask = ring_blocks - 1;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(s_mem) + kStages * kBox + kPitch + warp * (ring_blocks * 512u);
    const uint32_t first = active ? __ldg(a.off + group) : 0u, n_steps = active ? __ldg(a.off + group + 1) - first : 0u;
    const unsigned char* src = reinterpret_cast<const unsigned char*>(a.steps) + (size_t)first * 128 + lane * 16;
    auto fill = [&](uint32_t blk) {             // block blk of 4 steps; the array ends with room for a whole block
        if (blk < (n_steps + 3) / 4) cp_async16(ring + (blk & ring_mask) * 512u + lane * 16, src + (size_t)blk * 512);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t b = 0; b + 1 < kRing; ++b) fill(b);
    const uint32_t slot = group * kGroupRows + lane / 8;
    const uint2 ri = active && slot < a.m ? __ldg(a.rows + slot) : make_uint2(0u, 0u);
    uint32_t my_cnt = active && lane < a.chunks ? __ldg(a.cnt + (size_t)group * a.chunks + lane) : 0u;

    if (threadIdx.x == 0) {
#pragma unroll
        for (uint32_t s = 0; s < kStages; ++s) {
            spx::mbar_init(&s_bar[s], 1);
            spx::mbar_init(&s_free[s], nactive);
        }
        s_asked = min(kStages, a.chunks);
    }
    if (threadIdx.x < kPitch / 16)              // up to 16 threads: the row of zeros
        *reinterpret_cast<float4*>(s_mem + kStages * kBox + threadIdx.x * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    // an earlier CTA's (or call's) wait ran out: leave at once
    const bool bad = __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int*>(a.failed) != 0);
    spx::pdl_wait();
    spx::pdl_launch();
    if (bad) {                                  // this call's output is not written either: said again, for a graph's launches
        if (threadIdx.x == 0) *a.failed_host = 1;
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    auto ask = [&](uint32_t c) {                // by one thread: chunk c into stage c % kStages
        const uint32_t st = c % kStages;
        spx::mbar_expect_tx(&s_bar[st], kBox + a.missing);
        spx::tma_load_2d(s_mem + st * kBox, &tmap, (int)(slice * 32u * NV), (int)(c * kChunk), &s_bar[st]);
    };
    if (threadIdx.x == 0)
        for (uint32_t c = 0; c < min(kStages, a.chunks); ++c) ask(c);
    if (!active) return;

    const uint32_t r = lane / 8, l = lane & 7;
    const float b = (slot < a.m && a.bias) ? __ldg(a.bias + ri.x) : 0.0f;
    float4 acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = make_float4(b, b, b, b);
    const uint32_t xbase = (uint32_t)__cvta_generic_to_shared(s_mem) + l * 16;
    uint32_t step = 0;                          // of the group's stream
    bool landed = true;
    // kDeep.  Registers for two steps, the even and the odd ones of the stream: a step's operands are asked for before the
    // step in front of it is multiplied, its ids right after the operands of that step's predecessor, its weights once that
    // one is multiplied.  Operands only within a phase: the next chunk may not have landed (looking across it, with the wait
    // in the step, made every case slower, 11.2 to 14.2 us at 2048 x 2048, 30 %, C = 32).
    float4 w0, w1, k0, k1, x0[4][NV], x1[4][NV];
    auto place = [&](uint32_t st) { return ring + ((st % (4 * kRing)) * 128u) + r * 16; };
    auto next_block = [&](uint32_t blk) {       // entering it: it has landed, and the one before the last is free
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        fill(blk + 2);
    };
    auto ids = [&](float4& k, uint32_t st) {    // where the step's place in its block is not known
        if ((st & 3u) == 0) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            if (st) fill(st / 4 + 2);
        }
        k = lds128(place(st) + 64);
    };
    auto operands = [&](float4 (&x)[4][NV], const float4& k) {
        const uint32_t id[4] = {__float_as_uint(k.x), __float_as_uint(k.y), __float_as_uint(k.z), __float_as_uint(k.w)};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) x[u][v] = lds128(xbase + id[u] * (NV * 128u) + v * 128u);
    };
    auto multiply = [&](const float4& w, const float4 (&x)[4][NV]) {
        const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                acc[v].x = fmaf(wv[u], x[u][v].x, acc[v].x);
                acc[v].y = fmaf(wv[u], x[u][v].y, acc[v].y);
                acc[v].z = fmaf(wv[u], x[u][v].z, acc[v].z);
                acc[v].w = fmaf(wv[u], x[u][v].w, acc[v].w);
            }
    };
    // The stream's next step, POS % 4 of its block (kOdd: 1 or 3); whether another of the phase follows.
    constexpr int kOdd = 5;
    auto one = [&](auto pos, bool more) {
        constexpr int POS = decltype(pos)::value;
        float4 (&x)[4][NV] = POS & 1 ? x1 : x0;
        float4 (&xn)[4][NV] = POS & 1 ? x0 : x1;
        float4 &w = POS & 1 ? w1 : w0, &kn = POS & 1 ? k0 : k1;
        if (more) {
            operands(xn, kn);
            if (POS == 1 || (POS == kOdd && (step & 2u) == 0)) next_block((step + 3) / 4);
            kn = lds128(place(step + 3) + 64);
        }
        multiply(w, x);
        w = lds128(place(step + 2));
        ++step;
    };
    if constexpr (kDeep) {
        ids(k0, 0);
        ids(k1, 1);
        w0 = lds128(place(0));
        w1 = lds128(place(1));
    }
    for (uint32_t c = 0; c < a.chunks; ++c) {
        if (c && (c & 31u) == 0) my_cnt = c + lane < a.chunks ? __ldg(a.cnt + (size_t)group * a.chunks + c + lane) : 0u;
        const uint32_t all = __shfl_sync(0xffffffffu, my_cnt, c & 31u);
        if (landed) landed = spx::mbar_wait(&s_bar[c % kStages], (c / kStages) & 1u);
        if constexpr (kDeep) {
            using std::integral_constant;
            constexpr integral_constant<int, 0> p0{};
            constexpr integral_constant<int, 1> p1{};
            constexpr integral_constant<int, 2> p2{};
            constexpr integral_constant<int, 3> p3{};
            constexpr integral_constant<int, kOdd> p_odd{};
            uint32_t left = all;                // up to the end of a block, whole blocks, the rest
            if (left) {
                if (step & 1u) { operands(x1, k1); ids(k1, step + 2); one(p_odd, --left != 0); }
                else { operands(x0, k0); ids(k0, step + 2); }
                if (left && (step & 2u)) {
                    one(p2, --left != 0);
                    if (left) one(p3, --left != 0);
                }
                for (; left >= 4; left -= 4) {
                    one(p0, true);
                    one(p1, true);
                    one(p2, true);
                    one(p3, left > 4);
                }
                if (left) {
                    one(p0, --left != 0);
                    if (left) one(p1, --left != 0);
                    if (left) one(p2, false);
                }
            }
        } else {
            for (uint32_t s = 0; s < all;) {
                const uint32_t in_block = step & 3u, n = min(4u - in_block, all - s);
                if (in_block == 0) {                // entering a block of the ring: it has landed, and the one before is free
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncwarp();
                    fill(step / 4 + 1);
                }
                const uint32_t at = place(step);
                switch (n) {                        // unrolled: the hand-off and the gathers of a step run ahead of its FMAs
                case 1: tile_steps<NV, 1>(acc, at, xbase); break;
                case 2: tile_steps<NV, 2>(acc, at, xbase); break;
                case 3: tile_steps<NV, 3>(acc, at, xbase); break;
                default: tile_steps<NV, 4>(acc, at, xbase);
                }
                s += n;
                step += n;
            }
        }
        if (c + 1 < kWindow) continue;
        __syncwarp();
        // No later phase reads chunk c + 1 - kWindow: the last warp to get here asks for the chunk that takes its
        // place.  The arrival tells whether it is the last (one pending before it) and releases this warp's reads;
        // the test of the phase it has just completed acquires the other warps' arrivals, so that all reads of the
        // stage come before the copy unit's writes (3001 x 4999, 6 %, C = 77: 21.5 us; 24.6 with the whole bounded wait in its
        // place).  A fence and an atomic instead would wait for the warp's cp.async in flight, 1500 cycles per chunk.
        const uint32_t out = c + 1 - kWindow, st = out % kStages;
        if (lane == 0 && spx::mbar_arrive_pending(&s_free[st]) == 1u && landed && out + kStages < a.chunks) {
            spx::mbar_acquire(&s_free[st], (out / kStages) & 1u);
            ask(out + kStages);
            atomicAdd(&s_asked, 1u);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!landed) {
        *a.failed = 1;
        *a.failed_host = 1;
        // copies still in flight write this CTA's shared memory: one more bounded wait for each
        if (lane == 0) {
            const uint32_t asked = *reinterpret_cast<volatile uint32_t*>(&s_asked);
            for (uint32_t j = asked > kStages ? asked - kStages : 0; j < asked; ++j) (void)spx::mbar_wait(&s_bar[j % kStages], (j / kStages) & 1u);
        }
    }
    if (slot >= a.m) return;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const uint32_t col = slice * 32u * NV + v * 32u + l * 4u;
        if (col < a.C) {
            float4 o = acc[v];
            if (a.act != SPX_ACT_NONE) {
                o.x = spx::apply_act(o.x, a.act); o.y = spx::apply_act(o.y, a.act);
                o.z = spx::apply_act(o.z, a.act); o.w = spx::apply_act(o.w, a.act);
            }
            const size_t at = (size_t)(a.out.row0 + ri.x) * a.ldy + col;
            if (a.vec_out) {
                store_out(a.out, at, o);
            } else {
                store_out(a.out, at, o.x);
                if (col + 1 < a.C) store_out(a.out, at + 1, o.y);
                if (col + 2 < a.C) store_out(a.out, at + 2, o.z);
                if (col + 3 < a.C) store_out(a.out, at + 3, o.w);
            }
        }
    }
}

}  // namespace

namespace spx {

// The tiled form of a handle's matrix.  A group's steps are contiguous, chunk after chunk.
struct spx_tiles_impl {
    std::mutex mu;
    int calls = 0;              // SpMM calls that could have used the form
    std::atomic<int> state{0};  // 0: not built, 1: ready, 2: cannot be built
    uint32_t groups = 0, chunks = 0;
    uint64_t steps_bytes = 0;
    uint32_t* steps = nullptr;
    uint32_t* off = nullptr;
    uint32_t* cnt = nullptr;
};

void free_tiles(spx_ell* e)
{
    spx_tiles_impl* t = static_cast<spx_tiles_impl*>(e->tiles);
    if (!t) return;
    pool_free(t->steps, t->steps_bytes, nullptr);
    pool_free(t->off, (size_t)(t->groups + 1) * 4, nullptr);
    pool_free(t->cnt, (size_t)t->groups * t->chunks * 4, nullptr);
    delete t;
    e->tiles = nullptr;
}

void* new_tiles() { return new (std::nothrow) spx_tiles_impl(); }

static int build_tiles(spx_ell* e, spx_tiles_impl* t, cudaStream_t s)
{
    t->state = 2;
    t->groups = (e->m + kGroupRows - 1) / kGroupRows;
    t->chunks = (e->n + kChunk - 1) / kChunk;
    const size_t cells = (size_t)t->groups * t->chunks;
    ensure_tma_words(e);
    if (!e->tma_failed_dev || !e->tma_failed_mapped) return SPX_OK;
    void *pos = nullptr, *total = nullptr, *cnt = nullptr, *off = nullptr, *steps = nullptr;
    PinnedBlock stage;
    auto body = [&]() -> int {
        if (int rc = pool_alloc(&pos, cells * sizeof(uint4), e->device, s)) return rc;
        if (int rc = pool_alloc(&cnt, cells * 4, e->device, s)) return rc;
        if (int rc = pool_alloc(&total, (size_t)t->groups * 4, e->device, s)) return rc;
        if (int rc = pool_alloc(&off, (size_t)(t->groups + 1) * 4, e->device, s)) return rc;
        if (int rc = pinned_acquire((size_t)(t->groups + 1) * 4, &stage)) return rc;
        uint32_t* h = static_cast<uint32_t*>(stage.host);
        tile_count_kernel<<<(t->groups + 7) / 8, 256, 0, s>>>(e->idx, e->rows, e->m, e->pitch, t->groups, t->chunks,
                                                             static_cast<uint32_t*>(cnt), static_cast<uint4*>(pos), static_cast<uint32_t*>(total));
        SPX_LAUNCH_CHECK("tile_count_kernel");
        SPX_CUDA(cudaMemcpyAsync(h, total, (size_t)t->groups * 4, cudaMemcpyDeviceToHost, s));
        SPX_CUDA(cudaStreamSynchronize(s));
        uint64_t run = 0;
        for (uint32_t g = 0; g < t->groups; ++g) {
            const uint32_t n = h[g];
            h[g] = (uint32_t)run;
            run += n;
        }
        h[t->groups] = (uint32_t)run;
        if (run >= (1ull << 31)) return SPX_OK;
        t->steps_bytes = (run + 4) * kStepWords * 4;        // the ring copies whole blocks of 4 steps
        if (int rc = pool_alloc(&steps, t->steps_bytes, e->device, s)) return rc;
        SPX_CUDA(cudaMemcpyAsync(off, h, (size_t)(t->groups + 1) * 4, cudaMemcpyHostToDevice, s));
        tile_fill_kernel<<<(t->groups + 7) / 8, 256, 0, s>>>(e->Wd, e->idx, e->rows, e->m, e->pitch, t->groups, t->chunks,
                                                            static_cast<uint32_t*>(cnt), static_cast<uint4*>(pos), static_cast<uint32_t*>(off),
                                                            static_cast<uint32_t*>(steps));
        SPX_LAUNCH_CHECK("tile_fill_kernel");
        return SPX_OK;
    };
    const int rc = body();
    const cudaError_t err = cudaStreamSynchronize(s);       // complete for every stream, and for the blocks given back
    pool_free(pos, cells * sizeof(uint4), s);
    pool_free(total, (size_t)t->groups * 4, s);
    pinned_release(stage);
    if (rc != SPX_OK || err != cudaSuccess || !steps) {
        pool_free(cnt, cells * 4, s);
        pool_free(off, (size_t)(t->groups + 1) * 4, s);
        pool_free(steps, t->steps_bytes, s);
        if (err != cudaSuccess) return fail(SPX_ERR_CUDA, "spmm: building the tiled form failed: %s", cudaGetErrorString(err));
        return rc == SPX_ERR_OOM ? SPX_OK : rc;             // no room: the gather kernels need none
    }
    t->steps = static_cast<uint32_t*>(steps);
    t->off = static_cast<uint32_t*>(off);
    t->cnt = static_cast<uint32_t*>(cnt);
    t->state = 1;
    return SPX_OK;
}

template <int NV, int WARPS>
static int launch_tile_nv(const spx_ell* e, TileArgs a, const CUtensorMap& map, uint32_t warps, uint32_t slices, cudaStream_t s)
{
    a.row_blocks = (a.groups + warps - 1) / warps;
    size_t smem = (size_t)(kStages * kChunk + 1) * NV * 128 + (size_t)warps * kRingBlocks<WARPS> * 512;
    // One CTA to an SM where the grid is one wave: started while the kernel before still fills some of the SMs, two small ones
    // share one and take twice as long (435 x 3968, 35 %, C = 274, behind the copy of X: 61 us against 34).
    if (a.row_blocks * slices <= sm_count(e->device)) smem = std::max<size_t>(smem, 116 * 1024);
    if (int rc = allow_smem<spmm_tile_kernel<NV, WARPS>>(e->device)) return rc;
    SPX_CUDA(launch_pdl(spmm_tile_kernel<NV, WARPS>, dim3(a.row_blocks * slices), dim3(warps * 32), smem, s, a, map));
    count_launch();
    return SPX_OK;
}

namespace {

// The kernel for CTAs of `warps`: the one that keeps two steps' operands in registers, compiled for at most so many warps; 0: none.
constexpr uint32_t deep_limit(uint32_t NV, uint32_t warps) {
    return NV == 1 ? (warps <= 20 ? 20u : warps <= 24 ? 24u : 0u) : warps <= 16 ? 16u : 0u;
}

struct Plan {
    uint32_t slices, warps, deep;
    uint64_t waves;
    double us;
};

// Launch shape and expected time.  As few waves of CTAs as kMaxWarps warps each allow, and then equally
// many warps in every CTA.  Time: a third of a microsecond per phase (wait, hand-off, a block of steps cut short; more where
// X's rows do not begin on sectors, or end inside a line), and per step of a warp the
// larger of its latency and the shared-memory wavefronts of all the SM's warps (16 NV gathers + 4 of hand-off).
// A phase in which any row of a group has an entry due takes a step, however few they are: rows of less than a
// few entries per chunk are mostly empty slots (60000 x 4000, 8 entries a row, C = 33: 91 us against 30 gathered).
// The constants of both estimates are fitted to 593 measured shapes (256 to 150000 rows, 256 to 60000 columns, 4 to 3200
// entries a row, C = 1 to 1000): the kernel they choose takes 0.8 % longer than the fastest of the three (gathered, slices of
// 32 and of 64) on average, more than 10 % longer for 16 of them.
Plan plan_tiles(const spx_ell* e, uint32_t C, uint32_t NV, uint32_t sms, bool aligned, bool sectors)
{
    Plan p;
    const uint32_t groups = (e->m + kGroupRows - 1) / kGroupRows, chunks = (e->n + kChunk - 1) / kChunk;
    p.slices = (C + 32 * NV - 1) / (32 * NV);
    const uint64_t units = (uint64_t)groups * p.slices;
    p.waves = (units + (uint64_t)sms * kMaxWarps - 1) / ((uint64_t)sms * kMaxWarps);
    for (;; ++p.waves) {                        // whole CTAs: the slices' last ones are not full
        p.warps = (uint32_t)std::min<uint64_t>(kMaxWarps, (units + sms * p.waves - 1) / (sms * p.waves));
        const auto ctas = [&] { return (uint64_t)((groups + p.warps - 1) / p.warps) * p.slices; };
        while (p.warps < kMaxWarps && ctas() > p.waves * sms) ++p.warps;
        if (ctas() <= p.waves * sms) break;
    }
    p.deep = deep_limit(NV, p.warps);
    const double len = (double)e->nnz_total / e->m;
    const double steps = std::max((len + 1.1 * std::sqrt(len)) / 4.0, chunks * (1.0 - std::exp(-(double)kGroupRows * len / chunks)));
    const double chunk = !p.deep || p.warps <= 3 ? 0.365 : p.deep == 24 ? 0.333 : 0.313;     // few warps wait for the copies
    const double step = std::max(!p.deep ? 0.0 : NV == 1 ? 0.036 : 0.051, p.warps * (16.0 * NV + 4.0) / 2060.0);
    double rows = sectors ? 0.0 : 0.12;                     // us per chunk, for the copies of X's rows
    if (C < 32 && aligned) rows = (C % 8 ? 14.0 : 5.0) / C;     // shorter than a box is wide (2080 x 613, C = 4: 3 us a chunk)
    else if (C % 32 && C > 32) rows += 0.04;
    p.us = 0.6 + rows * chunks + (aligned ? 0.0 : 3.2) +
           p.waves * ((NV == 1 ? 1.9 : 2.6) + chunks * chunk + steps * step);
    return p;
}

// Expected time of gathering in vectors of V floats (spmm_rows, or spmm_gather_half): the warps' load instructions,
// which L1 passes at 4, 2 or 1 cycles and some, and up to 0.1 us of each warp's own; or the rounds of the longest row,
// for every wave of warps where the deep groups let only 8 per SM reside.
double gather_us(const spx_ell* e, uint32_t C, uint32_t V, bool half)
{
    const double sms = sm_count(e->device);
    const uint32_t q = (C + V - 1) / V, nv_max = V == 4 ? 2 : 3;
    const uint32_t NV = std::min(nv_max, (q + 31) / 32), panels = (q + 32 * NV - 1) / (32 * NV);
    const uint32_t RW = NV > 1 ? 1u : std::min(32 / q, 16u);
    const double per_sm = std::ceil((double)e->m / RW) * panels / sms;
    const bool brief = e->nnz_total < 100ull * e->m;
    const double load = V == 4 ? 3.15e-3 : V == 2 ? 1.7e-3 : 1.34e-3, off_lines = V == 4 ? 0.47e-3 : V == 2 ? 0.5e-3 : 0.39e-3;
    double loads = e->nnz_total / sms * panels * (load * NV / RW + (C % 32 ? off_lines : 0.0)) + (brief ? 0.037 : 0.10) * per_sm;
    // Two CTAs of 8 warps reside: a last round of a few takes as long as a full one.  From the second CTA on: by the average, matrices
    // with 8 to 12 warps per SM were expected in 0.8 of what gathering them takes (41 shapes).
    if (V == 4 && NV == 2 && per_sm > 8 && !brief)
        loads = e->nnz_total / sms * panels * (5.5e-3 + (C % 32 ? off_lines : 0.0)) * std::ceil(per_sm / 16.0) * 16.0 / per_sm;
    else if (V == 4 && NV == 2 && per_sm > 8 && per_sm < 12)
        loads *= 1.25;
    if (V == 4 && RW > 1 && !brief) {           // long rows side by side in a warp: half as if each took a power of two of lanes
        uint32_t lanes = 1;
        while (lanes < q) lanes *= 2;
        loads = e->nnz_total / sms * 2.0e-3 * (lanes / 32.0 + 1.0 / RW) + 0.10 * per_sm;
    }
    double rounds = e->max_nnz;
    if (V == 1 && per_sm < 12) rounds *= NV == 1 ? 0.0147 : 0.0115 * NV * (NV == 3 ? std::ceil(per_sm / 8.0) : 1.0);
    else rounds *= (NV == 1 ? 0.0168 * (V == 4 && RW > 1 && !brief ? 1.0 + 0.03 * RW : 1.0) : 0.0282) * (V > 1 && NV == 1 && (per_sm < 48 || !brief) ? std::max(1.0, std::ceil(per_sm / 8.0)) : 1.0);
    const double l2 = loads * loads, r2 = rounds * rounds;
    return (3.5 + std::sqrt(std::sqrt(l2 * l2 + r2 * r2))) * (half ? 0.98 : 1.0);
}

}  // namespace

// Returns -1 when the shape or the handle is not for this kernel.
int launch_spmm_tile(spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias, int act, const PeerOut& out,
                     uint64_t ldy, bool vec_x, bool vec_out, uint32_t V, bool half, bool again, cudaStream_t s)
{
    static const int env = [] { const char* v = getenv("SPX_SPMM_TILE"); return v ? atoi(v) : 1; }();
    if (!env || !e->tiles || !e->cols_ascending || e->tma_off || e->max_nnz == 0) return -1;
    const PFN_cuTensorMapEncodeTiled encode = tensor_map_encoder();
    if (!encode || ldx > 0xffffffffull || e->n > 65536 || C > (1u << 30) || (env != 2 && e->n < kChunk)) return -1;
    // Slices of 64 columns read the entries half as often, slices of 32 leave fewer columns idle and give the SMs more
    // warps.  Of 411 shapes with C > 32 (256 to 8192 rows and columns, 2 to 50 %), the narrow ones are faster by more than 2 %
    // for 191 (3001 x 4999, 6 %, C = 77 21.5 us against 25.6; 600 x 3000, 30 %, C = 128 18.6 / 25.1), the wide ones for 220
    // (4096 x 4096, 10 %, C = 100 33.4 / 37.7).  The choice takes 0.3 % longer than the better one on average.
    const uint32_t sms = sm_count(e->device);
    const bool sectors = !vec_x || (ldx % 8 == 0 && reinterpret_cast<uintptr_t>(X) % 32 == 0);
    Plan p = plan_tiles(e, C, 1, sms, vec_x, sectors);
    uint32_t NV = 1;
    static const int slices_env = [] { const char* v = getenv("SPX_SPMM_SLICES"); return v ? atoi(v) : 0; }();      // 32 or 64, for tests
    if (slices_env ? slices_env == 64 : C > 32) {
        const Plan wide = plan_tiles(e, C, 2, sms, vec_x, sectors);
        if (slices_env || p.us > wide.us) {
            p = wide;
            NV = 2;
        }
    }
    // By 1.2 us where gathering takes less than 4.5, 0.8 from 6 to 8, by none from 14 on: the estimates are fitted to calls of
    // 10 us and more, and one of 2 us takes 1 longer staged (245 shapes of up to 2500 rows and columns: 60 of the 130 that
    // gather in less than 4 us took 5 % longer without it, none with it), nor is it worth the form.
    const double gather = gather_us(e, C, V, half);
    const double by = 0.8 * std::clamp((14.0 - gather) / 6.0, 0.0, 1.0) + 0.4 * std::clamp((6.0 - gather) / 1.5, 0.0, 1.0);
    const bool faster = p.us + by <= gather;
    if ((uint64_t)p.slices * e->m > 0x7fffffffull) return -1;
    if (env != 2 && !faster) return -1;
    spx_tiles_impl* t = static_cast<spx_tiles_impl*>(e->tiles);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (t->state != 1 || !vec_x) {              // building and the scratch below allocate: not while a graph is captured
        if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) { (void)cudaGetLastError(); return -1; }
    }
    std::optional<RelaxedCapture> relaxed;      // s is not being captured; another stream may be, by this thread
    if (t->state != 1 || !vec_x) relaxed.emplace();
    if (t->state != 1) {
        std::lock_guard<std::mutex> lk(t->mu);
        if (t->state == 0) {
            if ((again ? t->calls : ++t->calls) < 2) return -1;     // a matrix that is multiplied once is not worth the second form
            if (int rc = build_tiles(e, t, s)) return rc;
        }
        if (t->state != 1) return -1;
    }
    void* aligned = nullptr;
    const uint32_t Cp = C < 32 ? 32u : round_up(C, 8u);
    if (!vec_x) {                               // bulk copies need 16-byte rows, and are faster with whole sectors: X moves into scratch that has them
        if (int rc = scratch_alloc(&aligned, (size_t)e->n * Cp * 4, e->device, s)) return rc == SPX_ERR_OOM ? -1 : rc;
        const uint64_t quads = (uint64_t)e->n * (Cp / 4);
        const unsigned blocks = (unsigned)std::min<uint64_t>((quads + 255) / 256, (uint64_t)sm_count(e->device) * 16);
        const cudaError_t err = launch_pdl(align_rows_kernel, dim3(blocks), dim3(256), 0, s, X, ldx, e->n, C, Cp, static_cast<float*>(aligned));
        if (err != cudaSuccess) { scratch_free(aligned, s); return fail(SPX_ERR_CUDA, "launch of align_rows_kernel failed: %s", cudaGetErrorString(err)); }
        count_launch();
        X = static_cast<const float*>(aligned);
        ldx = Cp;
    }
    CUtensorMap map;
    const cuuint64_t gdim[2] = {vec_x ? C : Cp, e->n};
    const cuuint64_t gstr[1] = {ldx * 4};
    const cuuint32_t box[2] = {32 * NV, kChunk};
    const cuuint32_t estr[2] = {1, 1};
    int rc = -1;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(X), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS) {
        TileArgs a{};
        a.steps = t->steps; a.off = t->off; a.cnt = t->cnt; a.rows = e->rows;
        a.m = e->m; a.groups = t->groups; a.chunks = t->chunks; a.C = C; a.vec_out = vec_out;
        a.bias = bias; a.act = act; a.ldy = ldy; a.out = out;
        a.failed = e->tma_failed_dev; a.failed_host = e->tma_failed_mapped;
        // SPX_SPMM_TMA_TEST_TIMEOUT=k: the waits of the process's k-th launch run out
        static const int timeout_env = [] { const char* v = getenv("SPX_SPMM_TMA_TEST_TIMEOUT"); return v ? atoi(v) : 0; }();
        static std::atomic<int> launches{0};
        if (timeout_env && ++launches == timeout_env) a.missing = 16;
        const auto launch = NV == 1 ? (p.deep == 20 ? launch_tile_nv<1, 20> : p.deep == 24 ? launch_tile_nv<1, 24> : launch_tile_nv<1, kMaxWarps>)
                                    : (p.deep == 16 ? launch_tile_nv<2, 16> : launch_tile_nv<2, kMaxWarps>);
        rc = launch(e, a, map, p.warps, p.slices, s);
    }
    scratch_free(aligned, s);
    return rc;
}

}  // namespace spx
