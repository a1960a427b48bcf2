// conv_tmem.cu -- sparse convolution with the input patch in tensor memory.
//
// conv.cu's kernels read every operand from shared memory, 128 bytes per clock and SM = 32 FMAs per clock, a quarter of
// what the FP32 units do; merging four output channels' columns lifts that by 1.36 at 80 % sparsity.  Here a chunk of
// the input patch sits in tensor memory: lane = batch entry (or batch entry and tile, for batches below 32), column =
// (channel, row, column of the patch).  The input under a tap is then the same column for all lanes of a warp, and
// consecutive output positions are consecutive columns: two loads of 8 columns bring a tap's operands for 2 x 8
// positions x 32 lanes, which 8 packed FMAs per lane use.  Per output element the entries come in storage order, one
// FMA each: bit-identical to the other kernels.
//
// A CTA: 16 warps multiply, each 4 output channels x 2 x 8 positions x 32 lanes (64 accumulators a thread); every
// quadrant holds the same patch (or one of two, where there are 32 output channels and less), so a CTA covers up to 64
// channels.  4 more warps, one per quadrant, copy the patch from shared memory, where bulk tensor copies bring it, into
// one half of the quadrant's columns while the other half is used.
//
// What bounds it: issue slots (71 % used, FMA pipe 50 %; nothing issues when an SM quarter's four warps wait at once).  A
// tap costs a warp 8 packed FMAs (16 clocks of the FMA pipe) and about 8 other instructions, 24 clocks with four warps to a
// quarter; filling costs 4 clocks per column, a shared-memory wavefront for each quadrant.  Measured, 256 -> 256 channels,
// 3 x 3, 56 x 56, batch 32: 80 % sparse 704 us (708 in a process of its own) against 1341 with conv_rbm_tile_kernel, 50 %
// 1362 / 2369, 95 % 399 / 464; batch 8 258 / 374; 64 -> 64, 112 x 112 203 / 377; 5 x 5, 64 -> 96, 28 x 28, batch 16 56 / 101.
// The halves of a last wave (RW = 2) spill 16 bytes, the whole units nothing.  Tried: scalar FMAs 1221 against 1021 us at
// the time, 4 x 8 positions and 2 channels a warp 1272 (spills), no warps of their own for the copying 1010 against 819 (its
// waits add up), entries read through L1 instead of shared memory 807 against 732, weights stored twice so that the packed
// FMA can take them as they are 760 against 732, CTAs that go on to further units by themselves 764 against 743.
#include "conv.cuh"
#include "tma.cuh"
#include "tmem.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>

namespace {

using spx::ConvParams;
using spx::ConvViews;
using spx::kTmemColumns;
using spx::round_up;

constexpr uint32_t kRows = 4;               // output channels per block of the entries' form
constexpr uint32_t kWarps = 16;             // that multiply
constexpr uint32_t kTH = 2, kTW = 8;        // output positions per tile
constexpr uint32_t kBuffers = 2;            // chunks in tensor memory
constexpr uint32_t kMaxStages = 5;          // chunks in shared memory
constexpr uint32_t kSmem = 220 * 1024;      // dynamic shared memory
constexpr uint32_t kMaxChunks = 2048;       // the form's builder keeps 5 words per chunk in shared memory
// Registers: (kWarps + 4) * 32 threads start with 96 each, 61440 in all, and share them out as 512 * 104 + 128 * 64.
constexpr int kMulRegs = 104, kFillRegs = 64;

// The entries' form.  Per block of 4 output channels a run of 16-byte units, chunk after chunk of CC input channels: a
// header (the four rows' counts, a byte each; the chunk's units; the next chunk's), then per row its entries in storage
// order, two to a unit: (weight, tensor-memory column of the first position's operand) twice.
struct FormShape {
    uint32_t kH, kW, dH, dW, TWin, THin, CC, chunk_cols;
    bool operator==(const FormShape& o) const { return std::memcmp(this, &o, sizeof(o)) == 0; }
};

// First entry of a row whose column is at least c.
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* __restrict__ k, uint32_t n, uint64_t c)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(k + mid) < c) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// One CTA per block; entries: [block][chunk] how many.  Shared memory: [chunks + 1][4] run starts, [chunks] first unit of each chunk.
__global__ void __launch_bounds__(256)
conv_form_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx, const uint32_t* __restrict__ nnz, uint32_t m, uint32_t pitch,
                 FormShape f, uint32_t chunks, uint32_t cap, uint4* __restrict__ units, uint32_t* __restrict__ entries)
{
    extern __shared__ uint32_t s_form[];
    __shared__ uint32_t total;
    uint32_t* start = s_form;
    uint32_t* first = s_form + (chunks + 1) * kRows;
    const uint32_t r0 = blockIdx.x * kRows;
    for (uint32_t i = threadIdx.x; i < (chunks + 1) * kRows; i += blockDim.x) {
        const uint32_t c = i / kRows, row = r0 + i % kRows;
        uint32_t v = 0;
        if (row < m) {
            const uint32_t len = nnz[row];
            v = c == chunks ? len : lower_bound(idx + (size_t)row * pitch, len, (uint64_t)c * f.CC * f.kH * f.kW);
        }
        start[i] = v;
    }
    __syncthreads();
    auto halves = [](uint32_t n) { return (n + 1) / 2; };
    auto count = [&](uint32_t c, uint32_t r) { return start[(c + 1) * kRows + r] - start[c * kRows + r]; };
    if (threadIdx.x < 32) {                     // exclusive scan of the chunks' units
        uint32_t run = 0;
        for (uint32_t c0 = 0; c0 < chunks; c0 += 32) {
            const uint32_t c = c0 + threadIdx.x;
            uint32_t n = 0;
            if (c < chunks) {
                n = 1;
                for (uint32_t r = 0; r < kRows; ++r) n += halves(count(c, r));
            }
            uint32_t inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
                if ((int)threadIdx.x >= o) inc += v;
            }
            if (c < chunks) first[c] = run + inc - n;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (threadIdx.x == 0) total = run;
    }
    __syncthreads();
    uint4* __restrict__ dst = units + (size_t)blockIdx.x * cap;
    auto end = [&](uint32_t i) { return i < chunks ? first[i] : total; };
    for (uint32_t c = threadIdx.x; c < chunks; c += blockDim.x) {
        uint32_t counts = 0, all = 0;
        for (uint32_t r = 0; r < kRows; ++r) {
            counts |= count(c, r) << (8 * r);
            all += count(c, r);
        }
        if (entries) entries[(size_t)blockIdx.x * chunks + c] = all;
        dst[first[c]] = make_uint4(counts, end(c + 1) - end(c), end(min(c + 2, chunks)) - end(c + 1), 0u);
    }
    const uint32_t taps = f.kH * f.kW;
    for (uint32_t r = 0; r < kRows && r0 + r < m; ++r) {
        const size_t base = (size_t)(r0 + r) * pitch;
        const uint32_t len = nnz[r0 + r];
        for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) {
            const uint32_t k = idx[base + j], cin = k / taps, kh = k / f.kW % f.kH, kw = k % f.kW, c = cin / f.CC;
            uint32_t at = first[c] + 1;
            for (uint32_t q = 0; q < r; ++q) at += halves(count(c, q));
            const uint32_t place = j - start[c * kRows + r];
            const uint32_t col = c % kBuffers * f.chunk_cols + ((cin - c * f.CC) * f.THin + kh * f.dH) * f.TWin + kw * f.dW;
            reinterpret_cast<uint2*>(dst + at + place / 2)[place & 1u] = make_uint2(__float_as_uint(Wd[base + j]), col);
        }
    }
}

// Clocks that a chunk takes a CTA: the larger of what its busiest quadrant multiplies (an entry of a warp, a block's four
// runs) or the latency of the longest block's own, and what its fillers copy (a column; the lane groups of a warp read
// the same banks), and their fixed costs.
constexpr float kEntryClocks = 23.5f, kRunClocks = 115.0f, kEntryLatency = 60.0f, kRunLatency = 150.0f, kChunkLatency = 300.0f;
constexpr float kCtaClocks = 9650.0f;
__host__ __device__ inline float fill_clocks(uint32_t chunk_cols, uint32_t S)
{
    const float groups = 4.4f * S;
    return chunk_cols * (groups > 7.7f ? groups : 7.7f) + 690.0f;
}
constexpr int kLaneGroups = 4;                  // S = 1, 2, 4, 8
struct CtaClocks {
    float c[2][kLaneGroups];                    // whole CTAs and halves; by S
};

// The clocks of a CTA of each group of `per_group` blocks, summed over its own chunks' entries, and per block the union
// columns and the entries.
__global__ void __launch_bounds__(128)
conv_load_kernel(const uint32_t* __restrict__ entries, const uint32_t* __restrict__ union_cols, const uint32_t* __restrict__ nnz, uint32_t m,
                 uint32_t chunks, uint32_t per_group, uint32_t chunk_cols, CtaClocks* __restrict__ ctas, uint2* __restrict__ blocks)
{
    __shared__ float s_part[4][2 * kLaneGroups];
    const uint32_t nblocks = (m + kRows - 1) / kRows, b0 = blockIdx.x * per_group, nq = per_group / 4;
    if (threadIdx.x < per_group && b0 + threadIdx.x < nblocks) {
        const uint32_t b = b0 + threadIdx.x;
        uint32_t all = 0;
        for (uint32_t r = b * kRows; r < min(m, (b + 1) * kRows); ++r) all += nnz[r];
        blocks[b] = make_uint2(union_cols[b], all);
    }
    float sum[2 * kLaneGroups] = {};
    for (uint32_t c = threadIdx.x; c < chunks; c += 128) {
        float mul = 0.0f;
        for (uint32_t q = 0; q < nq; ++q) {     // blocks q, q + nq, ... share a quadrant
            float quad = 0.0f;
            for (uint32_t b = b0 + q; b < min(nblocks, b0 + per_group); b += nq) {
                const float n = (float)entries[(size_t)b * chunks + c];
                quad += kEntryClocks * n + kRows * kRunClocks;
                mul = fmaxf(mul, kEntryLatency * n + kRows * kRunLatency + kChunkLatency);
            }
            mul = fmaxf(mul, quad);
        }
#pragma unroll
        for (int i = 0; i < kLaneGroups; ++i) {
            const float fill = fill_clocks(chunk_cols, 1u << i);
            sum[i] += fmaxf(mul, fill);
            sum[kLaneGroups + i] += fmaxf(mul / 2, fill);
        }
    }
#pragma unroll
    for (int i = 0; i < 2 * kLaneGroups; ++i) {
#pragma unroll
        for (int o = 16; o; o >>= 1) sum[i] += __shfl_down_sync(0xffffffffu, sum[i], o);
        if (threadIdx.x % 32 == 0) s_part[threadIdx.x / 32][i] = sum[i];
    }
    __syncthreads();
    if (threadIdx.x < 2 * kLaneGroups) {
        const uint32_t i = threadIdx.x;
        ctas[blockIdx.x].c[i / kLaneGroups][i % kLaneGroups] = kCtaClocks + s_part[0][i] + s_part[1][i] + s_part[2][i] + s_part[3][i];
    }
}

struct TmemArgs {
    ConvParams c;
    ConvViews v;
    const uint4* units;
    const float* bias;
    float* out;
    int act;
    uint32_t quads_out;                     // positions are contiguous in the output, in whole 16-byte quads
    uint32_t cap, slot;                     // units per block of the form; per slot of a chunk's units in shared memory
    uint32_t BT, S, QT;                     // batch entries per lane group; lane groups per warp; quadrants with patches of their own
    uint32_t TWin, CC, chunks, chunk_cols, row_cols;    // row_cols: columns from one row of positions to the next
    uint32_t tilesX, tiles, tile_units, groups, unit0;
    uint32_t box_bytes, sub_stage, stage, stages;       // bytes of a patch, from patch to patch, of a stage; stages
    int* failed;
    int* failed_host;
    uint32_t missing;                       // tests: bytes waited for that no copy brings
};

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t at) {
    uint4 d;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(d.x), "=r"(d.y), "=r"(d.z), "=r"(d.w) : "r"(at) : "memory");
    return d;
}
__device__ __forceinline__ float lds32(uint32_t at) {
    float d;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(d) : "r"(at) : "memory");
    return d;
}

__device__ __forceinline__ void fma_tile(float (&acc)[kTH][8], float w, const float (&x)[kTH][8])
{
#pragma unroll
    for (int g = 0; g < (int)kTH; ++g)
#pragma unroll
        for (int i = 0; i < 8; i += 2) spx::fma_pair(acc[g][i], acc[g][i + 1], w, x[g][i], x[g][i + 1]);
}

// Columns of `pitch` bytes (PITCH, or at run time) into tensor memory, 8 at a time, 32 on their way: a warp issues in
// order, so all loads of a batch come before its stores.
template <uint32_t PITCH>
__device__ __forceinline__ void fill_columns(uint32_t from, uint32_t pitch, uint32_t to, uint32_t columns)
{
    if (PITCH) pitch = PITCH;
    constexpr int N = 4;
    uint32_t n = columns / 8;
    for (; n >= N; n -= N, from += N * 8 * pitch, to += N * 8) {
        float v[N][8];
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) v[j][i] = lds32(from + (j * 8 + i) * pitch);
#pragma unroll
        for (int j = 0; j < N; ++j) spx::tmem_st8(to + j * 8, v[j]);
    }
    for (; n; --n, from += 8 * pitch, to += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = lds32(from + i * pitch);
        spx::tmem_st8(to, v);
    }
}

// Sigmoid and tanh: one copy of their code.  Inlined for each of a thread's 64 results they made the instruction cache
// miss at the end of every CTA: 256 -> 256, 56 x 56 742 against 697 us at the time, 3 -> 416, 80 x 80 242 against 147.  (The merged kernel's
// small cuts lose by the call, also where it is not made: 3 -> 160, 45 x 45, batch 30 30.4 against 33.1.)
__device__ __noinline__ float activate(float v, int act) { return spx::apply_act(v, act); }

// RW: output channels per warp (4, or half a block: the last wave of a launch on twice the CTAs); GP: row_cols, where
// it is known.  Work units are (group of output channels, tiles, batch entries), groups fastest, so that the CTAs that
// read the same patch run side by side.
template <int RW, int GP>
__global__ void __launch_bounds__((kWarps + 4) * 32, 1)
conv_tmem_kernel(const __grid_constant__ TmemArgs a, const __grid_constant__ CUtensorMap tmap)
{
    extern __shared__ __align__(128) unsigned char s_mem[];     // stages of the patches, then two slots of units per warp
    __shared__ __align__(8) uint64_t s_full[kMaxStages], s_free[kMaxStages];    // patches in shared memory
    __shared__ __align__(8) uint64_t t_full[4][kBuffers], t_free[4][kBuffers];  // chunks in a quadrant's columns
    __shared__ uint32_t s_tmem, s_asked;
    const ConvParams& p = a.c;
    const uint32_t lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), quad = warp & 3u, in_quad = warp >> 2;

    const uint32_t unit = a.unit0 + blockIdx.x;
    const uint32_t group = unit % a.groups, tile_unit = unit / a.groups % a.tile_units, bz = unit / a.groups / a.tile_units;
    const uint32_t subs = a.S * a.QT, first_tile = tile_unit * subs;
    const uint32_t sub = quad % a.QT * a.S + lane / a.BT;       // this lane's patch among the CTA's

    if (threadIdx.x == 32) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            spx::mbar_init(&s_full[s], 1);
            spx::mbar_init(&s_free[s], 4);
        }
        for (uint32_t q = 0; q < 4; ++q)
            for (uint32_t b = 0; b < kBuffers; ++b) {
                spx::mbar_init(&t_full[q][b], 1);
                spx::mbar_init(&t_free[q][b], kWarps / 4);
            }
        s_asked = min(a.stages, a.chunks);
    }
    // Tensor memory is taken after the predecessor's end: a CTA that held it and waited would stop for good a predecessor
    // that lets successors in before it takes its own.
    spx::pdl_wait();
    if (warp == 0) spx::tmem_alloc_all(&s_tmem);
    spx::tmem_fence_before();
    // an earlier CTA's (or call's) wait ran out: leave at once
    const bool bad = __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int*>(a.failed) != 0);
    spx::tmem_fence_after();
    const uint32_t tmem = s_tmem;
    spx::pdl_launch();
    if (bad) {                                  // this call's output is not written either: said again, for a graph's launches
        if (threadIdx.x == 0) *a.failed_host = 1;
        if (warp == 0) spx::tmem_free_all(tmem);
        return;
    }
    const uint32_t quad_base = tmem + (quad << 21);
    bool landed = true;
    if (warp >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFillRegs));
        // The quadrant's filler: brings chunk after chunk from shared memory into its columns.  Lane s asks for the
        // patch of the CTA's s-th tile.
        const uint32_t my_tile = min(first_tile + lane, a.tiles - 1);
        const int tx = (int)(my_tile % a.tilesX * kTW * p.sW) - (int)p.pW, ty = (int)(my_tile / a.tilesX * kTH * p.sH) - (int)p.pH;
        auto ask = [&](uint32_t c, uint32_t st) {           // by one warp: the patches of chunk c
            if (lane == 0) spx::mbar_expect_tx(&s_full[st], a.box_bytes * subs + a.missing);
            __syncwarp();
            if (lane < subs) spx::tma_load_4d(s_mem + st * a.stage + lane * a.sub_stage, &tmap, (int)(bz * a.BT), tx, ty, (int)(c * a.CC), &s_full[st]);
        };
        if (warp == kWarps)
            for (uint32_t c = 0; c < min(a.stages, a.chunks); ++c) ask(c, c);
        const uint32_t my_patch = (uint32_t)__cvta_generic_to_shared(s_mem) + sub * a.sub_stage + (lane % a.BT) * 4;
        uint32_t st = 0, phase = 0;
        for (uint32_t c = 0; c < a.chunks; ++c) {
            const uint32_t buf = c % kBuffers;
            if (landed && c >= kBuffers) landed = spx::mbar_wait(&t_free[quad][buf], (c / kBuffers - 1) & 1u);
            if (landed) landed = spx::mbar_wait(&s_full[st], phase);
            spx::tmem_fence_after();
            const uint32_t from = my_patch + st * a.stage, to = quad_base + buf * a.chunk_cols;
            if (a.BT == 32) fill_columns<128>(from, 128, to, a.chunk_cols);
            else fill_columns<0>(from, a.BT * 4, to, a.chunk_cols);
            spx::tmem_wait_st();
            spx::tmem_fence_before();
            __syncwarp();
            uint32_t last = 0;
            if (lane == 0) {
                spx::mbar_arrive(&t_full[quad][buf]);
                // the filler that is done with the stage last asks for the chunk that takes its place; the arrival tells
                // whether it is (one pending before it), the test of the phase it has completed acquires the others' reads
                if (landed && c + a.stages < a.chunks && spx::mbar_arrive_pending(&s_free[st]) == 1u) {
                    spx::mbar_acquire(&s_free[st], phase);
                    atomicAdd(&s_asked, 1u);
                    last = 1;
                }
            }
            if (__shfl_sync(0xffffffffu, last, 0)) ask(c + a.stages, st);
            if (++st == a.stages) {
                st = 0;
                phase ^= 1u;
            }
        }
        if (!landed) {
            *a.failed = 1;
            *a.failed_host = 1;
            if (lane == 0) {                    // copies still in flight write this CTA's shared memory: a bounded wait for each
                const uint32_t asked = *reinterpret_cast<volatile uint32_t*>(&s_asked);
                for (uint32_t j = asked > a.stages ? asked - a.stages : 0; j < asked; ++j)
                    (void)spx::mbar_wait(&s_full[j % a.stages], (j / a.stages) & 1u);
            }
        }
        __syncthreads();
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMulRegs));
    // the warp's rows: hb counts runs of RW rows
    const uint32_t hb = (group * kWarps + in_quad * 4) / a.QT + quad / a.QT;
    const uint32_t blk = hb * RW / kRows, sub_row = hb * RW % kRows, mo0 = blk * kRows + sub_row;
    const bool active = mo0 < p.Cout;
    // The warp's units of a chunk are brought into one of two slots in shared memory a chunk ahead.
    const uint32_t slots = (uint32_t)__cvta_generic_to_shared(s_mem) + a.stages * a.stage + warp * (2 * a.slot * 16u);
    const uint4* __restrict__ src = a.units + (size_t)(active ? blk : 0) * a.cap + lane;
    auto fetch = [&](uint32_t c, uint32_t n) {
        for (uint32_t i = 0; i < n; i += 32)
            if (i + lane < n) cp_async16(slots + ((c & 1u) * a.slot + i + lane) * 16, src + i);
        src += n;
    };
    // (a reduction, though all lanes hold the same: its result is known to be uniform, and the loops over it then are)
    if (active) fetch(0, __reduce_max_sync(0xffffffffu, __ldg(a.units + (size_t)blk * a.cap).y));
    float acc[RW][kTH][8];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float bv = (a.bias && mo0 + r < p.Cout) ? __ldg(a.bias + mo0 + r) : 0.0f;
#pragma unroll
        for (int g = 0; g < (int)kTH; ++g)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[r][g][i] = bv;
    }
    const uint32_t row_cols = GP ? (uint32_t)GP : a.row_cols;
    auto load = [&](float (&x)[kTH][8], uint32_t col) {
#pragma unroll
        for (int g = 0; g < (int)kTH; ++g) spx::tmem_ld8(x[g], quad_base + col + g * row_cols);
    };
    uint32_t u = 0;                             // address of the unit at hand
    uint4 e{};                                  // the unit: the one behind it is read while it is multiplied
    auto row = [&](float (&ac)[kTH][8], uint32_t n) {
        for (const uint32_t end = u + n / 2 * 16; u != end;) {
            float x0[kTH][8], x1[kTH][8];
            const float w0 = __uint_as_float(e.x), w1 = __uint_as_float(e.z);
            load(x0, e.y);
            load(x1, e.w);
            e = lds128(u += 16);
            spx::tmem_wait_ld(x0);
            spx::tmem_wait_ld(x1);
            fma_tile(ac, w0, x0);
            fma_tile(ac, w1, x1);
        }
        if (n & 1u) {
            float x0[kTH][8];
            const float w0 = __uint_as_float(e.x);
            load(x0, e.y);
            e = lds128(u += 16);
            spx::tmem_wait_ld(x0);
            fma_tile(ac, w0, x0);
        }
    };
    for (uint32_t c = 0; c < a.chunks; ++c) {
        if (landed) landed = spx::mbar_wait(&t_full[quad][c % kBuffers], (c / kBuffers) & 1u);
        spx::tmem_fence_after();
        if (active) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();                       // the chunk's units are there, and the other slot is no longer read
            u = slots + (c & 1u) * (a.slot * 16u);
            const uint4 h = lds128(u);
            const uint32_t counts = __reduce_max_sync(0xffffffffu, h.x);
            fetch(c + 1, __reduce_max_sync(0xffffffffu, h.z));
            u += 16;
            if (RW < (int)kRows)
#pragma unroll
                for (uint32_t r = 0; r + RW < kRows; ++r)
                    if (r < sub_row) u += ((counts >> (8 * r) & 255u) + 1) / 2 * 16;
            e = lds128(u);
#pragma unroll
            for (int r = 0; r < RW; ++r) row(acc[r], counts >> (8 * (sub_row + r)) & 255u);
        }
        spx::tmem_fence_before();
        __syncwarp();
        if (lane == 0) spx::mbar_arrive(&t_free[quad][c % kBuffers]);
    }
    if (!landed) {
        *a.failed = 1;
        *a.failed_host = 1;
    }
    const uint32_t tile = first_tile + sub, b = bz * a.BT + lane % a.BT;
    const uint32_t oh0 = tile / a.tilesX * kTH, ow0 = tile % a.tilesX * kTW;
    if (active && tile < a.tiles && b < a.v.b_out) {
        if (a.act == SPX_ACT_RELU) {
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int g = 0; g < (int)kTH; ++g)
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[r][g][i] = acc[r][g][i] > 0.0f ? acc[r][g][i] : 0.0f;
        } else if (a.act != SPX_ACT_NONE) {
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int g = 0; g < (int)kTH; ++g)
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[r][g][i] = activate(acc[r][g][i], a.act);
        }
        const int cols = (int)min(8u, p.Wo - ow0), rows = (int)min(kTH, p.Ho - oh0);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            if (mo0 + r >= p.Cout) break;
#pragma unroll
            for (int g = 0; g < (int)kTH; ++g) {
                if (g >= rows) break;
                float* __restrict__ o = a.out + (mo0 + r) * a.v.oC + (oh0 + g) * a.v.oH + ow0 * a.v.oW + b * a.v.oB;
                if (a.quads_out) {              // positions side by side: whole sectors per lane
                    reinterpret_cast<float4*>(o)[0] = make_float4(acc[r][g][0], acc[r][g][1], acc[r][g][2], acc[r][g][3]);
                    if (cols > 4) reinterpret_cast<float4*>(o)[1] = make_float4(acc[r][g][4], acc[r][g][5], acc[r][g][6], acc[r][g][7]);
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i, o += a.v.oW)
                    if (i < cols) *o = acc[r][g][i];
            }
        }
    }
    __syncthreads();                            // all loads are done, all copies have landed or been waited for
    spx::tmem_fence_after();
    if (warp == 0) spx::tmem_free_all(tmem);
}

}  // namespace

namespace spx {

// A handle's forms: one per kernel shape that it is used with, never changed once built (a captured graph may use one).
struct conv_tmem_impl {
    static constexpr int kForms = 4;
    struct Form {
        FormShape shape{};
        uint4* units = nullptr;
        size_t bytes = 0;
        uint32_t cap = 0;
        // what the CTAs' own entries are expected to take, here and in the merged kernel; not known without memory to find out
        bool loads = false;
        CtaClocks mean{}, worst{};
        MergedLoad merged[3];                   // CTAs of 16, 8 and 4 blocks
    };
    std::mutex mu;
    int count = 0;
    bool no_memory = false;     // an earlier attempt found none: a further one would wait for the whole device to give memory back
    Form forms[kForms];
};

void* new_conv_tmem() { return new (std::nothrow) conv_tmem_impl(); }

void free_conv_tmem(spx_ell* e)
{
    conv_tmem_impl* t = static_cast<conv_tmem_impl*>(e->conv_tmem);
    if (!t) return;
    for (int i = 0; i < t->count; ++i) pool_free(t->forms[i].units, t->forms[i].bytes, nullptr);
    delete t;
    e->conv_tmem = nullptr;
}

void merged_loads(const uint2* blocks, uint32_t nblocks, MergedLoad (&out)[3])
{
    for (int k = 0; k < 3; ++k) {
        const uint32_t nb = 16u >> k;
        MergedLoad& l = out[k];
        for (uint32_t b0 = 0; b0 < nblocks; b0 += nb) {
            double longest = 0.0, work = 0.0;
            for (uint32_t b = b0; b < std::min(nblocks, b0 + nb); ++b) {
                longest = std::max<double>(longest, blocks[b].x);
                work += 0.7 * blocks[b].x + 0.2 * blocks[b].y;
            }
            l.longest += longest;
            l.work += work;
            l.longest_worst = std::max(l.longest_worst, longest);
            l.work_worst = std::max(l.work_worst, work);
        }
        const uint32_t n = (nblocks + nb - 1) / nb;
        l.longest /= n;
        l.work /= n;
    }
}

static void read_loads(conv_tmem_impl::Form& form, const CtaClocks* ctas, uint32_t groups, uint32_t nblocks)
{
    for (int h = 0; h < 2; ++h)
        for (int i = 0; i < kLaneGroups; ++i) {
            double sum = 0.0;
            for (uint32_t g = 0; g < groups; ++g) {
                sum += ctas[g].c[h][i];
                form.worst.c[h][i] = std::max(form.worst.c[h][i], ctas[g].c[h][i]);
            }
            form.mean.c[h][i] = (float)(sum / groups);
        }
    merged_loads(reinterpret_cast<const uint2*>(ctas + groups), nblocks, form.merged);
    form.loads = true;
}

// The form for a shape, built where it is not there yet (the call then waits for its stream, so that every stream may
// use the form).  -1: it cannot be (no memory, too many shapes, or a graph is being captured).
static int find_form(spx_ell* e, const FormShape& f, uint32_t chunks, uint32_t per_group, cudaStream_t s, const conv_tmem_impl::Form** out)
{
    conv_tmem_impl* t = static_cast<conv_tmem_impl*>(e->conv_tmem);
    std::lock_guard<std::mutex> lk(t->mu);
    for (int i = 0; i < t->count; ++i)
        if (t->forms[i].shape == f) { *out = &t->forms[i]; return SPX_OK; }
    if (t->no_memory || t->count == conv_tmem_impl::kForms) return -1;
    cudaStreamCaptureStatus cap_status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap_status) != cudaSuccess || cap_status != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return -1;
    }
    RelaxedCapture relaxed;                     // s is not being captured; another stream may be, by this thread
    // The other kernel's weights, which a later call may take (another batch, say); how many columns they have is counted below.
    const int merged = ensure_rbm(e, f.kH, f.kW, s, nullptr);
    if (merged > 0) return merged;
    ensure_tma_words(e);
    if (!e->tma_failed_dev || !e->tma_failed_mapped) {
        t->no_memory = true;
        return -1;
    }
    const uint32_t blocks = (e->m + kRows - 1) / kRows;
    // per row at most one half-empty unit per chunk
    const uint64_t cap = chunks + kRows * (((uint64_t)e->max_nnz + chunks + 1) / 2);
    if (cap > 0x7fffffffull) return -1;
    conv_tmem_impl::Form& form = t->forms[t->count];
    form = conv_tmem_impl::Form{};
    form.shape = f;
    form.cap = (uint32_t)cap;
    form.bytes = (size_t)blocks * cap * 16;
    void* units = nullptr;
    if (pool_alloc(&units, form.bytes, e->device, s) != SPX_OK) {
        t->no_memory = true;
        return -1;
    }
    form.units = static_cast<uint4*>(units);
    // the loads' intermediate counts, and where the host finds them
    const uint32_t groups = (blocks + per_group - 1) / per_group;
    const size_t entries_bytes = (size_t)blocks * chunks * 4;
    void *entries = nullptr, *found = nullptr;
    PinnedBlock host;
    bool loads = merged == SPX_OK && pinned_acquire(groups * sizeof(CtaClocks) + blocks * sizeof(uint2), &host) == SPX_OK &&
                 cudaHostGetDevicePointer(&found, host.host, 0) == cudaSuccess &&
                 scratch_alloc(&entries, entries_bytes, e->device, s, true) == SPX_OK;
    if (!loads) (void)cudaGetLastError();
    const size_t smem = (size_t)((chunks + 1) * kRows + chunks) * 4;
    conv_form_kernel<<<blocks, 256, smem, s>>>(e->Wd, e->idx, e->nnz, e->m, e->pitch, f, chunks, form.cap, form.units, static_cast<uint32_t*>(entries));
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) count_launch();
    if (err == cudaSuccess && loads) {
        conv_load_kernel<<<groups, 128, 0, s>>>(static_cast<uint32_t*>(entries), e->conv->ncols, e->nnz, e->m, chunks, per_group, f.chunk_cols,
                                                static_cast<CtaClocks*>(found), reinterpret_cast<uint2*>(static_cast<CtaClocks*>(found) + groups));
        err = cudaGetLastError();
        if (err == cudaSuccess) count_launch();
    }
    scratch_free(entries, s);
    const cudaError_t done = cudaStreamSynchronize(s);
    if (err == cudaSuccess) err = done;
    if (err == cudaSuccess && loads) read_loads(form, static_cast<const CtaClocks*>(host.host), groups, blocks);
    pinned_release(host);
    if (err != cudaSuccess) {
        pool_free(form.units, form.bytes, s);
        return fail(SPX_ERR_CUDA, "conv2d: building the entries' form failed: %s", cudaGetErrorString(err));
    }
    ++t->count;
    *out = &form;
    return SPX_OK;
}

namespace {

// How a batch segment on lane groups of BT entries is cut.
struct Cut {
    uint32_t S, QT, subs, TWin, THin, CC, chunks, chunk_cols, stage, stages, slot, tilesX, tiles, tile_units, groups;
    uint64_t units;
};

bool plan(const ConvParams& p, uint32_t BT, uint32_t b_len, Cut& c)
{
    const uint32_t nblocks = (p.Cout + kRows - 1) / kRows, taps = p.kH * p.kW;
    c.S = 32 / BT;
    c.QT = nblocks > 8 ? 1 : 2;             // 29 to 32 output channels (fewer do not come here): two quadrants share a tile
    c.subs = c.S * c.QT;
    c.TWin = (kTW - 1) * p.sW + (p.kW - 1) * p.dW + 1;
    c.THin = (kTH - 1) * p.sH + (p.kH - 1) * p.dH + 1;
    if (p.sW != 1 || c.TWin > 256 || c.THin > 256) return false;    // a stride would take every other column
    const uint64_t patch = (uint64_t)c.TWin * c.THin;
    if (patch > kTmemColumns / kBuffers || taps > 255) return false;
    // channels per chunk: as many as fit half the columns, bytes of counts, and shared memory beside two stages
    // (nothing here depends on BT: one form serves all segments)
    for (c.CC = std::min<uint32_t>(p.Cin, kTmemColumns / kBuffers / (uint32_t)patch); c.CC; --c.CC) {
        c.chunks = (p.Cin + c.CC - 1) / c.CC;
        c.chunk_cols = round_up(c.CC * (uint32_t)patch, 8u);
        c.stage = c.chunk_cols * 128 * c.QT;
        c.slot = 1 + kRows * ((c.CC * taps + 1) / 2);
        const uint32_t slots = kWarps * 2 * c.slot * 16 + 16;
        c.stages = slots < kSmem ? std::min(std::min(kMaxStages, c.chunks), (kSmem - slots) / c.stage) : 0;
        if (c.CC * taps <= 255 && c.stages >= std::min(2u, c.chunks)) break;
    }
    if (!c.CC || c.chunks > kMaxChunks) return false;
    c.tilesX = (p.Wo + kTW - 1) / kTW;
    const uint64_t tiles = (uint64_t)c.tilesX * ((p.Ho + kTH - 1) / kTH);
    if (tiles > 0x3fffffffull) return false;
    c.tiles = (uint32_t)tiles;
    c.tile_units = (c.tiles + c.subs - 1) / c.subs;
    c.groups = (nblocks * c.QT + kWarps - 1) / kWarps;
    c.units = (uint64_t)c.tile_units * c.groups * (b_len / BT);
    return c.units <= 0x1fffffffull;
}

// The batch in segments: all multiples of 32 with an entry per lane, the rest on lane groups of 16, 8 and 4 entries.
template <class F>
int each_segment(uint32_t B, const F& f)
{
    uint32_t at = 0;
    for (uint32_t BT = 32; BT >= 4; BT /= 2) {
        const uint32_t len = (B - at) / BT * BT;
        if (!len) continue;
        if (int rc = f(BT, at, len)) return rc;
        at += len;
    }
    return SPX_OK;
}

// A launch whose last wave is under half full issues it as CTAs of half the output channels.
enum class Tail { none, split, all };
Tail tail_of(uint64_t units, uint32_t sms)
{
    if (units * 2 <= sms) return Tail::all;
    const uint32_t rem = (uint32_t)(units % sms);
    return units > sms && rem && rem * 2 <= sms ? Tail::split : Tail::none;
}

}  // namespace

// Expected time, by the density alone (iid entries) or, where a form is there, by its loads: waves of CTAs, and results
// that are not contiguous along the batch by the million, in quads or one by one.  Launches on less than half of the SMs
// count 15 % longer: the other kernel cuts finer.  Fitted with conv_rbm_us to 400 shapes of both kernels (3 to 512
// channels, 3 x 3 and 5 x 5, 7 x 7 to 112 x 112, batch 1 to 32, 5 to 50 % dense, all layouts).
static double conv_tmem_us(const spx_ell* e, const ConvParams& p, const ConvViews& v, const conv_tmem_impl::Form* form)
{
    const uint32_t sms = (uint32_t)sm_count(e->device);
    const double density = (double)e->nnz_total / ((double)e->m * e->n);
    double clocks = 0.0;
    const int rc = each_segment(p.B, [&](uint32_t BT, uint32_t, uint32_t len) {
        Cut c;
        if (!plan(p, BT, len, c)) return -1;
        const double run = c.CC * p.kH * p.kW * density;
        const int si = c.S == 1 ? 0 : c.S == 2 ? 1 : c.S == 4 ? 2 : 3;
        const auto cta = [&](uint32_t rows) -> double {
            if (form) return form->mean.c[rows < kRows][si];
            const double quad = std::min<double>(16.0, (p.Cout + kRows - 1) / kRows * c.QT * (kRows / rows)) / 4.0;
            const double mul = std::max(quad * rows * (kEntryClocks * run + kRunClocks), rows * (kEntryLatency * run + kRunLatency) + kChunkLatency);
            return kCtaClocks + c.chunks * std::max<double>(mul, fill_clocks(c.chunk_cols, c.S));
        };
        const Tail t = tail_of(c.units, sms);
        const double full = std::floor((double)c.units / sms), rem = (double)(c.units % sms);
        double seg = t == Tail::all ? 1.15 * cta(2) : t == Tail::split ? full * cta(4) + cta(2) + 1040.0 : (full + (rem > 0)) * cta(4);
        if (form) seg = std::max<double>(seg, t == Tail::all ? 1.15 * form->worst.c[1][si] : form->worst.c[0][si]);
        clocks += seg;
        return 0;
    });
    const double strided = v.oB == 1 ? 0.0 : p.Wo % 4 == 0 ? 1.15e-6 : 7.2e-6;
    return rc ? 1e30 : clocks / 1900.0 + strided * p.Cout * p.Ho * p.Wo * p.B;
}

// The rule.  By the density: below 0.92 of the other kernel's expected time (0.85 for a batch that leaves lanes to a second
// tile), and not for few output channels with a batch that is no multiple of 16.  On the 400 shapes it was the faster
// one every time it was taken, some 115 times; picking the faster each time would gain another 1.2 % on average.  Then,
// with the form built, by what the entries' places say: below 1.04 of the other kernel's (the estimates are that close).
// Weights that are not iid need it: of 1484 measured ones (see rbm_cut) the density alone made 184 more than 10 % slower
// than the other kernel (512 -> 512, 14 x 14, batch 32, rows that share their columns, 5 % dense 76 us against 140), both
// rules leave 20 (up to 1.9) and give away more than 10 % of what the density had gained in 7 (up to 1.4).
static bool worth_it(const spx_ell* e, const ConvParams& p, const ConvViews& v, const conv_tmem_impl::Form* form,
                     double (*other_us)(const spx_ell*, const ConvParams&, const MergedLoad*))
{
    const double us = conv_tmem_us(e, p, v, form);
    if (form) return us <= 1.04 * other_us(e, p, form->merged);
    return us < 1e30 && us <= (p.B % 32 ? 0.85 : 0.92) * other_us(e, p, nullptr);
}

static int tmem_env()
{
    // the switches that force the other kernels turn this one off
    static const int env = [] {
        if (const char* v = getenv("SPX_CONV_TMEM")) return atoi(v);
        for (const char* k : {"SPX_CONV_RBM", "SPX_CONV_RBM_MIN_SHARE", "SPX_CONV_RBM_SEGMENTS", "SPX_CONV_CUT", "SPX_CONV_TMA"})
            if (getenv(k)) return 0;
        return 1;
    }();
    return env;
}

// Below 25 million FMAs a CTA's fixed cost decides (the smallest gains seen were at 16 million), and a call of 4 us
// is the host's: it does without the estimates (3 -> 32, 21 x 21, batch 8 4.3 against 4.7 us).
static bool too_small(const spx_ell* e, const ConvParams& p)
{
    return (p.B % 16 && p.Cout <= 32) || (double)e->nnz_total * p.Ho * p.Wo * p.B < 25e6;
}

double conv_tmem_expected(const spx_ell* e, const ConvParams& p, const ConvViews& v, double (*other_us)(const spx_ell*, const ConvParams&, const MergedLoad*))
{
    Cut first;
    if (!tmem_env() || !e->conv_tmem || e->tma_off || p.B % 4 || too_small(e, p) || !plan(p, 4, p.B, first) || !worth_it(e, p, v, nullptr, other_us)) return 1e30;
    return conv_tmem_us(e, p, v, nullptr);
}

template <int RW, int GP>
static int launch_units(const spx_ell* e, const TmemArgs& a, const CUtensorMap& map, uint32_t ctas, cudaStream_t s)
{
    const size_t smem = (size_t)a.stages * a.stage + kWarps * 2 * a.slot * 16 + 16;     // a unit behind the last is read, not used
    if (int rc = allow_smem<conv_tmem_kernel<RW, GP>>(e->device)) return rc;
    const cudaError_t err = launch_pdl(conv_tmem_kernel<RW, GP>, dim3(ctas), dim3((kWarps + 4) * 32), smem, s, a, map);
    if (err != cudaSuccess) return fail(SPX_ERR_CUDA, "launch of conv_tmem_kernel failed: %s", cudaGetErrorString(err));
    count_launch();
    return SPX_OK;
}

template <int GP>
static int launch_cut(const spx_ell* e, TmemArgs a, const CUtensorMap& map, uint32_t units, cudaStream_t s)
{
    const uint32_t sms = (uint32_t)sm_count(e->device);
    const Tail t = tail_of(units, sms);
    const uint32_t halved = t == Tail::all ? units : t == Tail::split ? units % sms : 0;
    if (units > halved)
        if (int rc = launch_units<4, GP>(e, a, map, units - halved, s)) return rc;
    if (!halved) return SPX_OK;
    a.unit0 = (units - halved) * 2;             // groups are the fastest: unit u is units 2u and 2u + 1 of twice the groups
    a.groups *= 2;
    return launch_units<2, GP>(e, a, map, halved * 2, s);
}

int launch_conv_tmem(spx_ell* e, const ConvParams& p, const ConvViews& v, const float* in, const float* bias, int act, float* out,
                     double (*other_us)(const spx_ell*, const ConvParams&, const MergedLoad*), cudaStream_t s)
{
    const int env = tmem_env();
    const PFN_cuTensorMapEncodeTiled encode = tensor_map_encoder();
    if (!env || !e->conv_tmem || e->tma_off || e->max_nnz == 0 || p.B % 4 || !encode) return -1;
    if (env != 2 && too_small(e, p)) return -1;
    Cut first;                                  // what the form depends on is the same for all segments
    if (!plan(p, 4, p.B, first) || (env != 2 && !worth_it(e, p, v, nullptr, other_us))) return -1;
    const conv_tmem_impl::Form* form = nullptr;
    const FormShape f{p.kH, p.kW, p.dH, p.dW, first.TWin, first.THin, first.CC, first.chunk_cols};
    if (const int rc = find_form(e, f, first.chunks, 16 / first.QT, s, &form); rc != SPX_OK) return rc;
    if (env != 2 && form->loads && !worth_it(e, p, v, form, other_us)) return -1;
    static const int short_env = [] { const char* v = getenv("SPX_CONV_TMA_TEST_TIMEOUT"); return v ? atoi(v) : 0; }();
    bool launched = false;
    return each_segment(p.B, [&](uint32_t BT, uint32_t at, uint32_t len) -> int {
        Cut c;
        plan(p, BT, len, c);
        TmemArgs a{};
        a.c = p; a.v = v;
        a.v.b_out = v.b_out > at ? v.b_out - at : 0u;
        a.units = form->units; a.cap = form->cap; a.slot = c.slot;
        a.bias = bias; a.out = out + at * v.oB; a.act = act;
        a.quads_out = v.oW == 1 && p.Wo % 4 == 0 && (v.oB | v.oC | v.oH) % 4 == 0 && reinterpret_cast<uintptr_t>(a.out) % 16 == 0;
        a.BT = BT; a.S = c.S; a.QT = c.QT;
        a.TWin = c.TWin; a.CC = c.CC; a.chunks = c.chunks; a.chunk_cols = c.chunk_cols; a.row_cols = p.sH * c.TWin;
        a.tilesX = c.tilesX; a.tiles = c.tiles; a.tile_units = c.tile_units; a.groups = c.groups;
        a.box_bytes = c.CC * c.TWin * c.THin * BT * 4;
        a.sub_stage = c.chunk_cols * BT * 4;    // a multiple of 128 bytes
        a.stage = c.stage; a.stages = c.stages;
        a.failed = e->tma_failed_dev; a.failed_host = e->tma_failed_mapped;
        if (short_env) a.missing = 16;
        // dimensions, innermost first, [B][W][H][Cin]; positions outside the tensor read as zero, which is the halo.  The
        // innermost coordinate is a multiple of BT floats from a pointer moved by a multiple of 4, as the copy unit requires.
        CUtensorMap map;
        const cuuint64_t gdim[4] = {p.B - at, p.W, p.H, p.Cin};
        const cuuint64_t gstr[3] = {v.iW * 4, v.iH * 4, v.iC * 4};
        const cuuint32_t box[4] = {BT, c.TWin, c.THin, c.CC};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        int rc = -1;
        if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(in + at), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
            rc = a.row_cols == 10 ? launch_cut<10>(e, a, map, (uint32_t)c.units, s) : launch_cut<0>(e, a, map, (uint32_t)c.units, s);
        if (rc == -1 && launched) return fail(SPX_ERR_CUDA, "conv2d: a batch segment could not be launched");
        launched = true;
        return rc;
    });
}

}  // namespace spx
