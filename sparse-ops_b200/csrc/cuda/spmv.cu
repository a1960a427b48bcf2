// spmv.cu -- ELLPACK SpMV  y = bias + E * x  for sm_100a.
//
// Replaces ellpack_matvec of the reference (src/ellpack_matvec.cpp:20-147).  The reference
// gathers x[idx] for all r slots of a row into the Xt scratch, then runs a 16-lane FMA over
// the nnz[i] live entries and a horizontal reduce.  Here the gather goes straight to
// registers: x is staged once per CTA in shared memory (random 4-byte reads cost a few bank
// conflicts there instead of one L1 line each), LPR lanes share a row and stream its Wd / idx
// slab with coalesced 16-byte loads, partial sums are combined with warp shuffles.  The
// summation order differs from the reference's 16-partial-sum order, so results agree within
// the stated tolerance 1e-5 * sum|w||x|, not bit for bit.  Padding slots are never multiplied.
//
// HBM-bound: 8 bytes per nonzero streamed once.  The kernels that stage x are launched as programmatic
// dependents: what belongs to the handle (schedule, first slab vectors) is asked for while the predecessor in the
// stream drains, and only x, bias and y wait for it.
#include "common.cuh"

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdlib>

namespace {

template <int LPR>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Asks for x[0 .. n) in shared memory, by all threads of the CTA, asynchronously: every thread's copies are
// in flight together.  landed_x(): they have landed for the whole CTA.
__device__ __forceinline__ void stage_x(float* xs, const float* __restrict__ x, uint32_t n)
{
    const uint32_t n4 = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) ? (n >> 2) : 0;
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(xs);
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * i), "l"(x + 4 * (size_t)i) : "memory");
    for (uint32_t i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + 4 * i), "l"(x + i) : "memory");
}
__device__ __forceinline__ void landed_x()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

// x beyond the windowed kernel's reach, or columns that do not ascend: x gathered through L1 / L2.
template <int LPR>
__global__ void __launch_bounds__(512, 2)
spmv_ell_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                const uint32_t* __restrict__ nnz, const uint2* __restrict__ rows,
                uint32_t m, uint32_t n, uint32_t pitch,
                const float* __restrict__ x, const float* __restrict__ bias, float* __restrict__ y)
{
    const uint32_t lane = threadIdx.x & (LPR - 1);
    const uint32_t groups_per_block = blockDim.x / LPR;
    const uint32_t group = blockIdx.x * groups_per_block + threadIdx.x / LPR;
    const uint32_t stride = gridDim.x * groups_per_block;
    // All lanes of a warp run the same number of row iterations so that the shuffles below
    // always see the full warp.
    const uint32_t iters = (m + stride - 1) / stride;

    for (uint32_t it = 0; it < iters; ++it) {
        // slots of the sorted row schedule are dealt round-robin: every group gets long and short rows
        const uint32_t slot = group + it * stride;
        const bool live = slot < m;
        const uint2 ri = live ? __ldg(rows + slot) : make_uint2(0u, 0u);
        const uint32_t row = ri.x, nn = ri.y;
        const float4* __restrict__ w4 = reinterpret_cast<const float4*>(Wd + (size_t)row * pitch);
        const uint4* __restrict__ k4 = reinterpret_cast<const uint4*>(idx + (size_t)row * pitch);
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
        // UNR 16-byte vectors of Wd and of idx in flight per lane; entries >= nn are padding and
        // are neither loaded nor multiplied
        constexpr int UNR = 4;
        for (uint32_t j = lane * 4; j < nn; j += LPR * 4 * UNR) {
            float4 wv[UNR];
            uint4 kv[UNR];
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const uint32_t ju = j + u * LPR * 4;
                if (ju < nn) {
                    wv[u] = __ldcs(w4 + (ju >> 2));
                    kv[u] = __ldcs(k4 + (ju >> 2));
                } else {
                    wv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    kv[u] = make_uint4(0u, 0u, 0u, 0u);
                }
            }
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const uint32_t ju = j + u * LPR * 4;
                if (ju < nn) a0 = fmaf(wv[u].x, __ldg(x + kv[u].x), a0);
                if (ju + 1 < nn) a1 = fmaf(wv[u].y, __ldg(x + kv[u].y), a1);
                if (ju + 2 < nn) a2 = fmaf(wv[u].z, __ldg(x + kv[u].z), a2);
                if (ju + 3 < nn) a3 = fmaf(wv[u].w, __ldg(x + kv[u].w), a3);
            }
        }
        float acc = (a0 + a1) + (a2 + a3);
        acc = group_sum<LPR>(acc);
        if (live && lane == 0) y[row] = (bias ? __ldg(bias + row) : 0.0f) + acc;
    }
}

// spmv_staged_kernel: x fits in shared memory (n <= 51200).  One CTA per SM.  Staging x, the row
// schedule, the row length and the slabs would be four memory round trips in a row, so the kernel is
// software-pipelined: a group asks for its first row's id and length and for that row's first slab vectors
// BEFORE x is staged (none of them depends on x), and while a row is summed the next row's id, length and
// first vectors are already in flight.  rows may be null (rows of near-equal length): slot == row then, and
// one dependent load goes away.  Against a kernel that starts a row when the one before is done, for all
// n (it was used up to 8192 columns): 16384 x 16384, 90 / 95 / 99 % sparse 39.0 / 22.7 / 7.5 -> 33.7 / 18.4 /
// 4.5 us; 5000 x 40000, 95 %: 28 -> 15 us; 60000 x 50000, 97 %: 143 -> 133 us.
template <int LPR>
__global__ void __launch_bounds__(1024)
spmv_staged_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                const uint32_t* __restrict__ nnz, const uint2* __restrict__ rows,
                uint32_t m, uint32_t n, uint32_t pitch,
                const float* __restrict__ x, const float* __restrict__ bias, float* __restrict__ y)
{
    extern __shared__ __align__(16) float xs[];
    constexpr int UNR = 4;                       // 16-byte vectors of Wd and of idx in flight per lane
    constexpr uint32_t STEP = LPR * 4 * UNR;     // entries a group consumes per chunk
    const uint32_t lane = threadIdx.x & (LPR - 1);
    const uint32_t groups_per_block = blockDim.x / LPR;
    // neighbouring slots go to different CTAs, so that a last, partly filled round is spread over all SMs
    const uint32_t group = threadIdx.x / LPR * gridDim.x + blockIdx.x;
    const uint32_t stride = gridDim.x * groups_per_block;
    // All lanes of a warp run the same number of row iterations so that the shuffles below
    // always see the full warp.
    const uint32_t iters = (m + stride - 1) / stride;

    float4 wv[UNR];
    uint4 kv[UNR];
    // entries >= nn are padding and are neither loaded nor multiplied
    auto load_chunk = [&](uint32_t row, uint32_t nn, uint32_t j) {
        const float4* __restrict__ w4 = reinterpret_cast<const float4*>(Wd + (size_t)row * pitch);
        const uint4* __restrict__ k4 = reinterpret_cast<const uint4*>(idx + (size_t)row * pitch);
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const uint32_t ju = j + u * LPR * 4;
            if (ju < nn) {
                wv[u] = __ldcs(w4 + (ju >> 2));
                kv[u] = __ldcs(k4 + (ju >> 2));
            } else {
                wv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                kv[u] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    // slots of the sorted row schedule are dealt round-robin: every group gets long and short rows
    uint32_t slot = group;
    bool live = slot < m;
    // rows may be null: slot == row then
    auto row_info = [&](uint32_t sl) { return rows ? __ldg(rows + sl) : make_uint2(sl, __ldg(nnz + sl)); };
    uint2 ri = live ? row_info(slot) : make_uint2(0u, 0u);
    uint32_t row = ri.x, nn = ri.y;
    load_chunk(row, nn, lane * 4);

    spx::pdl_wait();                            // x, bias and y belong to the stream's order, the handle does not
    spx::pdl_launch();
    stage_x(xs, x, n);
    landed_x();

    for (uint32_t it = 0; it < iters; ++it) {
        // the next row's id and length travel while this row is summed
        const uint32_t slot_n = slot + stride;
        const bool live_n = (it + 1 < iters) && slot_n < m;
        ri = live_n ? row_info(slot_n) : make_uint2(0u, 0u);
        const uint32_t row_n = ri.x, nn_n = ri.y;
        const float b = (live && bias) ? __ldg(bias + row) : 0.0f;

        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
        for (uint32_t j = lane * 4; j < nn; j += STEP) {
            if (j != lane * 4) load_chunk(row, nn, j);          // the first chunk is already here
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const uint32_t ju = j + u * LPR * 4;
                if (ju < nn) a0 = fmaf(wv[u].x, xs[kv[u].x], a0);
                if (ju + 1 < nn) a1 = fmaf(wv[u].y, xs[kv[u].y], a1);
                if (ju + 2 < nn) a2 = fmaf(wv[u].z, xs[kv[u].z], a2);
                if (ju + 3 < nn) a3 = fmaf(wv[u].w, xs[kv[u].w], a3);
            }
        }
        load_chunk(row_n, nn_n, lane * 4);                      // first vectors of the next row
        float acc = (a0 + a1) + (a2 + a3);
        acc = group_sum<LPR>(acc);
        if (live && lane == 0) y[row] = b + acc;
        slot = slot_n; live = live_n; row = row_n; nn = nn_n;
    }
}

// ---------------------------------------------------------------------------------------------
// x larger than shared memory: the columns are cut into equal windows, two of which fit; the kernel runs
// one phase per window, with the next window's copy in flight behind it.  In a phase every row adds the
// products of its entries whose column lies in the window (a contiguous run, columns ascend; the run's ends
// come from a per-row split table built once per handle by binary search).  Each matrix entry is read once;
// y is written in phase 0 (bias + partial) and updated by the same lane in later phases.  A row's first slab
// vectors, the next row's run and the id of the row after it are on their way while a row is summed: that,
// not the windows, is what gains (65536 x 65536, 95 % sparse: 306 us with two windows and neither, 325 with
// double-buffered windows alone, 267 with both = the time a copy of the same bytes takes; 20000 x 60000, 90 %:
// 214 -> 150 us; gathering x through L1 / L2, 32-byte sectors for 4 useful bytes: 320 and 216 us).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
spmv_splits_kernel(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ nnz, uint32_t m, uint32_t pitch,
                   uint32_t win, uint32_t bounds, uint32_t* __restrict__ split)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)m * bounds) return;
    const uint32_t row = (uint32_t)(t % m), b = (uint32_t)(t / m);
    const uint32_t bound = (b + 1) * win;
    const uint32_t* __restrict__ k = idx + (size_t)row * pitch;
    uint32_t lo = 0, hi = nnz[row];
    while (lo < hi) {                           // first entry with column >= bound
        const uint32_t mid = (lo + hi) >> 1;
        if (k[mid] < bound) lo = mid + 1; else hi = mid;
    }
    split[t] = lo;
}

template <int LPR>
__global__ void __launch_bounds__(1024)
spmv_ell_windowed_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                         const uint32_t* __restrict__ nnz, const uint2* __restrict__ rows,
                         const uint32_t* __restrict__ split, uint32_t m, uint32_t n, uint32_t win, uint32_t pitch,
                         const float* __restrict__ x, const float* __restrict__ bias, float* __restrict__ y)
{
    extern __shared__ __align__(16) float xs_all[];        // two windows of x
    const uint32_t lane = threadIdx.x & (LPR - 1);
    const uint32_t groups_per_block = blockDim.x / LPR;
    // neighbouring slots go to different CTAs, so that a last, partly filled round is spread over all SMs
    const uint32_t group = threadIdx.x / LPR * gridDim.x + blockIdx.x;
    const uint32_t stride = gridDim.x * groups_per_block;
    const uint32_t iters = (m + stride - 1) / stride;
    const uint32_t phases = (n + win - 1) / win;
    spx::pdl_wait();
    spx::pdl_launch();

    constexpr int UNR = 4;                      // 16-byte vectors of Wd and of idx in flight per lane
    float4 wv[UNR];
    uint4 kv[UNR];
    // the vectors from entry j on of a run that ends at j1; entries outside the run belong to other phases
    auto load_chunk = [&](uint32_t row, uint32_t j, uint32_t j1) {
        const float4* __restrict__ w4 = reinterpret_cast<const float4*>(Wd + (size_t)row * pitch);
        const uint4* __restrict__ k4 = reinterpret_cast<const uint4*>(idx + (size_t)row * pitch);
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const uint32_t ju = j + u * LPR * 4;
            if (ju < j1) {
                wv[u] = __ldcs(w4 + (ju >> 2));
                kv[u] = __ldcs(k4 + (ju >> 2));
            }
        }
    };
    // ids only: carrying the lengths along costs the registers of a vector in flight (313 -> 332 us at
    // 65536 x 65536, 95 % sparse)
    auto id_of = [&](uint64_t slot) { return slot < m ? __ldg(&rows[slot].x) : 0u; };

    stage_x(xs_all, x, min(win, n));
    for (uint32_t p = 0; p < phases; ++p) {
        const uint32_t lo = p * win;
        const float* xs = xs_all + (p & 1u) * win;
        // this phase's run [j0, j1) of a row: split table entries p-1 and p (0 and nnz at the ends)
        auto run_of = [&](uint64_t slot, uint32_t r, uint32_t& b0, uint32_t& b1) {
            b0 = b1 = 0;
            if (slot >= m) return;
            b0 = p ? __ldg(split + (size_t)(p - 1) * m + r) : 0u;
            b1 = (p + 1 < phases) ? __ldg(split + (size_t)p * m + r) : __ldg(nnz + r);
        };
        // A row's first vectors, the next row's run and the id of the row after it are always on their way.
        uint32_t row = id_of(group), row_next = id_of((uint64_t)group + stride);
        uint32_t j0, j1;
        run_of(group, row, j0, j1);
        load_chunk(row, (j0 & ~3u) + lane * 4, j1);
        landed_x();                             // and nobody reads the other window any more: the next one goes there
        if (p + 1 < phases) stage_x(xs_all + ((p + 1) & 1u) * win, x + lo + win, min(win, n - lo - win));

        for (uint32_t it = 0; it < iters; ++it) {
            const uint64_t slot = group + (uint64_t)it * stride;
            uint32_t n0, n1;
            run_of(slot + stride, row_next, n0, n1);
            const uint32_t row_after = id_of(slot + 2 * (uint64_t)stride);
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
            const uint32_t first = (j0 & ~3u) + lane * 4;
            for (uint32_t j = first; j < j1; j += LPR * 4 * UNR) {
                if (j != first) load_chunk(row, j, j1);
#pragma unroll
                for (int u = 0; u < UNR; ++u) {
                    const uint32_t ju = j + u * LPR * 4;
                    if (ju >= j0 && ju < j1) a0 = fmaf(wv[u].x, xs[kv[u].x - lo], a0);
                    if (ju + 1 >= j0 && ju + 1 < j1) a1 = fmaf(wv[u].y, xs[kv[u].y - lo], a1);
                    if (ju + 2 >= j0 && ju + 2 < j1) a2 = fmaf(wv[u].z, xs[kv[u].z - lo], a2);
                    if (ju + 3 >= j0 && ju + 3 < j1) a3 = fmaf(wv[u].w, xs[kv[u].w - lo], a3);
                }
            }
            load_chunk(row_next, (n0 & ~3u) + lane * 4, n1);
            float acc = (a0 + a1) + (a2 + a3);
            acc = group_sum<LPR>(acc);
            if (slot < m && lane == 0) {
                if (p == 0) y[row] = (bias ? __ldg(bias + row) : 0.0f) + acc;
                else if (j1 > j0) y[row] += acc;
            }
            row = row_next; row_next = row_after; j0 = n0; j1 = n1;
        }
    }
}

// Reference-order variant: reproduces the summation order of the reference's AVX-512 path bit for
// bit (src/ellpack_matvec.cpp:72-99): sixteen partial sums, partial l takes entries j = l, l+16, ...
// with one FMA each starting from 0; then lanes l and l+8, l and l+4, the two horizontal adds, and
// finally bias + sum.  Sixteen lanes per row; slower than the others (4-byte loads, chains of
// nnz/16), meant for checking, not for throughput.
__global__ void __launch_bounds__(256)
spmv_reforder_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                     const uint32_t* __restrict__ nnz, uint32_t m, uint32_t pitch,
                     const float* __restrict__ x, const float* __restrict__ bias, float* __restrict__ y)
{
    const uint32_t l = threadIdx.x & 15;
    const uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const bool live = row < m;
    const uint32_t nn = live ? __ldg(nnz + row) : 0u;
    const float* __restrict__ w = Wd + (size_t)(live ? row : 0) * pitch;
    const uint32_t* __restrict__ k = idx + (size_t)(live ? row : 0) * pitch;
    float a = 0.0f;
    for (uint32_t j = l; j < nn; j += 16) a = fmaf(__ldg(w + j), __ldg(x + __ldg(k + j)), a);
    a = a + __shfl_xor_sync(0xffffffffu, a, 8);      // l with l+8
    a = a + __shfl_xor_sync(0xffffffffu, a, 4);      // l with l+4
    a = a + __shfl_xor_sync(0xffffffffu, a, 1);      // (0+1), (2+3)
    a = a + __shfl_xor_sync(0xffffffffu, a, 2);      // their sum
    if (live && l == 0) y[row] = (bias ? __ldg(bias + row) : 0.0f) + a;
}

int finish(cudaError_t err, const char* name)
{
    if (err != cudaSuccess) return spx::fail(SPX_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(err));
    spx::count_launch();
    return SPX_OK;
}

constexpr uint32_t kStaged = 200 * 1024 / sizeof(float);        // columns up to which all of x is staged

template <int LPR>
int launch_lpr(const spx_ell* e, const float* x, const float* bias, float* y, cudaStream_t s)
{
    const uint64_t sms = spx::sm_count(e->device);
    if (e->n <= kStaged) {
        // Rows of near-equal length need no schedule: slot == row saves one dependent load per row.
        const uint2* order = (e->max_nnz - e->min_nnz) * 8u <= e->max_nnz ? nullptr : e->rows;
        // One CTA on every SM, with as many groups as give each the same number of rows (64 registers a
        // thread: 1024 threads are all an SM holds); fewer threads leave room for the next launch's CTAs.
        const uint64_t per = (e->m + sms - 1) / sms;
        const uint64_t iters = (per * LPR + 1023) / 1024, groups = (per + iters - 1) / iters;
        const unsigned threads = (unsigned)((groups * LPR + 31) / 32 * 32);
        const size_t smem = (size_t)e->n * sizeof(float);
        if (int rc = spx::allow_smem<spmv_staged_kernel<LPR>>(e->device)) return rc;
        return finish(spx::launch_pdl(spmv_staged_kernel<LPR>, dim3((unsigned)std::min<uint64_t>(sms, e->m)), dim3(threads), smem, s, e->Wd, e->idx, e->nnz, order,
                                      e->m, e->n, e->pitch, x, bias, y), "spmv_staged_kernel");
    }
    if (e->spmv_split) {
        const size_t smem = (size_t)e->spmv_win * 2 * sizeof(float);
        if (int rc = spx::allow_smem<spmv_ell_windowed_kernel<LPR>>(e->device)) return rc;
        return finish(spx::launch_pdl(spmv_ell_windowed_kernel<LPR>, dim3((unsigned)std::min<uint64_t>(sms, e->m)), dim3(1024), smem, s, e->Wd, e->idx, e->nnz, e->rows,
                                      e->spmv_split, e->m, e->n, e->spmv_win, e->pitch, x, bias, y), "spmv_ell_windowed_kernel");
    }
    // as many CTAs as give every group the same number of rows
    const uint64_t per_block = 512 / LPR, rounds = (e->m + sms * 4 * per_block - 1) / (sms * 4 * per_block);
    const uint64_t blocks = (e->m + rounds * per_block - 1) / (rounds * per_block);
    spmv_ell_kernel<LPR><<<(unsigned)blocks, 512, 0, s>>>(e->Wd, e->idx, e->nnz, e->rows, e->m, e->n, e->pitch, x, bias, y);
    SPX_LAUNCH_CHECK("spmv_ell_kernel");
    return SPX_OK;
}

// Lanes per row.  A lane consumes 16 entries per round trip, so long rows want many lanes and short ones few.
// Staged x: all rows of an SM at once, if 1024 threads carry them that way, is best -- the fewest rounds and
// row changes (16384 x 16384, 90 %: 33.7 us with 8 lanes, 36 with 16 or 32; 33088 x 3904, 402 entries: 19.3 us
// with 4, 20.2 with 32) -- as long as a row takes at most 16 rounds (26877 x 24384, 2377 entries: 81 us with
// 8 lanes, 79 with 16) and no lane idles for most of a row.
int lanes_per_row(const spx_ell* e)
{
    const double windows = e->spmv_split ? (double)((e->n + e->spmv_win - 1) / e->spmv_win) : 1.0;
    const double mean = (double)e->nnz_total / e->m / windows;
    if (e->spmv_split) return mean > 300.0 ? 32 : mean > 100.0 ? 16 : mean > 40.0 ? 8 : 4;
    const uint64_t per = (e->m + spx::sm_count(e->device) - 1) / spx::sm_count(e->device);
    if (e->n > kStaged || per * 4 > 1024) return mean > 192.0 ? 32 : mean > 96.0 ? 16 : mean > 40.0 ? 8 : 4;
    int lpr = 32;
    while (lpr > 4 && (per * lpr > 1024 || (lpr > 8 && mean / 12.0 < lpr))) lpr /= 2;
    while (lpr < 32 && mean > 16.0 * 16 * lpr) lpr *= 2;
    return lpr;
}

}  // namespace

namespace spx {

int launch_spmv_reforder(const spx_ell* e, const float* x, const float* bias, float* y, cudaStream_t s)
{
    if (e->m == 0) return SPX_OK;
    const uint64_t threads = (uint64_t)e->m * 16;
    spmv_reforder_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(e->Wd, e->idx, e->nnz, e->m, e->pitch, x, bias, y);
    SPX_LAUNCH_CHECK("spmv_reforder_kernel");
    return SPX_OK;
}

// x beyond shared memory: up to kMaxWindows equal column windows of at most 104 KB (two at a time are
// staged); the per-row split table ((windows - 1) * m entries) is built on the first call and kept.
static int ensure_spmv_windows(spx_ell* e, cudaStream_t s)
{
    constexpr uint32_t kWinMax = 104 * 1024 / sizeof(float), kMaxWindows = 16;
    static const int enabled = [] { const char* v = getenv("SPX_SPMV_WINDOWED"); return v ? atoi(v) : 1; }();
    if (e->spmv_split || e->spmv_win == UINT32_MAX) return SPX_OK;
    e->spmv_win = UINT32_MAX;                                       // decided: stays "no" unless built below
    if (!enabled || !e->cols_ascending || e->n <= kStaged || e->max_nnz == 0) return SPX_OK;
    const uint32_t windows = (e->n + kWinMax - 1) / kWinMax;
    if (windows > kMaxWindows) return SPX_OK;
    const uint32_t win = round_up((e->n + windows - 1) / windows, 4u);
    const uint64_t entries = (uint64_t)e->m * (windows - 1);
    if (pool_alloc_now(reinterpret_cast<void**>(&e->spmv_split), entries * sizeof(uint32_t), e->device) != SPX_OK) {
        e->spmv_split = nullptr;
        return SPX_OK;                                              // no room: gather x from global memory
    }
    e->spmv_split_bytes = entries * sizeof(uint32_t);
    spmv_splits_kernel<<<(unsigned)((entries + 255) / 256), 256, 0, s>>>(e->idx, e->nnz, e->m, e->pitch, win, windows - 1,
                                                                       e->spmv_split);
    SPX_LAUNCH_CHECK("spmv_splits_kernel");
    e->spmv_win = win;
    return SPX_OK;
}

int launch_spmv(spx_ell* e, const float* x, const float* bias, float* y, cudaStream_t s)
{
    if (e->m == 0) return SPX_OK;
    static const bool exact = [] { const char* v = getenv("SPX_SPMV_REFERENCE_ORDER"); return v && v[0] == '1'; }();
    if (exact) return launch_spmv_reforder(e, x, bias, y, s);
    const int rcw = ensure_spmv_windows(e, s);
    if (rcw != SPX_OK) return rcw;
    switch (lanes_per_row(e)) {
    case 32: return launch_lpr<32>(e, x, bias, y, s);
    case 16: return launch_lpr<16>(e, x, bias, y, s);
    case 8:  return launch_lpr<8>(e, x, bias, y, s);
    default: return launch_lpr<4>(e, x, bias, y, s);
    }
}

}  // namespace spx
