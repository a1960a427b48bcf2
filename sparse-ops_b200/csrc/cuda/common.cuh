// common.cuh -- shared declarations of the CUDA side of libspx_b200.so (sm_100a only).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "spx_b200.h"

namespace spx {
struct PinnedBlock {
    void* host = nullptr;
    size_t bytes = 0;
};
struct ConvTables;
}  // namespace spx

// Device-resident ELLPACK (see include/spx_b200.h).  Row i occupies entries
// [i*pitch, i*pitch + nnz[i]) of Wd / idx; pitch is a multiple of 32 entries so that
// every row starts on a 128-byte boundary and float4 / uint4 loads are aligned.
struct spx_ell {
    int device = 0;
    uint32_t m = 0, n = 0, r = 0;
    uint32_t pitch = 0;          // row pitch in entries (0 when r == 0)
    uint64_t nnz_total = 0;
    uint32_t max_nnz = 0;        // longest row actually stored (<= r)
    uint32_t min_nnz = 0;        // shortest row
    float* Wd = nullptr;         // m * pitch floats
    uint32_t* idx = nullptr;     // m * pitch column ids
    uint32_t* nnz = nullptr;     // m counts
    // Row schedule: (row id, nnz) sorted by descending nnz (ties by ascending id).  Kernels that give
    // a warp one row take rows in this order, so the warps of a CTA get rows of equal length
    // (no warp idles behind a long row) and the longest rows start first.  The length sits beside the
    // id so that a warp needs one load, not two dependent ones, before it can ask for its slab.
    uint2* rows = nullptr;           // m entries
    uint32_t long_rows = 0;          // rows with at least 512 stored entries (a prefix of rows)
    // True when every row's stored column ids are strictly ascending (always so for handles made
    // from CSR, from a dense matrix or by the encoders; checked at upload for raw arrays).  The
    // tiled convolution kernels rely on it; without it the convolution takes the general kernel.
    bool cols_ascending = true;
    // Raised by a convolution kernel whose bounded wait for a bulk tensor copy ran out: a word in
    // device memory (read by the kernel's later CTAs) and a word in pinned host memory (its device
    // alias is tma_failed_mapped; read by the next convolution call on the handle).
    std::atomic<int*> tma_failed_host{nullptr};     // set last: the others are there when it is seen
    spx::PinnedBlock tma_failed_block;
    int* tma_failed_mapped = nullptr;
    int* tma_failed_dev = nullptr;
    std::atomic<bool> tma_off{false};
    // Tiled form of the matrix for spmm_tile.cu, built on the second SpMM call that can use it.
    void* tiles = nullptr;
    // Tap tables and merged weights of the convolution, and how the entries lie for it (conv.cuh).
    spx::ConvTables* conv = nullptr;
    // The convolution's entries for conv_tmem.cu, built on the first call that uses them.
    void* conv_tmem = nullptr;
    // SpMV with x larger than shared memory (spmv.cu): column window width and the per-row split
    // table, built on the first spx_spmv of such a handle.  spmv_win == UINT32_MAX: not applicable.
    uint32_t* spmv_split = nullptr;
    size_t spmv_split_bytes = 0;
    uint32_t spmv_win = 0;
    // Pinned + device staging for the host-buffer entry points (abi.cu), grown on demand.
    void* stage_dev = nullptr;
    size_t stage_dev_bytes = 0;
    // Streams of the pipelined host-buffer SpMM (copy in, exchange, multiply, copy out) and the events
    // that chain and time its stages, created on first use and kept.
    cudaStream_t pipe_streams[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t pipe_events[64] = {};
    // Row slices for the copy-engine exchange (spx_spmm_exchange, abi.cu): handles over contiguous
    // row ranges of this one that share its Wd / idx / nnz arrays and own only their row schedule
    // (view == true for such a handle).  slice_row0[k] is slice k's first row; the streams carry
    // the peer copies, the events chain them to the multiplications.
    bool view = false;
    uint32_t nslices = 0;
    spx_ell* slices[16] = {};
    uint32_t slice_row0[17] = {};
    cudaStream_t xchg_streams[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t xchg_events[24] = {};
};

namespace spx {

int fail(int code, const char* fmt, ...);
extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }
void count_launch_beside();     // of a kernel that runs at once although the call is being recorded: not one of the graph's
int sm_count(int device);

// Rounds up to a multiple of `to`.
template <class T> __host__ __device__ inline T round_up(T v, T to) { return (v + to - 1) / to * to; }

__device__ __forceinline__ float apply_act(float v, int act) {
    // Precise expf / tanhf: the library is built without fast-math so that sigmoid and tanh
    // stay within a few ulp of the C library results of the reference.
    switch (act) {
    case SPX_ACT_RELU:    return v > 0.0f ? v : 0.0f;
    case SPX_ACT_SIGMOID: return 1.0f / (1.0f + expf(-v));
    case SPX_ACT_TANH:    return tanhf(v);
    default:              return v;
    }
}

// Programmatic dependent launch: a kernel launched with launch_pdl() may start while its predecessor
// in the stream is still draining.  Before pdl_wait() it may only touch what no kernel of the stream
// writes -- the arrays of a finished handle; after it everything the predecessors wrote is visible.
// pdl_launch() lets the successor in as soon as every CTA of this grid has reached it; it comes after
// pdl_wait(), so that one successor waits and not a row of them (three that pile up: 645 x 5312, C = 32
// 24.3 us against 15.7).  Every thread calls pdl_wait() before it leaves.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// (a0, a1) += w * (x0, x1) with ONE instruction: sm_100a's packed fma.rn.f32x2.  Each half is an
// IEEE fused multiply-add rounded to nearest -- exactly fmaf -- so chains stay bit-identical while
// the FMA instruction count halves.  The 64-bit pairs are formed inside the block, which leaves
// the register allocator free to keep the operands in adjacent registers.
__device__ __forceinline__ void fma_pair(float& a0, float& a1, float w, float x0, float x1) {
    asm("{\n\t.reg .b64 pa, px, pw;\n\tmov.b64 pa, {%0, %1};\n\tmov.b64 px, {%3, %4};\n\tmov.b64 pw, {%2, %2};\n\t"
        "fma.rn.f32x2 pa, pw, px, pa;\n\tmov.b64 {%0, %1}, pa;\n\t}"
        : "+f"(a0), "+f"(a1) : "f"(w), "f"(x0), "f"(x1));
}

}  // namespace spx

#define SPX_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t _e = (call);                                                           \
        if (_e != cudaSuccess)                                                             \
            return spx::fail(_e == cudaErrorMemoryAllocation ? SPX_ERR_OOM : SPX_ERR_CUDA, \
                             "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e),       \
                             __FILE__, __LINE__);                                          \
    } while (0)

#define SPX_LAUNCH_CHECK(name)                                                             \
    do {                                                                                   \
        cudaError_t _e = cudaGetLastError();                                               \
        if (_e != cudaSuccess)                                                             \
            return spx::fail(SPX_ERR_CUDA, "launch of %s failed: %s", name,                \
                             cudaGetErrorString(_e));                                      \
        spx::count_launch();                                                               \
    } while (0)

// Kernel launchers implemented in the individual .cu files.
namespace spx {
// again: a further part of a call that has been counted (a matrix gets its block form on its second call).
int launch_spmm(const spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias,
                int act, float* Y, uint64_t ldy, cudaStream_t s, bool again = false);
int launch_spmm_bcast(const spx_ell* e, const float* X, uint32_t C, uint64_t ldx, const float* bias, int act,
                      float* const* Ys, uint32_t npeers, uint64_t row0, uint64_t ldy, cudaStream_t s, bool mcast = false,
                      bool again = false);
void* new_tiles();
void free_tiles(spx_ell* e);
int launch_spmv(spx_ell* e, const float* x, const float* bias, float* y, cudaStream_t s);
int launch_spmv_reforder(const spx_ell* e, const float* x, const float* bias, float* y, cudaStream_t s);
int launch_conv2d(spx_ell* e, const spx_conv_geom* g, int layout, const float* in, uint32_t B,
                  const float* bias, int act, float* out, cudaStream_t s);
int launch_eltwise(int op, const float* a, const float* b, float* out, uint64_t count, cudaStream_t s);
int encode_device(const float* dW, uint32_t m, uint32_t n, cudaStream_t s, spx_ell** out);
int decode_device(const spx_ell* e, float* dW, cudaStream_t s);
int csr_to_ell_device(spx_ell* e, const uint64_t* d_rowptr, const uint32_t* d_col, const float* d_val,
                      cudaStream_t s);
// zero_fill: whether the slabs and counts are cleared on s (a caller that writes every slot passes false).
int alloc_ell(uint32_t m, uint32_t n, uint32_t r, spx_ell** out, cudaStream_t s, bool zero_fill = true);
int check_current_device(const spx_ell* e, const char* what);
// Builds e->rows from host row counts (counting sort by length) and uploads it.
int set_row_order(spx_ell* e, const uint32_t* host_nnz);
// The sort behind it: fills order[m], and the handle's long_rows / min_nnz; e->rows is allocated.
int sort_rows(spx_ell* e, const uint32_t* host_nnz, uint2* order, cudaStream_t s);

// Lets a kernel have all the dynamic shared memory a CTA can get.  The limit belongs to the function and not to a
// launch: were it set to each launch's own size, another thread's call could lower it between this one's setting and
// its launch, which would be refused.  So it is set once per kernel and device, to the most.
int allow_smem(const void* kernel, int device, std::atomic<uint64_t>& done);     // mem.cu
template <auto Kernel>
int allow_smem(int device)
{
    static std::atomic<uint64_t> done{0};           // a bit per device
    if (device < 64 && (done.load(std::memory_order_relaxed) >> device & 1)) return SPX_OK;
    return allow_smem(reinterpret_cast<const void*>(Kernel), device, done);
}

// While it lives, this thread may allocate and wait although it is recording a graph on another stream (such a call
// would otherwise end that capture with an error).  What runs under it does not touch the stream being recorded.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    RelaxedCapture(const RelaxedCapture&) = delete;
};

// Device memory from the library's pool of the given device, stream-ordered (mem.cu).
int pool_alloc(void** p, size_t bytes, int device, cudaStream_t s, bool optional = false);   // optional: as below
void pool_free(void* p, size_t bytes, cudaStream_t s);      // bytes as allocated; p may be null
int scratch_alloc(void** p, size_t bytes, int device, cudaStream_t s, bool optional = false);   // for one call: allocated and freed in stream order
void scratch_free(void* p, cudaStream_t s);
int pool_alloc_now(void** p, size_t bytes, int device);     // usable on every stream at once
// Host -> device copy in stream order; pageable sources are staged by several threads (hostcopy.cu).
int copy_h2d(void* dst, const void* src, size_t bytes, cudaStream_t s);
// The same for rows of `row` bytes, `stride` bytes apart, to contiguous device memory.
int copy_h2d_rows(void* dst, const void* src, size_t rows, size_t row, size_t stride, cudaStream_t s);
bool pageable_memory(const void* p);            // host memory that is not page-locked
// Replaces a handle's scratch block by a larger one (waits for the device: kernels may still use the old one).
int grow_scratch(spx_ell* e, void** p, size_t* bytes, size_t need);
void wait_for_device();                         // for all work on the current device
void pool_trim(int device);                     // waits for the device, then gives all free memory back
// A non-blocking stream per device for small transfers beside the caller's stream, created once (mem.cu).
int side_stream(int device, cudaStream_t* out);
// The calling thread's streams for its host-buffer calls on a device: 0 for all of a call, or copies in (0),
// multiplies (1) and copies out (2).
int host_stream(int device, int which, cudaStream_t* out);
// Pinned host memory from a bounded free list (mem.cu).
int pinned_acquire(size_t bytes, PinnedBlock* out);
void pinned_release(const PinnedBlock& b);
}  // namespace spx
