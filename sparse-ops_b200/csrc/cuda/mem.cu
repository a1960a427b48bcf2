// mem.cu -- device and pinned-host memory that outlives a single call.
//
// Device: the arrays of an ELLPACK handle come from one CUDA memory pool per device.  cudaMalloc and
// cudaFree cost 50 us to several milliseconds each here (page mapping, and an implicit wait for the
// whole device in every free); a program that re-encodes a weight each step paid that a dozen times
// per handle (encode + decode + destroy of an 8192 x 8192 matrix: 2.4 ms, of which the kernels were
// 0.2 ms).  The pool keeps at most kPoolKeep bytes of freed memory per device, gives everything above
// that back at the next synchronisation, and all of it when an allocation of this library fails.
// The driver's pool is safe to use from several threads and streams.
//
// Pinned host: staging blocks for transfers, kept on a free list of at most kPinnedKeep bytes.
#include "common.cuh"
#include "tma.cuh"

#include <cstdlib>
#include <mutex>
#include <vector>

namespace spx {

namespace {

constexpr uint64_t kPoolKeep = 2ull << 30;          // of about 180 GB
// Larger blocks are mapped and unmapped directly: growing the pool by them takes longer than cudaMalloc
// (slabs of 2 x 323 MB: 9 ms against 5), and a few of them are all the pool would keep.
constexpr size_t kPoolBlock = 128u << 20;
constexpr size_t kPinnedKeep = 64u << 20;
constexpr int kMaxDevices = 64;

std::mutex g_pool_mu;
cudaMemPool_t g_pools[kMaxDevices] = {};

int device_pool(int device, cudaMemPool_t* out)
{
    if (device < 0 || device >= kMaxDevices) return fail(SPX_ERR_LIMIT, "device ordinal %d not supported", device);
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pools[device]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        SPX_CUDA(cudaMemPoolCreate(&p, &props));
        uint64_t keep = kPoolKeep;
        SPX_CUDA(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pools[device] = p;
    }
    *out = g_pools[device];
    return SPX_OK;
}

std::mutex g_pinned_mu;
std::vector<PinnedBlock> g_pinned;                  // free blocks
size_t g_pinned_bytes = 0;

}  // namespace

static int allocate(void** p, size_t bytes, int device, cudaStream_t s, bool pooled, bool trim = true)
{
    *p = nullptr;
    if (bytes == 0) return SPX_OK;
    cudaMemPool_t pool = nullptr;
    if (int rc = device_pool(device, &pool)) return rc;
    auto get = [&] { return pooled ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMalloc(p, bytes); };
    cudaError_t err = get();
    if (err == cudaErrorMemoryAllocation && trim) {
        (void)cudaGetLastError();
        pool_trim(device);
        err = get();
    }
    if (err != cudaSuccess) {
        (void)cudaGetLastError();
        *p = nullptr;
        return fail(err == cudaErrorMemoryAllocation ? SPX_ERR_OOM : SPX_ERR_CUDA, "device allocation of %zu bytes failed: %s",
                    bytes, cudaGetErrorString(err));
    }
    return SPX_OK;
}

// optional: the caller can do without, and is told at once; to give memory back first would wait for the whole device.
int pool_alloc(void** p, size_t bytes, int device, cudaStream_t s, bool optional) { return allocate(p, bytes, device, s, bytes <= kPoolBlock, !optional); }

// Scratch of one call, whatever its size: mapping and freeing memory directly would make the call wait for the device.
int scratch_alloc(void** p, size_t bytes, int device, cudaStream_t s, bool optional) { return allocate(p, bytes, device, s, true, !optional); }
void scratch_free(void* p, cudaStream_t s) { if (p) (void)cudaFreeAsync(p, s); }

void pool_free(void* p, size_t bytes, cudaStream_t s)
{
    if (p) (void)(bytes > kPoolBlock ? cudaFree(p) : cudaFreeAsync(p, s));
}

// Memory that is used on other streams than the one at hand, or while a stream is being captured: it comes
// through the side stream and is there when the call returns.
int pool_alloc_now(void** p, size_t bytes, int device)
{
    cudaStream_t side = nullptr;
    if (int rc = side_stream(device, &side)) return rc;
    if (int rc = pool_alloc(p, bytes, device, side)) return rc;
    if (bytes && cudaStreamSynchronize(side) != cudaSuccess) {
        (void)cudaGetLastError();
        pool_free(*p, bytes, side);
        *p = nullptr;
        return fail(SPX_ERR_CUDA, "device allocation of %zu bytes failed", bytes);
    }
    return SPX_OK;
}

// cudaDeviceSynchronize would end every stream capture in the process with an error, other threads' too; the free of
// mapped memory waits for the device as well and leaves their captures alone (4 us for the pair, as for the other).
// A small block that stays keeps their mapping: without it 0.7 ms.
void wait_for_device()
{
    static std::atomic<void*> anchors[kMaxDevices] = {};
    int device = -1;
    if (cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < kMaxDevices && !anchors[device].load()) {
        void *a = nullptr, *none = nullptr;
        if (cudaMalloc(&a, 256) == cudaSuccess && !anchors[device].compare_exchange_strong(none, a)) (void)cudaFree(a);
    }
    void* p = nullptr;
    if (cudaMalloc(&p, 256) == cudaSuccess && cudaFree(p) == cudaSuccess) return;
    (void)cudaGetLastError();
    (void)cudaDeviceSynchronize();
    (void)cudaGetLastError();
}

int grow_scratch(spx_ell* e, void** p, size_t* bytes, size_t need)
{
    if (*p) {
        wait_for_device();
        pool_free(*p, *bytes, nullptr);
    }
    *p = nullptr;
    *bytes = 0;
    if (int rc = pool_alloc_now(p, need, e->device)) return rc;
    *bytes = need;
    return SPX_OK;
}

void pool_trim(int device)
{
    if (device < 0 || device >= kMaxDevices) return;
    wait_for_device();
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pools[device]) (void)cudaMemPoolTrimTo(g_pools[device], 0);
}

static int kept_stream(cudaStream_t (&streams)[kMaxDevices], int device, cudaStream_t* out)
{
    if (device < 0 || device >= kMaxDevices) return fail(SPX_ERR_LIMIT, "device ordinal %d not supported", device);
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!streams[device]) SPX_CUDA(cudaStreamCreateWithFlags(&streams[device], cudaStreamNonBlocking));
    *out = streams[device];
    return SPX_OK;
}

int side_stream(int device, cudaStream_t* out)
{
    static cudaStream_t streams[kMaxDevices] = {};
    return kept_stream(streams, device, out);
}

int host_stream(int device, int which, cudaStream_t* out)
{
    struct Streams {                            // threads that make host-buffer calls do not wait for one another
        cudaStream_t s[3][kMaxDevices] = {};
        ~Streams() { for (auto& k : s) for (cudaStream_t st : k) if (st) (void)cudaStreamDestroy(st); }
    };
    thread_local Streams mine;
    return kept_stream(mine.s[which], device, out);
}

int pinned_acquire(size_t bytes, PinnedBlock* out)
{
    *out = PinnedBlock{};
    const size_t want = round_up<size_t>(bytes ? bytes : 1, 64 * 1024);
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        size_t best = SIZE_MAX;
        for (size_t i = 0; i < g_pinned.size(); ++i)        // smallest that fits and is not four times too large
            if (g_pinned[i].bytes >= want && g_pinned[i].bytes / 4 <= want && (best == SIZE_MAX || g_pinned[i].bytes < g_pinned[best].bytes))
                best = i;
        if (best != SIZE_MAX) {
            *out = g_pinned[best];
            g_pinned_bytes -= out->bytes;
            g_pinned[best] = g_pinned.back();
            g_pinned.pop_back();
            return SPX_OK;
        }
    }
    // portable: usable from every device's context; mapped: kernels may store small results into it
    SPX_CUDA(cudaHostAlloc(&out->host, want, cudaHostAllocPortable | cudaHostAllocMapped));
    out->bytes = want;
    return SPX_OK;
}

void pinned_release(const PinnedBlock& b)
{
    if (!b.host) return;
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        if (g_pinned_bytes + b.bytes <= kPinnedKeep) {
            g_pinned.push_back(b);
            g_pinned_bytes += b.bytes;
            return;
        }
    }
    (void)cudaFreeHost(b.host);
}

int allow_smem(const void* kernel, int device, std::atomic<uint64_t>& done)
{
    int most = 0;
    cudaFuncAttributes fa{};
    SPX_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    SPX_CUDA(cudaFuncGetAttributes(&fa, kernel));
    SPX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes));
    if (device < 64) done.fetch_or(1ull << device, std::memory_order_relaxed);
    return SPX_OK;
}

// Any of a handle's calls may be the first to need them, on any thread.
void ensure_tma_words(spx_ell* e)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    PinnedBlock block;
    if (e->tma_failed_host.load(std::memory_order_relaxed) || pinned_acquire(sizeof(int), &block) != SPX_OK) return;
    int* host = static_cast<int*>(block.host);
    *host = 0;                                  // (the block may have served before)
    cudaStream_t side = nullptr;
    if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&e->tma_failed_mapped), host, 0) != cudaSuccess ||
        side_stream(e->device, &side) != SPX_OK ||
        pool_alloc(reinterpret_cast<void**>(&e->tma_failed_dev), sizeof(int), e->device, side) != SPX_OK ||
        cudaMemsetAsync(e->tma_failed_dev, 0, sizeof(int), side) != cudaSuccess || cudaStreamSynchronize(side) != cudaSuccess) {
        e->tma_failed_mapped = nullptr;
        pool_free(e->tma_failed_dev, sizeof(int), side);
        e->tma_failed_dev = nullptr;
        (void)cudaGetLastError();
    }
    e->tma_failed_block = block;
    e->tma_failed_host.store(host, std::memory_order_release);
}

int check_tma_words(spx_ell* e, const char* what)
{
    volatile int* failed = e->tma_failed_host.load(std::memory_order_acquire);
    if (!failed || !*failed) return SPX_OK;
    *failed = 0;
    e->tma_off = true;
    return fail(SPX_ERR_CUDA, "%s: a bulk tensor copy of a call on this handle did not complete; that call's output is invalid", what);
}

PFN_cuTensorMapEncodeTiled tensor_map_encoder()
{
    static const PFN_cuTensorMapEncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(p);
    }();
    return fn;
}

}  // namespace spx
