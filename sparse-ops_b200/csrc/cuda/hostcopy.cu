// hostcopy.cu -- host -> device copies of ordinary (pageable) memory.
//
// cudaMemcpyAsync stages such memory through its own pinned buffer with ONE thread: 4 MB take 270 us
// (15 GB/s) where the PCIe link moves them in 87.  Here the calling thread and two helpers copy 256 KB
// pieces into a pinned ring and each piece is sent on as soon as it and its predecessors are there, so
// the link, not memcpy, decides the time: 4 MB in 125 us (183 us with stores that stay in the cores'
// caches, where the copy unit has to fetch them from; 3 to 11 helpers or pieces of 128 KB: no difference).
// The rows of a column panel are packed on the way.  Semantics are those of cudaMemcpyAsync from pageable
// memory: the source may be reused when the call returns, the device sees the data in stream order.
#include "common.cuh"

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#if defined(__x86_64__)
#include <immintrin.h>
#define SPX_PAUSE() _mm_pause()
#else
#define SPX_PAUSE() std::this_thread::yield()
#endif

namespace spx {

namespace {

constexpr size_t kPiece = 256 * 1024;
constexpr uint32_t kPieces = 16;                // per segment: half of the ring
constexpr size_t kSegment = kPiece * kPieces;
constexpr int kMaxDevices = 64;

// The copy unit reads what was just written: stores that bypass the caches leave it in memory, where it
// is fetched at link speed; from dirty lines of the cores' caches it comes at a third of that.
void copy_piece(char* dst, const char* src, size_t bytes)
{
#if defined(__SSE2__)
    size_t i = 0;
    if (reinterpret_cast<uintptr_t>(dst) & 15) {
        std::memcpy(dst, src, bytes);
        return;
    }
    for (; i + 64 <= bytes; i += 64) {
        const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i));
        const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 16));
        const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 32));
        const __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 48));
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i), a);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 32), c);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 48), d);
    }
    if (i < bytes) std::memcpy(dst + i, src + i, bytes - i);
#else
    std::memcpy(dst, src, bytes);
#endif
}

// Helpers for one copy at a time.  A ticket holds the number of pieces of the current segment beside the
// next piece to take, so whoever draws a valid one knows that the segment it read belongs to it:
// the segment's fields do not change until all its pieces are done.  The caller draws tickets too and
// waits only for pieces a helper has drawn, so a process without helpers (after a fork, or where
// threads cannot be started) makes the same progress alone.
class Helpers {
public:
    static Helpers& get() {
        static Helpers* h = new Helpers();      // never destroyed: its threads run until the process ends
        return *h;
    }
    std::mutex user;                            // held for the duration of a copy

    // `rows` rows of `row` bytes, `stride` bytes apart, to contiguous memory; `per` rows are a piece.
    void open(char* dst, const char* src, size_t rows, size_t row, size_t stride, size_t per) {
        dst_ = dst; src_ = src; rows_ = rows; row_ = row; stride_ = stride; per_ = per;
        const uint32_t n = (uint32_t)((rows + per - 1) / per);
        for (uint32_t i = 0; i < n; ++i) done_[i].store(0, std::memory_order_relaxed);
        ticket_.store((uint64_t)n << 32, std::memory_order_release);
        if (n > 1) {
            start();
            { std::lock_guard<std::mutex> lk(mu_); }
            cv_.notify_all();
        }
    }
    bool work() {                               // copies one piece, if there is one left to take
        const uint64_t v = ticket_.fetch_add(1, std::memory_order_acq_rel);
        const uint32_t i = (uint32_t)v;
        if (i >= (uint32_t)(v >> 32)) return false;
        const size_t r0 = i * per_, r1 = std::min(rows_, r0 + per_);
        if (row_ == stride_) copy_piece(dst_ + r0 * row_, src_ + r0 * row_, (r1 - r0) * row_);
        else for (size_t r = r0; r < r1; ++r) copy_piece(dst_ + r * row_, src_ + r * stride_, row_);
#if defined(__SSE2__)
        _mm_sfence();                           // the streaming stores, then the flag
#endif
        done_[i].store(1, std::memory_order_release);
        return true;
    }
    bool done(uint32_t i) const { return done_[i].load(std::memory_order_acquire) != 0; }

private:
    bool idle() const {
        const uint64_t v = ticket_.load(std::memory_order_acquire);
        return (uint32_t)v >= (uint32_t)(v >> 32);
    }
    void start() {
        if (started_) return;
        started_ = true;
        const unsigned hw = std::thread::hardware_concurrency();
        for (unsigned t = 0; t < (hw >= 8 ? 2u : hw >= 4 ? 1u : 0u); ++t) {
            try {
                std::thread([this] { loop(); }).detach();
            } catch (...) {
                break;
            }
        }
    }
    void loop() {
        for (;;) {
            while (work()) {}
            for (int spin = 0; spin < 2000 && idle(); ++spin) SPX_PAUSE();     // some tens of us: the next segment
            if (idle()) {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [this] { return !idle(); });
            }
        }
    }
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t rows_ = 0, row_ = 0, stride_ = 0, per_ = 1;
    std::atomic<uint64_t> ticket_{0};
    std::atomic<uint8_t> done_[kPieces] = {};
    std::mutex mu_;
    std::condition_variable cv_;
    bool started_ = false;
};

// Two segments of pinned memory for the whole process, and per device the events after which a half is free.
struct Ring {
    char* half[2] = {nullptr, nullptr};
    cudaEvent_t free_at[kMaxDevices][2] = {};
    int last_device[2] = {-1, -1};
    uint32_t turn = 0;
};
Ring g_ring;                                    // guarded by Helpers::user

}  // namespace

bool pageable_memory(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

// A copy that is being recorded into a graph stays one copy node on the caller's memory: what the ring holds and
// what its events stand for belong to this call, not to the graph's launches.
static bool being_captured(cudaStream_t s)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();
    return true;
}

// Whether the stream belongs to the device: the ring's events are made on the current one and can be recorded on no other's.
static bool stream_of(cudaStream_t s, int device)
{
    int owner = device;
    if (!s || s == cudaStreamLegacy || s == cudaStreamPerThread) return true;
    if (cudaStreamGetDevice(s, &owner) == cudaSuccess) return owner == device;
    (void)cudaGetLastError();
    return false;
}

int copy_h2d_rows(void* dst, const void* src, size_t rows, size_t row, size_t stride, cudaStream_t s)
{
    const size_t bytes = rows * row;
    if (bytes == 0) return SPX_OK;
    const auto plain = [&]() -> int {
        if (row == stride) SPX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
        else SPX_CUDA(cudaMemcpy2DAsync(dst, row, src, stride, row, rows, cudaMemcpyHostToDevice, s));
        return SPX_OK;
    };
    int device = -1;
    if (bytes < kPiece || row > kPiece || !pageable_memory(src) || being_captured(s) || cudaGetDevice(&device) != cudaSuccess ||
        device < 0 || device >= kMaxDevices || !stream_of(s, device))
        return plain();
    RelaxedCapture relaxed;                     // allocations and waits of the ring: no business of a capture on another stream
    Helpers& h = Helpers::get();
    std::unique_lock<std::mutex> lk(h.user, std::try_to_lock);
    if (lk.owns_lock() && !g_ring.half[0]) {
        void* p = nullptr;
        if (cudaHostAlloc(&p, 2 * kSegment, cudaHostAllocPortable) == cudaSuccess) {
            g_ring.half[0] = static_cast<char*>(p);
            g_ring.half[1] = g_ring.half[0] + kSegment;
        } else {
            (void)cudaGetLastError();
        }
    }
    if (!lk.owns_lock() || !g_ring.half[0]) return plain();     // another thread is copying: the driver's way
    const size_t per = kPiece / row, segment = per * kPieces;   // rows
    for (size_t r0 = 0; r0 < rows; r0 += segment) {
        const uint32_t half = g_ring.turn++ & 1u;
        const size_t len = std::min(segment, rows - r0);
        if (g_ring.last_device[half] >= 0) SPX_CUDA(cudaEventSynchronize(g_ring.free_at[g_ring.last_device[half]][half]));
        if (!g_ring.free_at[device][half]) SPX_CUDA(cudaEventCreateWithFlags(&g_ring.free_at[device][half], cudaEventDisableTiming));
        const uint32_t n = (uint32_t)((len + per - 1) / per);
        h.open(g_ring.half[half], static_cast<const char*>(src) + r0 * stride, len, row, stride, per);
        cudaError_t err = cudaSuccess;
        uint32_t sent = 0;
        auto send = [&] {                       // every piece at the front of the line that is there
            uint32_t to = sent;
            while (to < n && h.done(to)) ++to;
            if (to == sent) return;
            const size_t from = sent * per, end = std::min(len, to * per);
            if (err == cudaSuccess)
                err = cudaMemcpyAsync(static_cast<char*>(dst) + (r0 + from) * row, g_ring.half[half] + from * row, (end - from) * row,
                                      cudaMemcpyHostToDevice, s);
            sent = to;
        };
        while (h.work()) send();
        for (uint32_t spins = 0; sent < n; ++spins) {
            send();
            if (spins < 20000) SPX_PAUSE(); else std::this_thread::yield();
        }
        if (err == cudaSuccess) err = cudaEventRecord(g_ring.free_at[device][half], s);
        if (err != cudaSuccess) {               // no event tells when this half is free: it is when the stream has run dry
            (void)cudaStreamSynchronize(s);
            return fail(SPX_ERR_CUDA, "host to device copy failed: %s", cudaGetErrorString(err));
        }
        g_ring.last_device[half] = device;
    }
    return SPX_OK;
}

int copy_h2d(void* dst, const void* src, size_t bytes, cudaStream_t s)
{
    if (bytes < kPiece) {                       // one copy: each costs microseconds whatever its size
        if (bytes) SPX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
        return SPX_OK;
    }
    // as rows of 4 KB, and the rest
    const size_t whole = bytes / 4096 * 4096;
    if (int rc = copy_h2d_rows(dst, src, whole / 4096, 4096, 4096, s)) return rc;
    if (bytes > whole)
        SPX_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + whole, static_cast<const char*>(src) + whole, bytes - whole, cudaMemcpyHostToDevice, s));
    return SPX_OK;
}

}  // namespace spx
