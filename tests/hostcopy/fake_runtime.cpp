// A stand-in for the few CUDA runtime calls that hostcopy.cu makes, so that its bookkeeping can be tested without a
// device.  A copy from pageable memory reads its source at once; a copy from pinned memory is carried out as late as
// the runtime may: when its stream, or an event recorded behind it, is waited for.  A ring that is refilled too early
// therefore delivers wrong bytes here every time.  Streams belong to devices, events too.
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <vector>

#include "fake_runtime.hpp"

namespace fake {
std::recursive_mutex mu;
std::vector<std::pair<const char*, size_t>> pinned;
int current_device = 0;
int fail_copy_in = 0;               // the n-th asynchronous copy from now on fails (0: none)
thread_local bool recording_elsewhere = false, recording_broken = false;
thread_local cudaStreamCaptureMode thread_mode = cudaStreamCaptureModeThreadLocal;

bool is_pinned(const void* p)
{
    for (auto& b : pinned)
        if (p >= b.first && p < b.first + b.second) return true;
    return false;
}
Stream& of(cudaStream_t s)
{
    static Stream legacy;
    return s ? *reinterpret_cast<Stream*>(s) : legacy;
}
void Stream::drain(size_t upto)
{
    while (done < upto && !ops.empty()) {
        ops.front()();
        ops.pop_front();
        ++done;
    }
}
// What a thread that records a graph in thread-local mode may not do: it ends the capture with an error.
bool forbidden()
{
    const bool no = recording_elsewhere && thread_mode != cudaStreamCaptureModeRelaxed;
    recording_broken = recording_broken || no;
    return no;
}

struct Event {
    int device;
    Stream* stream = nullptr;
    size_t at = 0;
    bool captured = false;
};
}  // namespace fake

using namespace fake;
using Lock = std::lock_guard<std::recursive_mutex>;

namespace spx {
int fail(int code, const char*, ...) { return code; }
}  // namespace spx

static cudaError_t copy_op(Stream& st, const void* src, std::function<void()> op)
{
    if (fail_copy_in && --fail_copy_in == 0) return cudaErrorUnknown;
    if (st.capturing) {
        st.nodes.push_back({src, op});
        return cudaSuccess;
    }
    if (!is_pinned(src)) {          // read now, delivered in stream order
        st.drain(st.issued);
        op();
        return cudaSuccess;
    }
    st.ops.push_back(op);
    ++st.issued;
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s)
{
    Lock lk(mu);
    return copy_op(of(s), src, [=] { memcpy(dst, src, n); });
}
cudaError_t cudaMemcpy2DAsync(void* dst, size_t dp, const void* src, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t s)
{
    Lock lk(mu);
    return copy_op(of(s), src, [=] { for (size_t i = 0; i < h; ++i) memcpy((char*)dst + i * dp, (const char*)src + i * sp, w); });
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    Lock lk(mu);
    memset(a, 0, sizeof(*a));
    a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = current_device; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    Lock lk(mu);
    if (forbidden()) return cudaErrorStreamCaptureUnsupported;
    char* b = new char[n];
    pinned.push_back({b, n});
    *p = b;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* ev, unsigned)
{
    *ev = reinterpret_cast<cudaEvent_t>(new Event{current_device});
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t s)
{
    Lock lk(mu);
    Event& e = *reinterpret_cast<Event*>(ev);
    Stream& st = of(s);
    if (e.device != st.device) return cudaErrorInvalidResourceHandle;
    e.stream = &st;
    e.at = st.issued;
    e.captured = st.capturing;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev)
{
    Lock lk(mu);
    Event& e = *reinterpret_cast<Event*>(ev);
    if (forbidden()) return cudaErrorStreamCaptureUnsupported;
    if (e.captured) return cudaErrorCapturedEvent;
    if (e.stream) e.stream->drain(e.at);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    Lock lk(mu);
    if (forbidden() || of(s).capturing) return cudaErrorStreamCaptureUnsupported;
    of(s).drain(of(s).issued);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* out)
{
    Lock lk(mu);
    *out = of(s).capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamGetDevice(cudaStream_t s, int* d)
{
    Lock lk(mu);
    *d = of(s).device;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m)
{
    std::swap(*m, thread_mode);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
