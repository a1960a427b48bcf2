// Drives ensure_tma_words (mem.cu) from several threads on a stand-in for the CUDA runtime whose calls take their time; exits 0
// when every thread finds the words complete and none of them meets what a pinned block held before.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "common.cuh"
#include "tma.cuh"

#define CHECK(x) do { if (!(x)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #x); exit(1); } } while (0)

static void slowly() { std::this_thread::sleep_for(std::chrono::milliseconds(2)); }

namespace spx {
int fail(int code, const char*, ...) { return code; }
}  // namespace spx

extern "C" {
static cudaError_t get(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return get(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { slowly(); return get(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return get(p, n); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { slowly(); *d = h; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = reinterpret_cast<cudaMemPool_t>(1); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(2); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { slowly(); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes*, const void*) { return cudaErrorUnknown; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaErrorUnknown; }
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorUnknown; }
}

int main()
{
    for (int round = 0; round < 20; ++round) {
        spx::PinnedBlock used;                  // the free list's block has a value in it
        CHECK(spx::pinned_acquire(4, &used) == SPX_OK);
        memset(used.host, 0xff, used.bytes);
        spx::pinned_release(used);
        spx_ell e;
        std::vector<std::thread> threads;
        for (int i = 0; i < 4; ++i)
            threads.emplace_back([&] {
                spx::ensure_tma_words(&e);
                CHECK(e.tma_failed_host && e.tma_failed_dev && e.tma_failed_mapped);
                CHECK(*e.tma_failed_dev == 0);
            });
        threads.emplace_back([&] {              // a call that only asks
            for (int i = 0; i < 2000; ++i) CHECK(spx::check_tma_words(&e, "call") == SPX_OK);
        });
        for (auto& t : threads) t.join();
        CHECK(!e.tma_off);
        spx::pinned_release(e.tma_failed_block);
        free(e.tma_failed_dev);
    }
    return 0;
}
