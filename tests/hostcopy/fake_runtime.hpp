#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <deque>
#include <functional>
#include <mutex>
#include <utility>
#include <vector>

namespace fake {
struct Node {
    const void* src;
    std::function<void()> run;
};
struct Stream {
    int device = 0;
    bool capturing = false;
    std::vector<Node> nodes;                    // recorded while capturing
    std::deque<std::function<void()>> ops;      // copies from pinned memory, not carried out yet
    size_t issued = 0, done = 0;
    void drain(size_t upto);
    cudaStream_t handle() { return reinterpret_cast<cudaStream_t>(this); }
};
extern std::recursive_mutex mu;
extern std::vector<std::pair<const char*, size_t>> pinned;
extern int current_device, fail_copy_in;
extern thread_local bool recording_elsewhere, recording_broken;
bool is_pinned(const void* p);
}  // namespace fake
