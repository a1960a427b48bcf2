// conv.cuh -- what the convolution kernels' files share.
#pragma once

#include "common.cuh"

#include <mutex>

namespace spx {

struct ConvParams {
    uint32_t Cin, Cout, kH, kW, sH, sW, pH, pW, dH, dW, H, W, Ho, Wo, B;
};

// Strides in floats.  Input: the batch is contiguous, the other strides are multiples of 4.  Output: any
// layout; vec_out when the batch is contiguous there too and every position starts on 16 bytes.
struct ConvViews {
    uint64_t iC, iH, iW;
    uint64_t oB, oC, oH, oW;
    uint32_t b_out;     // batch entries that exist in the output (the input may be widened by up to 3)
    uint32_t vec_out;
};

// How a handle's entries lie in the merged kernel's CTAs (of 16, 8 or 4 row blocks): the union columns of the CTA's longest
// block and its work, 0.7 a union column and 0.2 an entry; on average and in the worst CTA.
struct MergedLoad {
    double longest = 0.0, work = 0.0, longest_worst = 0.0, work_worst = 0.0;
};

// From the blocks' (union columns, entries).
void merged_loads(const uint2* blocks, uint32_t nblocks, MergedLoad (&out)[3]);

// conv_tmem.cu: -1 when the shape or the handle is not for this kernel, or the other one's expected time is not above its own
// (load: for 16, 8 and 4 blocks; null: by the density).
int launch_conv_tmem(spx_ell* e, const ConvParams& p, const ConvViews& v, const float* in, const float* bias, int act, float* out,
                     double (*other_us)(const spx_ell*, const ConvParams&, const MergedLoad* load), cudaStream_t s);
// Its expected time where it might be taken, 1e30 where it is not.
double conv_tmem_expected(const spx_ell* e, const ConvParams& p, const ConvViews& v, double (*other_us)(const spx_ell*, const ConvParams&, const MergedLoad*));
// conv_gather.cu: whether the kernel takes the shape, in which form and what time is expected.
struct ConvGatherPlan {
    int form = 0;
    double us = 0.0;
};
bool plan_conv_gather(const spx_ell* e, const ConvParams& p, int layout, const float* in, const float* out, ConvGatherPlan& plan);
int launch_conv_gather(const spx_ell* e, const uint32_t* taps, const ConvParams& p, int layout, const float* in, const float* bias, int act, float* out,
                       const ConvGatherPlan& plan, cudaStream_t s);
// What a handle's convolutions share.  Built under the lock by whichever call first needs it, on any thread and stream; every
// call's stream is behind that, and a recorded call's table complete, before it is used.  Nothing is changed or given back before
// the handle is: calls in flight and recorded graphs may be using it.
struct ConvTables {
    struct Built {
        cudaEvent_t done = nullptr;
        bool pending = false;       // not known to be complete
    };
    struct Shape {                  // of a kernel
        uint32_t kH = 0, kW = 0;
        uint32_t* taps = nullptr;   // per slot of the slab: the column as cin << 16 | kh << 8 | kw
        uint2* hdr = nullptr;       // per merged column: (the same, bit r set when row r of the block stores it)
        Built taps_built, hdr_built;
        bool no_taps = false, no_hdr = false;   // an earlier call found no memory for them
        Shape* next = nullptr;
    };
    std::mutex mu;
    Shape* shapes = nullptr;        // as many as the handle is used with: divisors of its columns
    // Row-block-merged weights (conv.cu): per block of 4 rows the ascending union of their column ids.  Block b owns entries
    // [b * cap, b * cap + ncols[b]): the 4 rows' weights, 0.0f where a row has none, and the headers above.
    float* w = nullptr;             // built with the first shape's headers
    Shape* first = nullptr;
    uint32_t* ncols = nullptr;
    uint32_t cap = 0;
    std::atomic<bool> no_merged{false};     // an earlier call found no memory for them
    // How the entries lie for the merged kernel's CTAs of 16, 8 and 4 row blocks: read once they are counted.
    enum { unknown, counted, no_memory };
    std::atomic<int> loads_state{unknown};
    MergedLoad loads[3];
    // An input brought into [C,H,W,B4] order.  Calls that use it do not run side by side.
    struct Block {
        void* p = nullptr;
        size_t bytes = 0;
        Block* next = nullptr;
    };
    Block scratch;                  // next: smaller ones that recorded graphs use
    bool scratch_recorded = false;
};
ConvTables* new_conv_tables();
void free_conv_tables(spx_ell* e);
// conv.cu: the merged weights of conv_rbm_tile_kernel, for use on s, and (hdr may be null) their headers; -1 where there is no
// memory for them.
int ensure_rbm(spx_ell* e, uint32_t kH, uint32_t kW, cudaStream_t s, const uint2** hdr);
void* new_conv_tmem();
void free_conv_tmem(spx_ell* e);

}  // namespace spx
