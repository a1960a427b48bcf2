// conv_gather.cu -- sparse convolution that gathers its operands through L1, for small problems.
//
// The tiled kernels (conv.cu, conv_tmem.cu) bring a patch of the input into shared or tensor memory chunk by chunk, which pays
// where many output channels and batch entries share it.  With a batch of a few images, a stride of two or few channels
// that is mostly latency: a chunk is 250 to 500 clocks whatever is in it, half of the staged columns are skipped by a
// stride, the last three of four batch entries are padding, and NCHW images are copied first.  Here a warp takes one output
// channel at 32 V positions and loads each operand when it needs it: no staging, no copy, no padding, any batch and layout.
//
// Bound by issue slots (63 % used; 6 to 9 an operand, 200 to 400 a warp for its ends), L1 wavefronts (48 %; a stride
// of two or positions that are not neighbours in memory take two to 32 a load) and, with few warps, by the round trips of a
// row's entries, 8 at a time.  Measured against the tiled kernels: 64 -> 128 channels, 3 x 3, stride 2, 57 x 57, batch 3,
// NCHW 28 -> 15 us; 219 -> 32, 3 x 3, stride 2, 104 x 104, batch 1 100 -> 17; 384 -> 25, 3 x 3, 9 x 9, batch 27 300 -> 44; 96 -> 214,
// 1 x 1, stride 2, 36 x 36, batch 1, NCHW 23 -> 5.5; 64 -> 32, 3 x 3, 10 x 10, batch 1 14.6 -> 6.3.  Tried: places of the positions
// worked out by every warp (short rows 10 to 40 % slower), 8 loads of 2 positions a warp or 16 of one (1 to 2 % on average over
// the two forms here), branches around taps outside the image instead of predicates (10 to 60 % slower for long rows).
#include "conv.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

namespace {

using spx::ConvParams;

constexpr uint32_t kBatch = 32;             // entries that a warp decodes at a time, one a lane
constexpr uint32_t kWarps = 8;              // output channels of a CTA

struct GatherArgs {
    const float* Wd;
    const uint32_t* taps;
    const uint2* rows;
    uint32_t m, pitch;
    const float* in;
    const float* bias;
    float* out;
    int act;
    uint32_t kH, kW, sH, sW, pH, pW, dH, dW, H, W;
    uint32_t d0, d1, positions;             // positions in the order of the lanes: extents of the fastest and the next dimension
    uint32_t order;                         // 0: batch, column, row; 1: column, row, batch; 2: batch, row, column
    uint32_t iB, iC, iH, iW;
    uint32_t oB, oH, oW;
    uint64_t oC;
    uint32_t tiles;
};

// Predicated, not branched: the loads of a group are on their way together.  The tap's bit of the mask, which is moved to the
// sign by a tap's number (PACK), or met by its bit.
template <bool PACK, bool CHECK, int VEC>
__device__ __forceinline__ void load_vec(float (&d)[VEC], const void* __restrict__ p, uint32_t mask, uint32_t tap) {
    static_assert(PACK || VEC == 1);
    if constexpr (VEC == 4 && CHECK)
        asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tshf.l.wrap.b32 t, 0, %5, %6;\n\tsetp.lt.s32 p, t, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
            "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "l"(p), "r"(mask), "r"(tap));
    else if constexpr (VEC == 4)
        asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "l"(p));
    else if constexpr (CHECK && PACK)
        asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tshf.l.wrap.b32 t, 0, %2, %3;\n\tsetp.lt.s32 p, t, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "@p ld.global.nc.f32 %0, [%1];\n\t}" : "=f"(d[0]) : "l"(p), "r"(mask), "r"(tap));
    else if constexpr (CHECK)
        asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %2, %3;\n\tsetp.ne.u32 p, t, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "@p ld.global.nc.f32 %0, [%1];\n\t}" : "=f"(d[0]) : "l"(p), "r"(mask), "r"(tap));
    else
        asm("ld.global.nc.f32 %0, [%1];" : "=f"(d[0]) : "l"(p));
}

// A CTA computes 8 output channels, one a warp, at 32 V positions (of VEC batch entries each, where these are contiguous).
// The positions' places and the taps of each that lie inside the image are worked out once per CTA.  A row's entries are
// decoded 32 at a time, one a lane, to (weight, offset of the operand from that of the position's first tap) and the tap's bit,
// and read back as 16-byte broadcasts of two entries, or four bits where positions have taps outside.  Taps outside the image
// contribute w * 0 like everywhere.
template <int VEC, int V, int U, int MINB>
__global__ void __launch_bounds__(kWarps * 32, MINB)
conv_gather_kernel(const __grid_constant__ GatherArgs a)
{
    __shared__ __align__(16) uint2 s_entry[kWarps][2][kBatch];
    // Four positions a lane add a 32-bit offset an operand and meet the mask with the tap's bit, 5 instructions, at 16 bytes more
    // of shared memory for four entries: 721 -> 476 us (290 -> 501 channels, 5 x 5, 84 x 84, batch 1), 376 -> 248 (192 -> 64,
    // 3 x 3, 32 x 32, batch 20, NCHW).  The others keep offset and tap in one word, 7 instructions and fewer registers: with
    // the bits one position a lane took 15.4 -> 16.1 us, four batch entries up to 11 % longer.
    constexpr bool PACK = VEC == 4 || V == 1;
    __shared__ __align__(16) uint32_t s_tap[PACK ? 1 : kWarps][2][kBatch];
    __shared__ int s_in[32 * V];
    __shared__ uint32_t s_mask[32 * V], s_out[32 * V];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x % a.tiles, slot = blockIdx.x / a.tiles * kWarps + warp;
    spx::pdl_wait();
    spx::pdl_launch();
    const uint2 ri = slot < a.m ? __ldg(a.rows + slot) : make_uint2(0u, 0u);
    const uint32_t nn = ri.y;
    const float* __restrict__ wd = a.Wd + (size_t)ri.x * a.pitch;
    const uint32_t* __restrict__ tp = a.taps + (size_t)ri.x * a.pitch;
    uint32_t t = 0;
    float w = 0.0f;
    if (lane < nn) { t = __ldg(tp + lane); w = __ldg(wd + lane); }
    const float bias = a.bias && slot < a.m ? __ldg(a.bias + ri.x) : 0.0f;

    if (threadIdx.x < 32 * V) {
        const uint32_t p = min(tile * (32 * V) + threadIdx.x, a.positions - 1);
        const uint32_t q = p / a.d0, i0 = p - q * a.d0, i2 = q / a.d1, i1 = q - i2 * a.d1;
        const uint32_t b = a.order == 1 ? i2 : i0, ow = a.order == 0 ? i1 : a.order == 1 ? i0 : i2, oh = a.order == 0 ? i2 : i1;
        const int ih = (int)(oh * a.sH) - (int)a.pH, iw = (int)(ow * a.sW) - (int)a.pW;
        uint32_t mw = 0, m = 0;
        for (uint32_t k = 0; k < a.kW; ++k) mw |= (uint32_t)((unsigned)(iw + (int)(k * a.dW)) < a.W) << k;
        for (uint32_t k = 0; k < a.kH; ++k)
            if ((unsigned)(ih + (int)(k * a.dH)) < a.H) m |= mw << (k * a.kW);
        s_in[threadIdx.x] = ih * (int)a.iH + iw * (int)a.iW + (int)(b * a.iB);
        s_mask[threadIdx.x] = m;
        s_out[threadIdx.x] = oh * a.oH + ow * a.oW + b * a.oB;
    }
    __syncthreads();
    if (slot >= a.m) return;
    // the position's first tap, or its bytes from the input's start modulo 2^32 (it may lie before)
    std::conditional_t<PACK, const float*, uint32_t> base[V];
    uint32_t mask[V];
    const uint32_t all = 0xffffffffu >> (32 - a.kH * a.kW);
    bool inside = true;
    float acc[V][VEC];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if constexpr (PACK) base[v] = a.in + s_in[v * 32 + lane];
        else base[v] = 4u * (uint32_t)s_in[v * 32 + lane];
        mask[v] = s_mask[v * 32 + lane];
        inside = inside && mask[v] == all;
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[v][i] = bias;
    }
    auto load = [&](float (&x)[VEC], int v, uint32_t entry, uint32_t tap, auto check) {
        if constexpr (PACK) load_vec<PACK, decltype(check)::value, VEC>(x, base[v] + (entry >> 5), mask[v], entry);
        else load_vec<PACK, decltype(check)::value, VEC>(x, reinterpret_cast<const char*>(a.in) + (base[v] + entry), mask[v], tap);
    };
    auto group = [&](const uint2* __restrict__ e, const uint32_t* __restrict__ taps, auto check) {         // U entries
        uint2 en[U];
        uint32_t tap[U] = {};
        if constexpr (decltype(check)::value && !PACK) {
#pragma unroll
            for (int u = 0; u < U; u += 4) {
                const uint4 four = *reinterpret_cast<const uint4*>(taps + u);
                tap[u] = four.x; tap[u + 1] = four.y; tap[u + 2] = four.z; tap[u + 3] = four.w;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u += 2) {
            const uint4 two = *reinterpret_cast<const uint4*>(e + u);
            en[u] = make_uint2(two.x, two.y);
            en[u + 1] = make_uint2(two.z, two.w);
        }
        float x[U][V][VEC];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                load(x[u][v], v, en[u].y, tap[u], check);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int i = 0; i < VEC; ++i) acc[v][i] = fmaf(__uint_as_float(en[u].x), x[u][v][i], acc[v][i]);
    };
    auto run = [&](auto check) {
        for (uint32_t j = 0, buf = 0; j < nn; j += kBatch, buf ^= 1u) {
            uint2* __restrict__ e = s_entry[warp][buf];
            uint32_t* __restrict__ taps = s_tap[PACK ? 0 : warp][buf];
            const uint32_t kh = t >> 8 & 0xffu, kw = t & 0xffu;
            const uint32_t at = (t >> 16) * a.iC + kh * a.dH * a.iH + kw * a.dW * a.iW, tap = kh * a.kW + kw;
            e[lane] = make_uint2(__float_as_uint(w), PACK ? at << 5 | (31 - tap) : 4u * at);
            if constexpr (decltype(check)::value && !PACK) taps[lane] = 1u << tap;
            __syncwarp();
            if (j + kBatch + lane < nn) { t = __ldg(tp + j + kBatch + lane); w = __ldg(wd + j + kBatch + lane); }
            const uint32_t n = min(kBatch, nn - j);
            uint32_t u = 0;
            for (; u + U <= n; u += U) group(e + u, taps + u, check);
            for (; u < n; ++u) {
                const uint2 en = e[u];
                const uint32_t tap = decltype(check)::value && !PACK ? taps[u] : 0u;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float x[VEC];
                    load(x, v, en.y, tap, check);
#pragma unroll
                    for (int i = 0; i < VEC; ++i) acc[v][i] = fmaf(__uint_as_float(en.x), x[i], acc[v][i]);
                }
            }
        }
    };
    if (__all_sync(0xffffffffu, inside)) run(std::false_type());
    else run(std::true_type());
    float* __restrict__ out = a.out + ri.x * a.oC;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (tile * (32 * V) + v * 32 + lane >= a.positions) break;
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[v][i] = spx::apply_act(acc[v][i], a.act);
        float* __restrict__ o = out + s_out[v * 32 + lane];
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(o) = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
        else *o = acc[v][0];
    }
}

}  // namespace

namespace spx {

namespace {

// A form of the kernel and what it is expected to take: its own time, clocks of issue slots a warp, an entry and an
// operand, of an L1 wavefront, and of a round trip.  Fitted to 330 measured shapes (3 to 512 channels, 1 x 1 to 5 x 5, strides 1
// and 2, 7 x 7 to 112 x 112, batch 1 to 32, 5 to 50 % dense, all layouts): 0.9 to 1.1 of the time for half of them.
struct Form {
    uint32_t VEC, V, U;
    double us, warp, entry, operand, wavefront, trip;
};
constexpr Form kForms[4] = {{1, 1, 8, 3.5, 208, 3.2, 5.9, 0.42, 366}, {1, 4, 4, 2.8, 297, 3.5, 7.7, 0.42, 729},
                            {4, 2, 4, 2.0, 382, 6.3, 11.2, 0.40, 927}, {4, 1, 4, 2.5, 268, 5.5, 10.1, 0.43, 532}};

// The second one where neighbouring positions are neighbours in memory (elsewhere L1 wavefronts bound it, and the estimate
// above holds), fitted to 112 shapes with an SM's CTAs counted whole.
constexpr Form kNear = {1, 4, 4, 2.9, 364, 4.2, 4.9, 0.19, 325};

double form_us(const spx_ell* e, const ConvParams& p, int layout, const Form& f)
{
    const double sms = sm_count(e->device), len = (double)e->nnz_total / e->m;
    const uint64_t positions = (uint64_t)p.Ho * p.Wo * p.B / f.VEC;
    const double warps = (double)((positions + 32 * f.V - 1) / (32 * f.V)) * round_up(e->m, kWarps);
    // lines that a load touches: runs of neighbours, the gaps of a stride, the ends of rows
    double lines;
    if (layout == SPX_LAYOUT_FMAJOR) {
        const double run = std::min(32u * f.VEC, p.B);
        lines = 32.0 * f.VEC / run * (1.0 + (run - 1.0) / 32.0) * (1.0 + 2.0 / run);
    } else {
        lines = std::min(32.0, f.VEC * p.sW + 1.0 + 32.0 * f.VEC / ((double)p.Wo * (layout == SPX_LAYOUT_PF ? p.B : 1)));
    }
    double whole = 1.0;                         // the fullest SM's CTAs to the average
    if (&f == &kNear) {
        const double ctas = warps / kWarps / sms;
        whole = ctas <= 4.0 ? std::ceil(ctas) / ctas : (ctas + 0.5) / ctas;
    }
    const double busy = whole * (warps * (f.warp + len * (f.entry + f.operand * f.V)) / (4 * sms) + warps * len * f.V * lines * f.wavefront / sms);
    const double chain = 1000.0 + (e->max_nnz / f.U + 2.0) * f.trip;
    return f.us + std::sqrt(busy * busy + chain * chain) / 1900.0;
}

template <int VEC, int V, int U, int MINB>
int launch_form(const spx_ell* e, GatherArgs a, cudaStream_t s)
{
    a.tiles = (a.positions + 32 * V - 1) / (32 * V);
    const unsigned ctas = (unsigned)(a.tiles * ((e->m + kWarps - 1) / kWarps));
    const cudaError_t err = launch_pdl(conv_gather_kernel<VEC, V, U, MINB>, dim3(ctas), dim3(kWarps * 32), 0, s, a);
    if (err != cudaSuccess) return fail(SPX_ERR_CUDA, "launch of conv_gather_kernel failed: %s", cudaGetErrorString(err));
    count_launch();
    return SPX_OK;
}

}  // namespace

bool plan_conv_gather(const spx_ell* e, const ConvParams& p, int layout, const float* in, const float* out, ConvGatherPlan& plan)
{
    // the switches that force another kernel turn this one off
    static const int env = [] {
        if (const char* v = getenv("SPX_CONV_GATHER")) return atoi(v);
        for (const char* k : {"SPX_CONV_DIRECT", "SPX_CONV_TMEM", "SPX_CONV_RBM", "SPX_CONV_RBM_MIN_SHARE", "SPX_CONV_RBM_SEGMENTS", "SPX_CONV_CUT",
                              "SPX_CONV_TMA", "SPX_CONV_TMA_TEST_TIMEOUT", "SPX_CONV_SMALL_TILE", "SPX_CONV_CTAS", "SPX_CONV_WIDE_TILE"})
            if (getenv(k)) return 0;
        return 1;
    }();
    const uint64_t H = p.H, W = p.W, B = p.B, Cin = p.Cin, Ho = p.Ho, Wo = p.Wo;
    if (!env || p.kH * p.kW > 32) return false;             // a bit per tap
    // 27 bits of an entry's offset, 32 of an operand's in bytes and of a position's in the output
    const uint64_t iC = layout == SPX_LAYOUT_FMAJOR ? B : layout == SPX_LAYOUT_PF ? H * W * B : H * W;
    const uint64_t iH = layout == SPX_LAYOUT_FMAJOR ? Cin * B : layout == SPX_LAYOUT_PF ? W * B : W;
    const uint64_t iW = layout == SPX_LAYOUT_FMAJOR ? H * Cin * B : layout == SPX_LAYOUT_PF ? B : 1;
    if ((Cin - 1) * iC + (uint64_t)(p.kH - 1) * p.dH * iH + (uint64_t)(p.kW - 1) * p.dW * iW >= 1ull << 27) return false;
    if ((H + p.pH) * iH + (W + p.pW) * iW + Cin * H * W * B >= 1ull << 30 || p.Cout * Ho * Wo * B >= 1ull << 32) return false;
    if ((Ho * Wo * B + 31) / 32 * ((e->m + kWarps - 1) / kWarps) > 0x7fffffffull) return false;
    const bool vec = layout != SPX_LAYOUT_NCHW && B % 4 == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const int f0 = vec ? 2 : 0;
    const bool neighbours = layout != SPX_LAYOUT_FMAJOR && p.sW == 1;
    const Form& other = vec ? kForms[3] : neighbours ? kNear : kForms[1];
    const double us0 = form_us(e, p, layout, kForms[f0]), us1 = form_us(e, p, layout, other);
    plan.form = us1 < us0 ? f0 + 1 : f0;
    double us = std::min(us0, us1);
    // One batch entry a lane although four are contiguous: more warps, shorter round trips, fewer lanes idle.  Where it is expected
    // to be faster by a ninth: the estimates are a tenth off for half of the shapes.
    if (vec && layout == SPX_LAYOUT_PF) {
        const double one = form_us(e, p, layout, kForms[0]), four = neighbours ? form_us(e, p, layout, kNear) : 1e30;
        if (std::min(one, four) < 0.9 * us) { us = std::min(one, four); plan.form = four < one ? 1 : 0; }
    }
    plan.us = env == 2 ? 0.0 : us;
    return true;
}

int launch_conv_gather(const spx_ell* e, const uint32_t* taps, const ConvParams& p, int layout, const float* in, const float* bias, int act, float* out,
                       const ConvGatherPlan& plan, cudaStream_t s)
{
    const uint32_t H = p.H, W = p.W, Ho = p.Ho, Wo = p.Wo, B = p.B;
    GatherArgs a{};
    a.Wd = e->Wd; a.taps = taps; a.rows = e->rows; a.m = e->m; a.pitch = e->pitch;
    a.in = in; a.bias = bias; a.out = out; a.act = act;
    a.kH = p.kH; a.kW = p.kW; a.sH = p.sH; a.sW = p.sW; a.pH = p.pH; a.pW = p.pW; a.dH = p.dH; a.dW = p.dW; a.H = H; a.W = W;
    a.positions = Ho * Wo * B;
    if (layout == SPX_LAYOUT_PF) {
        a.order = 0; a.d0 = B; a.d1 = Wo;
        a.iB = 1; a.iW = B; a.iH = W * B; a.iC = H * W * B;
        a.oB = 1; a.oW = B; a.oH = Wo * B; a.oC = (uint64_t)Ho * Wo * B;
    } else if (layout == SPX_LAYOUT_NCHW) {
        a.order = 1; a.d0 = Wo; a.d1 = Ho;
        a.iW = 1; a.iH = W; a.iC = H * W; a.iB = p.Cin * H * W;
        a.oW = 1; a.oH = Wo; a.oC = (uint64_t)Ho * Wo; a.oB = p.Cout * Ho * Wo;
    } else {
        a.order = 2; a.d0 = B; a.d1 = Ho;
        a.iB = 1; a.iC = B; a.iH = p.Cin * B; a.iW = H * p.Cin * B;
        a.oB = 1; a.oC = B; a.oH = p.Cout * B; a.oW = Ho * p.Cout * B;
    }
    if (plan.form >= 2) {                       // four batch entries a lane
        a.d0 /= 4;
        a.positions /= 4;
        a.iB = a.oB = 4;
    }
    switch (plan.form) {
    case 0: return launch_form<1, 1, 8, 6>(e, a, s);
    case 1: return launch_form<1, 4, 4, 0>(e, a, s);
    case 2: return launch_form<4, 2, 4, 0>(e, a, s);
    default: return launch_form<4, 1, 4, 0>(e, a, s);
    }
}

}  // namespace spx
