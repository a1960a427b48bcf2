// encode.cu -- ELLPACK construction and decoding on the device.
//
// encode_device replaces convert_to_ellpack (src/ellpack_encoder.cpp:6-44) for a dense matrix
// that already lives in device memory: pass 1 counts v != 0.0f per row, the host finds r = the
// longest row, pass 2 packs values and column ids in ascending column order.  The result is
// bit-identical to the host encoder: -0.0f is dropped, NaN / inf / denormals are kept.
// decode_device replaces decode_from_ellpack (:46-60).  csr_to_ell_device fills the padded slabs
// from CSR arrays for matrices that never exist densely.
//
// The passes are bound by HBM: 4*m*n bytes read by the counter, 4*m*n written by the decoder, so the kernels move
// 16-byte vectors with several in flight per lane.  A large matrix is read once: the counter keeps the entries it finds,
// the packer fetches them from L2; a small one is read again, backwards: what the counter read last is then still in L2.
// Measured at 8192 x 8192, 10 % kept: count and keep 58 us, pack 29, decode 56 (6.0 TB/s); encode + decode + destroy
// through the C ABI 187 us (244 with two reads and a schedule sorted on the host).
#include "common.cuh"

#include <algorithm>
#include <vector>

namespace {

constexpr int kWarps = 8;
constexpr int kQuads = 4;       // 16-byte loads in flight per lane

// A warp's unit of work is one row, or, when the matrix has too few rows to fill the GPU, one of
// `segs` equal column segments of a row (`seg` columns each, a multiple of 4).  Rows start at any
// element offset, so a segment is walked in 16-byte quads aligned in memory: quads 0 .. count-1 from
// the aligned address `at`, of which only the first and the last can reach over an end of the
// segment.  Places in a segment count from its first column (n may be anything below 2^32, a segment's
// length is below 2^31: rows of 2^23 columns and more come in few enough to be cut): quad 0 starts at -lead.
struct Segment {
    uint32_t row;
    int64_t at;                 // element offset of quad 0 from W (may be below 0 or the segment's start)
    uint32_t c_lo;              // first column
    int32_t lead, len;          // elements of quad 0 before the segment; columns
    uint32_t quads;
};

__device__ __forceinline__ Segment segment_of(uint64_t unit, uint32_t mis, uint32_t n, uint32_t segs, uint32_t seg)
{
    Segment s;
    s.row = segs == 1 ? (uint32_t)unit : (uint32_t)(unit / segs);
    const uint64_t part = segs == 1 ? 0 : unit - (uint64_t)s.row * segs;
    s.c_lo = (uint32_t)min(part * seg, (uint64_t)n);
    s.len = (int32_t)(min((part + 1) * seg, (uint64_t)n) - s.c_lo);
    const uint64_t base = (uint64_t)s.row * n;
    const uint64_t first = base + s.c_lo + mis;             // counted from the aligned address W - mis
    s.at = (int64_t)(first & ~3ull) - (int64_t)mis;
    s.lead = (int32_t)(first & 3u);
    s.quads = (uint32_t)(s.lead + s.len + 3) >> 2;
    return s;
}

// Quad i of a segment; elements outside the segment read as 0.0f, which is "no entry".
__device__ __forceinline__ float4 load_quad(const float* __restrict__ W, const Segment& s, uint32_t i)
{
    const int32_t c = 4 * (int32_t)i - s.lead;
    const float* __restrict__ p = W + s.at + 4ull * i;
    if (c >= 0 && c + 4 <= s.len) return __ldg(reinterpret_cast<const float4*>(p));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= 0 && c < s.len) v.x = __ldg(p);
    if (c + 1 >= 0 && c + 1 < s.len) v.y = __ldg(p + 1);
    if (c + 2 >= 0 && c + 2 < s.len) v.z = __ldg(p + 2);
    if (c + 3 >= 0 && c + 3 < s.len) v.w = __ldg(p + 3);
    return v;
}

// Quads qb + lane + 32 u of the segment for u = 0 .. kQuads-1; whole blocks inside it without checks.
template <bool STREAM>              // read once: first to leave the caches
__device__ __forceinline__ void load_block(float4 (&v)[kQuads], const float* __restrict__ W, const Segment& s, uint32_t qb, int lane)
{
    if (qb > 0 && qb + 32 * kQuads < s.quads) {
        const float4* __restrict__ p = reinterpret_cast<const float4*>(W + s.at) + qb + lane;
#pragma unroll
        for (int u = 0; u < kQuads; ++u) v[u] = STREAM ? __ldcs(p + 32 * u) : __ldg(p + 32 * u);
        return;
    }
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
        const uint32_t i = qb + 32 * u + lane;
        v[u] = i < s.quads ? load_quad(W, s, i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__global__ void __launch_bounds__(kWarps * 32)
count_kernel(const float* __restrict__ W, uint32_t mis, uint32_t m, uint32_t n, uint32_t segs, uint32_t seg,
             uint32_t* __restrict__ counts)
{
    const int lane = threadIdx.x & 31;
    const uint64_t unit = (uint64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (unit >= (uint64_t)m * segs) return;
    const Segment s = segment_of(unit, mis, n, segs, seg);
    uint32_t cnt = 0;
    for (uint32_t qb = 0; qb < s.quads; qb += 32 * kQuads) {
        float4 v[kQuads];
        load_block<false>(v, W, s, qb, lane);
#pragma unroll
        for (int u = 0; u < kQuads; ++u)
            cnt += (v[u].x != 0.0f) + (v[u].y != 0.0f) + (v[u].z != 0.0f) + (v[u].w != 0.0f);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) counts[unit] = cnt;
}

// The counter that also keeps what it finds: per unit up to `cap` entries as (value, column) pairs in scratch, so that
// the matrix is read once.  A block of 512 elements is compacted in the warp's strip of shared memory (one scan of four
// byte-sized counts per lane gives all places) and leaves it in whole 8-byte rows of 32 lanes.  W is read with an
// evict-first hint, so that the pairs are still in L2 when pack_kernel fetches them.
// 8192 x 8192, 10 %: 58 us (count_kernel 53), and pack_kernel 29 instead of 67.
// A unit is given up where more than 17/64 of the columns seen so far (and 16) are entries: the pairs written until then
// are in vain.  It is marked in its first pair.  (Writing them up to a capacity of a quarter cost units that are denser 8
// to 12 %: 151 x 264025, 30 % 165 us, now 146, 143 without pairs.  The check costs 8192 x 8192, 10 % 1 us of 187.  A unit
// that is dense at its front only is read twice, as without pairs.)
constexpr uint32_t kNotKept = 0xffffffffu;                  // no column: n is at most this
constexpr uint32_t kKeepSlack = 16;
__host__ __device__ constexpr uint32_t keep_cap(uint32_t columns) { return columns / 64 * 17 + kKeepSlack; }

__global__ void __launch_bounds__(kWarps * 32)
count_keep_kernel(const float* __restrict__ W, uint32_t mis, uint32_t m, uint32_t n, uint32_t segs, uint32_t seg, uint32_t cap,
                  uint32_t* __restrict__ counts, uint2* __restrict__ kept)
{
    __shared__ __align__(16) uint2 strips[kWarps][128 * kQuads];
    const int lane = threadIdx.x & 31;
    uint2* strip = strips[threadIdx.x >> 5];
    const uint64_t unit = (uint64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (unit >= (uint64_t)m * segs) return;
    const Segment s = segment_of(unit, mis, n, segs, seg);
    uint2* __restrict__ dst = kept + unit * cap;
    uint32_t pos = 0;
    uint32_t qb = 0, most = kKeepSlack;
    bool keep = true;
    for (; keep && qb < s.quads; qb += 32 * kQuads) {
        float4 v[kQuads];
        load_block<true>(v, W, s, qb, lane);
        uint32_t own = 0;                                   // byte u: entries of this lane's quad u
#pragma unroll
        for (int u = 0; u < kQuads; ++u)
            own |= ((v[u].x != 0.0f) + (v[u].y != 0.0f) + (v[u].z != 0.0f) + (v[u].w != 0.0f)) << (8 * u);
        uint32_t upto = own;                                // at most 128 in a byte
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t b = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += b;
        }
        const uint32_t all = __shfl_sync(0xffffffffu, upto, 31), before = upto - own;
        uint32_t base = 0;
#pragma unroll
        for (int u = 0; u < kQuads; ++u) {
            uint32_t at = base + ((before >> (8 * u)) & 255u);
            const uint32_t col = s.c_lo + 4 * (qb + 32 * u + lane) - (uint32_t)s.lead;
            if (v[u].x != 0.0f) strip[at++] = make_uint2(__float_as_uint(v[u].x), col);
            if (v[u].y != 0.0f) strip[at++] = make_uint2(__float_as_uint(v[u].y), col + 1);
            if (v[u].z != 0.0f) strip[at++] = make_uint2(__float_as_uint(v[u].z), col + 2);
            if (v[u].w != 0.0f) strip[at] = make_uint2(__float_as_uint(v[u].w), col + 3);
            base += (all >> (8 * u)) & 255u;
        }
        __syncwarp();
        most = min(most + 34 * kQuads, cap);                // the next block's share
        keep = pos + base <= most;
        if (keep)
            for (uint32_t j = lane; j < base; j += 32) dst[pos + j] = strip[j];
        pos += base;
        __syncwarp();
    }
    if (!keep) {
        uint32_t cnt = 0;
        for (; qb < s.quads; qb += 32 * kQuads) {
            float4 v[kQuads];
            load_block<false>(v, W, s, qb, lane);           // pack_kernel reads it again
#pragma unroll
            for (int u = 0; u < kQuads; ++u)
                cnt += (v[u].x != 0.0f) + (v[u].y != 0.0f) + (v[u].z != 0.0f) + (v[u].w != 0.0f);
        }
        pos += __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) dst[0].y = kNotKept;                 // (a first pair was lane 0's store, too)
    }
    if (lane == 0) counts[unit] = pos;
}

// What the host has to know before the arrays can be allocated, where the device makes the row schedule (up to kRankRows
// rows of less than kRankColumns): one CTA adds up the rows' segments and leaves the result in page-locked memory, where
// the host finds it after one wait (instead of a copy of all counts and three loops over them).
constexpr uint32_t kRankRows = 15104, kRankColumns = 1u << 18;
struct RowStats {
    uint64_t total;
    uint32_t longest, shortest, long_rows, pad;
};

// A thread adds up a row, or a warp does, where rows come in many segments (16 and more, of at most some 600 rows then: as
// a chain of loads they cost 28 x 247446 48 us more; as warps, 8192 rows of 2 segments 2 us more).
template <bool WARPS>
__global__ void __launch_bounds__(1024)
row_stats_kernel(const uint32_t* __restrict__ counts, uint32_t m, uint32_t segs, uint32_t* __restrict__ keys, RowStats* __restrict__ out)
{
    __shared__ uint32_t s_hi[32], s_lo[32], s_long[32];
    __shared__ unsigned long long s_sum[32];
    uint32_t hi = 0, lo = 0xffffffffu, n_long = 0;
    unsigned long long sum = 0;
    constexpr uint32_t U = 8, lanes = WARPS ? 32 : 1;       // rows of a group of lanes in flight
    const uint32_t part = threadIdx.x % lanes, step = 1024 / lanes;
    for (uint32_t first = 0; first < m; first += step * U) {
        const uint32_t i0 = first + threadIdx.x / lanes;
        uint32_t len[U] = {};
        for (uint32_t k = part; k < segs; k += lanes)
#pragma unroll
            for (uint32_t u = 0; u < U; ++u)
                if (i0 + step * u < m) len[u] += __ldg(counts + (size_t)(i0 + step * u) * segs + k);
        for (uint32_t o = lanes / 2; o; o /= 2)
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) len[u] += __shfl_xor_sync(0xffffffffu, len[u], o);
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t i = i0 + step * u;
            if (i >= m || part) break;
            keys[i] = len[u] * kRankRows + (kRankRows - 1 - i);
            hi = max(hi, len[u]);
            lo = min(lo, len[u]);
            n_long += len[u] >= 512u;
            sum += len[u];
        }
    }
    auto reduce = [&] {
        hi = __reduce_max_sync(0xffffffffu, hi);
        lo = __reduce_min_sync(0xffffffffu, lo);
        n_long = __reduce_add_sync(0xffffffffu, n_long);
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    };
    reduce();
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { s_hi[w] = hi; s_lo[w] = lo; s_long[w] = n_long; s_sum[w] = sum; }
    __syncthreads();
    if (w) return;
    hi = s_hi[lane]; lo = s_lo[lane]; n_long = s_long[lane]; sum = s_sum[lane];
    reduce();
    if (lane == 0) *out = RowStats{sum, hi, lo, n_long, 0u};
}

// A row's place in the schedule (longest first, equal ones by id) is the number of rows with a larger key, length before
// reversed id.  4 lanes count for a row, over keys staged in shared memory (from global memory, one load after the
// other, 8192 rows took 110 us).
constexpr uint32_t kRankPerCta = kWarps * 32 / 4, kRankTile = 2048;
__device__ __forceinline__ void rank_rows(uint32_t cta, const uint32_t* __restrict__ keys, uint32_t m, uint2* __restrict__ rows, uint4* tile)
{
    const uint32_t i = cta * kRankPerCta + threadIdx.x / 4, part = threadIdx.x & 3;
    const uint32_t key = i < m ? __ldg(keys + i) : 0u;
    uint32_t rank = 0;
    for (uint32_t t0 = 0; t0 < m; t0 += kRankTile) {
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < kRankTile; j += kWarps * 32)
            reinterpret_cast<uint32_t*>(tile)[j] = t0 + j < m ? __ldg(keys + t0 + j) : 0u;     // 0 is larger than nothing
        __syncthreads();
#pragma unroll 8
        for (uint32_t q = part; q < kRankTile / 4; q += 4) {
            const uint4 o = tile[q];
            rank += (o.x > key) + (o.y > key) + (o.z > key) + (o.w > key);
        }
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    if (part == 0 && i < m) rows[rank] = make_uint2(i, key / kRankRows);
}

// Entries into their rows: from the pairs that the counter kept, or, where it gave the unit up (or kept none at all), out
// of the matrix again.  Unit u of the grid is the matrix's unit (last - u): the counter has just read the end
// of W.  The first rank_ctas CTAs make the row schedule.
__global__ void __launch_bounds__(kWarps * 32)
pack_kernel(const float* __restrict__ W, uint32_t mis, uint32_t m, uint32_t n, uint32_t segs, uint32_t seg,
            const uint32_t* __restrict__ counts, uint32_t pitch, float* __restrict__ Wd, uint32_t* __restrict__ idx,
            uint32_t* __restrict__ nnz, const uint2* __restrict__ kept, uint32_t cap, const uint32_t* __restrict__ keys,
            uint2* __restrict__ rows, uint32_t rank_ctas)
{
    __shared__ __align__(16) uint4 tile[kRankTile / 4];
    if (blockIdx.x < rank_ctas) {
        rank_rows(blockIdx.x, keys, m, rows, tile);
        return;
    }
    const int lane = threadIdx.x & 31;
    const uint64_t units = (uint64_t)m * segs;
    const uint64_t u_rev = (uint64_t)(blockIdx.x - rank_ctas) * kWarps + (threadIdx.x >> 5);
    if (u_rev >= units) return;
    const uint64_t unit = units - 1 - u_rev;
    const Segment s = segment_of(unit, mis, n, segs, seg);
    float* __restrict__ wd = Wd + (size_t)s.row * pitch;
    uint32_t* __restrict__ ix = idx + (size_t)s.row * pitch;
    const uint64_t first = (uint64_t)s.row * segs;
    uint32_t pos = 0;                                       // entries of the row in earlier segments
    if (segs > 1) {
        for (uint64_t k = first + lane; k < unit; k += 32) pos += counts[k];
        pos = __reduce_add_sync(0xffffffffu, pos);
    }
    const uint2* __restrict__ src = kept + unit * cap;
    const uint32_t mine = kept ? __ldg(counts + unit) : 0u, mark = kept ? __ldg(&src->y) : kNotKept;    // (one trip for both)
    if (kept && (mine == 0 || mark != kNotKept)) {
        constexpr uint32_t kRun = 4;                        // pairs per lane in flight
        for (uint32_t j0 = lane; j0 < mine; j0 += 32 * kRun) {
            uint2 p[kRun];
#pragma unroll
            for (uint32_t u = 0; u < kRun; ++u) if (j0 + 32 * u < mine) p[u] = __ldcs(src + j0 + 32 * u);
#pragma unroll
            for (uint32_t u = 0; u < kRun; ++u)
                if (j0 + 32 * u < mine) {
                    wd[pos + j0 + 32 * u] = __uint_as_float(p[u].x);
                    ix[pos + j0 + 32 * u] = p[u].y;
                }
        }
        pos += mine;
    } else {
        const uint32_t below = (1u << lane) - 1u;
        for (uint32_t qb = 0; qb < s.quads; qb += 32 * kQuads) {
            float4 v[kQuads];
            load_block<false>(v, W, s, qb, lane);
#pragma unroll
            for (int u = 0; u < kQuads; ++u) {
                const uint32_t b0 = __ballot_sync(0xffffffffu, v[u].x != 0.0f), b1 = __ballot_sync(0xffffffffu, v[u].y != 0.0f);
                const uint32_t b2 = __ballot_sync(0xffffffffu, v[u].z != 0.0f), b3 = __ballot_sync(0xffffffffu, v[u].w != 0.0f);
                // entries of the lanes below come first, then this lane's own in column order
                uint32_t at = pos + __popc(b0 & below) + __popc(b1 & below) + __popc(b2 & below) + __popc(b3 & below);
                const uint32_t col = s.c_lo + 4 * (qb + 32 * u + lane) - (uint32_t)s.lead;
                if (v[u].x != 0.0f) { wd[at] = v[u].x; ix[at++] = col; }
                if (v[u].y != 0.0f) { wd[at] = v[u].y; ix[at++] = col + 1; }
                if (v[u].z != 0.0f) { wd[at] = v[u].z; ix[at++] = col + 2; }
                if (v[u].w != 0.0f) { wd[at] = v[u].w; ix[at++] = col + 3; }
                pos += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
            }
        }
    }
    if (unit + 1 == first + segs) {                         // the row's last segment also owns its padding and count
        for (uint32_t j = pos + lane; j < pitch; j += 32) { wd[j] = 0.0f; ix[j] = 0u; }
        if (lane == 0) nnz[s.row] = pos;
    }
}

__global__ void __launch_bounds__(kWarps * 32)
csr_fill_kernel(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ col,
                const float* __restrict__ val, uint32_t m, uint32_t pitch,
                float* __restrict__ Wd, uint32_t* __restrict__ idx, uint32_t* __restrict__ nnz)
{
    const int lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (row >= m) return;
    const uint64_t b = rowptr[row], e = rowptr[row + 1];
    const uint32_t cnt = (uint32_t)(e - b);
    for (uint32_t j = lane; j < cnt; j += 32) {
        Wd[(size_t)row * pitch + j] = val[b + j];
        idx[(size_t)row * pitch + j] = col[b + j];
    }
    if (lane == 0) nnz[row] = cnt;
}

// Decoder for handles whose columns ascend: a warp rebuilds kDecode columns of a row at a time in
// its own shared-memory strip (cleared, then the run of entries that falls into it is scattered) and
// writes the strip out with 16-byte stores, so the dense matrix is written once; clearing it first
// and scattering 4-byte values into it moved twice the bytes.
constexpr uint32_t kDecode = 1024;

__global__ void __launch_bounds__(kWarps * 32)
decode_rows_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx, const uint32_t* __restrict__ nnz,
                   uint32_t mis, uint32_t m, uint32_t n, uint32_t segs, uint32_t seg, uint32_t pitch, float* __restrict__ W)
{
    __shared__ __align__(16) float strips[kWarps][kDecode];
    constexpr int kRun = 4;                                 // 32 entries each, in flight together
    const int lane = threadIdx.x & 31;
    float* strip = strips[threadIdx.x >> 5];
    const uint64_t unit = (uint64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (unit >= (uint64_t)m * segs) return;
    const Segment s = segment_of(unit, mis, n, segs, seg);
    const float* __restrict__ wd = Wd + (size_t)s.row * pitch;
    const uint32_t* __restrict__ ix = idx + (size_t)s.row * pitch;
    const uint32_t cnt = __ldg(nnz + s.row);
    uint32_t pos = 0;                                       // first entry of the segment: binary search
    if (s.c_lo > 0) {
        uint32_t end = cnt;
        while (pos < end) {
            const uint32_t mid = (pos + end) >> 1;
            if (__ldg(ix + mid) < s.c_lo) pos = mid + 1; else end = mid;
        }
    }
    for (uint32_t qb = 0; qb < s.quads; qb += kDecode / 4) {        // strip element i <-> place c0 + i of the segment
        const int32_t c0 = 4 * (int32_t)qb - s.lead, c1 = min(c0 + (int32_t)kDecode, s.len);
        uint32_t k[kRun];                                           // places; columns ascend, so all are at or behind the first
        float w[kRun];
        auto fetch = [&] {
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                const uint32_t j = pos + 32 * u + lane;
                k[u] = j < cnt ? __ldg(ix + j) - s.c_lo : 0xffffffffu;
                w[u] = j < cnt ? __ldg(wd + j) : 0.0f;
            }
        };
        fetch();
#pragma unroll
        for (uint32_t i = 0; i < kDecode / 128; ++i) reinterpret_cast<float4*>(strip)[i * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        for (;;) {
            uint32_t took = 0;
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                const bool in = k[u] < (uint32_t)c1;
                if (in) strip[(int32_t)k[u] - c0] = w[u];
                took += __popc(__ballot_sync(0xffffffffu, in));     // a prefix: columns ascend
            }
            pos += took;
            if (took < 32 * kRun) break;
            fetch();
        }
        __syncwarp();
        float* __restrict__ out = W + s.at + 4ull * qb;
        const uint32_t quads = min(kDecode / 4, s.quads - qb);
        for (uint32_t i = lane; i < quads; i += 32) {
            const int32_t c = c0 + 4 * (int32_t)i;
            const float4 v = reinterpret_cast<const float4*>(strip)[i];
            float* __restrict__ o = out + 4 * i;
            if (c >= 0 && c + 4 <= s.len) { __stcs(reinterpret_cast<float4*>(o), v); continue; }
            if (c >= 0 && c < s.len) o[0] = v.x;
            if (c + 1 >= 0 && c + 1 < s.len) o[1] = v.y;
            if (c + 2 >= 0 && c + 2 < s.len) o[2] = v.z;
            if (c + 3 >= 0 && c + 3 < s.len) o[3] = v.w;
        }
        __syncwarp();
    }
}

// Any column order (handles made from raw arrays), and few columns: scatter into a cleared matrix.
__global__ void __launch_bounds__(kWarps * 32)
decode_scatter_kernel(const float* __restrict__ Wd, const uint32_t* __restrict__ idx,
                      const uint32_t* __restrict__ nnz, uint32_t m, uint32_t n, uint32_t pitch,
                      float* __restrict__ W)
{
    const int lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (row >= m) return;
    const uint32_t cnt = nnz[row];
    for (uint32_t j = lane; j < cnt; j += 32)
        W[(size_t)row * n + idx[(size_t)row * pitch + j]] = Wd[(size_t)row * pitch + j];
}

// Column segments per row: one warp per row when that already is 64 warps per SM, else enough
// segments (of at least 1024 columns) to get there.
struct Split {
    uint32_t segs, seg;
    unsigned blocks;
};
Split split_rows(uint32_t m, uint32_t n, int sms)
{
    Split s;
    const uint64_t want = (uint64_t)sms * 64;
    const uint64_t most = std::max<uint64_t>(1, n / 1024);
    s.segs = (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(1, (want + m - 1) / m));
    s.seg = (uint32_t)spx::round_up<uint64_t>(((uint64_t)n + s.segs - 1) / s.segs, 4u);
    s.segs = (uint32_t)(((uint64_t)n + s.seg - 1) / s.seg);
    s.blocks = (unsigned)(((uint64_t)m * s.segs + kWarps - 1) / kWarps);
    return s;
}

inline uint32_t misalignment(const float* p) { return (uint32_t)((reinterpret_cast<uintptr_t>(p) & 15) / sizeof(float)); }

}  // namespace

namespace spx {

// Pairs kept by the counter: some more than a quarter of a unit's columns (denser units are read again, which is then no
// more to move than pairs would be), and no more scratch than the pool keeps for the next call in any case.  A matrix that
// stays in L2 is read again for less than the pairs cost, short units end in blocks of 512 columns that are mostly empty.  With
// many rows the schedule costs more (m comparisons a row on the device) or shows, where the host's sort no longer hides
// behind the packer: rows have to be longer then (5 %, with and without the pairs: 5000 x 5000 110 and 124 us, 3000 x 3000
// 73.5 and 71.5; 10000 x 2100 97 and 95, 14000 x 4096 133 and 140, x 8000 178 and 223; sorted by the host 16000 x 4096 161
// and 148, x 6000 183 and 195).
constexpr size_t kKeepBytes = 288u << 20, kKeepFrom = 64u << 20;
constexpr uint32_t kKeepColumns = 2048, kKeepColumnsRanked = 4096, kKeepColumnsHostSort = 4608;
// Without the pairs the packer takes longer and hides the host's sort of more rows: 8192 x 2000 98 us ranked, 109 sorted;
// 9472 x 3000 140 and 139; 16384 x 1000 140 and 129.
constexpr uint32_t kRankRowsReread = 8192;
// A handful of short rows is sorted by the host in less time than a kernel for it takes (4 x 4 38 us sorted, 41 ranked; 7 x 13
// 41 and 41); of long ones not, whose lengths it counts one by one (2 x 255065, 78 % 113 us sorted, 80 ranked).
constexpr uint32_t kRankFrom = 8, kRankLong = 8192;

// Device memory of one call beside the handle's own.
struct EncodeScratch {
    uint32_t* counts = nullptr;     // per unit
    uint32_t* keys = nullptr;       // per row, where the device ranks them: length * kRankRows + reversed id
    uint2* kept = nullptr;
    uint32_t cap = 0;
};

// Everything but the two passes is kept off the critical path: what the host must know (r fixes the pitch) is one wait
// away, the row schedule is made beside the packer -- on the device for few rows (a row costs m comparisons), else sorted
// on the host -- and the arrays come from the library's pool.
static int encode_rows(const float* dW, uint32_t m, uint32_t n, int device, cudaStream_t s, const PinnedBlock& stage, const Split& sp,
                       const EncodeScratch& sc, spx_ell** out)
{
    const uint32_t mis = misalignment(dW);
    const bool ranked = sc.keys != nullptr;
    uint32_t* h_counts = static_cast<uint32_t*>(stage.host);    // m * segs counts, then the schedule; or the statistics
    const size_t units = (size_t)m * sp.segs;
    if (sc.kept) count_keep_kernel<<<sp.blocks, kWarps * 32, 0, s>>>(dW, mis, m, n, sp.segs, sp.seg, sc.cap, sc.counts, sc.kept);
    else count_kernel<<<sp.blocks, kWarps * 32, 0, s>>>(dW, mis, m, n, sp.segs, sp.seg, sc.counts);
    SPX_LAUNCH_CHECK("count_kernel");
    if (ranked) {
        void* stats = nullptr;
        SPX_CUDA(cudaHostGetDevicePointer(&stats, stage.host, 0));
        const auto kernel = sp.segs >= 16 ? row_stats_kernel<true> : row_stats_kernel<false>;
        kernel<<<1, 1024, 0, s>>>(sc.counts, m, sp.segs, sc.keys, static_cast<RowStats*>(stats));
        SPX_LAUNCH_CHECK("row_stats_kernel");
    } else {
        SPX_CUDA(cudaMemcpyAsync(h_counts, sc.counts, units * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    }
    // A schedule from the host travels on a stream of its own, beside the packer: its block is allocated in that stream's
    // order too (the pool may hand out memory that work queued on another stream still uses, ordered behind it on the
    // allocating stream only), and here, where the host would wait anyway and no packer is queued to wait for.
    void* schedule = nullptr;
    cudaStream_t side = s;
    const size_t schedule_bytes = (size_t)m * sizeof(uint2);
    if (!ranked)
        if (int rc = side_stream(device, &side)) return rc;
    if (int rc = pool_alloc(&schedule, schedule_bytes, device, side)) return rc;
    const cudaError_t counted = cudaStreamSynchronize(s);
    uint32_t r = 0;
    uint64_t total = 0;
    if (counted == cudaSuccess && ranked) {
        r = static_cast<const RowStats*>(stage.host)->longest;
        total = static_cast<const RowStats*>(stage.host)->total;
    } else if (counted == cudaSuccess) {
        if (sp.segs > 1)
            for (uint32_t i = 0; i < m; ++i) {
                uint32_t c = h_counts[(size_t)i * sp.segs];
                for (uint32_t k = 1; k < sp.segs; ++k) c += h_counts[(size_t)i * sp.segs + k];
                h_counts[i] = c;                                    // in place: i <= i * segs
            }
        for (uint32_t i = 0; i < m; ++i) {
            r = std::max(r, h_counts[i]);
            total += h_counts[i];
        }
    }
    const int rc_ell = counted == cudaSuccess ? alloc_ell(m, n, r, out, s, r == 0)
                                              : fail(SPX_ERR_CUDA, "encode: count pass failed: %s", cudaGetErrorString(counted));
    if (rc_ell != SPX_OK) {
        pool_free(schedule, schedule_bytes, side);
        return rc_ell;
    }
    spx_ell* e = *out;
    e->rows = static_cast<uint2*>(schedule);
    e->nnz_total = total;
    e->max_nnz = r;
    const uint32_t rank_ctas = ranked ? (m + kRankPerCta - 1) / kRankPerCta : 0;
    const uint32_t pack_ctas = r ? sp.blocks : 0;
    if (rank_ctas + pack_ctas) {
        pack_kernel<<<rank_ctas + pack_ctas, kWarps * 32, 0, s>>>(dW, mis, m, n, sp.segs, sp.seg, sc.counts, e->pitch, e->Wd, e->idx, e->nnz,
                                                                  sc.kept, sc.cap, sc.keys, e->rows, rank_ctas);
        SPX_LAUNCH_CHECK("pack_kernel");
    }
    if (ranked) {
        const RowStats& st = *static_cast<const RowStats*>(stage.host);
        e->min_nnz = st.shortest;
        e->long_rows = st.long_rows;
    } else {
        uint2* h_order = reinterpret_cast<uint2*>(h_counts + round_up<size_t>(units, 2));
        if (int rc = sort_rows(e, h_counts, h_order, side)) return rc;
        SPX_CUDA(cudaMemcpyAsync(e->rows, h_order, schedule_bytes, cudaMemcpyHostToDevice, side));
        SPX_CUDA(cudaStreamSynchronize(side));
    }
    SPX_CUDA(cudaStreamSynchronize(s));         // the handle may be used on any stream from here on
    return SPX_OK;
}

int encode_device(const float* dW, uint32_t m, uint32_t n, cudaStream_t s, spx_ell** out)
{
    if (m == 0 || n == 0) {                     // no entries: only the counts and the (trivial) schedule
        int rc = alloc_ell(m, n, 0, out, s);
        if (rc == SPX_OK) rc = set_row_order(*out, std::vector<uint32_t>(m, 0u).data());
        if (rc == SPX_OK) SPX_CUDA(cudaStreamSynchronize(s));
        return rc;
    }
    int device = 0;
    SPX_CUDA(cudaGetDevice(&device));
    const Split sp = split_rows(m, n, sm_count(device));
    const size_t units = (size_t)m * sp.segs;
    EncodeScratch sc;
    sc.cap = keep_cap(sp.seg);
    const size_t keep = units * sc.cap * sizeof(uint2);
    bool keeps = sp.seg >= (m <= kRankRowsReread ? kKeepColumns : m <= kRankRows ? kKeepColumnsRanked : kKeepColumnsHostSort) &&
                 (size_t)m * n * sizeof(float) >= kKeepFrom && keep <= kKeepBytes;
    const bool ranked = (m >= kRankFrom || n >= kRankLong) && m <= (keeps ? kRankRows : kRankRowsReread) && n < kRankColumns;
    PinnedBlock stage;
    if (int rc = pinned_acquire(ranked ? sizeof(RowStats) : (units + 1) * sizeof(uint32_t) + m * sizeof(uint2), &stage)) return rc;
    // counts, the rows' keys, the pairs, each on a 16-byte boundary
    const size_t keys_at = round_up<size_t>(units * sizeof(uint32_t), 16), kept_at = keys_at + (ranked ? round_up<size_t>(m * sizeof(uint32_t), 16) : 0);
    void* scratch = nullptr;
    int rc = scratch_alloc(&scratch, kept_at + (keeps ? keep : 0), device, s, keeps);
    if (rc == SPX_ERR_OOM && keeps) {           // it goes without
        keeps = false;
        rc = scratch_alloc(&scratch, kept_at, device, s);
    }
    if (rc == SPX_OK) {
        unsigned char* base = static_cast<unsigned char*>(scratch);
        sc.counts = reinterpret_cast<uint32_t*>(base);
        if (ranked) sc.keys = reinterpret_cast<uint32_t*>(base + keys_at);
        if (keeps) sc.kept = reinterpret_cast<uint2*>(base + kept_at);
        rc = encode_rows(dW, m, n, device, s, stage, sp, sc, out);
    }
    if (rc != SPX_OK) {
        (void)cudaStreamSynchronize(s);         // nothing may still write the staging block
        if (*out) spx_ell_destroy(*out);
        *out = nullptr;
    }
    scratch_free(scratch, s);
    pinned_release(stage);
    return rc;
}

int decode_device(const spx_ell* e, float* dW, cudaStream_t s)
{
    if (e->m == 0 || e->n == 0) return SPX_OK;
    if (e->r == 0) {
        SPX_CUDA(cudaMemsetAsync(dW, 0, (size_t)e->m * e->n * sizeof(float), s));
        return SPX_OK;
    }
    // A row of a few columns is not worth a warp's strip: 100000 x 64 35 us through strips, 25 cleared and scattered;
    // 300000 x 100 95 and 93, 200000 x 200 74 and 88.  (Few rows: one launch is less than two, 64 x 64 14 us against 18.)
    if (e->cols_ascending && (e->n >= 128 || e->m < 32768)) {
        const Split sp = split_rows(e->m, e->n, sm_count(e->device));
        decode_rows_kernel<<<sp.blocks, kWarps * 32, 0, s>>>(e->Wd, e->idx, e->nnz, misalignment(dW), e->m, e->n, sp.segs, sp.seg,
                                                            e->pitch, dW);
        SPX_LAUNCH_CHECK("decode_rows_kernel");
        return SPX_OK;
    }
    SPX_CUDA(cudaMemsetAsync(dW, 0, (size_t)e->m * e->n * sizeof(float), s));
    decode_scatter_kernel<<<(e->m + kWarps - 1) / kWarps, kWarps * 32, 0, s>>>(e->Wd, e->idx, e->nnz, e->m, e->n, e->pitch, dW);
    SPX_LAUNCH_CHECK("decode_scatter_kernel");
    return SPX_OK;
}

int csr_to_ell_device(spx_ell* e, const uint64_t* d_rowptr, const uint32_t* d_col, const float* d_val,
                      cudaStream_t s)
{
    if (e->m == 0) return SPX_OK;
    csr_fill_kernel<<<(e->m + kWarps - 1) / kWarps, kWarps * 32, 0, s>>>(d_rowptr, d_col, d_val, e->m, e->pitch,
                                                                       e->Wd, e->idx, e->nnz);
    SPX_LAUNCH_CHECK("csr_fill_kernel");
    return SPX_OK;
}

}  // namespace spx
