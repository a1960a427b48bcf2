// Drives hostcopy.cu on the stand-in runtime; `main <scenario>` exits 0 when it holds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <thread>
#include <vector>

#include "fake_runtime.hpp"

namespace spx {
int copy_h2d(void* dst, const void* src, size_t bytes, cudaStream_t s);
int copy_h2d_rows(void* dst, const void* src, size_t rows, size_t row, size_t stride, cudaStream_t s);
}  // namespace spx

using fake::Stream;
using Bytes = std::vector<char>;

#define CHECK(x) do { if (!(x)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #x); exit(1); } } while (0)

static Bytes noise(size_t n, unsigned seed)
{
    std::mt19937 g(seed);
    Bytes b(n + 8);
    for (size_t i = 0; i < n; i += 4) { const uint32_t v = g(); memcpy(b.data() + i, &v, 4); }
    b.resize(n);
    return b;
}

// Copies of many sizes in a row, the source overwritten as soon as the call returns, all read back at the end.
static void contiguous(Stream& st, unsigned seed)
{
    const size_t K = 1024, M = K * K;
    const size_t sizes[] = {4, 256 * K - 4, 256 * K, 256 * K + 4, M, 4 * M, 4 * M + 4, 8 * M + 20, 13 * M + 4, 300 * K + 12};
    std::vector<Bytes> want, got;
    for (size_t n : sizes) {
        const size_t off = seed % 3 * 4 + 4;
        Bytes src = noise(n + off, seed + (unsigned)n);
        want.emplace_back(src.begin() + off, src.end());
        got.emplace_back(n);
        CHECK(spx::copy_h2d(got.back().data(), src.data() + off, n, st.handle()) == 0);
        memset(src.data(), 0x55, src.size());
    }
    CHECK(cudaStreamSynchronize(st.handle()) == cudaSuccess);
    for (size_t i = 0; i < want.size(); ++i) CHECK(want[i] == got[i]);
}

static void panels(Stream& st)
{
    struct P { size_t rows, row, stride; } ps[] = {{8192, 128, 256}, {5000, 300, 1200}, {40000, 512, 2048}, {3, 262144, 300000}, {2, 300000, 300004}, {70000, 4, 8}};
    std::vector<Bytes> want, got;
    unsigned seed = 1;
    for (auto& p : ps) {
        Bytes src = noise(p.rows * p.stride, seed++), w(p.rows * p.row);
        for (size_t r = 0; r < p.rows; ++r) memcpy(w.data() + r * p.row, src.data() + r * p.stride, p.row);
        want.push_back(w);
        got.emplace_back(w.size());
        CHECK(spx::copy_h2d_rows(got.back().data(), src.data(), p.rows, p.row, p.stride, st.handle()) == 0);
        memset(src.data(), 0x55, src.size());
    }
    CHECK(cudaStreamSynchronize(st.handle()) == cudaSuccess);
    for (size_t i = 0; i < want.size(); ++i) CHECK(want[i] == got[i]);
}

int main(int argc, char** argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    Stream a, b;
    if (what == "sizes") {
        contiguous(a, 1);
        contiguous(b, 2);
        contiguous(a, 3);
    } else if (what == "panels") {
        panels(a);
        panels(b);
    } else if (what == "threads") {
        std::vector<std::thread> ts;
        std::vector<Stream> ss(4);
        for (unsigned i = 0; i < 4; ++i) ts.emplace_back([&, i] { for (int k = 0; k < 3; ++k) contiguous(ss[i], 10 * i + k); });
        for (auto& t : ts) t.join();
    } else if (what == "capture") {
        // a recorded copy reads the caller's memory when the graph runs, whatever was copied in between
        Bytes src = noise(1 << 20, 7), dst(1 << 20);
        a.capturing = true;
        CHECK(spx::copy_h2d(dst.data(), src.data(), src.size(), a.handle()) == 0);
        a.capturing = false;
        CHECK(!a.nodes.empty());
        for (auto& n : a.nodes) CHECK(!fake::is_pinned(n.src));
        contiguous(b, 4);
        contiguous(a, 5);
        const Bytes later = noise(1 << 20, 8);
        memcpy(src.data(), later.data(), src.size());
        for (auto& n : a.nodes) n.run();
        CHECK(dst == src);
        // and a copy that has used the ring before
        a.nodes.clear();
        a.capturing = true;
        CHECK(spx::copy_h2d(dst.data(), src.data(), src.size(), a.handle()) == 0);
        a.capturing = false;
        contiguous(b, 6);
    } else if (what == "capture_elsewhere") {
        // the thread records a graph on one stream and copies on another
        fake::recording_elsewhere = true;
        Bytes src = noise(9 << 20, 9), dst(9 << 20);
        CHECK(spx::copy_h2d(dst.data(), src.data(), src.size(), a.handle()) == 0);
        CHECK(spx::copy_h2d(dst.data(), src.data(), src.size(), a.handle()) == 0);
        fake::recording_elsewhere = false;
        CHECK(!fake::recording_broken);
        CHECK(cudaStreamSynchronize(a.handle()) == cudaSuccess);
        CHECK(dst == src);
    } else if (what == "failed_copy") {
        // a copy that fails half way: what it had sent arrives intact although the ring is used again at once
        for (int nth = 2; nth <= 6; ++nth) {
            const size_t n = 12 << 20, piece = 256 * 1024;
            Bytes src = noise(n, 20 + nth), dst(n, 0x11), none(n, 0x11);
            fake::fail_copy_in = nth;
            const int rc = spx::copy_h2d(dst.data(), src.data(), n, a.handle());
            const bool failed = fake::fail_copy_in == 0;
            fake::fail_copy_in = 0;
            CHECK(failed ? rc != 0 : rc == 0);
            contiguous(b, nth);
            CHECK(cudaStreamSynchronize(a.handle()) == cudaSuccess);
            for (size_t at = 0; at < n; at += piece)
                CHECK(!memcmp(&dst[at], &src[at], piece) || !memcmp(&dst[at], &none[at], piece));
        }
    } else if (what == "other_device") {
        // streams of a device that is not current take copies as well
        b.device = 1;
        contiguous(a, 1);
        contiguous(b, 2);
        fake::current_device = 1;
        contiguous(a, 3);
        contiguous(b, 4);
    } else {
        printf("unknown scenario\n");
        return 2;
    }
    return 0;
}
