// CPU check of the threaded device-to-host reads (magnelio_b200/csrc/hostcopy.cuh)
// against a stand-in CUDA runtime (a header of its own beside the compiled
// copy of this file): every byte arrives once, at sizes around a piece and a
// lane; the stream's queued work is waited for once, before any piece is
// copied or any thread started; a thread that cannot be created, for want of
// a thread or of memory, leaves its pieces to the others; a missing
// page-locked allocation and a failing copy behave as documented.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "hostcopy.cuh"

// allocations from now that still succeed on the counting thread (< 0: all)
static thread_local long g_allocs = -1;
void* operator new(std::size_t n) {
    if (g_allocs == 0) throw std::bad_alloc();
    if (g_allocs > 0) --g_allocs;
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

static int run(size_t bytes, long allocs, bool no_pinned, long fail_copy) {
    std::vector<unsigned char> src(bytes), dst(bytes, 0xee);
    for (size_t q = 0; q < bytes; ++q) src[q] = (unsigned char)(q * 131 + (q >> 13));
    fake::reset();
    fake::no_pinned = no_pinned;
    fake::fail_copy = fail_copy;
    fitb::HostLanes lanes;
    std::vector<std::atomic<int>> seen(bytes / fitb::HostLanes::kPiece + 1);  // per piece
    const fitb::HostLanes::Sink sink = [&](size_t off, const void* p, size_t n) {
        memcpy(dst.data() + off, p, n);
        ++seen[off / fitb::HostLanes::kPiece];
    };
    int stream = 0;
    cudaError_t rc = cudaSuccess;
    bool threw = false;
    if (!no_pinned && allocs >= 0) lanes.prepare(fitb::HostLanes::kLanes);
    g_allocs = allocs;
    try {
        rc = lanes.read(0, src.data(), bytes, &stream, sink);
    } catch (const std::bad_alloc&) {
        threw = true;  // before any thread runs: an error of the call
    }
    g_allocs = -1;
    if (fail_copy >= 0) return rc == cudaErrorUnknown ? 0 : 1;
    if (threw) return 0;
    const bool twice = std::any_of(seen.begin(), seen.end(), [](const std::atomic<int>& c) { return c.load() > 1; });
    if (rc != cudaSuccess || twice || memcmp(src.data(), dst.data(), bytes)) return 1;
    if (!no_pinned && bytes && (fake::waits != 1 || fake::copies_before_wait != 0)) return 2;
    return 0;
}

int main() {
    const size_t P = fitb::HostLanes::kPiece, L = fitb::HostLanes::kLanes;
    int cases = 0;
    for (size_t bytes : {(size_t)16, P - 16, P, P + 16, 3 * P + 8, L * P, L * P + 16, 3 * L * P - 16}) {
        for (long allocs : {-1L, 0L, 1L, 2L, 3L, 5L, 9L, 13L})
            for (bool no_pinned : {false, true}) {
                if (no_pinned && allocs >= 0) continue;
                ++cases;
                if (const int e = run(bytes, allocs, no_pinned, -1)) {
                    std::printf("%zu bytes, %ld allocations, pinned %d: %d\n", bytes, allocs, !no_pinned, e);
                    return 1;
                }
            }
        ++cases;
        if (run(bytes, -1, false, (long)(bytes / P / 2))) {
            std::printf("%zu bytes: a failing copy was not reported\n", bytes);
            return 1;
        }
    }
    std::printf("ok %d reads\n", cases);
    return 0;
}
