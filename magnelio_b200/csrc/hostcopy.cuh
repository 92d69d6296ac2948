// Device-to-host reads of large results into the caller's pageable memory.
//
// A cudaMemcpy to pageable memory runs through the driver's staging buffer on
// one host thread, which also takes the page faults of a freshly allocated
// destination: 4.8 GB/s.  Here up to kLanes host threads each pull 1 MB pieces
// through a page-locked slot of their own and write them (converted if need
// be) to the destination, so the copy engine, the page faults and the host
// writes of different pieces overlap.  Measured on a 16-core host (ms):
// the fields of 16.8 M float32 cells (406 MB) 84 before, 23 now, of 49 M cells
// 245 and 65; nine components of 16 monitored frequencies on 256 x 256 cells
// 92 (with the caller's complex assembly) and 9.  Threads that sleep in the
// event wait instead of spinning give 42 / 120 / 17.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <exception>
#include <functional>
#include <thread>
#include <vector>

namespace fitb {

struct HostLanes {
    static constexpr int kLanes = 8;
    static constexpr size_t kPiece = 1 << 20;   // bytes of one piece
    static constexpr size_t kSmall = 512 << 10;  // up to here: one plain copy

    void* slots = nullptr;  // page-locked pieces, as many as a read has used at once
    int n_slots = 0;
    cudaEvent_t ev[kLanes] = {};
    HostLanes() = default;
    HostLanes(const HostLanes&) = delete;
    HostLanes& operator=(const HostLanes&) = delete;
    ~HostLanes() {
        if (slots) cudaFreeHost(slots);
        for (auto& e : ev)
            if (e) cudaEventDestroy(e);
    }
    cudaError_t prepare(int lanes) {
        if (lanes <= n_slots) return cudaSuccess;
        for (int q = 0; q < lanes; ++q) {
            if (ev[q]) continue;
            const cudaError_t rc = cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming);
            if (rc != cudaSuccess) return rc;
        }
        if (slots) cudaFreeHost(slots);
        slots = nullptr;
        n_slots = 0;
        const cudaError_t rc = cudaMallocHost(&slots, (size_t)lanes * kPiece);
        if (rc == cudaSuccess) n_slots = lanes;
        return rc;
    }

    // Reads `bytes` device bytes at `src` behind the work of stream `s`;
    // sink(offset, data, n) consumes the n bytes at `offset` and may run on
    // several threads at once, on disjoint ranges; it does not throw.  Pieces
    // are multiples of 16 bytes.  Returns when every byte is consumed (or with
    // the first error, after every thread has stopped).
    using Sink = std::function<void(size_t, const void*, size_t)>;
    cudaError_t read(int device, const void* src, size_t bytes, cudaStream_t s, const Sink& sink) {
        const size_t pieces = (bytes + kPiece - 1) / kPiece;
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        const int lanes = (int)std::min<size_t>({(size_t)kLanes, (size_t)hw, std::max<size_t>(1, pieces)});
        if (prepare(lanes) != cudaSuccess) {
            cudaGetLastError();
            return read_pageable(src, bytes, s, sink);
        }
        // one wait for the steps still queued: the threads spin in theirs
        const cudaError_t rc = cudaStreamSynchronize(s);
        if (rc != cudaSuccess) return rc;
        std::atomic<size_t> next{0};
        std::atomic<int> err{0};
        const auto work = [&](int lane) {
            char* slot = static_cast<char*>(slots) + (size_t)lane * kPiece;
            cudaError_t e = cudaSetDevice(device);
            while (e == cudaSuccess && err.load() == 0) {
                const size_t q = next.fetch_add(1);
                if (q >= pieces) break;
                const size_t off = q * kPiece, n = std::min(kPiece, bytes - off);
                e = cudaMemcpyAsync(slot, static_cast<const char*>(src) + off, n, cudaMemcpyDeviceToHost, s);
                if (e == cudaSuccess) e = cudaEventRecord(ev[lane], s);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[lane]);
                if (e == cudaSuccess) sink(off, slot, n);
            }
            if (e != cudaSuccess) err.store((int)e);
        };
        std::vector<std::thread> pool;
        pool.reserve(lanes);
        try {
            for (int t = 1; t < lanes; ++t) pool.emplace_back(work, t);
        } catch (const std::exception&) {
            // no thread or no memory for one: the others take its pieces
        }
        work(0);
        for (auto& t : pool) t.join();
        return (cudaError_t)err.load();
    }

    // Where no page-locked memory is to be had: one thread, a pageable piece.
    static cudaError_t read_pageable(const void* src, size_t bytes, cudaStream_t s, const Sink& sink) {
        std::vector<char> piece(std::min(kPiece, bytes));
        cudaError_t e = cudaSuccess;
        for (size_t off = 0; off < bytes && e == cudaSuccess; off += kPiece) {
            const size_t n = std::min(kPiece, bytes - off);
            e = cudaMemcpyAsync(piece.data(), static_cast<const char*>(src) + off, n, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e == cudaSuccess) sink(off, piece.data(), n);
        }
        return e;
    }
};

}  // namespace fitb
