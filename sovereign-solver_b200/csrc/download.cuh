// download.cuh -- a large result's way to ordinary host memory. The driver's
// copy into unpinned memory is one host thread's work, page faults of a fresh
// array included: 160 MB in 35 ms (4.6 GB/s). Here several threads each copy
// their pieces through two pinned pieces of their own, the next one on its way
// while the last is moved on.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

namespace pdhg {

// One per engine; its pinned pieces and streams are made by the first large
// download and freed with it. Not for use by two threads at once (as the
// engine's stream and buffers are not).
class Downloads {
   public:
    struct Part {
        void* dst;
        const void* src;
        size_t bytes;
    };

    Downloads() = default;
    Downloads(const Downloads&) = delete;
    Downloads& operator=(const Downloads&) = delete;
    ~Downloads() {
        for (Lane& l : lanes_) cudaStreamDestroy(l.stream);
        if (pinned_ != nullptr) cudaFreeHost(pinned_);
    }

    // Copies the parts (null destinations: none) after what `stream` holds, and
    // returns when they have arrived.
    cudaError_t run(const Part* parts, int count, int device, cudaStream_t stream) {
        std::vector<Part> staged;
        size_t total = 0;
        for (int i = 0; i < count; ++i) {
            const Part& p = parts[i];
            if (p.dst == nullptr || p.bytes == 0) continue;
            cudaPointerAttributes a{};
            const bool plain = p.bytes >= kPiece && cudaPointerGetAttributes(&a, p.dst) == cudaSuccess &&
                               a.type == cudaMemoryTypeUnregistered;
            if (plain) {
                staged.push_back(p);
                total += p.bytes;
            }
        }
        if (total < kLarge || !make_lanes()) staged.clear();
        for (int i = 0; i < count; ++i) {
            const Part& p = parts[i];
            if (p.dst == nullptr || p.bytes == 0) continue;
            bool here = true;
            for (const Part& s : staged) here = here && s.dst != p.dst;
            if (!here) continue;
            const cudaError_t e = cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, stream);
            if (e != cudaSuccess) return e;
        }
        const cudaError_t e = cudaStreamSynchronize(stream);
        return e != cudaSuccess || staged.empty() ? e : spread(staged, device);
    }

   private:
    // Pinned memory costs about 1 ms per MB to make: pieces of 256 KB, whose
    // copy (10 us) hides under the last one's move, 4 MB for all lanes. The
    // rule's line: a first download of 32 MB already wins back the 5 ms that
    // the lanes take (7 ms by the driver, 2 ms by the lanes); one of 11 MB
    // would gain 1 ms only once they are there.
    static constexpr size_t kPiece = size_t{256} << 10, kLarge = size_t{32} << 20;
    static constexpr size_t kMostLanes = 8;
    struct Lane {
        cudaStream_t stream = nullptr;
        unsigned char* piece[2] = {nullptr, nullptr};
    };
    std::vector<Lane> lanes_;
    unsigned char* pinned_ = nullptr;

    // False: no room for them, or too few host cores.
    bool make_lanes() {
        if (!lanes_.empty()) return true;
        size_t want = std::thread::hardware_concurrency() / 2;
        if (want > kMostLanes) want = kMostLanes;
        if (want < 2) return false;
        void* p = nullptr;
        if (cudaHostAlloc(&p, 2 * kPiece * want, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        pinned_ = static_cast<unsigned char*>(p);
        while (lanes_.size() < want) {
            Lane l;
            if (cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking) != cudaSuccess) {
                cudaGetLastError();  // fewer lanes
                break;
            }
            for (int i = 0; i < 2; ++i) l.piece[i] = pinned_ + (2 * lanes_.size() + i) * kPiece;
            lanes_.push_back(l);
        }
        if (!lanes_.empty()) return true;
        cudaFreeHost(pinned_);
        pinned_ = nullptr;
        return false;
    }

    cudaError_t spread(const std::vector<Part>& parts, int device) {
        struct Piece {
            unsigned char* dst;
            const unsigned char* src;
            size_t bytes;
        };
        std::vector<Piece> pieces;
        for (const Part& p : parts)
            for (size_t o = 0; o < p.bytes; o += kPiece)
                pieces.push_back({static_cast<unsigned char*>(p.dst) + o, static_cast<const unsigned char*>(p.src) + o,
                                  p.bytes - o < kPiece ? p.bytes - o : kPiece});
        std::atomic<size_t> next{0};
        std::atomic<int> error{static_cast<int>(cudaSuccess)};
        auto work = [&](Lane* l) {
            cudaError_t e = cudaSetDevice(device);
            size_t cur = next.fetch_add(1), q = 0;
            auto fetch = [&](size_t i, size_t w) {
                if (e == cudaSuccess && i < pieces.size())
                    e = cudaMemcpyAsync(l->piece[w], pieces[i].src, pieces[i].bytes, cudaMemcpyDeviceToHost, l->stream);
            };
            fetch(cur, q);
            while (e == cudaSuccess && cur < pieces.size()) {
                e = cudaStreamSynchronize(l->stream);
                const size_t then = next.fetch_add(1);
                fetch(then, q ^ 1);
                if (e == cudaSuccess) std::memcpy(pieces[cur].dst, l->piece[q], pieces[cur].bytes);
                cur = then;
                q ^= 1;
            }
            if (e != cudaSuccess) {
                cudaStreamSynchronize(l->stream);  // nothing still writes to the pieces
                error.store(static_cast<int>(e));
                next.store(pieces.size());
            }
        };
        const size_t n = lanes_.size();
        std::vector<std::thread> threads;
        threads.reserve(n);
        try {
            for (size_t i = 1; i < n; ++i) threads.emplace_back(work, &lanes_[i]);
        } catch (const std::exception&) {  // no more threads: those that run do it
        }
        work(&lanes_[0]);
        for (std::thread& t : threads) t.join();
        return static_cast<cudaError_t>(error.load());
    }
};

}  // namespace pdhg
