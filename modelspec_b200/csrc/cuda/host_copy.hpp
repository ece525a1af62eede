// Device-to-host copies into memory that is not pinned.
//
// The driver's own path for such a destination is one thread that copies through a small pinned
// buffer: 0.95 ms for 16 MB into touched pages, and 13 ms for the 62 MB of a prediction into pages
// the kernel still has to zero (4.6 GB/s; the same bytes reach pinned memory at 55 GB/s). Here
// several threads each move their share of 1 MB pieces through two pinned pieces of their own, so
// that the copies out of the staging memory and the page faults of a fresh destination overlap with
// one another and with the transfers.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace msx {

class HostCopier {
public:
    HostCopier() = default;
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;
    ~HostCopier() { release(); }

    // Copies `bytes` from the device to `host` behind what `stream` holds, and returns when they have
    // arrived. The first error of any thread is the result. A share whose thread cannot be started (a
    // process at its limit of threads or memory) is moved by the caller's.
    cudaError_t to_host(int device, void* host, const void* from, uint64_t bytes, cudaStream_t stream) {
        cudaPointerAttributes where;
        const bool pageable = bytes >= kSmallest && cudaPointerGetAttributes(&where, host) == cudaSuccess && where.type == cudaMemoryTypeUnregistered;
        // One staged copy at a time: the transfers of two would share the one bus anyway.
        std::unique_lock<std::mutex> held(mutex_, std::defer_lock);
        if (!pageable || !held.try_lock() || !prepare(lanes_for(bytes))) {
            cudaError_t e = cudaMemcpyAsync(host, from, bytes, cudaMemcpyDeviceToHost, stream);
            return e != cudaSuccess ? e : cudaStreamSynchronize(stream);
        }
        cudaError_t e = cudaEventRecord(ready_, stream);
        if (e != cudaSuccess) return e;
        const uint64_t pieces = (bytes + kPiece - 1) / kPiece;
        const uint32_t lanes = static_cast<uint32_t>(std::min<uint64_t>(lanes_for(bytes), lanes_.size()));
        std::atomic<int> failed{static_cast<int>(cudaSuccess)};
        auto work = [&](uint32_t l) {
            cudaError_t mine = cudaSetDevice(device);
            if (mine == cudaSuccess) mine = move_pieces(lanes_[l], static_cast<char*>(host), static_cast<const char*>(from), bytes, l, pieces, lanes);
            int none = static_cast<int>(cudaSuccess);
            if (mine != cudaSuccess) failed.compare_exchange_strong(none, static_cast<int>(mine));
        };
        std::thread others[kMostLanes];
        uint32_t started = 1;
        try {
            for (; started < lanes; ++started) others[started] = std::thread(work, started);
        } catch (const std::exception&) {
        }
        work(0);
        for (uint32_t l = started; l < lanes; ++l) work(l);
        for (std::thread& t : others)
            if (t.joinable()) t.join();
        return static_cast<cudaError_t>(failed.load());
    }

private:
    // Below kSmallest the driver's path is as fast; a lane needs a piece or two to be worth a thread.
    static constexpr uint64_t kSmallest = 256ull << 10, kPiece = 1ull << 20;
    static constexpr uint32_t kMostLanes = 8;

    struct Lane {
        char* piece[2] = {nullptr, nullptr};
        cudaEvent_t arrived[2] = {nullptr, nullptr};
        cudaStream_t stream = nullptr;
    };

    static uint32_t lanes_for(uint64_t bytes) {
        const uint32_t cores = std::max(1u, std::thread::hardware_concurrency());
        const uint64_t wanted = bytes / (2 * kPiece);
        return static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>({wanted, kMostLanes, cores})));
    }

    // Makes the lanes a copy needs (at most kMostLanes of two pieces each, kept for the next copy).
    bool prepare(uint32_t lanes) {
        if (!ready_ && cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming) != cudaSuccess) return false;
        while (lanes_.size() < lanes) {
            Lane lane;
            bool ok = cudaStreamCreateWithFlags(&lane.stream, cudaStreamNonBlocking) == cudaSuccess;
            for (int h = 0; h < 2 && ok; ++h)
                ok = cudaMallocHost(&lane.piece[h], kPiece) == cudaSuccess && cudaEventCreateWithFlags(&lane.arrived[h], cudaEventDisableTiming) == cudaSuccess;
            if (!ok) {
                drop(lane);
                cudaGetLastError();  // the plain copy takes over
                return !lanes_.empty();
            }
            lanes_.push_back(lane);
        }
        return true;
    }

    cudaError_t move_pieces(Lane& lane, char* host, const char* from, uint64_t bytes, uint64_t first, uint64_t pieces, uint64_t stride) {
        auto size_of = [&](uint64_t p) { return std::min<uint64_t>(kPiece, bytes - p * kPiece); };
        auto fetch = [&](uint64_t p, int h) {
            cudaError_t e = cudaMemcpyAsync(lane.piece[h], from + p * kPiece, size_of(p), cudaMemcpyDeviceToHost, lane.stream);
            return e != cudaSuccess ? e : cudaEventRecord(lane.arrived[h], lane.stream);
        };
        cudaError_t e = cudaStreamWaitEvent(lane.stream, ready_, 0);
        for (int h = 0; h < 2 && e == cudaSuccess; ++h)
            if (first + h * stride < pieces) e = fetch(first + h * stride, h);
        int h = 0;
        for (uint64_t p = first; p < pieces && e == cudaSuccess; p += stride, h ^= 1) {
            e = cudaEventSynchronize(lane.arrived[h]);
            if (e != cudaSuccess) break;
            std::memcpy(host + p * kPiece, lane.piece[h], size_of(p));
            if (p + 2 * stride < pieces) e = fetch(p + 2 * stride, h);
        }
        if (e != cudaSuccess) cudaStreamSynchronize(lane.stream);  // nothing of a failed copy is left in flight
        return e;
    }

    static void drop(Lane& lane) {
        if (lane.stream) cudaStreamDestroy(lane.stream);
        for (int h = 0; h < 2; ++h) {
            if (lane.piece[h]) cudaFreeHost(lane.piece[h]);
            if (lane.arrived[h]) cudaEventDestroy(lane.arrived[h]);
        }
        lane = Lane();
    }
    void release() {
        for (Lane& lane : lanes_) drop(lane);
        lanes_.clear();
        if (ready_) cudaEventDestroy(ready_);
        ready_ = nullptr;
    }

    std::mutex mutex_;
    std::vector<Lane> lanes_;
    cudaEvent_t ready_ = nullptr;
};

}  // namespace msx
