// Device-to-host copies into memory that is not pinned.
//
// The driver's own path for such a destination is one thread that copies through a small pinned
// buffer, faulting in the pages that nothing has touched yet: 60 us a MB into touched pages, 450 into fresh ones
// (3.7 ms for 8 MB, 28 ms for the 62 MB of a prediction; the same bytes reach pinned memory at 55 GB/s). Here
// several threads each move their share of the pieces through two pinned pieces of their own, so
// that the copies out of the staging memory and the page faults of a fresh destination overlap with
// one another and with the transfers. Measured on 16 cores, us a copy (driver's path, this one):
//
//   MB             0.25         1           2           4           8           12          16          62
//   fresh        102, 111   446, 398   1123, 412   2241, 944   3979, 1039  5731, 1516  7530, 1669  28618, 4985
//   touched     (the driver's path up to 12 MB: 34, 90, 153, 263, 508)    1211, 822   1320, 944   3993, 2387
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "pinned.hpp"

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
        // One staged copy at a time: the transfers of two would share the one bus anyway.
        std::unique_lock<std::mutex> held(mutex_, std::defer_lock);
        if (!pageable(host, bytes) || !held.try_lock() || !worth_staging(host, bytes)) {
            cudaError_t e = cudaMemcpyAsync(host, from, bytes, cudaMemcpyDeviceToHost, stream);
            return e != cudaSuccess ? e : cudaStreamSynchronize(stream);
        }
        cudaError_t e = cudaEventRecord(ready_, stream);
        if (e != cudaSuccess) return e;
        // All lanes from 2 MB on, with two pieces each where that leaves them large enough: below, the
        // threads would take as long to start as the one copies.
        const uint32_t lanes = bytes < kAllLanes ? 1 : static_cast<uint32_t>(lanes_.size());
        const uint64_t share = (bytes / (2 * lanes) + kPage - 1) / kPage * kPage;
        const uint64_t piece = std::min<uint64_t>(kPiece, std::max<uint64_t>(kSmallest, share));
        const uint64_t pieces = (bytes + piece - 1) / piece;
        std::atomic<int> failed{static_cast<int>(cudaSuccess)};
        auto work = [&](uint32_t l) {
            cudaError_t mine = cudaSetDevice(device);
            if (mine == cudaSuccess) mine = move_pieces(lanes_[l], static_cast<char*>(host), static_cast<const char*>(from), bytes, piece, l, pieces, lanes);
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
    static constexpr uint64_t kSmallest = 256ull << 10, kPiece = 1ull << 20, kAllLanes = 2ull << 20, kPage = 4096;
    static constexpr uint32_t kMostLanes = 8;
    // A staged copy is the faster one into fresh pages always, into touched ones from kTouched on (alone from
    // 12 MB on, as in the table above; behind a forward program in a process with other work 15 and 17 MB took
    // 2 to 4 % longer than by the driver, 19 and 20 MB 4 to 9 % less). Making the lanes takes 5 ms: what staging saves on one copy of kTouchedMakes bytes, or on
    // kFreshMakes of copies into fresh pages in all.
    static constexpr uint64_t kTouched = 18ull << 20, kTouchedMakes = 160ull << 20, kFreshMakes = 20ull << 20;

    struct Lane {
        char* piece[2] = {nullptr, nullptr};
        cudaEvent_t arrived[2] = {nullptr, nullptr};
        cudaStream_t stream = nullptr;
    };

    static bool pageable(const void* host, uint64_t bytes) {
        if (bytes < kSmallest) return false;
        cudaPointerAttributes where;
        if (cudaPointerGetAttributes(&where, host) == cudaSuccess) return where.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();  // the plain copy takes over
        return false;
    }

    // Whether the destination's pages exist, by the look of a few of them (half a microsecond each).
    static bool touched(const void* host, uint64_t bytes) {
        for (uint64_t i = 1; i <= 4; ++i) {
            unsigned char resident = 0;
            const uintptr_t at = (reinterpret_cast<uintptr_t>(host) + bytes / 5 * i) / kPage * kPage;
            if (mincore(reinterpret_cast<void*>(at), kPage, &resident) != 0 || !(resident & 1u)) return false;
        }
        return true;
    }

    bool worth_staging(const void* host, uint64_t bytes) {
        const bool there = touched(host, bytes);
        if (there && bytes < kTouched) return false;
        if (!lanes_.empty()) return true;
        if (!there) fresh_bytes_ += bytes;
        return (bytes >= kTouchedMakes || fresh_bytes_ >= kFreshMakes) && make_lanes();
    }

    // The lanes of all later copies: one block of pinned memory, a stream a lane.
    bool make_lanes() {
        const uint32_t lanes = std::min(kMostLanes, std::max(1u, std::thread::hardware_concurrency()));
        bool ok = pinned_.make(2 * lanes * kPiece) == cudaSuccess && cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming) == cudaSuccess;
        for (uint32_t l = 0; l < lanes && ok; ++l) {
            Lane lane;
            ok = cudaStreamCreateWithFlags(&lane.stream, cudaStreamNonBlocking) == cudaSuccess;
            for (uint32_t h = 0; h < 2; ++h) {
                lane.piece[h] = pinned_.data() + (2 * l + h) * kPiece;
                ok = ok && cudaEventCreateWithFlags(&lane.arrived[h], cudaEventDisableTiming) == cudaSuccess;
            }
            lanes_.push_back(lane);
        }
        if (ok) return true;
        release();
        cudaGetLastError();  // the plain copy takes over
        return false;
    }

    cudaError_t move_pieces(Lane& lane, char* host, const char* from, uint64_t bytes, uint64_t piece, uint64_t first, uint64_t pieces,
                            uint64_t stride) {
        auto size_of = [&](uint64_t p) { return std::min<uint64_t>(piece, bytes - p * piece); };
        auto fetch = [&](uint64_t p, int h) {
            cudaError_t e = cudaMemcpyAsync(lane.piece[h], from + p * piece, size_of(p), cudaMemcpyDeviceToHost, lane.stream);
            return e != cudaSuccess ? e : cudaEventRecord(lane.arrived[h], lane.stream);
        };
        cudaError_t e = cudaStreamWaitEvent(lane.stream, ready_, 0);
        for (int h = 0; h < 2 && e == cudaSuccess; ++h)
            if (first + h * stride < pieces) e = fetch(first + h * stride, h);
        int h = 0;
        for (uint64_t p = first; p < pieces && e == cudaSuccess; p += stride, h ^= 1) {
            e = cudaEventSynchronize(lane.arrived[h]);
            if (e != cudaSuccess) break;
            std::memcpy(host + p * piece, lane.piece[h], size_of(p));
            if (p + 2 * stride < pieces) e = fetch(p + 2 * stride, h);
        }
        if (e != cudaSuccess) cudaStreamSynchronize(lane.stream);  // nothing of a failed copy is left in flight
        return e;
    }

    void release() {
        for (Lane& lane : lanes_) {
            if (lane.stream) cudaStreamDestroy(lane.stream);
            for (cudaEvent_t e : lane.arrived)
                if (e) cudaEventDestroy(e);
        }
        lanes_.clear();
        if (ready_) cudaEventDestroy(ready_);
        ready_ = nullptr;
        pinned_.release();
    }

    std::mutex mutex_;
    PinnedBlock pinned_;
    uint64_t fresh_bytes_ = 0;  // copied into fresh pages while there were no lanes
    std::vector<Lane> lanes_;
    cudaEvent_t ready_ = nullptr;
};

}  // namespace msx
