// Pinned host memory that host and device share at one address.
//
// cudaMallocHost serves small requests out of 2 MB blocks it keeps (a microsecond each while a block has
// room, 1 to 2.5 ms when it needs another one) and pins larger ones a 4 KB page at a time: 2 MB takes 2 ms,
// 16 MB 6.5 to 8.7 ms, 64 MB 26 ms. The same bytes on huge pages, registered, take 0.6, 2.3 and 9 ms, are
// given back in half the time and copy at the same 55 GB/s.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdint>

namespace msx {

class PinnedBlock {
public:
    PinnedBlock() = default;
    PinnedBlock(const PinnedBlock&) = delete;
    PinnedBlock& operator=(const PinnedBlock&) = delete;
    ~PinnedBlock() { release(); }

    char* data() const { return data_; }

    // `bytes` of it in the place of what it held. Requests that the driver's blocks hold, and hosts that
    // give no huge pages or refuse to register them, get the driver's memory.
    cudaError_t make(uint64_t bytes) {
        release();
        if (bytes > kDriverBlock / 2 && on_huge_pages(bytes)) return cudaSuccess;
        const cudaError_t e = cudaMallocHost(&data_, bytes);
        if (e != cudaSuccess) data_ = nullptr;
        return e;
    }

    void release() {
        if (mapped_) {
            cudaHostUnregister(data_);
            munmap(data_, mapped_);
        } else if (data_) {
            cudaFreeHost(data_);
        }
        data_ = nullptr;
        mapped_ = 0;
    }

private:
    static constexpr uint64_t kDriverBlock = 2ull << 20, kHugePage = 2ull << 20;

    bool on_huge_pages(uint64_t bytes) {
        const uint64_t size = (bytes + kHugePage - 1) / kHugePage * kHugePage;
        void* const whole = mmap(nullptr, size + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (whole == MAP_FAILED) return false;
        char* const first = static_cast<char*>(whole);
        char* const at = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(first) + kHugePage - 1) / kHugePage * kHugePage);
        if (at != first) munmap(first, static_cast<uint64_t>(at - first));
        const uint64_t behind = static_cast<uint64_t>(first + kHugePage - at);
        if (behind) munmap(at + size, behind);
        madvise(at, size, MADV_HUGEPAGE);
        // A child process gets no copy: its first write, or the parent's, would move the pages away from
        // the ones the device knows.
        madvise(at, size, MADV_DONTFORK);
        void* seen = nullptr;
        const bool registered = cudaHostRegister(at, size, cudaHostRegisterDefault) == cudaSuccess;
        if (registered && cudaHostGetDevicePointer(&seen, at, 0) == cudaSuccess && seen == at) {
            data_ = at;
            mapped_ = size;
            return true;
        }
        if (registered) cudaHostUnregister(at);
        cudaGetLastError();  // the driver's memory takes over
        munmap(at, size);
        return false;
    }

    char* data_ = nullptr;
    uint64_t mapped_ = 0;  // bytes mapped and registered here; 0: the driver's
};

}  // namespace msx
